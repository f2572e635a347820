"""What calls into the libraries prepare and launch, seen by a CUDA runtime that runs nothing (fake_cudart.cpp), in a process of
its own that never loads the real one."""
import ctypes as C
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
P = 1 << 20  # an aligned address that nobody reads


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    from dejavu_b200 import build

    build.build()
    nvcc = Path(build._nvcc()).resolve()
    folder = tmp_path_factory.mktemp("fake")
    versions = folder / "versions"
    versions.write_text("libcudart.so.12 { global: *; };\n")
    out = folder / "libcudart.so.12"
    subprocess.run([shutil.which("g++"), "-std=c++17", "-shared", "-fPIC", "-I", str(nvcc.parent.parent / "include"),
                    str(ROOT / "tests" / "fake_cudart.cpp"), "-o", str(out), "-Wl,-soname,libcudart.so.12",
                    f"-Wl,--version-script={versions}"], check=True)
    return out


PRELUDE = """
import ctypes as C
fake = C.CDLL({fake!r}, mode=C.RTLD_GLOBAL)
fake.fake_notes.restype = C.c_char_p
P = {P}
L = C.c_longlong
def load(name):
    lib = C.CDLL({root!r} + "/dejavu_b200/" + name)
    lib.djv_last_error.restype = C.c_char_p
    return lib
def done(lib, rc):
    assert rc == 0, lib.djv_last_error()
def notes():
    out = [l.split() for l in fake.fake_notes().decode().splitlines()]
    fake.fake_clear()
    return [dict(what=l[0], device=int(l[1]), kernel=l[2], grid=int(l[3]) * int(l[4]) * int(l[5]), block=int(l[6]), smem=int(l[7]),
                 cluster=int(l[8]), watched=int(l[9]) if len(l) > 9 else None) for l in out]
ptr = C.c_void_p(P)
"""


def run(fake, body):
    code = PRELUDE.format(fake=str(fake), root=str(ROOT), P=P) + body
    r = subprocess.run([sys.executable, "-I", "-c", code], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


CALLS = {
    "fc2 of several rows": """
for B in (3, 16, 17, 32):
    done(lib, lib.djv_gather_transposed_gemv(ptr, ptr, ptr, ptr, None, B, 4096, 2048, L(4096), 0, ptr, C.c_size_t(1 << 30), None))
""",
    "products of several rows": """
for B in (5, 16, 24, 32):
    done(lib, lib.djv_gather_gemv(ptr, ptr, ptr, ptr, None, B, 4096, 8192, L(4096), 0, 1, None))
""",
    "sparse MLP in one pass": """
for B in (1, 2, 4):
    done(lib, lib.djv_mlp_sparse_fused(ptr, ptr, ptr, ptr, ptr, None, None, B, 4096, 512, 16384, L(4096), L(4096), 0, ptr, C.c_size_t(1 << 30), None))
""",
    "top-K of long vectors": """
for f32 in (0, 1):
    done(lib, lib.djv_topk(ptr, None, ptr, 200000, 512, f32, None))
""",
    "projections of a batch": """
for hd in (32, 64, 128):
    done(lib, lib.djv_attn_step_project_batch(ptr, ptr, None, ptr, ptr, ptr, ptr, ptr, None, 0, 512, 8, hd, 64, 8, None))
""",
}


@pytest.mark.parametrize("what", CALLS)
def test_kernels_are_prepared_on_every_device(fake, what):
    """Attributes of a kernel belong to a device: what the first call sets on one does not serve the other."""
    run(fake, 'lib = load("libdejavu_b200.so")\nfor device in (0, 1):\n    fake.fake_set_device(device)\n'
        + "".join("    " + line + "\n" for line in CALLS[what].strip().splitlines())
        + "    assert any(n['what'] == 'launch' and n['device'] == device and n['smem'] > 48 * 1024 for n in notes())\n")


def test_routed_products_count_on_blocks_that_fit(fake):
    """The grid is what is resident with the shared memory that is launched, and that is two blocks per multiprocessor."""
    run(fake, """
lib = load("libdejavu_b200_routed.so")
for E in (1, 8, 57, 112, 300, 1137):
    for top in sorted({1, min(4, E), min(16, E)}):
        for B in (2, 8, 16, 24, 32):
            done(lib, lib.djv_moe_decode(1, ptr, ptr, ptr, ptr, ptr, ptr, ptr, None, None, None, B, E, top, 1024, 512, 0, 512, 3, None))
            for n in notes():
                if n["what"] == "launch":
                    assert 2 * (n["smem"] + 1376) <= 228 * 1024 and n["grid"] <= 2 * 148, (E, top, B, n)
                    asked.setdefault(n["kernel"], n["smem"])
                else:
                    asked[n["kernel"]] = n["smem"]
                assert asked[n["kernel"]] == n["smem"], (E, top, B, n)
""".replace("lib = load", "asked = {}\nlib = load", 1))


def test_short_lists_of_several_rows_fill_no_ring(fake):
    run(fake, """
lib = load("libdejavu_b200.so")
def kernel(B, N, M):
    done(lib, lib.djv_gather_gemv(ptr, ptr, ptr, ptr, None, B, N, M, L(N), 0, 1, None))
    n = [n for n in notes() if n["what"] == "launch"]
    assert len(n) == 1
    return "short" if "rowdot_mma_short" in n[0]["kernel"] else "ring" if "rowdot_mma" in n[0]["kernel"] else "rowdot"
for B in (9, 16, 32):
    for N, M in ((768, 384), (1024, 1024), (2048, 2048), (4096, 1024), (12288, 512)):
        assert kernel(B, N, M) == "short", (B, N, M)
    for N, M in ((768, 8192), (4096, 4096), (12288, 4096)):
        assert kernel(B, N, M) == "ring", (B, N, M)
for B in (5, 8):
    for N, M in ((768, 256), (512, 2048), (2048, 11264)):
        assert kernel(B, N, M) == "short", (B, N, M)
    for N, M in ((2048, 2048), (2048, 8192), (4096, 11264)):
        assert kernel(B, N, M) == "ring", (B, N, M)
for B in (1, 2):
    assert kernel(B, 4096, 4096) == "rowdot"
""")


def test_rows_of_two_tokens_are_dealt_out_without_idle_warps(fake):
    """(rows, chunks per row, blocks per multiprocessor) of the product's kernel, and that its blocks have all rows."""
    run(fake, """
import re
lib = load("libdejavu_b200.so")
for B, N, M, form in ((1, 12288, 512, "2,4,4"), (1, 4096, 4096, "4,2,4"), (2, 12288, 512, "2,4,3"), (2, 4096, 4096, "2,4,4"),
                      (2, 12288, 4096, "2,4,4"), (2, 4096, 12352, "4,2,3"), (3, 4096, 512, "2,4,2"), (4, 12288, 512, "2,4,2"),
                      (3, 12288, 1024, "4,2,2")):
    done(lib, lib.djv_gather_gemv(ptr, ptr, ptr, ptr, None, B, N, M, L(N), 0, 1, None))
    n, = notes()
    rows, chunks, blocks = re.search("rowdot_kernelI.*Li[1248]ELi([24])ELi([24])ELi([0-9])ELi(?:8|128)EE", n["kernel"]).groups()
    assert ",".join((rows, chunks, blocks)) == form and n["grid"] <= 148 * int(blocks), (B, N, M, n)
""")


def test_projections_of_few_and_of_many_sequences(fake):
    run(fake, """
lib = load("libdejavu_b200.so")
def project(B, nheads, nnz, hd, d):
    done(lib, lib.djv_attn_step_project_batch(ptr, ptr, None, ptr, ptr, ptr, ptr, ptr, ptr, nnz, d, nheads, hd, 64, B, None))
    return [n for n in notes() if n["what"] == "launch"][-1]
assert "qkv_sparse" in project(2, 32, 12, 128, 4096)["kernel"]
assert "qkv_sparse" in project(3, 32, 12, 128, 4096)["kernel"]
assert "qkv_batch" in project(2, 12, 1, 64, 768)["kernel"]
assert "qkv_batch" in project(3, 72, 24, 128, 9216)["kernel"]
for B, shares in ((7, 1), (16, 2), (64, 4)):
    n = project(B, 12, 4, 64, 768)
    assert "qkv_batch" in n["kernel"] and n["grid"] == 12 * 3 * n["cluster"] * shares, n
""")


def test_rows_per_kernel_do_not_depend_on_the_environment(fake):
    """From which number of rows on the tensor-core kernels take fc2 and the output projection, whatever a sweep may have set."""
    run(fake, """
import os
os.environ.update(DJV_RAB="9", DJV_OPB="9")
lib = load("libdejavu_b200.so")
lib.djv_gather_transposed_gemv_scratch_bytes.restype = C.c_size_t
for B in range(1, 17):
    need = lib.djv_gather_transposed_gemv_scratch_bytes(B, 4096, 2048)
    done(lib, lib.djv_gather_transposed_gemv(ptr, ptr, ptr, ptr, None, B, 4096, 2048, L(4096), 0, ptr, C.c_size_t(need), None))
    assert any("rowaxpy_mma" in n["kernel"] for n in notes()) == (B >= 3), B
    done(lib, lib.djv_out_proj_sparse(ptr, ptr, ptr, ptr, None, None, B, 4096, 32, 128, 12, None))
    assert any("out_proj_mma" in n["kernel"] for n in notes()) == (B >= 5), B
""")


def test_rows_that_may_be_asked_for_ahead(fake):
    """The hint alone allows all that a list names where rows are asked for line by line, and nothing of unknown size in bulk; with the
    rows of the matrix said, those below that."""
    run(fake, """
lib = load("libdejavu_b200.so")
def ahead(B, listed=True):
    fake.fake_watch(9 if B <= 4 else 11)  # of rowdot_kernel and rowdot_mma_short_kernel
    done(lib, lib.djv_gather_gemv(ptr, ptr, ptr, ptr if listed else None, None, B, 1024, 512, L(1024), 0, 1, None))
    n, = notes()
    assert ("rowdot_mma_short" in n["kernel"]) == (B > 4), n
    return n["watched"]
for enabled, rows, few, many in ((0, 0, 0, 0), (0, 4096, 0, 0), (1, 0, 2 ** 31 - 1, 0), (7, 0, 2 ** 31 - 1, 0), (1, 4096, 4096, 4096), (1, 1, 1, 1)):
    lib.djv_set_early_weight_prefetch(enabled)
    lib.djv_set_early_weight_rows(rows)
    for B in (1, 2, 3, 4):
        assert ahead(B) == few, (enabled, rows, B)
        assert ahead(B, False) == 512
    for B in (9, 16, 32):
        assert ahead(B) == many, (enabled, rows, B)
        assert ahead(B, False) == 512
""")


def test_splits_of_cached_tokens(fake):
    """One per 128 tokens while that fits the device with a third of the heads in use; fewer, and none that saves no pass, where not."""
    run(fake, """
lib = load("libdejavu_b200.so")
def splits(B, nheads, hd, S, listed=0):
    if listed:
        done(lib, lib.djv_decode_attn(ptr, ptr, ptr, ptr, ptr, listed, B, nheads, hd, S, S, C.c_float(1), ptr, C.c_size_t(1 << 30), None))
    else:
        done(lib, lib.djv_attn_step_attend_batch(ptr, ptr, ptr, ptr, ptr, B, nheads, hd, S, C.c_float(1), ptr, C.c_size_t(1 << 30), None))
    n, = notes()
    assert n["grid"] == (listed or nheads) * B * n["cluster"], n
    return n["cluster"]
for S, most in ((1, 1), (128, 1), (129, 2), (600, 5), (1024, 8), (2064, 8), (100000, 8)):
    for B, nheads in ((1, 12), (1, 72), (1, 96), (2, 32), (2, 12)):
        assert splits(B, nheads, 128, S) == most, (B, nheads, S)
    for hd in (32, 64, 128):
        assert splits(300, 40, hd, S) == 1 and splits(65535, 1, hd, S) == 1
assert [splits(B, 32, 128, 2064) for B in (3, 4, 8, 16, 32)] == [8, 6, 3, 1, 1]
assert [splits(B, 32, 128, 145) for B in (4, 8, 16)] == [2, 2, 1]
assert splits(4, 40, 128, 700) == 3  # (5 of 6 fit: two passes, for which 3 do)
assert [splits(1, 72, 128, 1104, k) for k in (12, 24, 36, 72)] == [8, 8, 5, 3]
assert [splits(16, 12, hd, 2064) for hd in (32, 64, 128)] == [8, 8, 4]
""")


def test_bounds_of_what_is_asked_for_ahead(tmp_path):
    """Spans start and end on 16 bytes inside their row, do not overlap, and are all of it where nothing caps them; rows that a list
    may hold while it is being written are refused."""
    (tmp_path / "ahead.cpp").write_text(f'#include "{ROOT}/dejavu_b200/csrc/ahead.cuh"\n' + """
#include <limits.h>
#include <stdio.h>
#include <string>
#define CHECK(c) if (!(c)) { printf("%s: %d %d %d\\n", #c, bytes, n, k); return 1; }
using namespace djv;
int main() {
  int n = 0, k = 0;
  for (int bytes = 16; bytes <= 12 * AHEAD_PIECE; bytes += 16) {
    n = ahead_pieces(bytes);
    for (int row = 0; row < 3; ++row) {
      int at = 0;
      for (k = 0; k < n; ++k) {
        const AheadSpan s = ahead_piece(row * n + k, bytes);
        CHECK(s.row == row && s.offset == at && s.bytes > 0 && s.bytes % 16 == 0 && s.bytes <= AHEAD_PIECE);
        at += s.bytes;
      }
      CHECK(at == bytes);
    }
    for (n = 1; n <= 8; ++n) {
      int at = 0;
      for (k = 0; k < n; ++k) {
        const AheadSpan s = ahead_share(k, n, bytes);
        if (s.bytes <= 0) continue;
        CHECK(s.row == 0 && s.offset == at && s.bytes % 16 == 0 && s.bytes <= AHEAD_PIECE && s.offset + s.bytes <= bytes);
        at += s.bytes;
      }
      CHECK(at == (bytes < n * AHEAD_PIECE ? bytes : n * AHEAD_PIECE) || (at <= bytes && bytes > n * (AHEAD_PIECE - 16)));
    }
  }
  const int bytes = 0;
  for (long long r : {-1ll, 4096ll, 0x7f7f7f7fll, 0x7f7f7f7f7f7f7f7fll, LLONG_MIN, -4096ll, 1ll << 32}) CHECK(!ahead_takes(r, 4096));
  CHECK(ahead_takes(0, 4096) && ahead_takes(4095, 4096) && !ahead_takes(0, 0) && !ahead_takes(1, 1));
  return 0;
}
""")
    subprocess.run([shutil.which("g++"), "-std=c++17", "-O1", str(tmp_path / "ahead.cpp"), "-o", str(tmp_path / "ahead")], check=True)
    r = subprocess.run([str(tmp_path / "ahead")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
