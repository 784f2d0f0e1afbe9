"""SHA-256 of the host absorb (csrc/host_sha.cuh) on the CPU: both block functions against hashlib, every way a stream can be cut."""
import hashlib
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "%s/zklm_compile_b200/csrc/host_sha.cuh"
using namespace zkb;
extern "C" void blocks(int plain, u32* st, const unsigned char* p, size_t n) { if (plain) sha256_blocks_plain(st, p, n); else sha256_blocks_host(st, p, n); }
extern "C" void absorb(TrState* t, const void* p, size_t n) { tr_absorb_host(*t, p, n); }
"""
IV = [0x6A09E667, 0xBB67AE85, 0x3C6EF372, 0xA54FF53A, 0x510E527F, 0x9B05688C, 0x1F83D9AB, 0x5BE0CD19]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    import ctypes
    if not shutil.which("nvcc"):
        pytest.skip("nvcc not on PATH")
    d = tmp_path_factory.mktemp("sha")
    (d / "s.cu").write_text(SRC % ROOT)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "--extended-lambda", "-Xcompiler", "-fPIC", "-shared",
                    "-o", str(d / "s.so"), str(d / "s.cu")], check=True, capture_output=True)
    return ctypes.CDLL(str(d / "s.so"))


def padded(msg):
    return msg + b"\x80" + b"\0" * ((55 - len(msg)) % 64) + (8 * len(msg)).to_bytes(8, "big")


@pytest.mark.parametrize("n", [0, 1, 55, 56, 63, 64, 65, 127, 1000, 4096])
def test_both_block_functions_match_hashlib(lib, n):
    import ctypes as C
    msg = bytes(np.random.default_rng(n).integers(0, 256, n, dtype=np.uint8))
    want = hashlib.sha256(msg).digest()
    data = padded(msg)
    for plain in (0, 1):
        st = (C.c_uint32 * 8)(*IV)
        lib.blocks(plain, st, data, C.c_size_t(len(data) // 64))
        assert b"".join(int(w).to_bytes(4, "big") for w in st) == want
    for cut in {0, 1, 63, 64, n // 2, n}:
        if cut > n:
            continue
        t = np.zeros(28, np.uint32)                    # h[8], buflen, pad, total (64 bits), buf[64]
        t[:8] = IV
        for part in (data[:cut], data[cut:]):
            lib.absorb(t.ctypes.data_as(C.c_void_p), part, C.c_size_t(len(part)))
        assert t[8] == 0 and t[10] == len(data) and b"".join(int(w).to_bytes(4, "big") for w in t[:8]) == want
