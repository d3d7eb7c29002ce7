"""The radix sort and the prefix sums (csrc/radix_sort.cu) against numpy:
tile edges, both launch forms of the large scan, segments, in place, and
arrays that start 1 to 3 words past a 16-byte boundary."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
import build  # noqa: E402

pytestmark = pytest.mark.gpu

TILE = 4096
HARNESS = r"""
#include "radix_sort.cuh"
using namespace pm;
#define OUT extern "C" __attribute__((visibility("default")))
OUT unsigned long long sort_words(unsigned n) { return radix_sort_hist_words(n); }
OUT int sort(uint32_t *k, uint32_t *v, uint32_t *kt, uint32_t *vt, const uint32_t *n_dev, unsigned max_n, int b0, int b1,
             uint32_t *hist, const uint2 *seg, int *swapped) {
    uint32_t *ok = nullptr, *ov = nullptr;
    cudaError_t e = radix_sort_pairs_u32(k, v, kt, vt, n_dev, max_n, b0, b1, hist, 0, &ok, &ov, seg);
    *swapped = ok == kt;
    return e ? e : cudaDeviceSynchronize();
}
OUT int scan(const uint32_t *in, uint32_t *out, unsigned n, uint32_t *total, uint32_t *tmp) {
    cudaError_t e = exclusive_scan_u32_large(in, out, n, total, tmp, 0);
    return e ? e : cudaDeviceSynchronize();
}
OUT int scan_seg(const uint32_t *in, uint32_t *out, unsigned n, const uint2 *seg, uint32_t *tmp) {
    cudaError_t e = exclusive_scan_u32_segmented(in, out, n, seg, tmp, 0);
    return e ? e : cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("sort")
    src, so = d / "harness.cu", d / "libsort.so"
    src.write_text(HARNESS)
    subprocess.run([build.NVCC] + build.ARCH + ["-std=c++17", "-O2", "-shared", "-Xcompiler", "-fPIC", "-I",
                   build.CSRC, "-o", str(so), str(src), os.path.join(build.BUILD, "radix_sort.cu.o")], check=True)
    so = ctypes.CDLL(str(so))
    so.sort_words.restype = ctypes.c_ulonglong
    p, u = ctypes.c_void_p, ctypes.c_uint
    so.sort.argtypes = [p, p, p, p, p, u, ctypes.c_int, ctypes.c_int, p, p, p]
    so.scan.argtypes = [p, p, u, p, p]
    so.scan_seg.argtypes = [p, p, u, p, p]
    return so


class Words:
    """n device words that start `off` words past a 16-byte boundary, guarded
    by 64 words on both sides."""

    def __init__(self, a, off=0):
        self.n, self.off = len(a), 64 + off
        host = np.full(self.n + 132, 0xA5A5A5A5, np.uint32)
        host[self.off: self.off + self.n] = a
        self.t = torch.from_numpy(host.view(np.int32)).cuda()
        self.ptr = self.t.data_ptr() + 4 * self.off

    def get(self):
        h = self.t.cpu().numpy().view(np.uint32)
        assert (h[: self.off] == 0xA5A5A5A5).all() and (h[self.off + self.n:] == 0xA5A5A5A5).all()
        return h[self.off: self.off + self.n].copy()


def segments(tiles, rs):
    """Per tile: its segment's first tile and tile count."""
    tab, t = [], 0
    while t < tiles:
        c = min(int(rs.randint(1, 6)), tiles - t)
        tab += [(t, c)] * c
        t += c
    return np.array(tab, np.uint32)


@pytest.mark.parametrize("n,off,seg", [(1, 0, False), (4095, 1, False), (4096, 2, False), (4097, 3, False),
                                       (65539, 1, False), (300001, 3, False), (9 * TILE, 0, True), (30 * TILE, 2, True)])
def test_sort(lib, n, off, seg):
    rs = np.random.RandomState(n)
    bits = (0, 16) if n % 2 else (0, 31)
    k = rs.randint(0, 1 << bits[1], n, dtype=np.int64).astype(np.uint32)
    k[: n // 3] &= np.uint32(0xFF00)  # equal keys keep their order
    v = np.arange(n, dtype=np.uint32)
    keys, vals = Words(k, off), Words(v, (off + 1) % 4)
    kt, vt = Words(np.zeros(n, np.uint32), (off + 2) % 4), Words(np.zeros(n, np.uint32), off)
    hist = Words(np.zeros(lib.sort_words(n), np.uint32), off)
    n_dev = Words(np.array([n], np.uint32))
    tab = segments(n // TILE, rs) if seg else None
    segd = torch.from_numpy(tab.view(np.int32)).cuda() if seg else None
    swapped = ctypes.c_int()
    assert lib.sort(keys.ptr, vals.ptr, kt.ptr, vt.ptr, n_dev.ptr, n, bits[0], bits[1], hist.ptr,
                    segd.data_ptr() if seg else None, ctypes.byref(swapped)) == 0
    group = np.repeat(tab[:, 0], TILE) if seg else np.zeros(n, np.uint32)
    order = np.lexsort((k, group))
    hist.get()
    np.testing.assert_array_equal((kt if swapped.value else keys).get(), k[order])
    np.testing.assert_array_equal((vt if swapped.value else vals).get(), v[order])


@pytest.mark.parametrize("n,off_in,off_out,place", [(5, 1, 0, False), (65537, 0, 0, False), (65538, 1, 2, False),
                                                    (70003, 3, 3, True), (TILE * TILE, 0, 0, True),
                                                    (TILE * TILE + 5, 2, 1, False)])
def test_scan(lib, n, off_in, off_out, place):
    a = np.random.RandomState(n).randint(0, 100, n).astype(np.uint32)
    src = Words(a, off_in)
    dst = src if place else Words(np.zeros(n, np.uint32), off_out)
    total, tmp = Words(np.zeros(1, np.uint32)), Words(np.zeros(n // TILE + 2, np.uint32))
    assert lib.scan(src.ptr, dst.ptr, n, total.ptr, tmp.ptr) == 0
    c = np.cumsum(a.astype(np.uint64))
    np.testing.assert_array_equal(dst.get(), np.concatenate([[0], c[:-1]]).astype(np.uint32))
    assert total.get()[0] == c[-1]
    tmp.get()


@pytest.mark.parametrize("tiles,off", [(1, 0), (7, 1), (40, 2)])
def test_segmented_scan(lib, tiles, off):
    rs = np.random.RandomState(tiles)
    n = tiles * TILE
    a = rs.randint(0, 100, n).astype(np.uint32)
    tab = segments(tiles, rs)
    src, dst = Words(a, off), Words(np.zeros(n, np.uint32), (off + 1) % 4)
    segd, tmp = torch.from_numpy(tab.view(np.int32)).cuda(), Words(np.zeros(tiles + 1, np.uint32))
    assert lib.scan_seg(src.ptr, dst.ptr, n, segd.data_ptr(), tmp.ptr) == 0
    want = np.cumsum(a.astype(np.uint64)) - a
    want -= np.repeat(want[tab[:, 0].astype(np.int64) * TILE], TILE)
    np.testing.assert_array_equal(dst.get(), want.astype(np.uint32))
    tmp.get()
