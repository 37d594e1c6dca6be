"""Batched row scans of 32-disparity levels: scanlines that leave their 16-bit steps with copies of the
next steps' costs in flight (1 .. 8 steps before their end), followed by other scanlines of the same
warp, against the exact-integer recurrence. Two outstanding cp.async writes of one address have no order,
so a scanline has to wait for its own before the next one starts. The kernel is launched alone: no
image leads a batch to such scanlines at a chosen step."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from tests.test_init_wrap import scanline_minima

CSRC = Path(__file__).resolve().parent.parent / "fasterstereocuda_b200" / "csrc"
P1, P2, H, PF = 10, 150, 40, 8
LIMIT = 8192  # |m| up to which a block of 8 steps runs in 16 bits

HARNESS = r"""
#include <vector>
#include "sgm_batch_kernels.cuh"
using namespace sgm::batch;

// One launch of `blocks` blocks over n pairs of one view; their volumes lie behind each other, W[i]*H*32 bytes
// each, their bases W[i]*H each.
extern "C" int rows3_init(const unsigned char* cost, const short* init, unsigned char* lr, unsigned char* rl,
                          const int* W, int H, int n, int p1, int p2, int G, int blocks) {
  size_t px = 0;
  std::vector<BatchPair> pairs(n);
  std::vector<int> tab(2 * n + 2);  // ids, prefix, queue
  std::vector<size_t> at(n);
  const int S = 32 / G;
  for (int i = 0; i < n; ++i) {
    at[i] = px;
    px += (size_t)W[i] * H;
    tab[i] = i;
    tab[n + i + 1] = tab[n + i] * (i > 0) + (2 * H + S - 1) / S;
  }
  tab[n] = 0;
  unsigned char *dc, *dl, *dr;
  short* di;
  BatchPair* dp;
  int *dt, *dq;
  cudaError_t e = cudaSuccess;
  auto ok = [&](cudaError_t r) { if (e == cudaSuccess) e = r; return e == cudaSuccess; };
  if (!ok(cudaMalloc(&dc, px * 32)) || !ok(cudaMalloc(&dl, px * 32)) || !ok(cudaMalloc(&dr, px * 32)) ||
      !ok(cudaMalloc(&di, px * 2)) || !ok(cudaMalloc(&dp, n * sizeof(BatchPair))) ||
      !ok(cudaMalloc(&dt, tab.size() * 4)) || !ok(cudaMalloc(&dq, 4)))
    return (int)e;
  for (int i = 0; i < n; ++i) {
    BatchPair b{};
    b.cost = dc + at[i] * 32; b.lr = dl + at[i] * 32; b.rl = dr + at[i] * 32; b.init = di + at[i]; b.nv = 1;
    b.IP.W = W[i]; b.IP.H = H; b.IP.x0 = 0; b.IP.p1 = p1; b.IP.p1s = p1; b.IP.p2s = p2; b.IP.p2_div0 = -1;
    b.IP.invalid_cost = 255; b.IP.vstride = (size_t)W[i] * H * 32;
    pairs[i] = b;
  }
  ok(cudaMemcpy(dc, cost, px * 32, cudaMemcpyHostToDevice));
  ok(cudaMemcpy(di, init, px * 2, cudaMemcpyHostToDevice));
  ok(cudaMemcpy(dp, pairs.data(), n * sizeof(BatchPair), cudaMemcpyHostToDevice));
  ok(cudaMemcpy(dt, tab.data(), tab.size() * 4, cudaMemcpyHostToDevice));
  ok(cudaMemset(dq, 0, 4));
  if (e == cudaSuccess) {
    if (G == 2) kb_rows3_init<2, 8><<<blocks, 128>>>(dp, dt, dt + n, n, dq);
    else if (G == 4) kb_rows3_init<4, 8><<<blocks, 128>>>(dp, dt, dt + n, n, dq);
    else kb_rows3_init<8, 8><<<blocks, 128>>>(dp, dt, dt + n, n, dq);
    ok(cudaGetLastError());
    ok(cudaDeviceSynchronize());
  }
  ok(cudaMemcpy(lr, dl, px * 32, cudaMemcpyDeviceToHost));
  ok(cudaMemcpy(rl, dr, px * 32, cudaMemcpyDeviceToHost));
  cudaFree(dc); cudaFree(dl); cudaFree(dr); cudaFree(di); cudaFree(dp); cudaFree(dt); cudaFree(dq);
  return (int)e;
}
"""


def _line(rng, n):
    """costs and bases: every second pixel beyond the range of its neighbour and invalid (255)"""
    cost = rng.integers(0, 65, (n, 32)).astype(np.uint8)
    cost[1::2] = 255
    return cost, np.where(np.arange(n) % 2 == 0, 0, 2000).astype(np.int16)


def _widens_at(ms):
    """first step in 32 bits: the end of the first block of PF steps after which |m| is past the limit"""
    return next((s + 1 for s in range(PF - 1, len(ms), PF) if abs(ms[s]) > LIMIT), len(ms))


def _pairs():
    """(cost, bases) of the pairs: left-to-right scans that widen 1 .. 8 steps before their end"""
    rng = np.random.default_rng(17)
    cost, bases = _line(rng, 200)
    at = _widens_at(scanline_minima(cost, bases, P1, P2)[1])
    assert PF < at < 190
    out = []
    for left in range(1, PF + 1):
        lines = [_line(rng, at + left) for _ in range(H)]
        out.append((np.stack([c for c, _ in lines]), np.stack([b for _, b in lines])))
    return out


def test_the_scanlines_widen_before_their_end():
    pairs = _pairs()
    for left, (cost, bases) in enumerate(pairs, 1):
        at = {_widens_at(scanline_minima(cost[y], bases[y], P1, P2)[1]) for y in range(3)}
        assert any(0 < cost.shape[1] - a <= PF for a in at), (left, at)


@pytest.mark.gpu
@pytest.mark.parametrize("G", [2, 4, 8])
def test_paths_of_scanlines_after_one_that_widened(tmp_path, G):
    src, so = tmp_path / "rows.cu", tmp_path / "rows.so"
    src.write_text(HARNESS)
    subprocess.run(["nvcc", "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler",
                    "-fPIC", f"-I{CSRC}", str(src), "-o", str(so)], check=True)
    fn = C.CDLL(str(so)).rows3_init
    pairs = _pairs()
    cost = np.concatenate([c.reshape(-1) for c, _ in pairs])
    init = np.concatenate([b.reshape(-1) for _, b in pairs])
    W = np.array([c.shape[1] for c, _ in pairs], np.int32)
    lr, rl = np.zeros_like(cost), np.zeros_like(cost)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    # one block: four warps take all items in turn
    assert fn(p(cost), p(init), p(lr), p(rl), p(W), H, len(W), P1, P2, G, 1) == 0
    o = 0
    for c, b in pairs:
        n = c.shape[1]
        for y in range(H):
            sl = slice(o + y * n * 32, o + (y + 1) * n * 32)
            want = np.stack(scanline_minima(c[y], b[y], P1, P2)[0])
            assert np.array_equal(lr[sl].reshape(n, 32), want), (n, y)
            want = np.stack(scanline_minima(c[y][::-1], b[y][::-1], P1, P2)[0])[::-1]
            assert np.array_equal(rl[sl].reshape(n, 32), want), (n, y)
        o += H * n * 32
