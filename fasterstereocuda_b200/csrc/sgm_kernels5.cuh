// Plain-level scans at D = 256: one warp per scanline, eight disparities per lane in 16-bit halves
// (plain_step16 of sgm_kernels4.cuh, exact for P1 <= 127, P1 <= P2 <= 16383).
//
// Chunks of kC5 steps are staged through mbarriers, three buffers deep: a row chunk is one contiguous
// bulk copy, a column chunk one box of a tensor map (unswizzled: a pixel's 256 costs are wider than a
// swizzle's 128 bytes). Eight steps a chunk keep a warp's buffers at 6 KB (10 KB top to bottom), so
// that all 2880 row scans of a 1280x720 pair are resident at once; with sixteen the last 8 % of them
// ran alone. One 256-byte bulk copy per image row instead of the box was bound by the copies' issue
// (389 us bottom to top).
// One pair of 1280x720, a launch at a time under ncu: rows 335 us (1.82 GB, 5.4 TB/s, integer ALU 78 %
// busy), bottom to top 177 us (0.90 GB, 5.1 TB/s, 73 %), top to bottom with the WTA 312 us (1.90 GB,
// 6.1 TB/s, 69 %): the last at 94 % of the measured copy bandwidth, the others between that (84 and 79 %)
// and the integer ALU. The lane-per-disparity kernels they replace took 1582 us for the rows and 1961 us
// for the columns (32-bit values, plain loads per step). With three pairs in flight a match takes 1.03 ms.
#pragma once
#include "sgm_async.cuh"
#include "sgm_kernels4.cuh"

namespace sgm {

constexpr int kC5 = 8;           // steps per staged chunk
constexpr int kD5 = 256;         // disparities
constexpr int kBox5 = kC5 * kD5;  // bytes of a chunk
constexpr int kRowBufs5 = 3;      // rows, and columns bottom to top: path costs replace costs in place
constexpr int kDownBoxes5 = 2 + 3;  // top to bottom: two of cost, one of each stored path

// The kC5 steps of a chunk in shared memory: at step j this lane reads its 8 bytes of cost at at(j)
// and leaves its path costs there. start: step 0 begins the scanline (L = C).
template <typename At>
__device__ __forceinline__ void chunk5(At at, bool start, uint32_t (&L)[4], uint32_t& mm, const Consts16& q) {
  uint2 in[kC5];
#pragma unroll
  for (int j = 0; j < kC5; ++j) in[j] = *at(j);
#pragma unroll
  for (int j = 0; j < kC5; ++j) {
    const uint32_t c[4] = {widen_lo(in[j].x), widen_hi(in[j].x), widen_lo(in[j].y), widen_hi(in[j].y)};
    if (j == 0 && start) {
#pragma unroll
      for (int k = 0; k < 4; ++k) L[k] = c[k];
      mm = min16_both<4>(L);
    } else {
      plain_step16<4>(L, c, mm, q);
    }
    *at(j) = make_uint2(narrow(L[0], L[1]), narrow(L[2], L[3]));
  }
}

// Row scans: warp i of the grid owns scanline i = (view, direction, y) as in hpaths3_lane. A
// right-to-left scan places a short (last) chunk at the end of the buffer, so that step j of every
// chunk reads pixel kC5 - 1 - j; all kC5 steps run, those past a short chunk on bytes nothing stores.
constexpr int kWpb5 = 2;  // warps per block

__global__ void __launch_bounds__(32 * kWpb5) k_hscan_plain256(const uint8_t* __restrict__ cost,
                                                              uint8_t* __restrict__ lr, uint8_t* __restrict__ rl,
                                                              PlainParams P, int nviews) {
  constexpr int C = kC5, D = kD5, NB = kRowBufs5;
  __shared__ __align__(128) uint8_t cbuf[kWpb5][NB][kBox5];
  __shared__ __align__(8) uint64_t bars[kWpb5][NB];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int H = P.H, W = P.W, len = W - P.x0, nch = (len + C - 1) / C;
  const int i = blockIdx.x * kWpb5 + w;
  if (i >= nviews * 2 * H || len <= 0) return;  // the whole warp
  if (lane == 0) {
    for (int b = 0; b < NB; ++b) mbar_init(&bars[w][b], 1);
    mbar_fence_init();
  }
  __syncwarp();
  const int grp = 2 * P.view0 + i / H, y = i % H;
  const bool rtl = grp & 1;
  const size_t ro = (size_t)(grp >> 1) * P.vstride + (size_t)y * W * D;
  const uint8_t* crow = cost + ro;
  uint8_t* orow = (rtl ? rl : lr) + ro;
  auto chunk_n = [&](int c) { return min(C, len - c * C); };
  auto chunk_x = [&](int c) { return rtl ? W - (c * C + chunk_n(c)) : P.x0 + c * C; };
  auto place = [&](int c) { return cbuf[w][c % NB] + (rtl ? (C - chunk_n(c)) * D : 0); };
  auto issue = [&](int c) {  // lane 0
    const uint32_t bytes = (uint32_t)chunk_n(c) * D;
    mbar_expect_tx(&bars[w][c % NB], bytes);
    bulk_to_smem(place(c), crow + (size_t)chunk_x(c) * D, bytes, &bars[w][c % NB]);
  };
  if (lane == 0) {
    issue(0);
    if (nch > 1) issue(1);
  }
  const Consts16 q = consts16<8>(P.p1, P.p2);
  uint32_t L[4], mm = 0, phase = 0u;
  for (int c = 0; c < nch; ++c) {
    const int b = c % NB;
    if (!mbar_wait_warp(&bars[w][b], (phase >> b) & 1u)) {
      scan_give_up_mask(bars[w], phase, (1u << b) | (c + 1 < nch ? 1u << ((c + 1) % NB) : 0u));
      if (lane == 0) bulk_wait_all();
      return;
    }
    phase ^= 1u << b;
    __syncwarp();
    uint8_t* mine = cbuf[w][b] + lane * 8;
    if (rtl)
      chunk5([mine](int j) { return reinterpret_cast<uint2*>(mine + (C - 1 - j) * D); }, c == 0, L, mm, q);
    else
      chunk5([mine](int j) { return reinterpret_cast<uint2*>(mine + j * D); }, c == 0, L, mm, q);
    fence_proxy_async();  // the chunk's path costs (and its cost reads) before the bulk copies
    __syncwarp();
    if (lane == 0) {
      bulk_to_global(orow + (size_t)chunk_x(c) * D, place(c), (uint32_t)chunk_n(c) * D);
      bulk_commit();
      if (c + 2 < nch) {
        bulk_wait_read<1>();  // the store of chunk c - 1 has left the buffer chunk c + 2 goes to
        issue(c + 2);
      }
    }
  }
  if (lane == 0) bulk_wait_all();
}

// WTA of one pixel from its four path rows in shared memory, by four neighbouring lanes of 64
// disparities each: the sums S(d) <= 1020 in 16-bit halves, searched as keys S(d) * 64 + (d mod 64),
// then as S * 256 + d over the four. The 16-byte units of a lane's quarter are taken in an order of
// its own (k XORed in), so that the eight lanes of a shared-memory phase read different banks. The
// lowest tied d wins (tie rules kTieLowest, and kTieRefB200, which differs at D = 64 only); the rest
// as plain_wta_rows. Every lane of the warp calls it.
__device__ __forceinline__ float wta256(const uint8_t* a, const uint8_t* b, const uint8_t* c, const uint8_t* e,
                                        int min_d, const WtaParams& Q) {
  const int lane = threadIdx.x & 31, k = ((lane >> 1) & 1) | ((lane >> 1) & 2);
  uint32_t lo[4], hi[4];  // per word t: least keys of d = 4t (+2 in the high half) and 4t + 1 (+3)
#pragma unroll
  for (int t = 0; t < 4; ++t) lo[t] = hi[t] = 0xFFFFFFFFu;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int u = 4 * (lane & 3) + (j ^ k);
    const uint32_t kb = (uint32_t)(16 * (j ^ k)) * 0x10001u;
    const uint4 va = reinterpret_cast<const uint4*>(a)[u], vb = reinterpret_cast<const uint4*>(b)[u];
    const uint4 vc = reinterpret_cast<const uint4*>(c)[u], ve = reinterpret_cast<const uint4*>(e)[u];
    const uint32_t wa[4] = {va.x, va.y, va.z, va.w}, wb[4] = {vb.x, vb.y, vb.z, vb.w};
    const uint32_t wc[4] = {vc.x, vc.y, vc.z, vc.w}, we[4] = {ve.x, ve.y, ve.z, ve.w};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      uint32_t sl, sh;
      sum4_bytes(wa[t], wb[t], wc[t], we[t], sl, sh);
      lo[t] = min16x2(lo[t], sl * 64u + kb);
      hi[t] = min16x2(hi[t], sh * 64u + kb);
    }
  }
  uint32_t acc = 0xFFFFFFFFu;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const uint32_t dl = (uint32_t)(4 * t) * 0x10001u + 0x20000u;
    acc = __vimin3_u16x2(acc, lo[t] + dl, hi[t] + dl + 0x10001u);
  }
  const uint32_t key = hmin16(acc);
  uint32_t best = ((key >> 6) << 8) | (key & 63u) | (uint32_t)(64 * (lane & 3));
  best = min(best, __shfl_xor_sync(kFull, best, 1));
  best = min(best, __shfl_xor_sync(kFull, best, 2));
  const uint32_t m = best >> 8;
  const int ds = (int)(best & 255u);
  if (ds <= 0 || ds >= Q.dmax_excl) return kInvalidFloat;
  auto sum_at = [&](int d) { return (uint32_t)a[d] + b[d] + c[d] + e[d]; };
  const float c1 = (float)sum_at(ds - 1), c2 = (float)m, c3 = ds + 1 < kD5 ? (float)sum_at(ds + 1) : (float)ds;
  const float d12 = __fsub_rn(c1, c2), d32 = __fsub_rn(c3, c2);
  const float uq = d12 < d32 ? d12 : d32;
  if (uq <= __fmul_rn(c2, __fsub_rn(1.0f, Q.uniqueness))) return kInvalidFloat;
  return __fadd_rn((float)(ds + min_d), subpix_bias(c1, c2, c3));
}

// Column scans: warp (blockIdx.x * kWpb5 + w) owns column x of view blockIdx.y, over boxes as in
// k_vscan_plain4. PASS 1: bottom to top, storing bt (the top box, which may start above row 0, row by
// row). PASS 2: top to bottom, then per chunk the sum of the four paths and the WTA, four lanes per
// pixel. Rows outside the image read as zeros; their steps store nothing.
template <int PASS>
constexpr size_t vscan256_smem() { return (size_t)kWpb5 * (PASS == 1 ? kRowBufs5 : kDownBoxes5) * kBox5; }

template <int PASS>
__global__ void __launch_bounds__(32 * kWpb5)
    k_vscan_plain256(const __grid_constant__ CUtensorMap m_cost, const __grid_constant__ CUtensorMap m_bt,
                     const __grid_constant__ CUtensorMap m_lr, const __grid_constant__ CUtensorMap m_rl,
                     uint8_t* __restrict__ bt, float* __restrict__ disp, PlainParams P, WtaParams Q) {
  constexpr int C = kC5, D = kD5, NB = PASS == 1 ? kRowBufs5 : 2;
  extern __shared__ __align__(128) uint8_t smem5[];
  __shared__ __align__(8) uint64_t bars[kWpb5][4];  // 0 .. NB - 1: cost; 3: the stored paths
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int W = P.W, H = P.H, nch = (H + C - 1) / C;
  const int x = blockIdx.x * kWpb5 + w, view = P.view0 + blockIdx.y;
  if (x >= W) return;  // the whole warp
  disp += (size_t)view * Q.dstride + x;
  if (x < P.x0) {
    if (PASS == 2)
      for (int y = lane; y < H; y += 32) disp[(size_t)y * W] = kInvalidFloat;
    return;
  }
  if (lane == 0) {
    for (int b = 0; b < 4; ++b) mbar_init(&bars[w][b], 1);
    mbar_fence_init();
  }
  __syncwarp();
  uint8_t* buf = smem5 + (size_t)w * (PASS == 1 ? kRowBufs5 : kDownBoxes5) * kBox5;
  auto box_y = [&](int c) { return PASS == 1 ? H - C * (c + 1) : C * c; };  // image row of box row 0
  auto issue_cost = [&](int c) {  // lane 0
    uint64_t* bar = &bars[w][c % NB];
    mbar_expect_tx(bar, kBox5);
    tma_load_3d(buf + (c % NB) * kBox5, &m_cost, x * D, box_y(c), view, bar);
  };
  auto issue_paths = [&](int c) {  // lane 0
    uint64_t* bar = &bars[w][3];
    uint8_t* dst = buf + 2 * kBox5;
    mbar_expect_tx(bar, 3u * kBox5);
    tma_load_3d(dst, &m_bt, x * D, box_y(c), view, bar);
    tma_load_3d(dst + kBox5, &m_lr, x * D, box_y(c), view, bar);
    tma_load_3d(dst + 2 * kBox5, &m_rl, x * D, box_y(c), view, bar);
  };
  if (lane == 0) {
    issue_cost(0);
    if (nch > 1) issue_cost(1);
    if (PASS == 2) issue_paths(0);
  }
  const Consts16 q = consts16<8>(P.p1, P.p2);
  const bool col_ok = x >= Q.xlo && x <= Q.xhi;
  uint32_t L[4], mm = 0, phase = 0u;
  for (int c = 0; c < nch; ++c) {
    const int b = c % NB;
    if (!mbar_wait_warp(&bars[w][b], (phase >> b) & 1u)) {
      scan_give_up_mask(bars[w], phase,
                        (1u << b) | (c + 1 < nch ? 1u << ((c + 1) % NB) : 0u) | (PASS == 2 ? 8u : 0u));
      if (lane == 0) bulk_wait_all();
      return;
    }
    phase ^= 1u << b;
    __syncwarp();
    uint8_t* box = buf + b * kBox5;
    uint8_t* mine = box + lane * 8;
    if (PASS == 1)
      chunk5([mine](int j) { return reinterpret_cast<uint2*>(mine + (C - 1 - j) * D); }, c == 0, L, mm, q);
    else
      chunk5([mine](int j) { return reinterpret_cast<uint2*>(mine + j * D); }, c == 0, L, mm, q);
    if constexpr (PASS == 1) {
      fence_proxy_async();
      __syncwarp();
      const int y0 = box_y(c);
      if (y0 >= 0) {
        if (lane == 0) {
          tma_store_3d(&m_bt, x * D, y0, view, box);
          bulk_commit();
        }
      } else {  // the top box: its rows inside the image, 8 bytes a lane
        for (int r = -y0; r < C; ++r)
          *reinterpret_cast<uint2*>(bt + (size_t)view * P.vstride + ((size_t)(y0 + r) * W + x) * D + lane * 8) =
              *reinterpret_cast<const uint2*>(mine + r * D);
      }
      if (lane == 0 && c + 2 < nch) {
        bulk_wait_read<1>();  // the store of chunk c - 1 has left the box chunk c + 2 goes to
        issue_cost(c + 2);
      }
    } else {
      __syncwarp();  // the chunk's path costs, written by disparity, are read by pixel
      if (!mbar_wait_warp(&bars[w][3], (phase >> 3) & 1u)) {
        scan_give_up_mask(bars[w], phase, 8u | (c + 1 < nch ? 1u << ((c + 1) % NB) : 0u));
        return;
      }
      phase ^= 8u;
      const uint8_t* paths = buf + 2 * kBox5;
      const int r = lane >> 2, y = C * c + r, o = r * D;
      // a row outside the image or its border is searched too (its bytes are in the boxes)
      const float dv = wta256(box + o, paths + o, paths + kBox5 + o, paths + 2 * kBox5 + o, P.min_d, Q);
      const bool ok = col_ok && y >= Q.ylo && y <= Q.yhi && y < Q.rows;
      if (y < H && (lane & 3) == 0) disp[(size_t)y * W] = ok ? dv : kInvalidFloat;
      fence_proxy_async();  // the reads of the boxes before the copies that refill them
      __syncwarp();
      if (lane == 0) {
        if (c + 1 < nch) issue_paths(c + 1);
        if (c + 2 < nch) issue_cost(c + 2);
      }
    }
  }
  if (PASS == 1 && lane == 0) bulk_wait_all();
}

}  // namespace sgm
