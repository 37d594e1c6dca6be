// Latency form of the scans, variant 4: the 32-disparity pyramid levels (first half of this file)
// and plain levels with D <= 128 (second half).
//
// A pair alone on the GPU offers few scanlines (375 rows x 2 directions at 1242x375), so the time
// of a scan is its number of steps times the length of one step's dependency chain. Here one warp
// owns a scanline and holds its path costs in 32 bits, the reference's own arithmetic
// (Kernel_Aggregate_{Horizontal,Vertical}_Warp*, cusgm_ca.cu:1181-1888). At a 32-disparity level
// lane d holds disparity d and a step's chain is
//   m = prev_invalid ? 127 : min_d L(d)            one redux.sync, issued beside the shuffles
//   a, b = L(d + s - 1), L(d + s + 1)              two shuffles (s = base - last_base)
//   L'(d) = C(d) + min(L(d), a + P1, b + P1, m + P2') - m
// and everything that does not depend on L is taken off it:
//   * costs (and, for the top-to-bottom pass, the three stored paths) arrive in chunks of 32 steps
//     staged in shared memory by asynchronous copies completing on mbarriers: a row chunk is one
//     contiguous cp.async.bulk copy, a column chunk one box of a 3D tensor map
//     (cp.async.bulk.tensor, swizzled so that lanes reading consecutive box rows hit distinct
//     banks), issued ahead of use;
//   * the per-step bookkeeping of the initial disparities -- the realignment shift, P2' =
//     max(P1, P2 / |last_base - base + 1|), which steps are skipped for an INVALID base -- is
//     computed for a whole chunk at once, one step per lane (ballot for the last valid base), the
//     next chunk's beside the current chunk's steps;
//   * path costs leave per step (row scans at the 32-disparity levels) or per chunk with one bulk
//     or tensor store, and the top-to-bottom pass takes the WTA per chunk with lane = pixel.
// Every wait on an mbarrier is bounded: after kMaxWaitTries polls the warp records the timeout in
// g_scan_wait_timeouts (read by sgm_debug_wait_timeouts), waits (bounded again) for its copies in
// flight and stops.
#pragma once
#include <cuda.h>  // CUtensorMap

#include <type_traits>

#include "sgm_async.cuh"
#include "sgm_kernels3.cuh"

namespace sgm {

// Per-step parameters of a chunk, one step per lane (lane j = step j): packed as
// shift (8 bits, clamped to +-64: any |shift| > 33 puts both neighbours out of range) |
// kStepValid | kPrevInvalid, and P2'.
constexpr uint32_t kStepValid = 1u << 8, kPrevInvalid = 1u << 9;

struct ChunkState {
  int carry_base;      // base of the last step that set last_base before the chunk
  bool carry_invalid;  // the last step before the chunk was skipped (INVALID base)
};

// b: this lane's step base (INVALID for lanes past the chunk); gs0: global index of the chunk's
// first step; n: steps in the chunk; first_sets_base: the scanline's first pixel sets last_base
// (horizontal scans) or keeps the one given (vertical scans, cusgm_ca.cu:1291).
// p2tab: P2' by k = |last_base - base + 1| (fill_p2_table), in shared memory: the divisions are the
// longest part of a chunk's parameters.
__device__ __forceinline__ void chunk_params(int b, int gs0, int n, bool first_sets_base, const InitParams& P,
                                             const uint32_t* p2tab, ChunkState& st, uint32_t& flags, uint32_t& p2) {
  const int j = threadIdx.x & 31;
  const bool in = j < n;
  const bool first = gs0 + j == 0;
  const bool step_valid = in && !first && b != kInvalidShort;
  const bool sets_base = in && (step_valid || (first && first_sets_base));
  const unsigned vm = __ballot_sync(kFull, sets_base);
  const unsigned prev = vm & ((1u << j) - 1u);
  const int from_prev = __shfl_sync(kFull, b, prev ? 31 - __clz(prev) : 0);
  const int lb = prev ? from_prev : st.carry_base;
  const int s = b - lb;
  const int sc = s < -64 ? -64 : (s > 64 ? 64 : s);
  p2 = step_valid ? p2_term(p2tab, abs(lb - b + 1), P) : 0u;
  // the previous step was skipped: the chunk's carry for lane 0, the left neighbour's flag else
  const unsigned inv = __ballot_sync(kFull, in && !first && b == kInvalidShort);
  const bool prev_inv = j == 0 ? st.carry_invalid : ((inv >> (j - 1)) & 1u);
  flags = (uint32_t)(sc & 0xFF) | (step_valid ? kStepValid : 0u) | (prev_inv ? kPrevInvalid : 0u);
  const int last_set = __shfl_sync(kFull, b, vm ? 31 - __clz(vm) : 0);
  if (vm) st.carry_base = last_set;
  if (n > 0) st.carry_invalid = (inv >> (n - 1)) & 1u;
}

// One step of the scanline held by the warp (lane = disparity). L: this lane's state; c: its cost.
__device__ __forceinline__ void scan_step(uint32_t& L, uint32_t c, uint32_t flags, uint32_t p2, uint32_t p1) {
  const int lane = threadIdx.x & 31;
  const int s = (int)(int8_t)(flags & 0xFFu);
  const uint32_t mr = __reduce_min_sync(kFull, L);
  const int i1 = lane + s - 1, i2 = lane + s + 1;
  const uint32_t a = __shfl_sync(kFull, L, i1 & 31);
  const uint32_t b = __shfl_sync(kFull, L, i2 & 31);
  const uint32_t m = (flags & kPrevInvalid) ? kInvalidCost : mr;
  const uint32_t A = (unsigned)i1 < 32u ? a + p1 : kInvalidCost;
  const uint32_t B = (unsigned)i2 < 32u ? b + p1 : kInvalidCost;
  const uint32_t t = min(__vimin3_u32(L, A, B), m + p2);
  const uint32_t Ln = c + (t - m);
  if (flags & kStepValid) L = Ln;
}

// scan_step for a step that is valid and follows a valid one (no INVALID base at either): the
// same result with P1 added before the shuffles and the m + P2' bound taken off their path.
__device__ __forceinline__ void scan_step_fast(uint32_t& L, uint32_t c, int s, uint32_t p2, uint32_t p1) {
  const int lane = threadIdx.x & 31;
  const uint32_t m = __reduce_min_sync(kFull, L);
  const uint32_t Lp = L + p1;
  const int i1 = lane + s - 1, i2 = lane + s + 1;
  const uint32_t a = __shfl_sync(kFull, Lp, i1 & 31);
  const uint32_t b = __shfl_sync(kFull, Lp, i2 & 31);
  const uint32_t A = (unsigned)i1 < 32u ? a : kInvalidCost;
  const uint32_t B = (unsigned)i2 < 32u ? b : kInvalidCost;
  const uint32_t t = __vimin3_u32(__viaddmin_u32(m, p2, L), A, B);
  L = c + t - m;
}

// ---------------------------------------------------------------------------------------------
// Horizontal scans: warp w of the grid owns scanline i = (view, dir, y) as in hpaths3_lane. A
// chunk is 32 consecutive pixels of the row, one contiguous bulk copy (double-buffered).
// Right-to-left scans place a short (last) chunk at the end of the buffer, so that step j of every
// chunk reads row 31 - j; every chunk runs all 32 steps (the steps past a short chunk are marked
// skipped and keep the state). Each step stores its 32 path costs straight to global memory (one
// 32-byte segment per warp). The step parameters of the next chunk are computed beside the steps
// of this one (they do not depend on the path costs), and a chunk whose steps all have valid bases
// (the usual case) runs scan_step_fast. Step parameters: the shift (fast chunks) or kStepValid,
// kPrevInvalid and the shift in bits 0-9; P2'.
// A large level is bound by its integer operations (half rate: selects, compares, minima), then by
// how many warps are there to issue them. So the two directions are separate code (constant
// offsets), the parameters arrive ready to use, and a step's costs and parameters are read from
// shared memory kGroup4 steps ahead, not a chunk (152 -> 96 registers, 12 -> 20 warps an SM; 80
// registers spill): 4800x3409 pyramid, three levels of row scans 2432 -> 2008 us beside the
// bottom-to-top columns.
// ---------------------------------------------------------------------------------------------
constexpr int kGroup4 = 8;

template <int WPB>
__global__ void __launch_bounds__(32 * WPB, 1) k_hscan_init4(const uint8_t* __restrict__ cost,
                                                          const int16_t* __restrict__ init_l,
                                                          const int16_t* __restrict__ init_r,
                                                          uint8_t* __restrict__ lr, uint8_t* __restrict__ rl,
                                                          InitParams P, int nviews) {
  constexpr int D = kLevelRange, C = kScanChunk, NB = 2, R = kGroup4;
  __shared__ __align__(128) uint8_t cbuf[WPB][NB][C * D];
  __shared__ __align__(8) uint64_t bars[WPB][NB];
  __shared__ __align__(16) uint2 par[WPB][2][C];
  __shared__ uint32_t p2tab[kP2Tab];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    for (int b = 0; b < NB; ++b) mbar_init(&bars[w][b], 1);
    mbar_fence_init();
  }
  fill_p2_table(p2tab, P, threadIdx.x, 32 * WPB);
  __syncthreads();
  const int H = P.H, W = P.W;
  const int i = blockIdx.x * WPB + w;
  if (i >= nviews * 2 * H) return;  // the whole warp
  const int grp = i / H, y = i - grp * H;
  const int view = grp >> 1;
  const int len = W - P.x0;
  if (len <= 0) return;
  const size_t ro = (size_t)view * P.vstride + (size_t)y * W * D;
  const uint8_t* crow = cost + ro;
  const int16_t* ib = (view == 0 ? init_l : init_r) + (size_t)y * W;
  const int nch = (len + C - 1) / C;
  auto scan = [&](auto right_to_left) {
    constexpr bool kLeft = decltype(right_to_left)::value;
    constexpr int r0 = kLeft ? (C - 1) * D : 0, dr = kLeft ? -D : D;  // row of step j: r0 + j * dr
    uint8_t* orow = (kLeft ? rl : lr) + ro;
    // chunk c: steps [c*C, c*C + n), pixels [chunk_x, chunk_x + n) in memory order (n <= 0: none)
    auto chunk_n = [&](int c) { return min(C, len - c * C); };
    auto chunk_x = [&](int c) { return kLeft ? W - (c * C + chunk_n(c)) : P.x0 + c * C; };
    auto issue = [&](int c) {  // lane 0
      const int b = c % NB, n = chunk_n(c);
      mbar_expect_tx(&bars[w][b], (uint32_t)n * D);
      bulk_to_smem(cbuf[w][b] + (kLeft ? (C - n) * D : 0), crow + (size_t)chunk_x(c) * D, (uint32_t)n * D, &bars[w][b]);
    };
    auto base_of = [&](int c) {  // this lane's step of chunk c
      if (lane >= chunk_n(c)) return (int)kInvalidShort;
      return (int)ib[kLeft ? W - 1 - (c * C + lane) : P.x0 + c * C + lane];
    };
    ChunkState st{0, false};
    // parameters of chunk c to every lane (lane j: step j); whether it takes the fast path
    auto params = [&](int c, int bse) {
      uint32_t flags, p2;
      chunk_params(bse, c * C, chunk_n(c), true, P, p2tab, st, flags, p2);
      const bool fast =
          __all_sync(kFull, (flags & (kStepValid | kPrevInvalid)) == kStepValid || (c == 0 && lane == 0));
      par[w][c & 1][lane] = make_uint2(fast ? (uint32_t)(int)(int8_t)(flags & 0xFFu) : flags, p2);
      return fast;
    };
    if (lane == 0) {
      issue(0);
      if (nch > 1) issue(1);
    }
    bool fast = params(0, base_of(0));
    int bnext = base_of(1);
    uint32_t phase = 0u;  // bit b: parity of buffer b's next phase
    uint32_t L = 0;
    for (int c = 0; c < nch; ++c) {
      const int b = c % NB, n = chunk_n(c);
      if (!mbar_wait_warp(&bars[w][b], (phase >> b) & 1u)) {
        scan_give_up_mask(bars[w], phase, (1u << b) | (c + 1 < nch ? 1u << ((c + 1) % NB) : 0u));
        return;
      }
      phase ^= 1u << b;
      __syncwarp();
      const uint8_t* cb = cbuf[w][b] + lane + r0;
      const uint2* pq = par[w][c & 1];
      uint8_t* op = orow + (size_t)chunk_x(c) * D + lane + (kLeft ? (n - 1) * D : 0);  // step 0's byte
      const int bn = bnext;
      bnext = base_of(c + 2);  // a chunk ahead (no load past the scanline)
      const bool run_fast = fast;
      // groups of R steps; a group's costs and parameters are read during the group before
      uint32_t cv[R];
      uint2 q[R];
      auto read = [&](int g) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
          cv[j] = cb[(g + j) * dr];
          q[j] = pq[g + j];
        }
      };
      auto free_buffer = [&]() {
        fence_proxy_async();  // this lane's reads of the buffer before the copy that refills it
        __syncwarp();
        if (lane == 0 && c + 2 < nch) issue(c + 2);
      };
      read(0);
      fast = params(c + 1, bn);
      if (run_fast) {  // a full chunk (a short one has skipped steps)
#pragma unroll
        for (int g = 0; g < C; g += R) {
          uint32_t cc[R];
          uint2 qq[R];
#pragma unroll
          for (int j = 0; j < R; ++j) {
            cc[j] = cv[j];
            qq[j] = q[j];
          }
          if (g + R < C) read(g + R);
          if (g + R == C) free_buffer();
#pragma unroll
          for (int j = 0; j < R; ++j) {
            uint32_t Ls = L;
            scan_step_fast(Ls, cc[j], (int)qq[j].x, qq[j].y, P.p1);
            L = (g + j == 0 && c == 0) ? cc[0] : Ls;  // the first pixel of the scanline starts it
            op[(g + j) * dr] = (uint8_t)L;
          }
        }
      } else {
        for (int g = 0; g < C; g += R) {
          if (g) read(g);
#pragma unroll
          for (int j = 0; j < R; ++j) {
            uint32_t Ls = L;
            scan_step(Ls, cv[j], q[j].x, q[j].y, P.p1);
            L = (g + j == 0 && c == 0) ? cv[0] : Ls;
            // a skipped step past a short chunk keeps L: it rewrites the chunk's last pixel
            op[min(g + j, n - 1) * dr] = (uint8_t)L;
          }
        }
        free_buffer();
      }
    }
  };
  if (grp & 1) scan(std::true_type{});
  else scan(std::false_type{});
}

// The 32 steps of a column chunk: a step's path costs overwrite its costs at at(j). Groups of kGroup4
// steps; a group's costs and parameters are read during the group before.
template <typename At>
__device__ __forceinline__ void scan_chunk_cols(uint32_t& L, const uint2* par, At at, bool fast, bool first,
                                                uint32_t p1) {
  constexpr int C = kScanChunk, R = kGroup4;
  uint32_t cv[R];
  uint2 q[R];
#pragma unroll
  for (int j = 0; j < R; ++j) {
    cv[j] = *at(j);
    q[j] = par[j];
  }
  auto chunk = [&](auto step) {
#pragma unroll
    for (int g = 0; g < C; g += R) {
      uint32_t cc[R];
      uint2 qq[R];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        cc[j] = cv[j];
        qq[j] = q[j];
      }
      if (g + R < C) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
          cv[j] = *at(g + R + j);
          q[j] = par[g + R + j];
        }
      }
#pragma unroll
      for (int j = 0; j < R; ++j) {
        step(g + j, cc[j], qq[j]);
        *at(g + j) = (uint8_t)L;
      }
    }
  };
  if (fast) {
    chunk([&](int, uint32_t c, uint2 q) { scan_step_fast(L, c, (int)q.x, q.y, p1); });
  } else {
    chunk([&](int j, uint32_t c, uint2 q) {
      if (j == 0 && first) L = c;
      else scan_step(L, c, q.x, q.y, p1);
    });
  }
}

// ---------------------------------------------------------------------------------------------
// Vertical scans: warp (blockIdx.x * WPB + w) owns column x of view blockIdx.y and stores its path
// costs: PASS 1 bottom to top (bt), PASS 3 top to bottom (tb); the WTA follows in k_wta_init4, so
// both passes can run beside the row scans. Both start last_base from row 0's base
// (cusgm_ca.cu:1291); the first pixel of a vertical path does not set it. Chunks are swizzled
// tensor-map boxes of 32 rows x 32 bytes, as in k_vscan_plain4: PASS 1 boxes end at rows H - 32c
// (the last one starts above row 0 and reads zeros there; its steps past row 0 are marked
// skipped), PASS 3 boxes start at rows 32c. A step's path costs overwrite its costs in the box,
// which then leaves with one tensor store (a box that reaches past the column, row by row). Chunks
// of valid bases run scan_step_fast, as in the row scans.
// ---------------------------------------------------------------------------------------------
// m_out / out: the volume the pass stores (bt or tb) as a tensor map and as a pointer.
template <int WPB, int PASS>
__global__ void __launch_bounds__(32 * WPB, 1)
    k_vscan_init4(const __grid_constant__ CUtensorMap m_cost, const __grid_constant__ CUtensorMap m_out,
                  const int16_t* __restrict__ init_l, const int16_t* __restrict__ init_r, uint8_t* __restrict__ out,
                  InitParams P) {
  static_assert(PASS == 1 || PASS == 3, "bottom-to-top or top-to-bottom");
  constexpr int D = kLevelRange, C = kScanChunk, BOX = C * D;
  constexpr int NB = 3;  // chunks in flight
  constexpr bool kUp = PASS == 1;
  __shared__ __align__(1024) uint8_t cbuf[WPB][NB][BOX];
  __shared__ __align__(8) uint64_t bars[WPB][NB];
  __shared__ __align__(16) uint2 par[WPB][C];
  __shared__ uint32_t p2tab[kP2Tab];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    for (int b = 0; b < NB; ++b) mbar_init(&bars[w][b], 1);
    mbar_fence_init();
  }
  fill_p2_table(p2tab, P, threadIdx.x, 32 * WPB);
  __syncthreads();
  const int W = P.W, H = P.H;
  const int x = blockIdx.x * WPB + w;
  const int view = blockIdx.y;
  if (x >= W || x < P.x0) return;  // the whole warp
  // the swizzle pattern is a function of the shared address: the boxes must start on 1 KB
  if (smem_u32(&cbuf[0][0][0]) & 1023u) {
    if (lane == 0) atomicAdd(&g_scan_wait_timeouts, 1u);
    return;
  }
  const int16_t* ib = (view == 0 ? init_l : init_r) + x;
  const int nch = (H + C - 1) / C;
  auto chunk_n = [&](int c) { return min(C, H - c * C); };
  auto row_of = [&](int s) { return kUp ? H - 1 - s : s; };
  auto box_y = [&](int c) { return kUp ? H - C * (c + 1) : C * c; };  // first row of chunk c's box
  auto issue = [&](int c) {  // lane 0
    const int b = c % NB;
    mbar_expect_tx(&bars[w][b], BOX);
    tma_load_3d(cbuf[w][b], &m_cost, x * D, box_y(c), view, &bars[w][b]);
  };
  auto base_of = [&](int c) {
    const int n = chunk_n(c);
    return lane < n ? (int)ib[(size_t)row_of(c * C + lane) * W] : (int)kInvalidShort;
  };
  if (lane == 0) {
    issue(0);
    if (nch > 1) issue(1);
  }
  uint32_t phase = 0u;  // bit b: parity of buffer b's next phase
  ChunkState st{(int)ib[0], false};  // row 0's base
  int bnext = base_of(0);
  uint32_t L = 0;
  const int lo0 = lane, lo1 = lane ^ 16;  // this lane's byte of a box row under the two swizzles
  for (int c = 0; c < nch; ++c) {
    const int b = c % NB, n = chunk_n(c);
    const int bcur = bnext;
    if (c + 1 < nch) bnext = base_of(c + 1);
    uint32_t flags, p2;
    chunk_params(bcur, c * C, n, false, P, p2tab, st, flags, p2);
    const bool fast = __all_sync(kFull, (flags & (kStepValid | kPrevInvalid)) == kStepValid);
    par[w][lane] = make_uint2(fast ? (uint32_t)(int)(int8_t)(flags & 0xFFu) : flags, p2);
    if (!mbar_wait_warp(&bars[w][b], (phase >> b) & 1u)) {
      scan_give_up_mask(bars[w], phase, (1u << b) | (c + 1 < nch ? 1u << ((c + 1) % NB) : 0u));
      if (lane == 0) bulk_wait_all();
      return;
    }
    phase ^= 1u << b;
    __syncwarp();
    uint8_t* box = cbuf[w][b];
    // step j: box row C - 1 - j (PASS 1) or j (PASS 3); this lane's byte of it
    auto at = [&](int j) {
      const int r = kUp ? C - 1 - j : j;
      return box + r * D + (box_sw<D>(r) ? lo1 : lo0);
    };
    // all 32 steps run (steps past a short last chunk are marked skipped)
    scan_chunk_cols(L, par[w], at, fast, c == 0, P.p1);
    fence_proxy_async();
    __syncwarp();
    const int y0 = box_y(c);
    if (y0 >= 0 && y0 + C <= H) {
      if (lane == 0) {
        tma_store_3d(&m_out, x * D, y0, view, box);
        bulk_commit();
      }
    } else {  // a box reaching past row 0 or row H - 1: its rows inside the column, one per lane
      const int y = y0 + lane;
      if (y >= 0 && y < H) {
        const uint4* src = reinterpret_cast<const uint4*>(box + lane * D);
        uint4* dst = reinterpret_cast<uint4*>(out + (size_t)view * P.vstride + ((size_t)y * W + x) * D);
        const int sw = box_sw<D>(lane);
        const uint4 v0 = src[sw], v1 = src[sw ^ 1];
        dst[0] = v0;
        dst[1] = v1;
      }
    }
    if (lane == 0 && c + 2 < nch) {
      bulk_wait_read<1>();  // the store of chunk c - 1 has left the box chunk c + 2 goes to
      issue(c + 2);
    }
  }
  if (lane == 0) bulk_wait_all();
}

// WTA of one pixel of an initial-disparity level from its four stored path rows (32 bytes each,
// in global memory; S(d) = sum of the four): Kernel_ComputeDisparityByWTA for initial disparities
// (cusgm_ca.cu:3425-3512). d* <= 1 or d* >= 31 -> INVALID; uniqueness and the +0.5-shifted
// parabola as in wta_pixel; tie rules: kTieRefB200 the lowest tied d whose candidate is valid
// (every tied lane stores its own result there, a valid one wins), 1 / 2 the highest tied d, 0 / 3
// the lowest (one disparity per lane: lane order is disparity order). A row is read as two 16-byte
// words (unit u at u ^ sw: rows of a swizzled box); S(d) is summed in 16-bit halves, its minimum
// taken by SIMD minima and the tied set kept as a bit mask; S at a candidate's neighbours comes from
// single bytes.
__device__ __forceinline__ float init_wta_rows(const uint8_t* a, const uint8_t* b, const uint8_t* c,
                                               const uint8_t* e, int base, const WtaParams& Q, int sw = 0) {
  constexpr int D = kLevelRange;
  uint32_t lo[D / 4], hi[D / 4];  // lo[k] = S(4k) | S(4k + 2) << 16, hi[k] = S(4k + 1) | S(4k + 3) << 16
#pragma unroll
  for (int q = 0; q < D / 16; ++q) {
    const int u = q ^ sw;
    const uint4 va = reinterpret_cast<const uint4*>(a)[u], vb = reinterpret_cast<const uint4*>(b)[u];
    const uint4 vc = reinterpret_cast<const uint4*>(c)[u], ve = reinterpret_cast<const uint4*>(e)[u];
    const uint32_t wa[4] = {va.x, va.y, va.z, va.w}, wb[4] = {vb.x, vb.y, vb.z, vb.w};
    const uint32_t wc[4] = {vc.x, vc.y, vc.z, vc.w}, we[4] = {ve.x, ve.y, ve.z, ve.w};
#pragma unroll
    for (int t = 0; t < 4; ++t) sum4_bytes(wa[t], wb[t], wc[t], we[t], lo[4 * q + t], hi[4 * q + t]);
  }
  uint32_t mm = __vminu2(lo[0], hi[0]);
#pragma unroll
  for (int k = 1; k < D / 4; ++k) mm = __vminu2(mm, __vminu2(lo[k], hi[k]));
  const uint32_t m = min(mm & 0xFFFFu, mm >> 16), m2 = m * 0x10001u;
  uint32_t tied = 0;  // bit d: S(d) == m
#pragma unroll
  for (int k = 0; k < D / 4; ++k) {
    const uint32_t el = __vcmpeq2(lo[k], m2), eh = __vcmpeq2(hi[k], m2);
    tied |= ((el & 1u) | ((eh & 1u) << 1) | ((el >> 14) & 4u) | ((eh >> 13) & 8u)) << (4 * k);
  }
  const float ut = __fsub_rn(1.0f, Q.uniqueness);
  auto sum_at = [&](int d) {
    const int o = d ^ (sw << 4);
    return (uint32_t)a[o] + b[o] + c[o] + e[o];
  };
  auto candidate = [&](int d) {
    if (d <= 1 || d >= Q.dmax_excl) return kInvalidFloat;
    const float c1 = (float)sum_at(d - 1), c2 = (float)m, c3 = (float)sum_at(d + 1);
    const float d12 = __fsub_rn(c1, c2), d32 = __fsub_rn(c3, c2);
    const float uq = d12 < d32 ? d12 : d32;
    if (uq <= __fmul_rn(c2, ut)) return kInvalidFloat;
    return __fadd_rn((float)(d + base), subpix_bias(c1, c2, c3));
  };
  if (Q.tie_rule == kTieRefB200) {
    while (tied) {
      const float v = candidate(__ffs(tied) - 1);
      if (v != kInvalidFloat) return v;
      tied &= tied - 1u;
    }
    return kInvalidFloat;
  }
  const bool high = Q.tie_rule == kTieHighest || Q.tie_rule == kTieLaneHigh;
  return candidate(high ? 31 - __clz(tied) : __ffs(tied) - 1);
}

// WTA of an initial-disparity level, one thread per pixel, from the four stored path volumes:
// INVALID left of x0, on the image border, in rows >= Q.rows and where the pixel's base is
// INVALID.
__global__ void __launch_bounds__(128) k_wta_init4(const uint8_t* __restrict__ bt, const uint8_t* __restrict__ tb,
                                                   const uint8_t* __restrict__ lr, const uint8_t* __restrict__ rl,
                                                   const int16_t* __restrict__ init_l,
                                                   const int16_t* __restrict__ init_r, float* __restrict__ disp,
                                                   InitParams P, WtaParams Q) {
  constexpr int D = kLevelRange;
  const int x = blockIdx.x * 128 + threadIdx.x, y = blockIdx.y, view = blockIdx.z;
  const int W = P.W;
  if (x >= W) return;
  float dv = kInvalidFloat;
  if (x >= P.x0 && x >= Q.xlo && x <= Q.xhi && y >= Q.ylo && y <= Q.yhi && y < Q.rows) {
    const int base = (view == 0 ? init_l : init_r)[(size_t)y * W + x];
    if (base != kInvalidShort) {
      const size_t o = (size_t)view * P.vstride + ((size_t)y * W + x) * D;
      dv = init_wta_rows(tb + o, bt + o, lr + o, rl + o, base, Q);
    }
  }
  disp[(size_t)view * Q.dstride + (size_t)y * W + x] = dv;
}

// Top-to-bottom scan of a 32-disparity level with the WTA: as k_vscan_init4 with PASS 3, but a chunk's
// pixels take their WTA, one lane each, from the chunk's path costs and the boxes of the three stored
// paths, so the level needs no top-to-bottom volume and moves 4 bytes a voxel where PASS 3 and
// k_wta_init4 move 6; it can only follow the row scans, where PASS 3 runs beside them. Bound by issue and
// by the steps' chains: 24 warps an SM (80 registers; 12 at 135, 32 spill) and scan_step_fast took the
// 4800x3409 pyramid's three launches 1637 -> 1290 us.
template <int WPB>
__global__ void __launch_bounds__(32 * WPB, 24 / WPB)
    k_vscan_wta_init4(const __grid_constant__ CUtensorMap m_cost, const __grid_constant__ CUtensorMap m_bt,
                      const __grid_constant__ CUtensorMap m_lr, const __grid_constant__ CUtensorMap m_rl,
                      const int16_t* __restrict__ init_l, const int16_t* __restrict__ init_r,
                      float* __restrict__ disp, InitParams P, WtaParams Q) {
  constexpr int D = kLevelRange, C = kScanChunk, BOX = C * D, NB = 3;
  __shared__ __align__(1024) uint8_t cbuf[WPB][NB + 3][BOX];  // cost; bt, lr, rl
  __shared__ __align__(8) uint64_t bars[WPB][NB + 1];         // bars[NB]: the stored paths
  __shared__ __align__(16) uint2 par[WPB][C];
  __shared__ uint32_t p2tab[kP2Tab];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    for (int b = 0; b <= NB; ++b) mbar_init(&bars[w][b], 1);
    mbar_fence_init();
  }
  fill_p2_table(p2tab, P, threadIdx.x, 32 * WPB);
  __syncthreads();
  const int W = P.W, H = P.H;
  const int x = blockIdx.x * WPB + w, view = blockIdx.y;
  if (x >= W) return;  // the whole warp
  disp += (size_t)view * Q.dstride + x;
  if (x < P.x0) {
    for (int y = lane; y < H; y += 32) disp[(size_t)y * W] = kInvalidFloat;
    return;
  }
  // the swizzle pattern is a function of the shared address: the boxes must start on 1 KB
  if (smem_u32(&cbuf[0][0][0]) & 1023u) {
    if (lane == 0) atomicAdd(&g_scan_wait_timeouts, 1u);
    return;
  }
  const int16_t* ib = (view == 0 ? init_l : init_r) + x;
  const int nch = (H + C - 1) / C;
  auto issue_cost = [&](int c) {  // lane 0
    const int b = c % NB;
    mbar_expect_tx(&bars[w][b], BOX);
    tma_load_3d(cbuf[w][b], &m_cost, x * D, C * c, view, &bars[w][b]);
  };
  auto issue_paths = [&](int c) {  // lane 0
    mbar_expect_tx(&bars[w][NB], 3 * BOX);
    tma_load_3d(cbuf[w][NB + 0], &m_bt, x * D, C * c, view, &bars[w][NB]);
    tma_load_3d(cbuf[w][NB + 1], &m_lr, x * D, C * c, view, &bars[w][NB]);
    tma_load_3d(cbuf[w][NB + 2], &m_rl, x * D, C * c, view, &bars[w][NB]);
  };
  auto base_of = [&](int c) {
    const int y = C * c + lane;
    return y < H ? (int)ib[(size_t)y * W] : (int)kInvalidShort;
  };
  if (lane == 0) {
    issue_cost(0);
    if (nch > 1) issue_cost(1);
    issue_paths(0);
  }
  const bool col_ok = x >= Q.xlo && x <= Q.xhi;
  uint32_t phase = 0u;  // bit b: parity of buffer b's next phase
  ChunkState st{(int)ib[0], false};  // row 0's base
  int bnext = base_of(0);
  uint32_t L = 0;
  const int lo0 = lane, lo1 = lane ^ 16;  // this lane's byte of a box row under the two swizzles
  for (int c = 0; c < nch; ++c) {
    const int b = c % NB;
    const int bcur = bnext;
    if (c + 1 < nch) bnext = base_of(c + 1);
    uint32_t flags, p2;
    chunk_params(bcur, c * C, min(C, H - c * C), false, P, p2tab, st, flags, p2);
    const bool fast = __all_sync(kFull, (flags & (kStepValid | kPrevInvalid)) == kStepValid);
    par[w][lane] = make_uint2(fast ? (uint32_t)(int)(int8_t)(flags & 0xFFu) : flags, p2);
    if (!mbar_wait_warp(&bars[w][b], (phase >> b) & 1u)) {
      scan_give_up_mask(bars[w], phase, (1u << NB) | (1u << b) | (c + 1 < nch ? 1u << ((c + 1) % NB) : 0u));
      return;
    }
    phase ^= 1u << b;
    __syncwarp();
    uint8_t* box = cbuf[w][b];
    auto at = [&](int j) { return box + j * D + (box_sw<D>(j) ? lo1 : lo0); };
    scan_chunk_cols(L, par[w], at, fast, c == 0, P.p1);
    __syncwarp();  // the chunk's path costs, written by disparity, are read by pixel
    if (!mbar_wait_warp(&bars[w][NB], (phase >> NB) & 1u)) {
      scan_give_up_mask(bars[w], phase, (1u << NB) | (c + 1 < nch ? 1u << ((c + 1) % NB) : 0u));
      return;
    }
    phase ^= 1u << NB;
    const int y = C * c + lane, o = lane * D;
    if (y < H) {
      float dv = kInvalidFloat;
      if (col_ok && y >= Q.ylo && y <= Q.yhi && y < Q.rows && bcur != kInvalidShort)
        dv = init_wta_rows(box + o, cbuf[w][NB] + o, cbuf[w][NB + 1] + o, cbuf[w][NB + 2] + o, bcur, Q,
                           box_sw<D>(lane));
      disp[(size_t)y * W] = dv;
    }
    fence_proxy_async();  // the accesses of the boxes before the copies that refill them
    __syncwarp();
    if (lane == 0) {
      if (c + 1 < nch) issue_paths(c + 1);
      if (c + 2 < nch) issue_cost(c + 2);
    }
  }
}

}  // namespace sgm

namespace sgm {

// =============================================================================================
// Plain levels (no initial disparities), latency form. One warp owns a scanline; lane l holds the
// K consecutive disparities d = K l + k in 32 bits, the reference's lane mapping
// (Kernel_Aggregate_*_Warpfor{32,64,128}, cusgm_ca.cu:1343-1888). A step:
//   m = min_d L(d)                       one redux.sync of the lanes' K-wide minima
//   L(d - 1) + P1, L(d + 1) + P1         in the lane, or one shuffle up / down at its edges
//   L'(d) = C(d) + min(L(d), L(d-1) + P1 | 127, L(d+1) + P1 | 127, m + P2) - m
// and a lane moves its K bytes of costs and path costs as one 8/16/32-bit shared access.
// Chunks of 32 steps move between global and shared memory with bulk async copies; a step's path
// costs overwrite its costs in the chunk buffer, which then leaves with a bulk store (rows: one
// contiguous copy; columns: one tensor-map box of 32 rows), three buffers deep so a load never
// waits for the store of the chunk before. Every chunk runs all 32 steps: the steps past a scanline's end read and
// write rows of the buffer that hold nothing of this scanline and are neither stored nor used.
// The WTA of the top-to-bottom pass runs per chunk with lane = pixel.
// =============================================================================================

// A lane's K bytes of a step row, as one shared-memory word.
template <int K>
using LaneBytes = std::conditional_t<K == 1, uint8_t, std::conditional_t<K == 2, uint16_t, uint32_t>>;

template <int K>
__device__ __forceinline__ void unpack_bytes(uint32_t w, uint32_t (&c)[K]) {
#pragma unroll
  for (int k = 0; k < K; ++k) c[k] = k == 0 && K == 1 ? w : __byte_perm(w, 0u, 0x4440u + k);
}
template <int K>
__device__ __forceinline__ uint32_t pack_bytes(const uint32_t (&L)[K]) {
  if constexpr (K == 1) return L[0];
  if constexpr (K == 2) return __byte_perm(L[0], L[1], 0x0040u);
  if constexpr (K == 4) return __byte_perm(__byte_perm(L[0], L[1], 0x0040u), __byte_perm(L[2], L[3], 0x0040u), 0x5410u);
  return 0u;
}

template <int K>
__device__ __forceinline__ void plain_step4(uint32_t (&L)[K], const uint32_t (&c)[K], uint32_t p1, uint32_t p2) {
  const int lane = threadIdx.x & 31;
  uint32_t lm = L[0];
#pragma unroll
  for (int k = 1; k < K; ++k) lm = min(lm, L[k]);
  const uint32_t m = __reduce_min_sync(kFull, lm);
  uint32_t Lp[K];
#pragma unroll
  for (int k = 0; k < K; ++k) Lp[k] = L[k] + p1;
  const uint32_t up = __shfl_up_sync(kFull, Lp[K - 1], 1);  // L(K l - 1) + P1 from lane l - 1
  const uint32_t dn = __shfl_down_sync(kFull, Lp[0], 1);    // L(K l + K) + P1 from lane l + 1
  const uint32_t a0 = lane > 0 ? up : kInvalidCost;
  const uint32_t bK = lane < 31 ? dn : kInvalidCost;
  const uint32_t l4 = m + p2;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const uint32_t A = k == 0 ? a0 : Lp[k - 1];
    const uint32_t B = k == K - 1 ? bK : Lp[k + 1];
    const uint32_t t = min(__vimin3_u32(L[k], A, B), l4);
    L[k] = c[k] + t - m;
  }
}

// The same recurrence in 16-bit halves: lane l holds its K disparities as K / 2 words (u16x2), exact
// for P1 <= 127, P1 <= P2 <= 16383 (host: narrow4_ok). A GPU full of scans is bound by the integer ALU
// (DPX minima, byte permutes and selects all issue at half rate), so what counts is ALU operations
// per step: about 10 instead of 15 at K = 2, 19 instead of 29 at K = 4. 1242x375, D = 64, one pair
// alone: rows 110 -> 92 us, columns 47 + 66 -> 39 + 60 us; 32 pairs in flight 166 -> 153 us a pair
// (D = 128, 957x541: 344 -> 294 us). Two things keep the count down:
//   * the minimum over the lane's halves is taken in both halves (min(v, v with halves swapped)),
//     so one REDUX returns m in both halves and m never has to be spread;
//   * the candidate 127 beyond d = 0 and d = D - 1 rides on the jump candidate: x is
//     min(L(d-1), L(d+1), min(m + P2 - P1, cap)) with cap = 127 - P1 there, and x + P1 follows. At
//     K = 2 the edge lanes' shuffles return the lane's own word, whose half is the other neighbour, a
//     candidate anyway; wider lanes put all ones there (sgm_kernels5.cuh holds eight disparities a lane the same way).
struct Consts16 {
  uint32_t p1x2, p2m1x2, cap_lo, cap_hi;  // cap of the lane's first and last word (K = 2: both in cap_lo)
};
template <int K>
__device__ __forceinline__ Consts16 consts16(uint32_t p1, uint32_t p2) {
  const int lane = threadIdx.x & 31;
  const uint32_t cap = (kInvalidCost - p1) & 0xFFFFu;
  Consts16 q;
  q.p1x2 = rep16(p1);
  q.p2m1x2 = rep16(p2 - p1);
  q.cap_lo = lane == 0 ? 0xFFFF0000u | cap : 0xFFFFFFFFu;
  q.cap_hi = lane == 31 ? (cap << 16) | 0xFFFFu : 0xFFFFFFFFu;
  if (K == 2) q.cap_lo &= q.cap_hi;
  return q;
}
// min over the scanline of L, in both halves
template <int NW>
__device__ __forceinline__ uint32_t min16_both(const uint32_t (&L)[NW]) {
  uint32_t v = L[0];
  if constexpr (NW == 2) v = min16x2(L[0], L[1]);
  if constexpr (NW == 4) v = min16x2(__vimin3_u16x2(L[0], L[1], L[2]), L[3]);
  return __reduce_min_sync(kFull, min16x2(v, __byte_perm(v, v, 0x1032)));
}
// mm: m in both halves, of the state before and after the step
template <int NW>
__device__ __forceinline__ void plain_step16(uint32_t (&L)[NW], const uint32_t (&c)[NW], uint32_t& mm,
                                             const Consts16& q) {
  const int lane = threadIdx.x & 31;
  uint32_t ln = __shfl_up_sync(kFull, L[NW - 1], 1), rn = __shfl_down_sync(kFull, L[0], 1);
  if constexpr (NW > 1) {
    ln = lane == 0 ? 0xFFFFFFFFu : ln;
    rn = lane == 31 ? 0xFFFFFFFFu : rn;
  }
  uint32_t b[NW + 1];  // b[k], b[k + 1]: the words of d - 1 and d + 1 of word k
  b[0] = __byte_perm(ln, L[0], 0x5432);
#pragma unroll
  for (int k = 1; k < NW; ++k) b[k] = __byte_perm(L[k - 1], L[k], 0x5432);
  b[NW] = __byte_perm(L[NW - 1], rn, 0x5432);
  // m + P2 - P1 (no half reaches 2^16), capped where the word holds an end of the range
  const uint32_t first = __viaddmin_u16x2(mm, q.p2m1x2, q.cap_lo);
  const uint32_t last = NW > 1 ? __viaddmin_u16x2(mm, q.p2m1x2, q.cap_hi) : first;
  const uint32_t mid = NW > 2 ? mm + q.p2m1x2 : 0u;
#pragma unroll
  for (int k = 0; k < NW; ++k) {
    const uint32_t x = __vimin3_u16x2(b[k], b[k + 1], k == 0 ? first : (k == NW - 1 ? last : mid));
    L[k] = __viaddmin_u16x2(x, q.p1x2, L[k]) + c[k] - mm;
  }
  mm = min16_both<NW>(L);
}

// The state of a scanline: 32-bit costs, or 16-bit halves and their minimum.
template <int K, bool N16>
struct Plain4 {
  uint32_t L[N16 ? K / 2 : K], mm = 0;
  Consts16 q;
  uint32_t p1, p2;
  __device__ __forceinline__ Plain4(const PlainParams& P) : p1(P.p1), p2(P.p2) {
    if constexpr (N16) q = consts16<K>(P.p1, P.p2);
  }
  // one step from the lane's K cost bytes; start: L = C
  __device__ __forceinline__ uint32_t advance(uint32_t w, bool start) {
    if constexpr (N16) {
      uint32_t c[K / 2];
      c[0] = widen_lo(w);
      if constexpr (K == 4) c[1] = widen_hi(w);
      if (start) {
#pragma unroll
        for (int k = 0; k < K / 2; ++k) L[k] = c[k];
        mm = min16_both<K / 2>(L);
      } else {
        plain_step16<K / 2>(L, c, mm, q);
      }
      return K == 4 ? narrow(L[0], L[K / 2 - 1]) : __byte_perm(L[0], 0u, 0x4420);
    } else {
      uint32_t c[K];
      unpack_bytes<K>(w, c);
      if (start) {
#pragma unroll
        for (int k = 0; k < K; ++k) L[k] = c[k];
      } else {
        plain_step4<K>(L, c, p1, p2);
      }
      return pack_bytes<K>(L);
    }
  }
};

// The 32 steps of a chunk held in shared memory: at step j this lane reads its K bytes of costs
// at at(j) (a LaneBytes<K> pointer) and leaves its path costs there. first: step 0 starts the
// scanline (L = C). Costs are read R steps ahead.
template <int K, bool N16, typename At>
__device__ __forceinline__ void plain_chunk(At at, bool first, Plain4<K, N16>& st) {
  constexpr int C = kScanChunk, R = 16;
  uint32_t ring[R];
#pragma unroll
  for (int j = 0; j < R; ++j) ring[j] = *at(j);
#pragma unroll
  for (int j = 0; j < C; ++j) {
    const uint32_t w = ring[j % R];
    if (j + R < C) ring[j % R] = *at(j + R);
    *at(j) = (LaneBytes<K>)st.advance(w, j == 0 && first);
  }
}

// Horizontal scans of a plain level; warp (blockIdx.x * WPB + w) owns scanline i = (view, dir, y)
// as in hpaths3_lane. A chunk is 32 consecutive pixels of the row: one contiguous bulk copy in,
// one out. Right-to-left scans place a short (last) chunk at the end of the buffer, so that step
// j of every chunk reads row 31 - j.
template <int K>
__host__ __device__ constexpr int hscan_plain4_warps() { return K == 4 ? 2 : 4; }

template <int K, bool N16, int WPB = hscan_plain4_warps<K>()>
__global__ void __launch_bounds__(32 * WPB) k_hscan_plain4(const uint8_t* __restrict__ cost, uint8_t* __restrict__ lr,
                                                           uint8_t* __restrict__ rl, PlainParams P, int nviews) {
  constexpr int D = 32 * K, C = kScanChunk, NB = 3;
  __shared__ __align__(128) uint8_t cbuf[WPB][NB][C * D];
  __shared__ __align__(8) uint64_t bars[WPB][NB];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    for (int b = 0; b < NB; ++b) mbar_init(&bars[w][b], 1);
    mbar_fence_init();
  }
  __syncwarp();
  const int H = P.H, W = P.W;
  const int i = blockIdx.x * WPB + w;
  if (i >= nviews * 2 * H) return;  // the whole warp
  const int grp = i / H, y = i - grp * H;
  const int view = P.view0 + (grp >> 1), dir = grp & 1;
  const int len = W - P.x0;
  if (len <= 0) return;
  const size_t ro = (size_t)view * P.vstride + (size_t)y * W * D;
  const uint8_t* crow = cost + ro;
  uint8_t* orow = (dir == 0 ? lr : rl) + ro;
  const int nch = (len + C - 1) / C;
  auto chunk_n = [&](int c) { return min(C, len - c * C); };
  auto chunk_x = [&](int c) { return dir == 0 ? P.x0 + c * C : W - (c * C + chunk_n(c)); };
  auto chunk_off = [&](int c) { return dir == 0 ? 0 : (C - chunk_n(c)) * D; };  // bytes into the buffer
  auto issue = [&](int c) {  // lane 0
    const int b = c % NB;
    const uint32_t bytes = (uint32_t)chunk_n(c) * D;
    mbar_expect_tx(&bars[w][b], bytes + (c == 0 && g_short_copy ? 16u : 0u));
    bulk_to_smem(cbuf[w][b] + chunk_off(c), crow + (size_t)chunk_x(c) * D, bytes, &bars[w][b]);
  };
  if (lane == 0) {
    issue(0);
    if (nch > 1) issue(1);
  }
  uint32_t phase = 0u;
  Plain4<K, N16> st(P);
  for (int c = 0; c < nch; ++c) {
    const int b = c % NB, n = chunk_n(c);
    if (!mbar_wait_warp(&bars[w][b], (phase >> b) & 1u)) {
      scan_give_up_mask(bars[w], phase, (1u << b) | (c + 1 < nch ? 1u << ((c + 1) % NB) : 0u));
      if (lane == 0) bulk_wait_all();
      return;
    }
    phase ^= 1u << b;
    __syncwarp();
    LaneBytes<K>* lb = reinterpret_cast<LaneBytes<K>*>(cbuf[w][b]) + lane;
    if (dir == 0)
      plain_chunk<K, N16>([lb](int j) { return lb + j * 32; }, c == 0, st);
    else
      plain_chunk<K, N16>([lb](int j) { return lb + (C - 1 - j) * 32; }, c == 0, st);
    fence_proxy_async();  // the chunk's path costs (and its cost reads) before the bulk copies
    __syncwarp();
    if (lane == 0) {
      bulk_to_global(orow + (size_t)chunk_x(c) * D, cbuf[w][b] + chunk_off(c), (uint32_t)n * D);
      bulk_commit();
      if (c + 2 < nch) {
        bulk_wait_read<1>();  // the store of chunk c - 1 has left the buffer chunk c + 2 goes to
        issue(c + 2);
      }
    }
  }
  if (lane == 0) bulk_wait_all();
}

// WTA of one plain-level pixel from its four path rows (D bytes each), by one lane:
// Kernel_ComputeDisparityByWTA_Warpfor{32,64,128} (cusgm_ca.cu:3514-3809). S(d) (at most 4 x 255)
// is summed in 16-bit halves and searched as the 16-bit key S(d) * 64 + (d mod 64) -- the lowest
// key of a block of 64 disparities is its minimum at its lowest d (with 63 - (d mod 64): at its
// highest d). d* = 0 or d* >= Q.dmax_excl -> INVALID; c3 at d* = D - 1 is the index itself;
// uniqueness and the +0.5-shifted parabola as in wta_pixel. Tie rules: kTieRefB200 at D = 64
// (A = {t < 32 : S(t) = m}, B = {t < 32 : S(t + 32) = m, S(t) != m}; even rows of the launch take
// the lowest of B (+ 32) if any, else of A; odd rows the lowest of A if any, else of B (+ 32));
// kTieHighest the highest tied d; the rest the lowest.
// a, b, c, e: the pixel's rows in four swizzled boxes (16-byte unit u of the row at u ^ sw).
template <int D>
__device__ __forceinline__ float plain_wta_rows(const uint8_t* a, const uint8_t* b, const uint8_t* c,
                                                const uint8_t* e, int sw, int min_d, int y, const WtaParams& Q) {
  constexpr int SPLIT = D == 64 ? 32 : 64;  // first d of the second key block (D = 64: A / B halves)
  const bool high = Q.tie_rule == kTieHighest;
  const uint32_t flip = high ? 63u * 0x10001u : 0u;
  uint32_t acc0 = 0xFFFFFFFFu, acc1 = 0xFFFFFFFFu;
#pragma unroll
  for (int q = 0; q < D / 16; ++q) {
    const int u = q ^ sw;
    const uint4 va = reinterpret_cast<const uint4*>(a)[u], vb = reinterpret_cast<const uint4*>(b)[u];
    const uint4 vc = reinterpret_cast<const uint4*>(c)[u], ve = reinterpret_cast<const uint4*>(e)[u];
    const uint32_t wa[4] = {va.x, va.y, va.z, va.w}, wb[4] = {vb.x, vb.y, vb.z, vb.w};
    const uint32_t wc[4] = {vc.x, vc.y, vc.z, vc.w}, we[4] = {ve.x, ve.y, ve.z, ve.w};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int d0 = 16 * q + 4 * t;  // the word's first disparity
      // lo = S(d0) | S(d0 + 2) << 16, hi = S(d0 + 1) | S(d0 + 3) << 16
      uint32_t lo, hi;
      sum4_bytes(wa[t], wb[t], wc[t], we[t], lo, hi);
      const uint32_t dlo = (uint32_t)(d0 & 63) | ((uint32_t)((d0 + 2) & 63) << 16);
      const uint32_t dhi = dlo + 0x10001u;
      const uint32_t klo = lo * 64u + (dlo ^ flip), khi = hi * 64u + (dhi ^ flip);
      if (d0 < SPLIT) acc0 = __vimin3_u16x2(acc0, klo, khi);
      else acc1 = __vimin3_u16x2(acc1, klo, khi);
    }
  }
  const uint32_t k0 = min(acc0 & 0xFFFFu, acc0 >> 16), k1 = min(acc1 & 0xFFFFu, acc1 >> 16);
  const uint32_t s0 = k0 >> 6, s1 = k1 >> 6;
  // the disparities of the two keys (block 1 of D = 128 starts at 64; D = 64's halves share d mod 64 = d)
  const int t0 = (int)((k0 & 63u) ^ (flip & 63u)), t1 = (D == 128 ? 64 : 0) + (int)((k1 & 63u) ^ (flip & 63u));
  uint32_t m;
  int ds;
  if constexpr (D == 32) {
    m = s0;
    ds = t0;
  } else {
    m = min(s0, s1);
    // the lowest (highest) tied d of the two blocks
    ds = s0 < s1 || (s0 == s1 && !high) ? t0 : t1;
    if (D == 64 && Q.tie_rule == kTieRefB200 && s0 == s1) {
      // both halves hold the minimum: odd rows take A's lowest (t0); even rows B's lowest if B is
      // not empty (a t with S(t + 32) = m and S(t) != m; rare, searched directly)
      ds = t0;
      if ((y & 1) == 0) {
        for (int t = 0; t < 32; ++t) {
          const int ob = (t + 32) ^ (sw << 4), oa = t ^ (sw << 4);
          const uint32_t sb = (uint32_t)a[ob] + b[ob] + c[ob] + e[ob];
          const uint32_t sa = (uint32_t)a[oa] + b[oa] + c[oa] + e[oa];
          if (sb == m && sa != m) {
            ds = t + 32;
            break;
          }
        }
      }
    }
  }
  if (ds <= 0 || ds >= Q.dmax_excl) return kInvalidFloat;
  auto sum_at = [&](int d) {
    const int o = d ^ (sw << 4);
    return (uint32_t)a[o] + b[o] + c[o] + e[o];
  };
  const float c1 = (float)sum_at(ds - 1);
  const float c2 = (float)m;
  const float c3 = (ds + 1 < D) ? (float)sum_at(ds + 1) : (float)ds;
  const float d12 = __fsub_rn(c1, c2), d32 = __fsub_rn(c3, c2);
  const float uq = d12 < d32 ? d12 : d32;
  if (uq <= __fmul_rn(c2, __fsub_rn(1.0f, Q.uniqueness))) return kInvalidFloat;
  return __fadd_rn((float)(ds + min_d), subpix_bias(c1, c2, c3));
}

// Warps per CTA of the column kernels (shared memory per warp: PASS 1 three boxes, PASS 2 two
// boxes of costs and three of stored paths, C x D bytes each).
template <int K>
__host__ __device__ constexpr int vscan_plain4_warps() { return K == 4 ? 2 : 4; }

// Vertical scans of a plain level: warp (blockIdx.x * WPB + w) owns column x of view P.view0 + blockIdx.y.
// PASS 1: bottom to top over boxes ending at rows H - 32c (the last one starts above row 0 and
// reads zeros there), storing its path costs (bt) box by box -- the last box row by row. PASS 2:
// top to bottom over boxes starting at rows 32c, then per box the WTA of its pixels with lane =
// pixel (rows >= Q.rows INVALID, as the reference's two-row WTA blocks leave them; border and
// columns left of x0 INVALID). Maps: the cost, bt, lr and rl volumes, [views][H][W * D] bytes.
template <int K, int PASS, bool N16>
__global__ void __launch_bounds__(32 * vscan_plain4_warps<K>())
    k_vscan_plain4(const __grid_constant__ CUtensorMap m_cost, const __grid_constant__ CUtensorMap m_bt,
                   const __grid_constant__ CUtensorMap m_lr, const __grid_constant__ CUtensorMap m_rl,
                   uint8_t* __restrict__ bt, float* __restrict__ disp, PlainParams P, WtaParams Q) {
  constexpr int D = 32 * K, C = kScanChunk, BOX = C * D, NSW = D / 16;
  constexpr int WPB = vscan_plain4_warps<K>();
  constexpr int NB = PASS == 1 ? 3 : 2;  // cost boxes
  constexpr int NS = PASS == 1 ? 0 : 3;  // stored-path boxes (bt, lr, rl)
  __shared__ __align__(1024) uint8_t cbuf[WPB][NB + NS][BOX];
  __shared__ __align__(8) uint64_t bars[WPB][NB + 1];  // bars[NB]: the stored paths
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    for (int b = 0; b <= NB; ++b) mbar_init(&bars[w][b], 1);
    mbar_fence_init();
  }
  __syncwarp();
  const int W = P.W, H = P.H;
  const int x = blockIdx.x * WPB + w;
  const int view = P.view0 + blockIdx.y;
  if (x >= W) return;  // the whole warp
  float* dout = disp + (size_t)view * Q.dstride + x;
  if (x < P.x0) {
    if (PASS == 2)
      for (int y = lane; y < H; y += 32) dout[(size_t)y * W] = kInvalidFloat;
    return;
  }
  // the swizzle pattern is a function of the shared address: the boxes must start on 1 KB
  if (smem_u32(&cbuf[0][0][0]) & 1023u) {
    if (lane == 0) atomicAdd(&g_scan_wait_timeouts, 1u);
    return;
  }
  const int nch = (H + C - 1) / C;
  auto box_y = [&](int c) { return PASS == 1 ? H - C * (c + 1) : C * c; };  // first row of chunk c's box
  auto issue_cost = [&](int c) {  // lane 0
    const int b = c % NB;
    mbar_expect_tx(&bars[w][b], BOX);
    tma_load_3d(cbuf[w][b], &m_cost, x * D, box_y(c), view, &bars[w][b]);
  };
  auto issue_paths = [&](int c) {  // lane 0
    mbar_expect_tx(&bars[w][NB], 3 * BOX);
    tma_load_3d(cbuf[w][NB + 0], &m_bt, x * D, box_y(c), view, &bars[w][NB]);
    tma_load_3d(cbuf[w][NB + 1], &m_lr, x * D, box_y(c), view, &bars[w][NB]);
    tma_load_3d(cbuf[w][NB + 2], &m_rl, x * D, box_y(c), view, &bars[w][NB]);
  };
  if (lane == 0) {
    issue_cost(0);
    if (nch > 1) issue_cost(1);
    if (PASS == 2) issue_paths(0);
  }
  // this lane's K bytes of a box row under each of the NSW swizzle patterns
  int lane_off[NSW];
#pragma unroll
  for (int v = 0; v < NSW; ++v) lane_off[v] = (K * lane) ^ (v << 4);
  uint32_t phase = 0u;  // bit b: parity awaited on bars[w][b]
  Plain4<K, N16> st(P);
  const bool col_ok = x >= Q.xlo && x <= Q.xhi;
  for (int c = 0; c < nch; ++c) {
    const int b = c % NB;
    const uint32_t pend_cost = (1u << b) | (c + 1 < nch ? 1u << ((c + 1) % NB) : 0u);
    if (!mbar_wait_warp(&bars[w][b], (phase >> b) & 1u)) {
      scan_give_up_mask(bars[w], phase, pend_cost | (PASS == 2 ? 1u << NB : 0u));
      if (lane == 0) bulk_wait_all();
      return;
    }
    phase ^= 1u << b;
    __syncwarp();
    uint8_t* box = cbuf[w][b];
    // step j: box row C - 1 - j (PASS 1) or j (PASS 2)
    plain_chunk<K, N16>(
        [&](int j) {
          const int r = PASS == 1 ? C - 1 - j : j;
          return reinterpret_cast<LaneBytes<K>*>(box + r * D + lane_off[box_sw<D>(r)]);
        },
        c == 0, st);
    if constexpr (PASS == 1) {
      fence_proxy_async();
      __syncwarp();
      const int y0 = box_y(c);
      if (y0 >= 0) {
        if (lane == 0) {
          tma_store_3d(&m_bt, x * D, y0, view, box);
          bulk_commit();
        }
      } else if (lane < C + y0) {  // the top box: rows 0 .. C + y0 - 1 of the column, one per lane
        const int r = lane - y0;     // box row of image row `lane`
        const uint4* src = reinterpret_cast<const uint4*>(box + r * D);
        uint4* dst = reinterpret_cast<uint4*>(bt + (size_t)view * P.vstride + ((size_t)lane * W + x) * D);
#pragma unroll
        for (int u = 0; u < NSW; ++u) dst[u] = src[u ^ box_sw<D>(r)];
      }
      if (lane == 0 && c + 2 < nch) {
        bulk_wait_read<1>();  // the store of chunk c - 1 has left the box chunk c + 2 goes to
        issue_cost(c + 2);
      }
    } else {
      __syncwarp();  // the chunk's path costs, written by disparity, are read by pixel
      if (!mbar_wait_warp(&bars[w][NB], (phase >> NB) & 1u)) {
        scan_give_up_mask(bars[w], phase, (1u << NB) | (c + 1 < nch ? 1u << ((c + 1) % NB) : 0u));
        return;
      }
      phase ^= 1u << NB;
      const int y = C * c + lane;
      if (y < H) {
        float dv = kInvalidFloat;
        if (col_ok && y >= Q.ylo && y <= Q.yhi && y < Q.rows)
          dv = plain_wta_rows<D>(box + lane * D, cbuf[w][NB] + lane * D, cbuf[w][NB + 1] + lane * D,
                                 cbuf[w][NB + 2] + lane * D, box_sw<D>(lane), P.min_d, y, Q);
        dout[(size_t)y * W] = dv;
      }
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
