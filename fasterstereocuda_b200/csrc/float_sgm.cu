// Differentiable float32 SGM: 4-path hard-min recurrence with per-pixel P1/P2 maps, summed over the
// paths, followed by a soft-argmin disparity; and its adjoint.
//
// No counterpart in the reference (it is the training/serving addition beside the bit-exact path).
// The recurrence is the reference's path recurrence (cusgm_ca.cu:1517-1564) in float with the
// penalties read at the current pixel and +inf beyond d = 0 and d = D-1:
//   L_p(d) = C_p(d) + min(L_q(d), L_q(d-1)+P1(p), L_q(d+1)+P1(p), m_q+P2(p)) - m_q,  m_q = min_k L_q(k)
//   S(p,d) = ((L_0 + L_1) + L_2) + L_3;  disp(p) = sum_d d * softmax_d(-S(p,d)/T)
// Ties of the hard minima are broken in the fixed order same d, d-1, d+1, jump (lowest k for m_q).
//
// Mapping, forward: one warp per scanline, lane l holding the K = D/32 consecutive disparities
// K l .. K l + K - 1; the per-pixel minimum is one REDUX on the floats, the d +- 1 terms stay in the
// lane except at its edges (one shuffle up, one down). Inputs move in chunks of kFC positions: a row
// chunk is one contiguous bulk copy, a column chunk one box of a 3D tensor map (TMA),
// double-buffered on mbarriers with bounded waits; the penalties are loaded one chunk ahead. A row
// scan is a chain of W dependent steps, so everything that does not depend on the path costs is
// kept off it.
// All four directions run in ONE launch (their blocks side by side, the long row scans first),
// each writing its own path volume; the soft-argmin kernel adds the four in path order. The
// backward launch likewise runs the four adjoint scans at once, each writing its own gradient
// volume and penalty-map gradients, and a last kernel adds them in path order.
//
// Backward: the forward scans record which candidate gave every L_p(d) and where m_q lies (2 bits
// per voxel and a byte per pixel of each path: a quarter of one volume pass for all four paths), and
// the adjoint routes the gradient of every L_p(d) to C_p(d), to P1(p) or P2(p) and to L_q by them.
// Storing path states every 8 pixels and repeating the recurrence in the backward read the cost
// volume a second time and ran the longer half of the backward's chain: 4 x 1242x375 x 64, scan
// 1576 -> 772 us (eight lanes a line then), with the recording forward scan at 640 us (645 before it).
// Mapping, backward: a scanline is held by G lanes of a warp, kBwdK disparities per lane (16 lanes at
// D = 64), sums by butterflies; the gradient of S is copied kBwdPF - 1 steps ahead. At that size
// 3.93 GB in 735 us, 5.3 TB/s; one image alone is bound by its row steps (~270 ns each).
//
// Layouts: cost/sum/grad volumes float [B][H][W][D] (16-byte aligned); maps float [B][H][W];
// records in four slabs of ckpt, one per path. Paths: 0 top->bottom, 1 left->right,
// 2 bottom->top, 3 right->left.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <string>
#include <type_traits>

#include "../../include/sgm_b200.h"
#include "sgm_async.cuh"
#include "sgm_tma.h"

void sgm_set_process_error(const char* msg);

namespace {

constexpr unsigned kFullMask = 0xFFFFFFFFu;
constexpr int kK = 8;       // disparities per lane of the soft-argmin kernels
constexpr int kSeg = 8;     // positions per segment of recorded choices
constexpr int kBwdK = 4;    // disparities per lane of the backward scans
constexpr int kBwdPF = 8;   // slots of the backward scans' copies ahead (divides kSeg)
constexpr int kWarps = 4;   // warps per block of the scan kernels
constexpr int kFC = 16;     // steps per staged chunk of the forward scans (a multiple of kSeg)
#define kInf __int_as_float(0x7f800000)

struct Geo {
  int B, H, W, D;
  int dir;
  int lines, len, nseg;
};

__host__ __device__ inline Geo make_geo(int B, int H, int W, int D, int dir) {
  Geo g;
  g.B = B; g.H = H; g.W = W; g.D = D; g.dir = dir;
  const bool horiz = dir == 1 || dir == 3;
  g.lines = horiz ? B * H : B * W;
  g.len = horiz ? W : H;
  g.nseg = (g.len + kSeg - 1) / kSeg;
  return g;
}

template <int G>
__device__ __forceinline__ float group_min(float v) {
#pragma unroll
  for (int o = G / 2; o; o >>= 1) v = fminf(v, __shfl_xor_sync(kFullMask, v, o));
  return v;
}
template <int G>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = G / 2; o; o >>= 1) v += __shfl_xor_sync(kFullMask, v, o);
  return v;
}

// minimum of K values as a balanced tree
template <int K>
__device__ __forceinline__ float minK(const float (&v)[K]) {
  float t[K];
#pragma unroll
  for (int i = 0; i < K; ++i) t[i] = v[i];
#pragma unroll
  for (int w = 1; w < K; w *= 2)
#pragma unroll
    for (int i = 0; i + w < K; i += 2 * w) t[i] = fminf(t[i], t[i + w]);
  return t[0];
}

template <int K>
__device__ __forceinline__ void loadK(const float* p, float (&v)[K]) {
#pragma unroll
  for (int h = 0; h < K / 4; ++h) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p) + h);
    v[4 * h] = a.x; v[4 * h + 1] = a.y; v[4 * h + 2] = a.z; v[4 * h + 3] = a.w;
  }
}
template <int K>
__device__ __forceinline__ void storeK(float* p, const float (&v)[K]) {
#pragma unroll
  for (int h = 0; h < K / 4; ++h)
    reinterpret_cast<float4*>(p)[h] = make_float4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
}

// Blocks of the four directions side by side in one grid: slot i (direction order[i]) owns blocks
// [first_block[i], first_block[i + 1]).
struct Grid4 {
  Geo g[4];
  int order[4];
  int first_block[5];
};

struct Line {
  int dir, line;
  bool live;  // false for the padding lanes of a warp past the direction's last line
};

// The line of this thread; false if the whole warp is past the direction's lines.
template <int G>
__device__ __forceinline__ bool locate(const Grid4& q, Line& ln, Geo& g) {
  const int b = blockIdx.x;
  const int slot = (b >= q.first_block[1]) + (b >= q.first_block[2]) + (b >= q.first_block[3]);
  ln.dir = q.order[slot];
  g = q.g[ln.dir];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wline = ((b - q.first_block[slot]) * kWarps + warp) * (32 / G);
  if (wline >= g.lines) return false;
  const int mine = wline + lane / G;
  ln.live = mine < g.lines;
  ln.line = ln.live ? mine : g.lines - 1;
  return true;
}

// The adjoint needs, per pixel and path, which of the four candidates gave every L_p(d) (2 bits) and
// the lowest k with L_q(k) = m_q: the forward scans record both, so that the backward scans neither
// read the cost volume nor repeat the recurrence. Records of a direction live in its checkpoint slab
// (slab_elems floats), per line and segment of kSeg positions:
//   codes  32 words (one per forward lane, 2K bits per slot: 32 bits at D = 64, 16 at D = 32)
//   argmin kSeg bytes
// Slot t of a segment is the t-th pixel in the order in which the adjoint walks it (against the
// path): position 7 - t on paths of ascending position, t on descending ones.
// codes: 0 same d, 1 d-1, 2 d+1, 3 jump (the first of equal candidates; 0 unless another is smaller, so
// also where L_q(d) is NaN, after a pixel whose costs are all infinite).
template <int K>
using CodeWord = typename std::conditional<K == 2, uint32_t, uint16_t>::type;

template <int K>
__host__ __device__ constexpr size_t code_bytes(size_t lines, size_t nseg) {
  return lines * nseg * 32 * sizeof(CodeWord<K>);
}

struct FwdArgs {
  const float* cost;
  const float* p1;
  const float* p2;
  float* out[4];   // path volumes, one per direction
  float* rec[4];   // record slabs, one per direction
  Grid4 q;         // one line per warp
};

__device__ __forceinline__ float warp_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

// The records of one line being written: the current segment's codes of this lane and argmins.
struct Rec {
  uint32_t code = 0, arg[2] = {0, 0};
};

// One forward step of a warp-held scanline (lane l: d = K l + j) into slot `slot` of r.
// At K = 2 the edge lanes' shuffles return their own value: lane 0's "d-1" is then its own d+1
// candidate and lane 31's "d+1" its own d-1 candidate, so no minimum changes and no select is
// needed; only lane 0's code says 1 for 2, which store_rec puts right.
template <int K, bool REC>
__device__ __forceinline__ void fstep_warp(float (&L)[K], const float (&c)[K], float& m, float p1, float p2, Rec& r,
                                           int slot) {
  const int lane = threadIdx.x & 31;
  const float jump = m + p2;
  if constexpr (REC) {
    uint32_t arg;  // lowest k with L(k) = m
    if constexpr (K == 2) {
      const uint32_t e0 = __ballot_sync(kFullMask, L[0] == m), e1 = __ballot_sync(kFullMask, L[1] == m);
      const int first = __ffs(e0 | e1) - 1;
      arg = 2 * first + (((e0 >> (first & 31)) & 1u) ^ 1u);
    } else {
      arg = __ffs(__ballot_sync(kFullMask, L[0] == m)) - 1;
    }
    r.arg[slot / 4] |= (arg & 0xffu) << (8 * (slot % 4));
  }
  float lm[K], lp[K];
  if constexpr (K == 2) {
    const float2 a = __fadd2_rn(make_float2(L[0], L[1]), make_float2(p1, p1));
    lm[0] = __shfl_up_sync(kFullMask, a.y, 1);
    lp[1] = __shfl_down_sync(kFullMask, a.x, 1);
    lp[0] = a.y;
    lm[1] = a.x;
  } else {
    const float a = L[0] + p1;
    const float left = __shfl_up_sync(kFullMask, a, 1), right = __shfl_down_sync(kFullMask, a, 1);
    lm[0] = lane > 0 ? left : kInf;
    lp[0] = lane < 31 ? right : kInf;
  }
  float t[K];
#pragma unroll
  for (int j = 0; j < K; ++j) {
    t[j] = fminf(fminf(fminf(L[j], lm[j]), lp[j]), jump);
    if constexpr (REC) {
      const int sh = 2 * K * slot + 2 * j;
      const bool q0 = t[j] < L[j], q1 = q0 && lm[j] != t[j], q2 = q1 && lp[j] != t[j];
      if (q0) r.code += 1u << sh;
      if (q1) r.code += 1u << sh;
      if (q2) r.code += 1u << sh;
    }
  }
  if constexpr (K == 2) {
    const float2 n = __fadd2_rn(__fadd2_rn(make_float2(c[0], c[1]), make_float2(t[0], t[1])), make_float2(-m, -m));
    L[0] = n.x;
    L[1] = n.y;
    m = warp_min(fminf(n.x, n.y));
  } else {
    L[0] = c[0] + t[0] - m;
    m = warp_min(L[0]);
  }
}

template <int K>
__device__ __forceinline__ void ld_lane(const float* p, float (&v)[K]) {
  if constexpr (K == 2) {
    const float2 x = *reinterpret_cast<const float2*>(p);
    v[0] = x.x;
    v[1] = x.y;
  } else {
    v[0] = p[0];
  }
}
template <int K>
__device__ __forceinline__ void st_lane(float* p, const float (&v)[K]) {
  if constexpr (K == 2)
    *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  else
    p[0] = v[0];
}

// Pixel index of position 0 of a line and the pixel stride of one position (positions ascend with
// x or y; paths 2 and 3 run through them downwards).
__device__ __forceinline__ void line_positions(const Geo& g, int line, long long& base, long long& step) {
  if (g.dir == 1 || g.dir == 3) {  // line = b*H + y
    base = (long long)line * g.W;
    step = 1;
  } else {  // line = b*W + x
    const int b = line / g.W;
    base = (long long)b * g.H * g.W + (line - b * g.W);
    step = g.W;
  }
}

// Shared memory of the forward kernel: per warp two chunk buffers of kFC x D floats.
template <int K>
constexpr size_t fwd_smem_bytes() {
  return (size_t)kWarps * 2 * kFC * 32 * K * sizeof(float);
}

// tm_cost: the cost volume as a 3D tensor map (floats of a row, rows, images), boxes of D x kFC x 1.
template <int K, bool REC>
__global__ void __launch_bounds__(kWarps * 32) k_float_fwd(const __grid_constant__ CUtensorMap tm_cost,
                                                           const FwdArgs a) {
  constexpr int D = 32 * K, C = kFC, NB = 2;
  extern __shared__ __align__(128) float fsm[];
  __shared__ __align__(8) uint64_t bars[kWarps][NB];
  __shared__ float2 pens[kWarps][NB][C];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    for (int b = 0; b < NB; ++b) sgm::mbar_init(&bars[w][b], 1);
    sgm::mbar_fence_init();
  }
  __syncwarp();
  Line ln;
  Geo g;
  if (!locate<32>(a.q, ln, g)) return;  // the whole warp
  long long base, step;
  line_positions(g, ln.line, base, step);
  const bool horiz = g.dir == 1 || g.dir == 3;
  const bool rev = g.dir == 2 || g.dir == 3;
  float* box0 = fsm + (size_t)w * NB * C * D;
  const int len = g.len, nch = (len + C - 1) / C;
  // chunk c holds positions cC .. cC + n - 1 in buffer rows 0 .. n - 1; descending paths take the
  // chunks, and the positions in them, from the end
  auto chunk_at = [&](int it) { return rev ? nch - 1 - it : it; };
  auto chunk_n = [&](int c) { return min(C, len - c * C); };
  auto issue = [&](int it) {  // lane 0
    const int b = it % NB, c = chunk_at(it);
    float* dst = box0 + b * C * D;
    if (horiz) {
      const uint32_t bytes = (uint32_t)(chunk_n(c) * D * sizeof(float));
      sgm::mbar_expect_tx(&bars[w][b], bytes);
      sgm::bulk_to_smem(dst, a.cost + (base + (long long)c * C) * D, bytes, &bars[w][b]);
    } else {  // column x of image bi; rows past the image read as zeros
      const int bi = ln.line / g.W, x = ln.line - bi * g.W;
      sgm::mbar_expect_tx(&bars[w][b], (uint32_t)(C * D * sizeof(float)));
      sgm::tma_load_3d(dst, &tm_cost, x * D, c * C, bi, &bars[w][b]);
    }
  };
  // the penalties of position `lane` of the chunk of iteration it
  auto pen = [&](int it, float2& q) {
    q = make_float2(0.f, 0.f);
    const int c = chunk_at(it);
    if (it < nch && lane < chunk_n(c)) {
      const long long p = base + ((long long)c * C + lane) * step;
      q = make_float2(__ldg(a.p1 + p), __ldg(a.p2 + p));
    }
  };
  if (lane == 0) {
    issue(0);
    if (nch > 1) issue(1);
  }
  float2 pq;
  pen(0, pq);
  uint32_t phase = 0u;  // bit b: parity of buffer b's next phase
  float L[K], m = 0.f;
  const long long od = step * D;
  auto* codes = reinterpret_cast<CodeWord<K>*>(a.rec[g.dir]) + (size_t)ln.line * g.nseg * 32 + lane;
  uint2* args = reinterpret_cast<uint2*>(reinterpret_cast<char*>(a.rec[g.dir]) + code_bytes<K>(g.lines, g.nseg)) +
                (size_t)ln.line * g.nseg;
  auto run = [&](auto rev_c, float* out) {
    constexpr bool REV = decltype(rev_c)::value;
    for (int it = 0; it < nch; ++it) {
      const int b = it % NB, c = chunk_at(it), n = chunk_n(c);
      if (lane < C) pens[w][b][lane] = pq;
      pen(it + 1, pq);  // a chunk ahead
      if (!sgm::mbar_wait_warp(&bars[w][b], (phase >> b) & 1u)) {
        sgm::scan_give_up_mask(bars[w], phase, (1u << b) | (it + 1 < nch ? 1u << ((it + 1) % NB) : 0u));
        return;
      }
      phase ^= 1u << b;
      __syncwarp();
      const float* bx = box0 + b * C * D + lane * K;
      float cv[C][K];
#pragma unroll
      for (int j = 0; j < C; ++j) ld_lane<K>(bx + j * D, cv[j]);
      sgm::fence_proxy_async();  // this lane's reads of the buffer before the copy that refills it
      __syncwarp();
      if (lane == 0 && it + 2 < nch) issue(it + 2);
      float* op = out + (base + (long long)c * C * step) * D;  // position 0 of the chunk
      const int first = REV ? len - 1 - c * C : -c * C;        // the path's first pixel, as a row of this chunk
      Rec r;
      auto one = [&](int j) {
        const int slot = REV ? j % kSeg : kSeg - 1 - j % kSeg;
        if (j == first) {
#pragma unroll
          for (int t = 0; t < K; ++t) L[t] = cv[j][t];
          m = warp_min(minK<K>(L));
        } else {
          const float2 P = pens[w][b][j];
          fstep_warp<K, REC>(L, cv[j], m, P.x, P.y, r, slot);
        }
        st_lane<K>(op + j * od, L);
      };
      auto store_rec = [&](int h) {  // segment h of the chunk
        if (!REC) return;
        const int seg = c * (C / kSeg) + h;
        if (seg < g.nseg) {
          if (K == 2 && lane == 0) {  // d = 0 has no d-1: its code 1 is the d+1 candidate
            const uint32_t x = r.code & ~(r.code >> 1) & 0x11111111u;
            r.code ^= 3u * x;
          }
          codes[(size_t)seg * 32] = (CodeWord<K>)r.code;
          if (lane == 0) args[seg] = make_uint2(r.arg[0], r.arg[1]);
        }
        r = Rec();
      };
      const bool whole = n == C && (first < 0 || first >= C);
      if (whole) {
#pragma unroll
        for (int i = 0; i < C; ++i) {
          const int j = REV ? C - 1 - i : i;
          const int slot = REV ? j % kSeg : kSeg - 1 - j % kSeg;
          const float2 P = pens[w][b][j];
          fstep_warp<K, REC>(L, cv[j], m, P.x, P.y, r, slot);
          st_lane<K>(op + j * od, L);
          if (i % kSeg == kSeg - 1) store_rec(j / kSeg);
        }
      } else {  // a short chunk, or the one with the path's first pixel
#pragma unroll
        for (int i = 0; i < C; ++i) {
          const int j = REV ? C - 1 - i : i;
          if (j < n) one(j);
          if (i % kSeg == kSeg - 1) store_rec(j / kSeg);
        }
      }
    }
  };
  if (rev)
    run(std::true_type{}, a.out[g.dir] + lane * K);
  else
    run(std::false_type{}, a.out[g.dir] + lane * K);
}

// S = ((L0 + L1) + L2) + L3, written over L0 for a backward pass; disp = sum_d d softmax(-S/T)
template <int G, bool STORE>
__global__ void __launch_bounds__(256) k_soft_argmin_fwd(float* __restrict__ sum, const float* __restrict__ l1,
                                                         const float* __restrict__ l2, const float* __restrict__ l3,
                                                         float* __restrict__ disp, size_t npix, float inv_t) {
  constexpr int D = G * kK;
  const size_t first = ((size_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * (32 / G);
  if (first >= npix) return;
  const size_t mine = first + (threadIdx.x & 31) / G;
  const bool live = mine < npix;
  const size_t p = live ? mine : npix - 1;
  const int gl = threadIdx.x % G;
  const size_t off = p * D + gl * kK;
  float S[kK], b[kK], c[kK], d[kK];
  loadK<kK>(sum + off, S);
  loadK<kK>(l1 + off, b);
  loadK<kK>(l2 + off, c);
  loadK<kK>(l3 + off, d);
#pragma unroll
  for (int j = 0; j < kK; ++j) S[j] = ((S[j] + b[j]) + c[j]) + d[j];
  if (STORE && live) storeK<kK>(sum + off, S);
  const float mn = group_min<G>(minK<kK>(S));
  float z = 0.f, num = 0.f;
#pragma unroll
  for (int j = 0; j < kK; ++j) {
    const float e = expf(-(S[j] - mn) * inv_t);
    z += e;
    num += e * (float)(gl * kK + j);
  }
  z = group_sum<G>(z);
  num = group_sum<G>(num);
  if (live && gl == 0) disp[p] = num / z;
}

// dS = -gdisp/T * w(d) * (d - disp), w = softmax(-S/T)
template <int G>
__global__ void __launch_bounds__(256) k_soft_argmin_bwd(const float* __restrict__ sum,
                                                         const float* __restrict__ gdisp, float* __restrict__ gsum,
                                                         size_t npix, float inv_t) {
  constexpr int D = G * kK;
  const size_t first = ((size_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * (32 / G);
  if (first >= npix) return;
  const size_t mine = first + (threadIdx.x & 31) / G;
  const bool live = mine < npix;
  const size_t p = live ? mine : npix - 1;
  const int gl = threadIdx.x % G;
  const size_t off = p * D + gl * kK;
  float S[kK], e[kK];
  loadK<kK>(sum + off, S);
  const float mn = group_min<G>(minK<kK>(S));
  float z = 0.f, num = 0.f;
#pragma unroll
  for (int j = 0; j < kK; ++j) {
    e[j] = expf(-(S[j] - mn) * inv_t);
    z += e[j];
    num += e[j] * (float)(gl * kK + j);
  }
  z = group_sum<G>(z);
  num = group_sum<G>(num);
  const float dd = num / z;
  const float gd = __ldg(gdisp + p);
  const float scale = -gd * inv_t / z;
  float gs[kK];
#pragma unroll
  for (int j = 0; j < kK; ++j) gs[j] = scale * e[j] * ((float)(gl * kK + j) - dd);
  if (live) storeK<kK>(gsum + off, gs);
}

struct BwdArgs {
  const float* gsum;
  const float* rec[4];  // the forward scans' records
  float* gout[4];       // gradient volumes, one per direction (written)
  float* gp1[4];        // penalty-map gradients, one per direction (written)
  float* gp2[4];
  Grid4 q;
};

// Codes of the lane's K disparities over one segment: K / 2 words; the two bits of voxel t in slot j.
template <int FK>
__device__ __forceinline__ constexpr int code_shift(int t, int j) {
  return FK == 2 ? 4 * j + 2 * (t & 1) : 16 * (t & 1) + 2 * j;
}

// Sums over the line's G lanes of 2 kSeg values per lane: afterwards lane gl holds in v[0 ..
// 2 kSeg / G) the sums of values gl * 2 kSeg / G onwards.
template <int G>
__device__ __forceinline__ void reduce_segment(float (&v)[2 * kSeg], int gl) {
  int n = 2 * kSeg;
#pragma unroll
  for (int o = G / 2; o; o >>= 1) {
    n /= 2;
    const bool hi = gl & o;
#pragma unroll
    for (int i = 0; i < kSeg; ++i)
      if (i < n) {
        const float send = hi ? v[i] : v[i + n], keep = hi ? v[i + n] : v[i];
        v[i] = keep + __shfl_xor_sync(kFullMask, send, o);
      }
  }
}

// Adjoint of the four paths. A line is walked against its path; every step adds the gradient that
// arrives at L_p from its successor to the one of S, writes it (the gradient of C_p) and routes it to
// the predecessor by the recorded choices: gv goes to L_q(d), L_q(d-1), L_q(d+1) or to m_q, and
// subtracting m_q takes the sum of all that did not jump from L_q(argmin).
//
// The gradient of S arrives kBwdPF - 1 steps ahead by asynchronous copies (cp.async, one group a step):
// a warp's lanes copy the step's 512 bytes in 16-byte units side by side and read their own unit after a
// warp barrier. As a ring of registers the loads shared scoreboards with younger loads and with the
// step's shuffles, and a row step took ~750 cycles.
// Four disparities per lane: with eight, twice the lines fit a warp, but a step is twice the
// instructions for one warp to issue, and the row scans take as long as their steps do (both with the
// copies ahead: one 1242x375 image, D = 64, backward pass 581 -> 479 us; four 1294 -> 1274 us, and at
// D = 32 803 -> 722 us). From the ring of registers with eight: one 627 -> 481, four 1330 -> 1272, but eight
// 320x240 images 411 -> 426.
template <int G>
__global__ void __launch_bounds__(kWarps * 32, 4) k_float_bwd(const BwdArgs a) {
  constexpr int K = kBwdK, D = G * K, FK = D / 32, PF = kBwdPF;
  Line ln;
  Geo g;
  if (!locate<G>(a.q, ln, g)) return;
  const int lane = threadIdx.x & 31, gl = lane % G;
  long long base, step;
  line_positions(g, ln.line, base, step);
  const bool down = ln.dir < 2;  // paths of ascending position are walked downwards
  const int len = g.len, nseg = g.nseg;
  const long long sd = step * D;
  static_assert(K == 4, "a unit of 16 bytes a lane and step");
  __shared__ __align__(16) float4 ring[kWarps][PF][32];
  float4(*rows)[32] = ring[threadIdx.x >> 5];
  const float* gs = a.gsum + base * D + gl * K;  // this lane's unit of a step
  float* go = a.gout[ln.dir] + base * D + gl * K;
  float* gp1 = a.gp1[ln.dir];
  float* gp2 = a.gp2[ln.dir];
  const uint2* codes = reinterpret_cast<const uint2*>(reinterpret_cast<const CodeWord<FK>*>(a.rec[ln.dir]) +
                                                      (size_t)ln.line * nseg * 32) + gl;
  const uint2* args = reinterpret_cast<const uint2*>(reinterpret_cast<const char*>(a.rec[ln.dir]) +
                                                     code_bytes<FK>(g.lines, nseg)) + (size_t)ln.line * nseg;
  const bool live = ln.live;
  float gn[K];  // gradient arriving from the successor
#pragma unroll
  for (int t = 0; t < K; ++t) gn[t] = 0.f;
  auto segment = [&](int si) { return down ? nseg - 1 - si : si; };
  auto position = [&](int seg, int slot) { return seg * kSeg + (down ? kSeg - 1 - slot : slot); };
  // gradient of S at a slot of segment si into ring row r; nothing past the line; a group either way
  auto fetch = [&](int r, int si, int slot) {
    if (si < nseg) {
      const int pos = position(segment(si), slot);
      if (pos < len) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sgm::smem_u32(rows[r] + lane)), "l"(gs + pos * sd)
                     : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // before slot j of segment si: its row is there for every lane; the row of the slot before is refilled
  auto turn = [&](int si, int j) {
    asm volatile("cp.async.wait_group %0;" ::"n"(PF - 2) : "memory");
    __syncwarp();
    const int ahead = j + PF - 1;
    fetch(ahead % PF, ahead < kSeg ? si : si + 1, ahead % kSeg);
  };
#pragma unroll
  for (int j = 0; j < PF - 1; ++j) fetch(j, 0, j);
  uint2 cw = __ldg(codes + (size_t)segment(0) * G);
  uint2 aw = __ldg(args + segment(0));
  for (int si = 0; si < nseg; ++si) {
    const int seg = segment(si);
    const uint32_t w[K / 2] = {cw.x, cw.y}, ar[2] = {aw.x, aw.y};
    if (si + 1 < nseg) {
      cw = __ldg(codes + (size_t)segment(si + 1) * G);
      aw = __ldg(args + segment(si + 1));
    }
    float part[2 * kSeg];  // this lane's share of the P1 and P2 gradients of each slot
    auto step_at = [&](int j, bool start) {
      turn(si, j);
      const long long off = position(seg, j) * sd;
      float gv[K];
      const float4 x = rows[j % PF][lane];
      const float2 lo = __fadd2_rn(make_float2(x.x, x.y), make_float2(gn[0], gn[1]));
      const float2 hi = __fadd2_rn(make_float2(x.z, x.w), make_float2(gn[2], gn[3]));
      gv[0] = lo.x;
      gv[1] = lo.y;
      gv[2] = hi.x;
      gv[3] = hi.y;
      if (live) storeK<K>(go + off, gv);
      part[2 * j] = part[2 * j + 1] = 0.f;
      if (start) return;  // the path's first pixel: nothing before it
      float same[K], dn[K], up[K];  // flows to L_q(d), L_q(d-1), L_q(d+1)
      float2 kept = make_float2(0.f, 0.f), side = kept, jumped = kept;
#pragma unroll
      for (int t = 0; t < K; t += 2) {
        float lo[2], hi[2], ju[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int sh = code_shift<FK>(t + h, j);
          const bool b0 = (w[(t + h) / 2] >> sh) & 1u, b1 = (w[(t + h) / 2] >> sh) & 2u;
          const float v = gv[t + h];
          lo[h] = b1 ? 0.f : v;  // codes 0 and 1
          hi[h] = b1 ? v : 0.f;  // codes 2 and 3
          same[t + h] = b0 ? 0.f : lo[h];
          dn[t + h] = b0 ? lo[h] : 0.f;
          up[t + h] = b0 ? 0.f : hi[h];
          ju[h] = b0 ? hi[h] : 0.f;
        }
        const float2 u = make_float2(up[t], up[t + 1]);
        kept = __fadd2_rn(kept, __fadd2_rn(make_float2(lo[0], lo[1]), u));
        side = __fadd2_rn(side, __fadd2_rn(make_float2(dn[t], dn[t + 1]), u));
        jumped = __fadd2_rn(jumped, make_float2(ju[0], ju[1]));
      }
      part[2 * j] = side.x + side.y;
      part[2 * j + 1] = jumped.x + jumped.y;
      const float all_kept = group_sum<G>(kept.x + kept.y);
      float from_up = __shfl_down_sync(kFullMask, dn[0], 1), from_dn = __shfl_up_sync(kFullMask, up[K - 1], 1);
      if (gl == G - 1) from_up = 0.f;
      if (gl == 0) from_dn = 0.f;
      const int at = (int)((ar[j / 4] >> (8 * (j % 4))) & 0xffu) - gl * K;
#pragma unroll
      for (int t = 0; t < K; ++t) {
        float v = same[t] + (t < K - 1 ? dn[t + 1] : from_up);
        v += t > 0 ? up[t - 1] : from_dn;
        if (t == at) v -= all_kept;
        gn[t] = v;
      }
    };
    const int p0 = seg * kSeg;
    const int start = down ? (seg == 0 ? kSeg - 1 : -1) : (seg == nseg - 1 ? len - 1 - p0 : -1);  // its slot
    if (p0 + kSeg <= len && start < 0) {
#pragma unroll
      for (int j = 0; j < kSeg; ++j) step_at(j, false);
    } else {
#pragma unroll
      for (int j = 0; j < kSeg; ++j) {
        part[2 * j] = part[2 * j + 1] = 0.f;
        if (position(seg, j) < len)
          step_at(j, j == start);
        else
          turn(si, j);
      }
    }
    reduce_segment<G>(part, gl);
    if constexpr (G == 2 * kSeg) {  // one value a lane
      const int pos = position(seg, gl / 2);
      if (live && pos < len) (gl & 1 ? gp2 : gp1)[base + pos * step] = part[0];
    } else {
#pragma unroll
      for (int i = 0; i < kSeg / G; ++i) {
        const int pos = position(seg, gl * (kSeg / G) + i);
        if (live && pos < len) {
          gp1[base + pos * step] = part[2 * i];
          gp2[base + pos * step] = part[2 * i + 1];
        }
      }
    }
  }
}

// grad_cost = ((G0 + G1) + G2) + G3 in place over G0; grad_p = (((0 + a0) + a1) + a2) + a3
struct SumArgs {
  float4* g0;
  const float4* g1;
  const float4* g2;
  const float4* g3;
  size_t n4;
  float* gp1;
  float* gp2;
  const float* a1[4];
  const float* a2[4];
  size_t npix;
};

__global__ void __launch_bounds__(256) k_grad_sum(const SumArgs a) {
  const size_t n = a.n4 + a.npix;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    if (i < a.n4) {
      float4 x = a.g0[i];
      const float4 y = __ldg(a.g1 + i), z = __ldg(a.g2 + i), w = __ldg(a.g3 + i);
      x.x = ((x.x + y.x) + z.x) + w.x;
      x.y = ((x.y + y.y) + z.y) + w.y;
      x.z = ((x.z + y.z) + z.z) + w.z;
      x.w = ((x.w + y.w) + z.w) + w.w;
      a.g0[i] = x;
    } else {
      const size_t p = i - a.n4;
      a.gp1[p] = (((0.f + a.a1[0][p]) + a.a1[1][p]) + a.a1[2][p]) + a.a1[3][p];
      a.gp2[p] = (((0.f + a.a2[0][p]) + a.a2[1][p]) + a.a2[2][p]) + a.a2[3][p];
    }
  }
}

int check(const char* what) {
  const cudaError_t st = cudaGetLastError();
  if (st != cudaSuccess) {
    std::string m = std::string(what) + ": " + cudaGetErrorString(st);
    sgm_set_process_error(m.c_str());
    return SGM_ERR_CUDA;
  }
  return SGM_OK;
}

int validate(int B, int H, int W, int D, float temperature) {
  if (B <= 0 || H <= 0 || W <= 0 || (D != 32 && D != 64)) {
    sgm_set_process_error("float SGM: B, H, W > 0 and D in {32, 64} required");
    return SGM_ERR_ARG;
  }
  if (!(temperature > 0.0f) || !std::isfinite(1.0f / temperature)) {
    sgm_set_process_error("float SGM: temperature must be > 0 with a finite reciprocal");
    return SGM_ERR_ARG;
  }
  // B*H*W*D voxels, bounded factor by factor so that no product can wrap
  const uint64_t kMaxVoxels = (uint64_t)1 << 40;
  uint64_t n = 1;
  for (const int32_t f : {B, H, W, D}) {
    if ((uint64_t)f > kMaxVoxels / n) {
      sgm_set_process_error("float SGM: volume too large");
      return SGM_ERR_ARG;
    }
    n *= (uint64_t)f;
  }
  return SGM_OK;
}

int check_present(std::initializer_list<const void*> ptrs) {
  for (const void* p : ptrs)
    if (!p) {
      sgm_set_process_error("float SGM: null device pointer");
      return SGM_ERR_ARG;
    }
  return SGM_OK;
}

int check_aligned(std::initializer_list<const void*> ptrs) {
  for (const void* p : ptrs)
    if (reinterpret_cast<uintptr_t>(p) & 15) {
      sgm_set_process_error("float SGM: cost, sum, gradient and workspace arrays must be 16-byte aligned");
      return SGM_ERR_ARG;
    }
  return SGM_OK;
}

size_t slab_elems(int B, int H, int W, int D) { return sgm_float_checkpoint_elems(B, H, W, D) / 4; }

// The four directions of one launch, row scans first (their scanlines are the longest).
template <int G>
Grid4 make_grid(int B, int H, int W, int D) {
  Grid4 q;
  const int order[4] = {1, 3, 0, 2};
  const int lines_per_block = kWarps * (32 / G);
  q.first_block[0] = 0;
  for (int i = 0; i < 4; ++i) {
    q.order[i] = order[i];
    q.g[i] = make_geo(B, H, W, D, i);  // indexed by direction
  }
  for (int i = 0; i < 4; ++i)
    q.first_block[i + 1] = q.first_block[i] + (q.g[order[i]].lines + lines_per_block - 1) / lines_per_block;
  return q;
}

// The cost volume [B][H][W][D] floats as a 3D tensor map (floats of a row, rows, images) with
// boxes of D x kFC x 1: the forward column scans' chunks.
int cost_map(const float* cost, int B, int H, int W, int D, CUtensorMap* map) {
  const sgm::EncodeTiledFn fn = sgm::encode_tiled();
  if (!fn) {
    sgm_set_process_error("float SGM: cuTensorMapEncodeTiled is not available from the driver");
    return SGM_ERR_CUDA;
  }
  const cuuint64_t dims[3] = {(cuuint64_t)W * D, (cuuint64_t)H, (cuuint64_t)B};
  const cuuint64_t strides[2] = {(cuuint64_t)W * D * sizeof(float), (cuuint64_t)H * W * D * sizeof(float)};
  const cuuint32_t box[3] = {(cuuint32_t)D, (cuuint32_t)kFC, 1u};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(cost), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    sgm_set_process_error("float SGM: cuTensorMapEncodeTiled failed for the cost volume");
    return SGM_ERR_CUDA;
  }
  return SGM_OK;
}

// REC: the records (in ckpt) are written for a backward pass.
template <int K, bool REC>
int forward_impl(const float* cost, const float* p1, const float* p2, int B, int H, int W, float inv_t, float* sum,
                 float* ckpt, float* work, float* disp, cudaStream_t s) {
  constexpr int D = 32 * K;
  const size_t V = (size_t)B * H * W * D, npix = (size_t)B * H * W;
  FwdArgs a;
  a.cost = cost;
  a.p1 = p1;
  a.p2 = p2;
  a.out[0] = sum;
  for (int i = 1; i < 4; ++i) a.out[i] = work + (i - 1) * V;
  const size_t slab = slab_elems(B, H, W, D);
  for (int i = 0; i < 4; ++i) a.rec[i] = REC ? ckpt + slab * i : nullptr;
  a.q = make_grid<32>(B, H, W, D);
  CUtensorMap tm;
  int st = cost_map(cost, B, H, W, D, &tm);
  if (st) return st;
  constexpr size_t smem = fwd_smem_bytes<K>();
  static_assert(smem <= 48 * 1024, "no opt-in for more shared memory needed");
  k_float_fwd<K, REC><<<a.q.first_block[4], kWarps * 32, smem, s>>>(tm, a);
  st = check("float forward");
  if (st) return st;
  constexpr int GS = D / kK;  // lanes per pixel of the soft-argmin kernels
  const size_t px_per_block = 8 * (32 / GS);
  k_soft_argmin_fwd<GS, REC><<<(unsigned)((npix + px_per_block - 1) / px_per_block), 256, 0, s>>>(
      sum, a.out[1], a.out[2], a.out[3], disp, npix, inv_t);
  return check("soft argmin");
}

template <int G>
int backward_impl(int B, int H, int W, float inv_t, const float* sum, const float* ckpt, const float* grad_disp,
                  float* grad_sum, float* work, float* grad_cost, float* grad_p1, float* grad_p2, cudaStream_t s) {
  constexpr int D = G * kBwdK;
  const size_t V = (size_t)B * H * W * D, npix = (size_t)B * H * W;
  constexpr int GS = D / kK;  // lanes per pixel of the soft-argmin kernels
  const size_t px_per_block = 8 * (32 / GS);
  k_soft_argmin_bwd<GS><<<(unsigned)((npix + px_per_block - 1) / px_per_block), 256, 0, s>>>(
      sum, grad_disp, grad_sum, npix, inv_t);
  int st = check("soft argmin backward");
  if (st) return st;
  BwdArgs a;
  a.gsum = grad_sum;
  const size_t slab = slab_elems(B, H, W, D);
  float* maps = work + 3 * V;
  for (int i = 0; i < 4; ++i) {
    a.rec[i] = ckpt + slab * i;
    a.gout[i] = i == 0 ? grad_cost : work + (i - 1) * V;
    a.gp1[i] = maps + i * npix;
    a.gp2[i] = maps + (4 + i) * npix;
  }
  a.q = make_grid<G>(B, H, W, D);
  k_float_bwd<G><<<a.q.first_block[4], kWarps * 32, 0, s>>>(a);
  if ((st = check("float backward"))) return st;
  SumArgs r;
  r.g0 = reinterpret_cast<float4*>(grad_cost);
  r.g1 = reinterpret_cast<const float4*>(a.gout[1]);
  r.g2 = reinterpret_cast<const float4*>(a.gout[2]);
  r.g3 = reinterpret_cast<const float4*>(a.gout[3]);
  r.n4 = V / 4;
  r.gp1 = grad_p1;
  r.gp2 = grad_p2;
  for (int i = 0; i < 4; ++i) {
    r.a1[i] = a.gp1[i];
    r.a2[i] = a.gp2[i];
  }
  r.npix = npix;
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  k_grad_sum<<<nsm * 8, 256, 0, s>>>(r);
  return check("float backward sum");
}

}  // namespace

// Waits of the forward scans that ran out (sgm_debug_wait_timeouts adds them to the engine's).
int64_t sgm_float_wait_timeouts() {
  unsigned int n = 0;
  if (cudaMemcpyFromSymbol(&n, sgm::g_scan_wait_timeouts, sizeof(n)) != cudaSuccess) return -1;
  return n;
}

extern "C" {

size_t sgm_float_checkpoint_elems(int32_t B, int32_t H, int32_t W, int32_t D) {
  size_t n = 0;
  for (int dir = 0; dir < 4; ++dir) {
    const Geo g = make_geo(B, H, W, D, dir);
    n = n > (size_t)g.lines * g.nseg * D ? n : (size_t)g.lines * g.nseg * D;
  }
  return 4 * n;
}

size_t sgm_float_workspace_elems(int32_t B, int32_t H, int32_t W, int32_t D) {
  return 3 * (size_t)B * H * W * D + 8 * (size_t)B * H * W;
}

int sgm_float_forward(const float* cost, const float* p1, const float* p2, int32_t B, int32_t H, int32_t W,
                      int32_t D, float temperature, float* sum, float* ckpt, float* work, float* disp, void* stream) {
  int st = validate(B, H, W, D, temperature);
  if (st || (st = check_present({cost, p1, p2, sum, ckpt, work, disp})) ||
      (st = check_aligned({cost, sum, ckpt, work})))
    return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const float inv_t = 1.0f / temperature;
  return D == 64 ? forward_impl<2, true>(cost, p1, p2, B, H, W, inv_t, sum, ckpt, work, disp, s)
                 : forward_impl<1, true>(cost, p1, p2, B, H, W, inv_t, sum, ckpt, work, disp, s);
}

int sgm_float_disparity(const float* cost, const float* p1, const float* p2, int32_t B, int32_t H, int32_t W,
                        int32_t D, float temperature, float* sum, float* work, float* disp, void* stream) {
  int st = validate(B, H, W, D, temperature);
  if (st || (st = check_present({cost, p1, p2, sum, work, disp})) || (st = check_aligned({cost, sum, work})))
    return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const float inv_t = 1.0f / temperature;
  return D == 64 ? forward_impl<2, false>(cost, p1, p2, B, H, W, inv_t, sum, nullptr, work, disp, s)
                 : forward_impl<1, false>(cost, p1, p2, B, H, W, inv_t, sum, nullptr, work, disp, s);
}

int sgm_float_backward(const float* cost, const float* p1, const float* p2, int32_t B, int32_t H, int32_t W, int32_t D,
                       float temperature, const float* sum, const float* ckpt, const float* grad_disp,
                       float* grad_sum, float* work, float* grad_cost, float* grad_p1, float* grad_p2, void* stream) {
  int st = validate(B, H, W, D, temperature);
  if (st || (st = check_present({cost, p1, p2, sum, ckpt, grad_disp, grad_sum, work, grad_cost, grad_p1, grad_p2})) ||
      (st = check_aligned({cost, sum, ckpt, grad_sum, work, grad_cost})))
    return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const float inv_t = 1.0f / temperature;
  return D == 64 ? backward_impl<64 / kBwdK>(B, H, W, inv_t, sum, ckpt, grad_disp, grad_sum, work, grad_cost, grad_p1,
                                             grad_p2, s)
                 : backward_impl<32 / kBwdK>(B, H, W, inv_t, sum, ckpt, grad_disp, grad_sum, work, grad_cost, grad_p1,
                                             grad_p2, s);
}

}  // extern "C"
