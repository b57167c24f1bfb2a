// Gapless low-rank correlation prefilter: the quantity of sseqs/fft.cu:17-415
// with sseqs/filter.cu:92-159, computed directly instead of by FFT.
//
// For a query q (Lq residues), rank-k look-up tables A (query side) and B
// (database side), a segment t (Lt <= N bytes) and N a power of two:
//   a_r[i] = A_r[pos(q[Lq-1-i])] (i < Lq),   b_r[i] = B_r[pos(t[i])] (i < Lt),
//   y      = sum_r a_r (*) b_r                (cyclic convolution of length N)
//   score  = fp16( 0.5 * max over even s of y[s] )
// pos() maps ARNDCQEGHILKMFPSTWYV to 0..19, X - * to 20 and any other byte to
// 21; B_r[21] is B_{r+1}[0] (the reference reads one entry past the row,
// sseqs/fft.cu:91,124) and 0 for the last rank.
//
// Direct form.  With j = Lq-1-i the forward query position, the linear
// correlation c[m] = sum_i a[i] b[m-i] is the sum of P(j, t[p]) along the
// diagonal p - j = m - (Lq-1) of the Lq x Lt matrix, where
//   P(j, c) = sum_r A_r[pos(q[j])] * B_r[c]
// is a per-query profile; and the cyclic y folds c once: y[s] = c[s] +
// c[s+N] (c has Lq+Lt-1 <= 2N entries), with y[s] = 0 for lags that no
// diagonal reaches.  So every score is a set of fp32 diagonal sums: one add
// per (query, target) cell, about Lq*Lt/2 useful ones per segment, instead of
// k+1 transforms of length N (N is set by the longest segment of the batch).
//
// B200 mapping: one warp per segment, lane l holding C = ceil(Lq/32)
// consecutive query columns (the query is left-padded to 32C columns with
// zero profile entries), D(j) the running sum of the diagonal ending at
// (row, j).  A row is D(j) <- D(j-1) + P(j, t[row]): a shift by one column
// (one shuffle crosses the lane boundary) and C adds.  Reading the profile
// is what bounds the kernel (shared-memory bandwidth: a profile entry per
// cell), so it is stored as fp16 -- half the bytes -- and each add takes the
// fp16 entry and the fp32 running sum in one instruction (add.f32.f16; the
// sums stay fp32).  The profile sits in shared memory, 32C entries per class,
// each lane's columns padded to an odd number of 16-byte units so the
// 128-bit loads of a warp do not conflict.  The value leaving the last column at row s is c[s]; it enters
// the maximum at once unless its partner c[s+N] exists, in which case it is
// parked in a per-warp shared array until the segment's last row, when the
// remaining diagonals (m >= Lt) are read off every column.
//
// Tensor-core form (rank k <= 4; the reference's default rank is 4): the even
// lags of the convolution as one matrix product per group of 128 segments on
// tcgen05, D[segment, lag] = sum_(p, r) b_r[p] * a_r[(lag - p) mod N], see
// prefilter_tc_kernel.
#include <cuda_fp16.h>

#include <algorithm>
#include <array>
#include <mutex>
#include <utility>

#include "tcgen05.cuh"

namespace sseqs {
namespace {

constexpr int kMaxRank = 20;
constexpr int kPfClasses = 22;

__device__ __forceinline__ int pf_pos(uint8_t c) {
  const uint8_t k = ascii_class(c);
  if (k < kNumAA) return k;
  return (c == 'X' || c == '-' || c == '*') ? 20 : 21;
}

struct PfArgs {
  const uint8_t* ascii;
  const int64_t* offsets;
  const int32_t* lengths;
  int64_t n;
  const float* A;           // [k][21] query side
  const float* B;           // [k][21] database side
  const uint8_t* qrev;      // query positions, reversed, already mapped (0..20)
  int Lq;
  int k;
  int N;                    // cyclic length
  __half* out;              // [n]
};

template <int C>
struct PfShape {
  static constexpr int NV = (C + 7) / 8;                       // 128-bit loads per row
  static constexpr int LW = ((NV % 2) ? NV : NV + 1) * 8;      // fp16 entries per lane (odd x 16 B)
  static constexpr int ROW = 32 * LW;                          // entries per class
  static constexpr int WARPS = C <= 32 ? 16 : 8;
  static constexpr int PARK = 16 * C;                          // parked c[s] per warp (even s)
  static constexpr size_t smem = sizeof(__half) * (size_t)kPfClasses * ROW +
                                 sizeof(float) * (size_t)WARPS * PARK + 256;
};

// fp32 + fp16 -> fp32 in one instruction
__device__ __forceinline__ float add_f32_f16(float acc, unsigned short h) {
  float r;
  asm("add.rn.f32.f16 %0, %1, %2;" : "=f"(r) : "h"(h), "f"(acc));
  return r;
}

template <int C>
__global__ void __launch_bounds__(32 * PfShape<C>::WARPS) prefilter_kernel(PfArgs a) {
  using S = PfShape<C>;
  constexpr int J = 32 * C;
  extern __shared__ float4 smem_pf[];
  __half* prof = reinterpret_cast<__half*>(smem_pf);               // [22][ROW]
  float* park_all = reinterpret_cast<float*>(prof + kPfClasses * S::ROW);   // [WARPS][PARK]
  uint8_t* lut = reinterpret_cast<uint8_t*>(park_all + S::WARPS * S::PARK);

  for (int i = threadIdx.x; i < 256; i += blockDim.x) lut[i] = (uint8_t)pf_pos((uint8_t)i);
  // profile: column j of lane l = j / C sits at l*LW + j % C; real query
  // column jr = j - (J - Lq) (left padding), its residue q[jr] = qrev[Lq-1-jr]
  const int pad = J - a.Lq;
  for (int i = threadIdx.x; i < kPfClasses * S::ROW; i += blockDim.x) {
    const int c = i / S::ROW, r = i - c * S::ROW;
    const int l = r / S::LW, v = r - l * S::LW;
    const int jr = l * C + v - pad;
    float p = 0.f;
    if (v < C && jr >= 0) {
      const int qa = a.qrev[a.Lq - 1 - jr];
      for (int rk = 0; rk < a.k; ++rk) {
        const float bv = c < 21 ? a.B[rk * 21 + c] : (rk + 1 < a.k ? a.B[(rk + 1) * 21] : 0.f);
        p = fmaf(a.A[rk * 21 + qa], bv, p);
      }
    }
    prof[i] = __float2half_rn(p);
  }
  __syncthreads();

  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  float* park = park_all + wib * S::PARK;
  const uint4* myprof = reinterpret_cast<const uint4*>(prof + lane * S::LW);
  const int64_t nwarps = (int64_t)gridDim.x * S::WARPS;
  const int N = a.N, Lq = a.Lq;
  const uintptr_t au = reinterpret_cast<uintptr_t>(a.ascii);
  const uint32_t* abase = reinterpret_cast<const uint32_t*>(au & ~(uintptr_t)3);
  const int64_t aoff = (int64_t)(au & 3);

  for (int64_t s = (int64_t)blockIdx.x * S::WARPS + wib; s < a.n; s += nwarps) {
    const int len = min((int)a.lengths[s], N);
    const int64_t base = a.offsets[s];
    // lags s' <= nlim have both c[s'] and c[s'+N]
    const int nlim = Lq + len - 2 - N;
    float D[C];
#pragma unroll
    for (int k = 0; k < C; ++k) D[k] = 0.f;
    float best = -INFINITY;
    for (int i0 = 0; i0 < len; i0 += 4) {
      // four target bytes from the two aligned words that hold them (a word
      // is read only when it holds a byte of the segment)
      const int64_t ap = base + i0 + aoff;
      const int64_t wi = ap >> 2;
      const uint32_t w0 = __ldg(abase + wi);
      const uint32_t w1 = ((wi + 1) << 2) < base + len + aoff ? __ldg(abase + wi + 1) : 0u;
      const uint32_t raw = __funnelshift_r(w0, w1, (uint32_t)(ap & 3) * 8u);
      const int rows = min(4, len - i0);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (r < rows) {
          const int cls = lut[(raw >> (8 * r)) & 0xffu];
          const uint4* pr = myprof + cls * (S::ROW / 8);
          unsigned short P[S::NV * 8];
#pragma unroll
          for (int v = 0; v < S::NV; ++v) {
            const uint4 x = pr[v];
            const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int h = 0; h < 4; ++h)
              asm("mov.b32 {%0, %1}, %2;" : "=h"(P[8 * v + 2 * h]), "=h"(P[8 * v + 2 * h + 1])
                  : "r"(w[h]));
          }
          float left = __shfl_up_sync(0xffffffffu, D[C - 1], 1);
          if (lane == 0) left = 0.f;
#pragma unroll
          for (int k = C - 1; k > 0; --k) D[k] = add_f32_f16(D[k - 1], P[k]);
          D[0] = add_f32_f16(left, P[0]);
          const int row = i0 + r;
          if (lane == 31 && (row & 1) == 0) {          // c[row] leaves the last column
            if (row <= nlim) park[row >> 1] = D[C - 1];
            else best = fmaxf(best, D[C - 1]);
          }
        }
      }
    }
    __syncwarp();
    // diagonals m = len + Lq - 2 - jr ending on the last row (jr <= Lq - 2)
    if (len > 0) {
#pragma unroll
      for (int k = 0; k < C; ++k) {
        const int jr = lane * C + k - (J - Lq);
        const int m = len + Lq - 2 - jr;
        if (jr >= 0 && jr <= Lq - 2 && (m & 1) == 0) {
          float v = D[k];
          if (m >= N) v += park[(m - N) >> 1];
          best = fmaxf(best, v);
        }
      }
    }
    // even lags that no diagonal reaches have y = 0 (all of them when the
    // query or the segment is empty)
    if (len == 0 || Lq == 0 || Lq + len - 1 <= N - 2) best = fmaxf(best, 0.f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
    if (lane == 0) a.out[s] = __float2half_rn(0.5f * best);
    __syncwarp();
  }
}

// ------------------------------------------------------- tensor-core form
// One matrix product per group of 128 segments: D[segment, lag] over the even
// lags, K = (target position, rank), fp16 factors, fp32 accumulators in
// tensor memory (128 lanes x up to 512 columns).
//
// Both operands use the no-swizzle K-major layout of 8-row x 16-byte core
// matrices.  A 16-byte chunk of K holds 2 target positions x 4 ranks, so the
// query operand needs no Toeplitz matrix: with arr[x] = (a_0 .. a_3)[-x mod N]
// (8 bytes per x) row n of the operand is lag S - 2 - 2n and starts 16 bytes
// after row n - 1, and the next chunk of K starts 16 bytes further too.  The
// descriptors' strides (16 bytes from chunk to chunk, 128 from 8 rows to 8
// rows) read the one 16N-byte array in place, for every lag and position; and
// as arr is periodic in N, the cyclic fold y[s] = c[s] + c[s + N] happens in
// the accumulation.
//
// A CTA (one per SM) takes every gridDim.x-th run of 32 segments, a window of
// them at a time, and sorts the window by length (counting sort in shared
// memory), so that the 128 segments of a group have nearly the same length:
// a group costs its longest segment.  Warps 4-11 build the segment operand,
// 32 positions to a 32 KB stage (one thread per segment: 32-byte loads, a
// table of the 4 factors of every letter, replicated over the 32 lanes so that
// no two lanes of a look-up share a bank); one thread of warp 12 issues the
// MMAs; warps 0-3 read the accumulators (lane = segment, so the maximum over
// lags needs no exchange between lanes).  Lags that a stage's positions
// cannot reach are skipped in units of 16 columns, so the work follows
// Lq * Lt, not the transform length.  A group of at most 256 even lags uses
// half of the tensor memory, so that the next one's products overlap its
// epilogue; one of more than 512 (N = 2048) takes two passes.
//
// Waits are bounded; one that runs out adds to the device's count of failures
// (sseqs_prefilter_failures), the CTA stops and its segments score NaN.
//
// Measured (300k segments of 30..1000 residues, rank 4) against the per-warp
// mma.sync form it replaced, which built every segment's Toeplitz operand
// (4600 warp instructions a segment): query length 858 2.04 -> 0.29 ms,
// 100k segments at 1501 (N = 2048) 1.45 -> 0.23 ms.  At 858 the tensor pipe's
// own time is 0.18 ms and shared memory, which feeds both operands and holds
// the look-ups, is the next bound; below ~400 residues (0.15-0.17 ms) the issue of the
// MMAs and the look-ups bound it.  tcgen05 runs the overlapping query
// operand at its full rate (N = 256: 128 clocks per MMA, 64: 48).  A third
// team of producers gained nothing.
constexpr int kTcRank = 4;             // ranks of the tensor-core form
constexpr int kTcGroup = 128;          // segments per group (MMA rows)
constexpr int kTcPos = 32;             // target positions per stage
constexpr int kTcStages = 4;
constexpr int kTcStageBytes = kTcGroup * kTcPos * 8;
constexpr int kTcWindow = 4096;        // segments sorted at a time
constexpr int kTcCols = 512;           // tensor-memory columns (fp32 lags)
constexpr int kTcEpiWarps = 4, kTcProducers = 2;      // producers: teams of 4 warps
constexpr int kTcProdWarps = 4 * kTcProducers;
constexpr int kTcThreads = 32 * (kTcEpiWarps + kTcProdWarps + 1);
// look-up entries: bytes 64..95, then a position past the end, '-' or '*',
// any other byte
constexpr int kTcZero = 32, kTcGap = 33, kTcOther = 34, kTcEntries = 35;
constexpr int kTcBins = 256;
// Halves of the operands' shared-memory descriptors (fields as umma_desc):
// the low one holds the start address and the K stride (segments: one chunk of
// all 128; query: 16 bytes), the high one the 8-row stride (128 bytes) and the
// version.
constexpr uint32_t kDescLoA = (uint32_t)(kTcGroup * 16 / 16) << 16, kDescLoB = 1u << 16;
constexpr uint32_t kDescHi = (128u >> 4) | (1u << 14);

inline size_t tc_smem(int N) {
  return (size_t)kTcStages * kTcStageBytes + (size_t)2 * N * 8 + kTcEntries * 32 * 8 +
         kTcWindow * 2 + kTcBins * 4 + (kTcWindow / kTcGroup) * 4 + 128;
}

// Sizes of one group: even lags (rows of the query operand), stages, passes.
struct TcGroup {
  int S, R, stages, passes;
  __device__ TcGroup(int N, int Lq, int longest) {
    S = min(N, max(32, (Lq + longest - 1 + 31) & ~31));   // lags computed: 0 .. S - 1
    R = S >> 1;
    stages = max(1, (longest + kTcPos - 1) / kTcPos);
    passes = (R + kTcCols - 1) / kTcCols;
  }
};

__global__ void __launch_bounds__(kTcThreads, 1) prefilter_tc_kernel(PfArgs a, unsigned* failures) {
  using namespace tc;
  extern __shared__ __align__(128) unsigned char pf_sm[];
  const int N = a.N, Lq = a.Lq, K = a.k;
  unsigned char* stages = pf_sm;
  uint2* arr = reinterpret_cast<uint2*>(stages + kTcStages * kTcStageBytes);   // [2N]
  uint2* lut = arr + 2 * N;                                                    // [35][32]
  uint16_t* order = reinterpret_cast<uint16_t*>(lut + kTcEntries * 32);
  int* hist = reinterpret_cast<int*>(order + kTcWindow);
  int* gmax = hist + kTcBins;
  __shared__ __align__(8) uint64_t full[kTcStages], empty[kTcStages];
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2], mma_done;
  __shared__ uint32_t tmem_base_s;
  __shared__ int valid_s;
  __shared__ volatile int abort_s;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int mma_warp = kTcEpiWarps + kTcProdWarps;
  if (warp == mma_warp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(&tmem_base_s)), "r"(kTcCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  if (tid == 0) {
    auto init = [](uint64_t* b, int count) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(b)), "r"(count));
    };
    for (int s = 0; s < kTcStages; ++s) { init(&full[s], 4); init(&empty[s], 1); }
    for (int h = 0; h < 2; ++h) { init(&acc_full[h], 1); init(&acc_empty[h], kTcEpiWarps); }
    init(&mma_done, 1);
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // query residues and factors, staged where the segment operand goes later
  uint8_t* tq = stages;
  __half* ta = reinterpret_cast<__half*>(stages + 2048);
  for (int i = tid; i < Lq; i += kTcThreads) tq[i] = a.qrev[i];
  for (int i = tid; i < kTcRank * 21; i += kTcThreads)
    ta[i] = __float2half_rn(i / 21 < K ? a.A[i] : 0.f);
  for (int i = tid; i < kTcEntries * 32; i += kTcThreads) {
    const int e = i >> 5;
    const int c = e == kTcGap ? 20 : e >= kTcZero ? 21 : pf_pos((uint8_t)(64 + e));
    __half h[kTcRank];
#pragma unroll
    for (int r = 0; r < kTcRank; ++r) {
      float v = 0.f;
      if (r < K && e != kTcZero) v = c < 21 ? a.B[r * 21 + c] : (r + 1 < K ? a.B[(r + 1) * 21] : 0.f);
      h[r] = __float2half_rn(v);
    }
    lut[i] = make_uint2(__half_as_ushort(h[0]) | ((uint32_t)__half_as_ushort(h[1]) << 16),
                        __half_as_ushort(h[2]) | ((uint32_t)__half_as_ushort(h[3]) << 16));
  }
  __syncthreads();
  for (int i = tid; i < 2 * N; i += kTcThreads) {
    const int x = i - N, j = x <= 0 ? -x : N - x;       // a[-x mod N]
    uint32_t v[2] = {0u, 0u};
    if (j >= 0 && j < Lq) {
      const int c = tq[j];
      v[0] = __half_as_ushort(ta[c]) | ((uint32_t)__half_as_ushort(ta[21 + c]) << 16);
      v[1] = __half_as_ushort(ta[42 + c]) | ((uint32_t)__half_as_ushort(ta[63 + c]) << 16);
    }
    arr[i] = make_uint2(v[0], v[1]);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;
  auto fail = [&]() {
    abort_s = 1;
    atomicAdd(failures, 1u);
  };

  // segment j of this CTA: runs of 32, gridDim.x apart
  const int64_t runs = (a.n + 31) >> 5;
  const int64_t mine = ((runs - blockIdx.x + gridDim.x - 1) / gridDim.x) << 5;
  auto segment = [&](int64_t j) -> int64_t {
    return ((((j >> 5) * gridDim.x) + blockIdx.x) << 5) + (j & 31);
  };

  // pipeline positions, kept by every role over all groups
  uint32_t it = 0;                  // stages so far
  uint32_t half = 0, uses[2] = {0, 0};
  bool issued = false;
  for (int64_t w0 = 0; w0 < mine; w0 += kTcWindow) {
    // -------------------------------------------------- sort the window
    const int cnt = (int)min((int64_t)kTcWindow, mine - w0);
    for (int i = tid; i < kTcBins; i += kTcThreads) hist[i] = 0;
    if (tid < kTcWindow / kTcGroup) gmax[tid] = 0;
    __syncthreads();
    auto length_of = [&](int64_t g) { return max(0, min((int)a.lengths[g], N)); };
    auto bin_of = [](int len) { return kTcBins - 1 - min(kTcBins - 1, len >> 3); };
    for (int i = tid; i < cnt; i += kTcThreads) {
      const int64_t g = segment(w0 + i);
      if (g < a.n) atomicAdd(&hist[bin_of(length_of(g))], 1);
    }
    __syncthreads();
    if (warp == 0) {
      int v[kTcBins / 32], sum = 0;
#pragma unroll
      for (int k = 0; k < kTcBins / 32; ++k) {
        v[k] = hist[lane * (kTcBins / 32) + k];
        sum += v[k];
      }
      int x = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) valid_s = x;
      int run = x - sum;
#pragma unroll
      for (int k = 0; k < kTcBins / 32; ++k) {
        hist[lane * (kTcBins / 32) + k] = run;
        run += v[k];
      }
    }
    __syncthreads();
    for (int i = tid; i < cnt; i += kTcThreads) {
      const int64_t g = segment(w0 + i);
      if (g < a.n) {
        const int len = length_of(g);
        const int at = atomicAdd(&hist[bin_of(len)], 1);
        order[at] = (uint16_t)i;
        atomicMax(&gmax[at / kTcGroup], len);
      }
    }
    __syncthreads();
    const int valid = valid_s, groups = (valid + kTcGroup - 1) / kTcGroup;

    if (warp >= kTcEpiWarps && warp < mma_warp) {
      // ------------------------------------------------ segment operand
      const uint32_t wg = (uint32_t)(warp - kTcEpiWarps) >> 2;   // team: every second stage
      const int slot = (warp & 3) * 32 + lane;
      // this thread's segment of a group (length 0 past the last one)
      struct Seg { const uint8_t* src; int len; };
      auto seg_of = [&](int g) -> Seg {
        const int at = g * kTcGroup + slot;
        if (g >= groups || at >= valid) return {a.ascii, 0};
        const int64_t sg = segment(w0 + order[at]);
        return {a.ascii + a.offsets[sg], length_of(sg)};
      };
      auto stages_of = [&](int g) {
        const TcGroup G(N, Lq, gmax[g]);
        return G.stages * G.passes;
      };
      // the bytes of a stage: the two aligned 32-byte chunks that cover its 32
      // positions, read only where they hold a byte of the segment
      struct Raw { uint32_t w[16]; };
      auto fetch = [&](const Seg& s, int p0) -> Raw {
        Raw r;
        const uintptr_t at = (reinterpret_cast<uintptr_t>(s.src) & ~(uintptr_t)31) + p0;
        const int sh = (int)(reinterpret_cast<uintptr_t>(s.src) & 31);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          uint32_t* w = r.w + 8 * k;
#pragma unroll
          for (int q = 0; q < 8; ++q) w[q] = 0;
          if (p0 < s.len && p0 + 32 * k - sh < s.len)
            asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]),
                           "=r"(w[6]), "=r"(w[7])
                         : "l"(at + 32 * k));
        }
        return r;
      };
      // the bytes of the next stage and the next group's segment are fetched
      // before the current stage is waited for, so that their latency is hidden
      bool ok = true;
      int g = 0, total = 0, t = 0;
      Seg cur = {a.ascii, 0}, nxt = seg_of(0);
      // (g, t) := the first stage at or after (g, t) in the order of stages
      auto settle = [&]() {
        while (g < groups && t >= total) {
          t -= total;
          ++g;
          cur = nxt;
          if (g < groups) total = stages_of(g);
          nxt = seg_of(g + 1);
        }
      };
      if (groups > 0) {
        total = stages_of(0);
        cur = nxt;
        nxt = seg_of(1);
        const uint32_t first = it;
        t = (int)((wg + kTcProducers - first % kTcProducers) % kTcProducers);
        uint32_t done = first + (uint32_t)t;   // stages done of this team's
        settle();
        Raw raw = {};
        int p0 = 0;
        if (g < groups) {
          p0 = (t % max(1, TcGroup(N, Lq, gmax[g]).stages)) * kTcPos;
          raw = fetch(cur, p0);
        }
        while (g < groups && ok) {
          const Seg now = cur;
          const int pos = p0;
          uint32_t w[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) w[k] = raw.w[k];
          t += kTcProducers;
          settle();
          if (g < groups) {
            p0 = (t % TcGroup(N, Lq, gmax[g]).stages) * kTcPos;
            raw = fetch(cur, p0);
          }
          const uint32_t stage = done % kTcStages;
          if (!mbar_wait(smem_u32(&empty[stage]), ((done / kTcStages) & 1u) ^ 1u)) {
            fail();
            ok = false;
          }
          uint4* dst = reinterpret_cast<uint4*>(stages + stage * kTcStageBytes) + slot;
          const int left = now.len - pos;       // positions of the segment from here on
          if (left <= 0) {
#pragma unroll
            for (int c = 0; c < kTcPos / 2; ++c) dst[c * kTcGroup] = make_uint4(0, 0, 0, 0);
          } else {
            const int sh = (int)(reinterpret_cast<uintptr_t>(now.src) & 31);
            if (sh & 16) {
#pragma unroll
              for (int k = 0; k < 12; ++k) w[k] = w[k + 4];
            }
            if (sh & 8) {
#pragma unroll
              for (int k = 0; k < 10; ++k) w[k] = w[k + 2];
            }
            if (sh & 4) {
#pragma unroll
              for (int k = 0; k < 9; ++k) w[k] = w[k + 1];
            }
            const uint32_t bits = (uint32_t)(sh & 3) * 8u;
#pragma unroll
            for (int k = 0; k < 8; ++k) w[k] = __funnelshift_r(w[k], w[k + 1], bits);
            // bytes of word k before the end of the segment
            auto keep = [&](int k) {
              const int r = left - 4 * k;
              return r >= 4 ? 0xffffffffu : r <= 0 ? 0u : (1u << (8 * r)) - 1u;
            };
            if (left < kTcPos) {
#pragma unroll
              for (int k = 0; k < 8; ++k) w[k] = (w[k] & keep(k)) | (0x40404040u & ~keep(k));
            }
            uint32_t odd = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) odd |= (w[k] ^ 0x40404040u) & 0xe0e0e0e0u;
            if (odd == 0) {
#pragma unroll
              for (int k = 0; k < 8; ++k) w[k] &= 0x1f1f1f1fu;
            } else {
              // some byte is outside 64..95
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                uint32_t e = 0;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                  const uint32_t c = (w[k] >> (8 * b)) & 0xffu;
                  const uint32_t v = (c & 0xe0u) == 0x40u   ? (c & 31u)
                                     : (c == '-' || c == '*') ? (uint32_t)kTcGap
                                                              : (uint32_t)kTcOther;
                  e |= v << (8 * b);
                }
                w[k] = e;
              }
            }
            if (left < kTcPos) {                // past the end: the zero entry
#pragma unroll
              for (int k = 0; k < 8; ++k)
                w[k] = (w[k] & keep(k)) | ((uint32_t)kTcZero * 0x01010101u & ~keep(k));
            }
            const uint2* my = lut + lane;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const uint2 f0 = my[(w[k] & 0x3fu) * 32], f1 = my[((w[k] >> 8) & 0x3fu) * 32];
              const uint2 f2 = my[((w[k] >> 16) & 0x3fu) * 32], f3 = my[(w[k] >> 24) * 32];
              dst[(2 * k) * kTcGroup] = make_uint4(f0.x, f0.y, f1.x, f1.y);
              dst[(2 * k + 1) * kTcGroup] = make_uint4(f2.x, f2.y, f3.x, f3.y);
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&full[stage]));
          done += kTcProducers;
          if (abort_s) ok = false;
        }
        // stages of the whole window, for the next one
        for (int q = 0; q < groups; ++q) it += (uint32_t)stages_of(q);
      }
    } else if (warp == mma_warp) {
      // ---------------------------------------------------- MMA issue
      // The whole warp runs this loop and one elected lane's instructions
      // take effect: with the values the same in every lane (broadcast
      // explicitly where they come from memory) the compiler keeps the
      // operands in uniform registers, where the instruction wants them.
      bool ok = true;
      const uint32_t leader = elect_one();
      const uint32_t arr0 = smem_u32(arr) >> 4, stage0 = smem_u32(stages) >> 4;
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
      for (int g = 0; g < groups && ok; ++g) {
        const int longest = __shfl_sync(0xffffffffu, gmax[g], 0);
        const TcGroup G(N, Lq, longest);
        for (int p = 0; p < G.passes && ok; ++p) {
          const int row0 = p * kTcCols, rows = min(kTcCols, G.R - row0);
          const bool narrow = rows <= kTcCols / 2;
          if (narrow ? !mbar_wait(smem_u32(&acc_empty[half]), (uses[half] & 1u) ^ 1u)
                     : !(mbar_wait(smem_u32(&acc_empty[0]), (uses[0] & 1u) ^ 1u) &&
                         mbar_wait(smem_u32(&acc_empty[1]), (uses[1] & 1u) ^ 1u))) {
            fail();
            ok = false;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t dcol = tm + (narrow ? half * (kTcCols / 2) : 0u) - (uint32_t)row0;
          for (int t = 0; t < G.stages && ok; ++t, ++it) {
            const uint32_t stage = it % kTcStages;
            if (!mbar_wait(smem_u32(&full[stage]), (it / kTcStages) & 1u)) {
              fail();
              ok = false;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t da = (stage0 + stage * (kTcStageBytes / 16)) | kDescLoA;
            const int k0 = t * kTcPos;
            const int nks = max(1, min(kTcPos / 4, (longest - k0 + 3) / 4));
            // row r of the query operand at positions k0 ..: arr0 + (.. + 2r) / 2
            const uint32_t db0 = (arr0 + (uint32_t)((N + k0 - (G.S - 2)) >> 1)) | kDescLoB;
            // one MMA: rows from r0 of the query operand, K step ks (4
            // positions: two chunks of the segment operand, 32 bytes of arr)
            auto mma = [&](int r0, int ks, uint32_t idesc, uint32_t accum) {
              asm volatile(
                  "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
                  "setp.ne.b32 p, %4, 0;\n\t"
                  "mov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %5};\n\t"
                  "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t}\n"
                  :: "r"(dcol + (uint32_t)r0), "r"(da + (uint32_t)(ks * (2 * kTcGroup))),
                     "r"(db0 + (uint32_t)(r0 + ks * 2)), "r"(idesc), "r"(accum), "n"(kDescHi));
            };
            // rows [r0, r1) times K steps [ka, kb); whole stages unrolled, as
            // the issuing thread's own instructions are what bounds short
            // queries
            auto product = [&](int r0, int r1, int ka, int kb, uint32_t accum) {
              r0 = max(r0, row0);
              r1 = min(r1, row0 + rows);
              for (; r0 < r1; r0 += 256) {
                const uint32_t nn = (uint32_t)min(256, r1 - r0);
                const uint32_t idesc = (1u << 4) | ((nn >> 3) << 17) |
                                       ((uint32_t)(kTcGroup >> 4) << 24);
                if (ka == 0 && kb == kTcPos / 4) {
                  if (leader) {
#pragma unroll
                    for (int ks = 0; ks < kTcPos / 4; ++ks) mma(r0, ks, idesc, 1u);
                  }
                } else {
                  for (int ks = ka; ks < kb; ++ks)
                    if (leader) mma(r0, ks, idesc, accum);
                }
                __syncwarp();
              }
            };
            int ka = 0;
            if (t == 0) {            // the first step writes every column
              product(0, G.R, 0, 1, 0u);
              ka = 1;
            }
            // lags these positions reach: [k0, k0 + 31 + Lq - 1], and, past
            // the end of the cycle, those up to k0 + 30 + Lq - N
            const int hi = min(k0 + kTcPos - 2 + Lq, G.S - 2) & ~1;
            const int rA0 = ((G.S - 2 - hi) >> 1) & ~15;
            const int rA1 = min(G.R, (((G.S - 2 - k0) >> 1) + 16) & ~15);
            product(rA0, rA1, ka, nks, 1u);
            const int wrap = k0 + kTcPos - 2 + Lq - N;
            if (wrap >= 0) {
              const int rW0 = (max(0, G.S - 2 - (wrap & ~1)) >> 1) & ~15;
              product(max(rW0, rA1), G.R, ka, nks, 1u);
            }
            commit_to(smem_u32(&empty[stage]), leader);
            issued = true;
          }
          if (abort_s) ok = false;
          if (narrow) {
            commit_to(smem_u32(&acc_full[half]), leader);
            ++uses[half];
            half ^= 1u;
          } else {
            commit_to(smem_u32(&acc_full[0]), leader);
            commit_to(smem_u32(&acc_full[1]), leader);
            ++uses[0];
            ++uses[1];
          }
        }
      }
      __syncwarp();
    } else {
      // ------------------------------------------------------ epilogue
      const int slot = warp * 32 + lane;
      bool ok = true;
      for (int g = 0; g < groups && ok; ++g) {
        const TcGroup G(N, Lq, gmax[g]);
        float best = -INFINITY;
        for (int p = 0; p < G.passes && ok; ++p) {
          const int rows = min(kTcCols, G.R - p * kTcCols);
          const bool narrow = rows <= kTcCols / 2;
          const uint32_t h0 = narrow ? half : 0u, h1 = narrow ? half : 1u;
          for (uint32_t h = h0; h <= h1; ++h) {
            if (!mbar_wait(smem_u32(&acc_full[h]), uses[h] & 1u)) { fail(); ok = false; }
            ++uses[h];
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t col = tmem + ((uint32_t)(warp * 32) << 16) +
                               (narrow ? half * (kTcCols / 2) : 0u);
          for (int c = 0; c < rows; c += 32) {
            uint32_t v[32];
            // rows is a multiple of 16: the second half of the last read may
            // lie past it, inside the allocation, and is not used
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,"
                "%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, "
                "[%32];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]),
                  "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
                  "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]),
                  "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
                  "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
                  "=r"(v[30]), "=r"(v[31])
                : "r"(col + (uint32_t)c));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            float m0 = __uint_as_float(v[0]), m1 = __uint_as_float(v[1]);
#pragma unroll
            for (int k = 2; k < 16; k += 2) {
              m0 = fmaxf(m0, __uint_as_float(v[k]));
              m1 = fmaxf(m1, __uint_as_float(v[k + 1]));
            }
            if (c + 16 < rows) {
#pragma unroll
              for (int k = 16; k < 32; k += 2) {
                m0 = fmaxf(m0, __uint_as_float(v[k]));
                m1 = fmaxf(m1, __uint_as_float(v[k + 1]));
              }
            }
            best = fmaxf(best, fmaxf(m0, m1));
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0)
            for (uint32_t h = h0; h <= h1; ++h) mbar_arrive(smem_u32(&acc_empty[h]));
          if (narrow) half ^= 1u;
        }
        const int at = g * kTcGroup + slot;
        if (at < valid) {
          const int64_t sg = segment(w0 + order[at]);
          // even lags that no diagonal reaches have y = 0
          if (Lq + length_of(sg) - 1 <= N - 2) best = fmaxf(best, 0.f);
          a.out[sg] = __float2half_rn(0.5f * best);
        }
        if (abort_s) ok = false;
      }
    }
    __syncthreads();
    if (abort_s) break;
  }
  // every MMA issued is complete before the tensor memory is freed
  if (issued) {
    commit_to(smem_u32(&mma_done), elect_one());
    if (!mbar_wait(smem_u32(&mma_done), 0)) fail();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_s) {
    for (int64_t j = tid; j < mine; j += kTcThreads) {
      const int64_t sg = segment(j);
      if (sg < a.n) a.out[sg] = __ushort_as_half((unsigned short)0x7fff);
    }
  }
  if (warp == mma_warp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(kTcCols));
}

// Waits of this kernel that ran out on each device since the library was loaded.
// A count of its own, never cleared: searches in several threads compare it with
// what it was before them, so that none takes another's failure away.
__device__ unsigned g_pf_failures;

unsigned* pf_failures() {
  static std::mutex mu;
  static unsigned* addr[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lk(mu);
  if (!addr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_pf_failures) != cudaSuccess) return nullptr;
    addr[dev] = static_cast<unsigned*>(p);
  }
  return addr[dev];
}

int launch_pf_tc(const PfArgs& a, cudaStream_t stream) {
  unsigned* failures = pf_failures();
  if (!failures) return SSEQS_ERR_CUDA;
  const size_t smem = tc_smem(a.N);
  if (cudaFuncSetAttribute((const void*)prefilter_tc_kernel,
                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return SSEQS_ERR_CUDA;
  const int64_t groups = (a.n + kTcGroup - 1) / kTcGroup;
  const int grid = (int)std::min<int64_t>(groups, device_sm_count());
  { prefilter_tc_kernel<<<grid, kTcThreads, smem, stream>>>(a, failures); count_launches(1); }
  return status_of(cudaGetLastError());
}

// ------------------------------------------------------------ dispatch
using PfFn = void (*)(PfArgs);
struct PfInfo {
  PfFn fn;
  size_t smem;
  int threads;
};

template <int... I>
std::array<PfInfo, sizeof...(I)> pf_table(std::integer_sequence<int, I...>) {
  return {{PfInfo{prefilter_kernel<I + 1>, PfShape<I + 1>::smem, 32 * PfShape<I + 1>::WARPS}...}};
}

int launch_pf(const PfArgs& a, cudaStream_t stream) {
  // Ranks up to 4 fit the 16-byte operand chunks of the tensor-core form,
  // which is faster at every size (its note has the figures); higher ranks and
  // empty queries take the direct sums.
  if (a.k <= kTcRank && a.Lq >= 1) return launch_pf_tc(a, stream);
  static const auto table = pf_table(std::make_integer_sequence<int, 64>{});
  const int C = std::max(1, (a.Lq + 31) / 32);
  const PfInfo& info = table[C - 1];
  if (cudaFuncSetAttribute((const void*)info.fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)info.smem) != cudaSuccess)
    return SSEQS_ERR_CUDA;
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, (const void*)info.fn, info.threads,
                                                    info.smem) != cudaSuccess || nb < 1)
    return SSEQS_ERR_CUDA;
  const int warps = info.threads / 32;
  const int64_t need = (a.n + warps - 1) / warps;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(need, (int64_t)device_sm_count() * nb));
  { info.fn<<<grid, info.threads, info.smem, stream>>>(a); count_launches(1); }
  return status_of(cudaGetLastError());
}

}  // namespace
}  // namespace sseqs

using namespace sseqs;

extern "C" size_t sseqs_prefilter_workspace_bytes(int n, int k) {
  if (n < 2 || k < 1) return 0;
  return 256;
}

extern "C" int sseqs_prefilter(const uint8_t* ascii, const int64_t* offsets, const int32_t* lengths,
                               int64_t n_segments, const uint8_t* query_pos_reversed,
                               int query_len, const float* lut_a, const float* lut_b, int k,
                               int n, void* out_scores, void* workspace, size_t ws_bytes,
                               cudaStream_t stream) {
  if (n_segments < 0 || query_len < 0 || k < 1 || k > kMaxRank) return SSEQS_ERR_ARG;
  if (n < 64 || n > 2048 || (n & (n - 1)) != 0) return SSEQS_ERR_UNSUPPORTED;
  if (query_len > n) return SSEQS_ERR_ARG;
  if (!lut_a || !lut_b || (query_len > 0 && !query_pos_reversed)) return SSEQS_ERR_ARG;
  if (n_segments > 0 && (!ascii || !offsets || !lengths || !out_scores)) return SSEQS_ERR_ARG;
  if (!workspace || ws_bytes < sseqs_prefilter_workspace_bytes(n, k)) return SSEQS_ERR_WORKSPACE;
  if (n_segments == 0) return SSEQS_OK;
  PfArgs a{ascii, offsets, lengths, n_segments, lut_a, lut_b, query_pos_reversed, query_len, k, n,
           reinterpret_cast<__half*>(out_scores)};
  return launch_pf(a, stream);
}

extern "C" int sseqs_prefilter_failures(uint32_t* out, cudaStream_t stream) {
  if (!out) return SSEQS_ERR_ARG;
  const unsigned* failures = pf_failures();
  if (!failures) return SSEQS_ERR_CUDA;
  return status_of(cudaMemcpyAsync(out, failures, sizeof(uint32_t), cudaMemcpyDefault, stream));
}
