// Affine local alignment with traceback (replaces the Triton kernels
// sseqs/sw.py:408-563 and :569-768 driven by sseqs/sw.py:27-219).
//
// Recurrence (textbook Gotoh, gaps open from H), i = query, j = target:
//   M(i,j)  = s(q_i, t_j) + H(i-1,j-1)
//   Ix(i,j) = max(H(i-1,j) - open, Ix(i-1,j) - ext)     Ix(0,j) := -16384
//   Iy(i,j) = max(H(i,j-1) - open, Iy(i,j-1) - ext)     Iy(i,0) := -16384
//   H(i,j)  = max(0, M, Ix, Iy),  H = 0 on row 0 and column 0,
// s = BLOSUM62 for two upper-case standard residues, else -5.  The end cell
// is the first cell in query-major order whose H equals the best score; the
// walk back takes, at every cell, the first state equal to H in the order M,
// Ix, Iy (diagonal, up, left) and stops at H == 0 or a border.  At every
// cell that state's own back-pointer condition holds by construction (M is
// s + H(i-1,j-1); Ix and Iy are the max of their two sources), so a 2-bit
// code per cell (stop / diag / up / left) carries the whole walk.
//
// B200 mapping: one block per target.  A lane holds 4 query rows and a warp 128
// (a row block), swept along the target as a wavefront: lane l computes
// column s - l at step s and receives H and Ix of the row above from lane l - 1
// (two shuffles for 4 cells).  The warps of a block take consecutive row blocks
// and run in phases of 32 steps, each two phases behind the one before it, whose last
// row it reads from a ring in shared memory; more than 1024 rows take several
// sweeps, the row between two of them kept in the workspace.  A step's 4 scores
// are one 32-bit shared-memory word (per lane and residue class), its 4 codes go to
// 4 registers, written as one 16-byte tile of 4 rows x 16 columns, so the walk
// back loads once per tile.
//
// Measured on 1024 targets of up to 500 residues and a 413-residue query: 1.45 ms
// with one warp per target and one row per lane (bound by the chain of dependent
// steps), now 0.37: half of it the issue of about 85 instructions for a step's
// 128 cells, then the walk of the longest paths by one thread each.
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace sseqs {
namespace {

constexpr int kNegBorder = -16384;

struct TbArgs {
  const uint8_t* q;
  int Lq;
  const uint8_t* tbytes;
  const int64_t* toff;
  const int32_t* tlen;
  int B;
  int go, ge;
  uint4* dir;               // workspace: codes, dir_stride tiles per target
  int64_t dir_stride;
  int2* top;                // workspace: last row (H, Ix) of a sweep, top_stride per target
  int64_t top_stride;
  int32_t* best;            // [B]
  int32_t* info;            // [B][5]: alen, q_start, q_end, t_start, t_end
  uint8_t* q_al;            // [B][cap], filled from the end
  uint8_t* t_al;
  int cap;
  int32_t* mfull;           // optional [B][Lq+1][tcols]
  int tcols;
  int tmax;                 // longest target the workspace was sized for
};

__device__ __forceinline__ int tb_class(uint8_t c) {
  return ascii_class(c) < kNumAA ? (int)ascii_class(c) : -1;
}

constexpr int kTbRows = 4;                       // query rows per lane
constexpr int kTbBlock = 32 * kTbRows;           // rows per warp
constexpr int kTbMaxWarps = 8;
constexpr int kTbRing = 128;                     // columns of a ring (a power of two)
constexpr int kTbClasses = 21;
// Scores are held times 4, the low two bits of a candidate for H naming its
// state, so that one maximum decides both (ties: stop, M, Ix, Iy, in this order)
// and the code is the maximum's low bits.  That leaves 2^29 for a score: gap
// costs below 0 (bonuses) can go past it, and then scores are held as they are and
// the state is found by comparisons (TAGGED false, chosen at the launch).
constexpr int kTagStop = 3, kTagM = 2, kTagX = 1, kTagY = 0;

// Shared memory per warp: scores [class][lane] (4 int8 each), and the ring its
// first lane reads.
constexpr size_t kTbWarpBytes = kTbClasses * 32 * 4 + kTbRing * sizeof(int2);

__device__ __forceinline__ int byte_of(uint32_t w, int r) {      // sign-extended byte r
  return (int)(w << (24 - 8 * r)) >> 24;
}

template <bool MATRIX, bool TAGGED>
__global__ void __launch_bounds__(32 * kTbMaxWarps, MATRIX ? 2 : 4) traceback_kernel(TbArgs a) {
  constexpr int SHIFT = TAGGED ? 2 : 0;
  constexpr int M_TAG = TAGGED ? kTagM : 0, X_TAG = TAGGED ? kTagX : 0, Y_TAG = TAGGED ? kTagY : 0;
  constexpr int kNegIx = (1 << SHIFT) * kNegBorder + X_TAG;
  constexpr int kNegIy = (1 << SHIFT) * kNegBorder + Y_TAG;
  extern __shared__ int2 tb_sm[];
  __shared__ uint8_t scls[256];
  __shared__ int8_t sb62[400];
  __shared__ int red[kTbMaxWarps][3];
  const int b = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
  const int Lq = a.Lq;
  const int Lt = a.tlen[b];
  if (Lt < 0 || Lt > a.tmax) {   // outside the workspace the caller sized
    if (tid == 0) {
      a.best[b] = -1;
      for (int k = 0; k < 5; ++k) a.info[(int64_t)b * 5 + k] = -1;
    }
    return;
  }
  int2* rings = tb_sm;                                                  // [nw][kTbRing]
  uint32_t* prof = reinterpret_cast<uint32_t*>(rings + nw * kTbRing) + w * (kTbClasses * 32);
  for (int i = tid; i < 256; i += blockDim.x) {
    const int c = tb_class((uint8_t)i);
    scls[i] = (uint8_t)(c < 0 ? kTbClasses - 1 : c);
  }
  for (int i = tid; i < 400; i += blockDim.x) sb62[i] = blosum62(i / 20, i % 20);
  __syncthreads();

  const uint8_t* t = a.tbytes + a.toff[b];
  const int ge = (1 << SHIFT) * a.ge;
  const int open_x = X_TAG - (1 << SHIFT) * a.go, open_y = Y_TAG - (1 << SHIFT) * a.go;
  const int own_phases = (Lt + 31 + 31) >> 5;         // a row block's Lt + 31 steps
  const int words = 2 * own_phases;                   // its code words
  uint4* dir = a.dir + (int64_t)b * a.dir_stride;
  int2* top = a.top + (int64_t)b * a.top_stride;
  int32_t* mf = MATRIX ? a.mfull + (int64_t)b * (Lq + 1) * a.tcols : nullptr;

  int bestv = 0, bi = 0x7fffffff, bj = 0x7fffffff;
  const int nblocks = (Lt > 0) ? (Lq + kTbBlock - 1) / kTbBlock : 0;
  for (int sweep = 0; sweep < nblocks; sweep += nw) {
    const int blk = sweep + w;
    const bool live = blk < nblocks;
    const int active = min(nw, nblocks - sweep);      // warps of this sweep
    const int i0 = blk * kTbBlock + lane * kTbRows;   // row r of the lane: i0 + r + 1 (1-based)
    int rbest[kTbRows], rbj[kTbRows], hl[kTbRows], yl[kTbRows];
    uint32_t codes[kTbRows];
    if (live) {
      int qc[kTbRows];
#pragma unroll
      for (int r = 0; r < kTbRows; ++r) {
        const bool ok = i0 + r < Lq;
        qc[r] = ok ? tb_class(a.q[i0 + r]) : -1;
        rbest[r] = ok ? 0 : 0x7fffffff;               // rows past the query never win
        rbj[r] = 0x7fffffff;
        hl[r] = 0;                                    // H(i, 0)
        yl[r] = kNegIy;                               // Iy(i, 0)
        codes[r] = 0;
      }
      for (int c = 0; c < kTbClasses; ++c) {
        uint32_t v = 0;
#pragma unroll
        for (int r = 0; r < kTbRows; ++r) {
          const int s = (qc[r] >= 0 && c < kNumAA) ? sb62[qc[r] * 20 + c] : -5;
          v |= (uint32_t)(uint8_t)(int8_t)((1 << SHIFT) * s + M_TAG) << (8 * r);
        }
        prof[c * 32 + lane] = v;
      }
    }
    __syncwarp();
    int hrow = 0, xrow = kNegIx;                      // the lane's last row, previous step
    int hdiag = 0;                                    // H of the row above, previous column
    const int phases = own_phases + 2 * (active - 1);
    for (int ph = 0; ph < phases; ++ph) {
      const int s0 = (ph - 2 * w) * 32;
      if (live && s0 >= 0 && s0 < Lt + 31) {
        int2* in = rings + w * kTbRing;
        int2* out = rings + (w + 1 < nw ? w + 1 : 0) * kTbRing;
        const bool to_ring = w + 1 < active, to_top = !to_ring && blk + 1 < nblocks;
        // the row above the first warp's block: constant, or the last sweep's row
        if (w == 0) {
          const int c = s0 + lane;
          in[c & (kTbRing - 1)] = (sweep > 0 && c < Lt) ? top[c] : make_int2(0, kNegIx);
          __syncwarp();
        }
        // residue classes of columns s0 - 32 .. s0 + 31 (0-based), a lane each
        const int ca = s0 - 32 + lane, cb = s0 + lane;
        const int clsA = ca >= 0 && ca < Lt ? scls[__ldg(t + ca)] : 0;
        const int clsB = cb < Lt ? scls[__ldg(t + cb)] : 0;
        // this lane's next column's class, moved along the warp
        int cls = __shfl_sync(0xffffffffu, clsA, (31 - lane) & 31);   // column s0 - 1 - lane
        // One step of the wavefront.  CHECK: some lane may be before its first
        // column or past its last one.
        auto step = [&](auto check, int k) {
          constexpr bool CHECK = decltype(check)::value;
          const int j = s0 + k - lane + 1;            // this lane's column (1-based)
          const int fresh = __shfl_sync(0xffffffffu, clsB, k);
          const int cls_up = __shfl_up_sync(0xffffffffu, cls, 1);
          const int h_up = __shfl_up_sync(0xffffffffu, hrow, 1);
          const int x_up = __shfl_up_sync(0xffffffffu, xrow, 1);
          const int2 ring = in[(s0 + k) & (kTbRing - 1)];
          cls = lane == 0 ? fresh : cls_up;
          const int hup = lane == 0 ? ring.x : h_up, xup = lane == 0 ? ring.y : x_up;
          const bool on = !CHECK || (j >= 1 && j <= Lt);
          uint32_t code[kTbRows] = {};
          if (CHECK) {
            hrow = 0;
            xrow = kNegIx;
          }
          if (on) {
            const uint32_t sc = prof[cls * 32 + lane];
            int diag = hdiag, hu = hup, xu = xup;
#pragma unroll
            for (int r = 0; r < kTbRows; ++r) {
              // floor (tag 3) and M (2), Ix (1), Iy (0): the largest tagged value is
              // the cell's H and, in its low bits, the state that gave it
              const int sm = byte_of(sc, r);
              const int m = __viaddmax_s32(diag, sm, TAGGED ? kTagStop : 0);
              const int x = __viaddmax_s32(hu, open_x, xu - ge);
              const int y = __viaddmax_s32(hl[r], open_y, yl[r] - ge);
              const int v = __vimax3_s32(m, x, y);
              const int h = TAGGED ? v & ~3 : v;
              code[r] = TAGGED   ? (uint32_t)v
                        : v == 0 ? (uint32_t)kTagStop
                        : v == m ? (uint32_t)kTagM
                                 : (uint32_t)(v == x ? kTagX : kTagY);
              if (h > rbest[r]) { rbest[r] = h; rbj[r] = j; }
              if constexpr (MATRIX) {
                if (i0 + r < Lq) mf[(int64_t)(i0 + r + 1) * a.tcols + j] = (sm + diag) >> SHIFT;
              }
              diag = hl[r];
              hl[r] = h;
              yl[r] = y;
              hu = h;
              xu = x;
            }
            hrow = hu;
            xrow = xu;
            if (lane == 31) {
              if (to_ring) out[(j - 1) & (kTbRing - 1)] = make_int2(hrow, xrow);
              else if (to_top) top[j - 1] = make_int2(hrow, xrow);
            }
          }
#pragma unroll
          for (int r = 0; r < kTbRows; ++r) codes[r] = __funnelshift_r(codes[r], code[r], 2);
          hdiag = !CHECK || j >= 1 ? hup : 0;
        };
        // 16 steps' codes make one word a row: a tile, stored by the whole warp
        auto flush = [&](int word) {
          dir[((int64_t)blk * words + word) * 32 + lane] =
              make_uint4(codes[0], codes[1], codes[2], codes[3]);
        };
        if (s0 >= 31 && s0 + 32 <= Lt) {              // every lane inside the target
#pragma unroll 1
          for (int h = 0; h < 2; ++h) {
#pragma unroll 2
            for (int k = 0; k < 16; ++k) step(std::false_type{}, 16 * h + k);
            flush((s0 >> 4) + h);
          }
        } else {
#pragma unroll 1
          for (int h = 0; h < 2; ++h) {
#pragma unroll 1
            for (int k = 0; k < 16; ++k) step(std::true_type{}, 16 * h + k);
            flush((s0 >> 4) + h);
          }
        }
      }
      __syncthreads();
    }
    if (live) {
#pragma unroll
      for (int r = 0; r < kTbRows; ++r) {
        const int i = i0 + r + 1;
        if (i <= Lq && rbest[r] > 0 &&
            (rbest[r] > bestv || (rbest[r] == bestv && (i < bi || (i == bi && rbj[r] < bj))))) {
          bestv = rbest[r];
          bi = i;
          bj = rbj[r];
        }
      }
    }
  }
  // best value, then the first cell in query-major order: over the warp, then
  // over the warps
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const int ov = __shfl_xor_sync(0xffffffffu, bestv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    const int oj = __shfl_xor_sync(0xffffffffu, bj, o);
    if (ov > bestv || (ov == bestv && (oi < bi || (oi == bi && oj < bj)))) {
      bestv = ov; bi = oi; bj = oj;
    }
  }
  if (lane == 0) { red[w][0] = bestv; red[w][1] = bi; red[w][2] = bj; }
  __syncthreads();
  if (tid != 0) return;
  for (int v = 1; v < nw; ++v) {
    const int ov = red[v][0], oi = red[v][1], oj = red[v][2];
    if (ov > bestv || (ov == bestv && (oi < bi || (oi == bi && oj < bj)))) {
      bestv = ov; bi = oi; bj = oj;
    }
  }
  bestv >>= SHIFT;
  a.best[b] = bestv;
  int32_t* inf = a.info + (int64_t)b * 5;
  inf[0] = 0; inf[1] = -1; inf[2] = -1; inf[3] = -1; inf[4] = -1;
  if (!(bestv > 0 && Lq > 0 && Lt > 0)) return;
  uint8_t* qa = a.q_al + (int64_t)b * a.cap;
  uint8_t* ta = a.t_al + (int64_t)b * a.cap;
  int ci = bi, cj = bj, n = 0;
  while (ci > 0 && cj > 0) {
    // the tile of cell (ci, cj): lane l of row block (ci - 1) / 128 computed the
    // cell at step cj - 1 + l; walked until the path leaves it
    const int group = (ci - 1) >> 2, l = group & 31, word = (cj - 1 + l) >> 4;
    const uint4 tile = dir[((int64_t)((ci - 1) / kTbBlock) * words + word) * 32 + l];
    bool stop = false;
    do {
      const int r = (ci - 1) & 3;
      const uint32_t row = r == 0 ? tile.x : r == 1 ? tile.y : r == 2 ? tile.z : tile.w;
      const int code = (int)(row >> (((cj - 1 + l) & 15) * 2)) & 3;
      if (code == kTagStop) { stop = true; break; }
      const int pos = a.cap - 1 - n;
      qa[pos] = code == kTagY ? (uint8_t)'-' : a.q[ci - 1];
      ta[pos] = code == kTagX ? (uint8_t)'-' : t[cj - 1];
      ci -= code != kTagY;
      cj -= code != kTagX;
      ++n;
    } while (cj > 0 && ((ci + 3) >> 2) == group + 1 && ((cj - 1 + l) >> 4) == word);
    if (stop) break;
  }
  if (n > 0) {
    inf[0] = n; inf[1] = ci; inf[2] = bi - 1; inf[3] = cj; inf[4] = bj - 1;
  }
}

}  // namespace
}  // namespace sseqs

using namespace sseqs;

namespace {
// Code tiles (4 rows x 16 steps) of one target: a row block's 32 lanes by its
// words (two a phase, tmax + 31 steps).
inline int64_t dir_tiles(int query_len, int tmax) {
  return (int64_t)((query_len + kTbBlock - 1) / kTbBlock) * 32 * (2 * ((tmax + 62) / 32));
}
}  // namespace

extern "C" size_t sseqs_backtrack_workspace_bytes(int query_len, int max_target_len, int B) {
  if (B < 0 || query_len < 0 || max_target_len < 0) return 0;
  return (size_t)B * (16 * (size_t)dir_tiles(query_len, max_target_len) +
                      sizeof(int2) * ((size_t)max_target_len + 1)) + 256;
}

extern "C" int sseqs_backtrack_affine(const uint8_t* query, int query_len, const uint8_t* tbytes,
                                      const int64_t* toff, const int32_t* tlen, int max_target_len,
                                      int B, int gap_open, int gap_extend, int32_t* best,
                                      int32_t* info, uint8_t* q_aligned, uint8_t* t_aligned,
                                      int cap, int32_t* m_full, int tcols, void* workspace,
                                      size_t ws_bytes, cudaStream_t stream) {
  if (B < 0 || query_len < 0 || max_target_len < 0) return SSEQS_ERR_ARG;
  if (B == 0) return SSEQS_OK;
  if (!tbytes || !toff || !tlen || !best || !info || !q_aligned || !t_aligned ||
      (query_len > 0 && !query))
    return SSEQS_ERR_ARG;
  if (cap < query_len + max_target_len) return SSEQS_ERR_ARG;
  if (m_full && tcols < max_target_len + 1) return SSEQS_ERR_ARG;
  if (!workspace || ws_bytes < sseqs_backtrack_workspace_bytes(query_len, max_target_len, B))
    return SSEQS_ERR_WORKSPACE;
  // tiles first, on a 16-byte boundary (the size has 256 bytes to spare)
  uint4* dir = reinterpret_cast<uint4*>((reinterpret_cast<uintptr_t>(workspace) + 15) &
                                        ~(uintptr_t)15);
  const int64_t ds = dir_tiles(query_len, max_target_len);
  int2* top = reinterpret_cast<int2*>(dir + (int64_t)B * ds);
  // The tagged form, unless a step's largest gain (11, or a gap that is a bonus) over
  // the longest path could come near 2^26.  Below that a gap cost of 2^26 or more
  // makes a state negative and less than its other source whatever its
  // size, so larger ones are cut to it.
  const int64_t gain = std::max<int64_t>({11, -(int64_t)gap_open, -(int64_t)gap_extend});
  const bool tagged = gain * ((int64_t)query_len + max_target_len + 2) < (1 << 26) + kNegBorder;
  auto cost = [&](int g) { return tagged ? std::min(1 << 26, g) : g; };
  TbArgs a{query, query_len, tbytes, toff, tlen, B, cost(gap_open), cost(gap_extend), dir, ds,
           top, (int64_t)max_target_len + 1, best, info, q_aligned, t_aligned, cap, m_full, tcols,
           max_target_len};
  const int warps = std::max(1, std::min(kTbMaxWarps, (query_len + kTbBlock - 1) / kTbBlock));
  auto fn = m_full ? (tagged ? traceback_kernel<true, true> : traceback_kernel<true, false>)
                   : (tagged ? traceback_kernel<false, true> : traceback_kernel<false, false>);
  { fn<<<B, 32 * warps, warps * kTbWarpBytes, stream>>>(a); count_launches(1); }
  return status_of(cudaGetLastError());
}
