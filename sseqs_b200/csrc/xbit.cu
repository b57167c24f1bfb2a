// xbit 5-bit codec (layout of sseqs/xbit.cu:8-62): 8 symbols per 5 bytes,
// first symbol in the high bits of a big-endian 40-bit window, symbol s is
// the byte s + 64.
//
// Decoding is HBM-bound (0.625 B read + 1 B written per symbol).  A block
// stages a tile of packed bytes in shared memory with 16-byte loads of the
// aligned chunks that cover it (every chunk read holds at least one byte of
// the tile, so no load leaves the caller's 16-byte chunks), then every thread
// decodes 4 groups (32 symbols, 20 bytes, as words: a stride of 5 words is
// conflict-free) and writes them as two 16-byte stores.
//
// Loading a batch needs the '@' positions of the decoded bytes besides: the
// same pass keeps one bit per symbol ('@' or not), a count per tile and the
// last other symbol, so that the positions come from 1/8 of the bytes and the
// decoded batch is not read again.
#include <algorithm>

#include "common.cuh"

namespace sseqs {
namespace {

constexpr int kDecThreads = 256;
constexpr int kGroupsPerThread = 4;                                // 32 symbols
constexpr int kTileGroups = kDecThreads * kGroupsPerThread;        // 1024 groups
constexpr int kTileBytes = kTileGroups * 5;                        // 5120 B in
constexpr int kTileChunks = kTileBytes / 16 + 2;                   // staged chunks

// The four 5-bit codes of 20 bits, the first in the high bits, as bytes from
// the low one up.
__device__ __forceinline__ uint32_t spread4(uint32_t v) {
  return ((v >> 15) & 31u) | ((v >> 2) & 0x1f00u) | ((v << 11) & 0x1f0000u) |
         ((v << 24) & 0x1f000000u);
}

// Bit i: byte i of the codes is 0 (bytes hold 0..31).
__device__ __forceinline__ uint32_t zero_bytes(uint32_t c) {
  const uint32_t z = (~(c + 0x7f7f7f7fu) >> 7) & 0x01010101u;
  return (z * 0x01020408u) >> 24 & 0xfu;
}

struct ScanOut {
  uint32_t* bits;        // [tiles][kDecThreads]: bit k of word t: symbol 32t + k is '@'
  int32_t* count;        // [tiles]
  int64_t* info;         // [0]: last symbol that is not '@' (preset to -1)
};

// in: packed stream starting at symbol 0; n_groups_total = ceil(n_syms / 8)
template <bool kAlignedOut, bool kScan>
__global__ void __launch_bounds__(kDecThreads)
    xbit_decode_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, int64_t n_syms,
                       ScanOut scan) {
  __shared__ uint4 stage[kTileChunks];
  __shared__ int warp_count[kDecThreads / 32];
  const uint32_t* swords = reinterpret_cast<const uint32_t*>(stage);
  const int64_t n_groups = (n_syms + 7) / 8;
  const int64_t n_tiles = (n_groups + kTileGroups - 1) / kTileGroups;
  const uintptr_t iu = reinterpret_cast<uintptr_t>(in);
  const uint4* abase = reinterpret_cast<const uint4*>(iu & ~(uintptr_t)15);
  const int64_t ioff = (int64_t)(iu & 15);
  int64_t last = -1;

  for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int64_t g0 = tile * kTileGroups;
    const int64_t ng = min((int64_t)kTileGroups, n_groups - g0);
    const int64_t byte0 = g0 * 5 + ioff;          // aligned coordinates
    // exclusive end, clipped to the packed stream's (5n+7)/8 bytes
    const int64_t byte1 = min((g0 + ng) * 5, (n_syms * 5 + 7) / 8) + ioff;
    const int64_t c0 = byte0 >> 4, c1 = (byte1 + 15) >> 4;
    __syncthreads();
    for (int64_t c = c0 + threadIdx.x; c < c1; c += blockDim.x) stage[c - c0] = __ldg(abase + c);
    __syncthreads();
    // this thread's 20 bytes as 5 words (the groups past the stream's end hold
    // whatever the stage held; their symbols are not written)
    const int at = (int)(byte0 - (c0 << 4)) + (int)threadIdx.x * (kGroupsPerThread * 5);
    const uint32_t sh = (uint32_t)(at & 3) * 8u;
    uint32_t b[6], w[2 * kGroupsPerThread];
#pragma unroll
    for (int k = 0; k < 6; ++k) b[k] = swords[(at >> 2) + k];
#pragma unroll
    for (int k = 0; k < 5; ++k)                   // big-endian, so that codes run downwards
      b[k] = __byte_perm(__funnelshift_r(b[k], b[k + 1], sh), 0u, 0x0123u);
    w[0] = spread4(b[0] >> 12);
    w[1] = spread4(((b[0] << 8) | (b[1] >> 24)) & 0xfffffu);
    w[2] = spread4((b[1] >> 4) & 0xfffffu);
    w[3] = spread4(((b[1] << 16) | (b[2] >> 16)) & 0xfffffu);
    w[4] = spread4(((b[2] << 4) | (b[3] >> 28)) & 0xfffffu);
    w[5] = spread4((b[3] >> 8) & 0xfffffu);
    w[6] = spread4(((b[3] << 12) | (b[4] >> 20)) & 0xfffffu);
    w[7] = spread4(b[4] & 0xfffffu);
    const int64_t s0 = (g0 + (int64_t)threadIdx.x * kGroupsPerThread) * 8;   // first symbol
    if constexpr (kScan) {
      uint32_t at_bits = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) at_bits |= zero_bytes(w[k]) << (4 * k);
      const int64_t left = n_syms - s0;
      const uint32_t live = left >= 32 ? 0xffffffffu : left <= 0 ? 0u : (1u << left) - 1u;
      const uint32_t other = ~at_bits & live;
      if (other) last = max(last, s0 + 31 - __clz((int)other));
      at_bits &= live;
      scan.bits[tile * kDecThreads + threadIdx.x] = at_bits;
      const int c = __reduce_add_sync(0xffffffffu, __popc(at_bits));
      if ((threadIdx.x & 31) == 0) warp_count[threadIdx.x >> 5] = c;
      __syncthreads();
      if (threadIdx.x == 0) {
        int t = 0;
        for (int k = 0; k < kDecThreads / 32; ++k) t += warp_count[k];
        scan.count[tile] = t;
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) w[k] += 0x40404040u;
    if (kAlignedOut && s0 + 32 <= n_syms) {
      uint4* o = reinterpret_cast<uint4*>(out + s0);
      o[0] = make_uint4(w[0], w[1], w[2], w[3]);
      o[1] = make_uint4(w[4], w[5], w[6], w[7]);
    } else {
#pragma unroll
      for (int k = 0; k < 32; ++k)
        if (s0 + k < n_syms) out[s0 + k] = (uint8_t)(w[k >> 2] >> ((k & 3) * 8));
    }
  }
  if constexpr (kScan) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
    if ((threadIdx.x & 31) == 0 && last >= 0)
      atomicMax(reinterpret_cast<long long*>(scan.info), (long long)last);
  }
}

// Exclusive scan of the tiles' counts (one block) into off; total -> info[1].
constexpr int kScanThreads = 1024;
template <class T>
__device__ __forceinline__ int64_t scan_block(T v, int64_t* excl) {
  __shared__ int64_t sums[kScanThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int64_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sums[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int64_t s = lane < (int)(blockDim.x >> 5) ? sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    sums[lane] = s;
  }
  __syncthreads();
  *excl = (wid == 0 ? 0 : sums[wid - 1]) + x - v;
  const int64_t total = sums[(blockDim.x >> 5) - 1];
  __syncthreads();
  return total;
}

__global__ void __launch_bounds__(kScanThreads)
    tile_scan_kernel(const int32_t* count, int64_t tiles, int64_t* off, int64_t* total) {
  constexpr int PER = 8;
  int64_t carry = 0;
  for (int64_t base = 0; base < tiles; base += (int64_t)kScanThreads * PER) {
    const int64_t i0 = base + (int64_t)threadIdx.x * PER;
    int32_t v[PER];
    int64_t sum = 0, ex;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      v[k] = i0 + k < tiles ? count[i0 + k] : 0;
      sum += v[k];
    }
    const int64_t all = scan_block(sum, &ex);
    ex += carry;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      if (i0 + k < tiles) off[i0 + k] = ex;
      ex += v[k];
    }
    carry += all;
  }
  if (threadIdx.x == 0) *total = carry;
}

// Positions of the first nd '@' from the bits, a tile a block.
__global__ void __launch_bounds__(kDecThreads)
    delim_scatter_kernel(const uint32_t* bits, const int64_t* off, int64_t tiles, int64_t nd,
                         int32_t* out) {
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    uint32_t m = bits[tile * kDecThreads + threadIdx.x];
    int64_t ex;
    scan_block(__popc(m), &ex);
    int64_t o = off[tile] + ex;
    const int64_t s0 = (tile * kDecThreads + threadIdx.x) * 32;
    while (m && o < nd) {
      out[o++] = (int32_t)(s0 + __ffs((int)m) - 1);
      m &= m - 1;
    }
  }
}

// ---- segment table of one batch from its delimiters (sseqs/msa.py:237-267)
constexpr int kSegThreads = 256, kSegItems = 8, kSegTile = kSegThreads * kSegItems;

struct SegArgs {
  const int32_t* delim;
  int64_t nd, nseg;          // delimiters; segments (nd, or nd + 1 with a trailing one)
  int64_t n;                 // symbols
  __device__ int32_t length(int64_t k) const {
    const int64_t prev = k == 0 ? -1 : (int64_t)delim[k - 1];
    return (int32_t)((k < nd ? (int64_t)delim[k] : n) - prev - 1);
  }
};

// Per tile: non-empty segments and the sum of their lengths + 1; info[0..2]:
// maximum length and total residues by atomics ([0] is set by the scan).
__global__ void __launch_bounds__(kSegThreads)
    seg_count_kernel(SegArgs a, int64_t tiles, int64_t* cnt, int64_t* sum, int64_t* info) {
  int longest = 0;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    int c = 0;
    int64_t s = 0;
#pragma unroll
    for (int i = 0; i < kSegItems; ++i) {
      const int64_t k = tile * kSegTile + i * kSegThreads + threadIdx.x;
      const int len = k < a.nseg ? a.length(k) : 0;
      c += len != 0;
      s += len != 0 ? len + 1 : 0;
      longest = max(longest, len);
    }
    int64_t ex;
    const int64_t ct = scan_block(c, &ex);
    const int64_t st = scan_block(s, &ex);
    if (threadIdx.x == 0) { cnt[tile] = ct; sum[tile] = st; }
  }
  longest = __reduce_max_sync(0xffffffffu, longest);
  if ((threadIdx.x & 31) == 0 && longest > 0)
    atomicMax(reinterpret_cast<long long*>(info + 1), (long long)longest);
}

// Both per-tile arrays to exclusive offsets in place (one block); info[0] =
// segments, info[2] = residues.
__global__ void __launch_bounds__(kScanThreads)
    seg_scan_kernel(int64_t* cnt, int64_t* sum, int64_t tiles, int64_t* info) {
  int64_t cc = 0, cs = 0;
  for (int64_t base = 0; base < tiles; base += kScanThreads) {
    const int64_t i = base + threadIdx.x;
    const int64_t c = i < tiles ? cnt[i] : 0, s = i < tiles ? sum[i] : 0;
    int64_t ec, es;
    const int64_t tc = scan_block(c, &ec);
    const int64_t ts = scan_block(s, &es);
    if (i < tiles) { cnt[i] = cc + ec; sum[i] = cs + es; }
    cc += tc;
    cs += ts;
  }
  if (threadIdx.x == 0) { info[0] = cc; info[2] = cs - cc; }
}

__global__ void __launch_bounds__(kSegThreads)
    seg_scatter_kernel(SegArgs a, int64_t tiles, const int64_t* cnt, const int64_t* sum,
                       int32_t* seg_index, int32_t* lengths, int64_t* offsets) {
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t k0 = tile * kSegTile + (int64_t)threadIdx.x * kSegItems;
    int32_t len[kSegItems];
    int c = 0;
    int64_t s = 0;
#pragma unroll
    for (int i = 0; i < kSegItems; ++i) {
      len[i] = k0 + i < a.nseg ? a.length(k0 + i) : 0;
      c += len[i] != 0;
      s += len[i] != 0 ? len[i] + 1 : 0;
    }
    int64_t ec, es;
    scan_block(c, &ec);
    scan_block(s, &es);
    int64_t o = cnt[tile] + ec, at = sum[tile] + es;
#pragma unroll
    for (int i = 0; i < kSegItems; ++i) {
      if (len[i] != 0) {
        seg_index[o] = (int32_t)(k0 + i);
        lengths[o] = len[i];
        offsets[o] = at;
        ++o;
        at += len[i] + 1;
      }
    }
  }
}

__global__ void xbit_encode_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out,
                                   int64_t n_syms) {
  const int64_t n_groups = (n_syms + 7) / 8;
  const int64_t out_bytes = (n_syms * 5 + 7) / 8;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_groups;
       t += (int64_t)gridDim.x * blockDim.x) {
    uint64_t w = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint8_t s = (t * 8 + k < n_syms) ? (uint8_t)(in[t * 8 + k] - 64u) : 0;
      w |= (uint64_t)(s & 31u) << (35 - 5 * k);
    }
#pragma unroll
    for (int b = 0; b < 5; ++b)
      if (t * 5 + b < out_bytes) out[t * 5 + b] = (uint8_t)(w >> (32 - 8 * b));
  }
}

}  // namespace
}  // namespace sseqs

using namespace sseqs;

namespace {
template <bool kScan>
int launch_decode(const uint8_t* in, uint8_t* out, int64_t n_syms, ScanOut scan,
                  cudaStream_t stream) {
  const int64_t n_groups = (n_syms + 7) / 8;
  const int64_t n_tiles = (n_groups + kTileGroups - 1) / kTileGroups;
  const int grid = (int)std::min<int64_t>(n_tiles, (int64_t)device_sm_count() * 8);
  if ((reinterpret_cast<uintptr_t>(out) & 15) == 0)
    { xbit_decode_kernel<true, kScan><<<grid, kDecThreads, 0, stream>>>(in, out, n_syms, scan); count_launches(1); }
  else
    { xbit_decode_kernel<false, kScan><<<grid, kDecThreads, 0, stream>>>(in, out, n_syms, scan); count_launches(1); }
  return status_of(cudaGetLastError());
}

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
inline int64_t decode_tiles(int64_t n) { return std::max<int64_t>(1, (n + kTileGroups * 8 - 1) / (kTileGroups * 8)); }
inline int64_t seg_tiles(int64_t n) { return std::max<int64_t>(1, (n + kSegTile - 1) / kSegTile); }

// Workspace of a batch being loaded: bits, tile counts, tile offsets.
struct LoadSpace {
  uint32_t* bits;
  int32_t* count;
  int64_t* off;
  static size_t bytes(int64_t n) {
    const size_t t = (size_t)decode_tiles(n);
    return align256(t * kDecThreads * 4) + align256(t * 4) + align256(t * 8);
  }
  LoadSpace(void* ws, int64_t n) {
    const size_t t = (size_t)decode_tiles(n);
    char* p = static_cast<char*>(ws);
    bits = reinterpret_cast<uint32_t*>(p);
    p += align256(t * kDecThreads * 4);
    count = reinterpret_cast<int32_t*>(p);
    p += align256(t * 4);
    off = reinterpret_cast<int64_t*>(p);
  }
};
}  // namespace

extern "C" int sseqs_xbit_decompress(const uint8_t* packed, uint8_t* out, int64_t n_syms,
                                     int64_t lo_bytes, cudaStream_t stream) {
  if (n_syms < 0 || lo_bytes < 0) return SSEQS_ERR_ARG;
  if (n_syms == 0) return SSEQS_OK;
  if (!packed || !out) return SSEQS_ERR_ARG;
  return launch_decode<false>(packed + lo_bytes, out, n_syms, ScanOut{}, stream);
}

extern "C" size_t sseqs_decode_scan_workspace_bytes(int64_t n_syms) {
  return n_syms < 0 ? 0 : LoadSpace::bytes(n_syms);
}

extern "C" int sseqs_decode_scan(const uint8_t* packed, uint8_t* out, int64_t n_syms,
                                 int64_t lo_bytes, int64_t* info, void* workspace,
                                 size_t ws_bytes, cudaStream_t stream) {
  if (n_syms < 0 || lo_bytes < 0) return SSEQS_ERR_ARG;
  if (!info || (n_syms > 0 && (!packed || !out))) return SSEQS_ERR_ARG;
  if (!workspace || ws_bytes < sseqs_decode_scan_workspace_bytes(n_syms)) return SSEQS_ERR_WORKSPACE;
  if (cudaMemsetAsync(info, 0xff, sizeof(int64_t), stream) != cudaSuccess) return SSEQS_ERR_CUDA;
  if (n_syms == 0) return status_of(cudaMemsetAsync(info + 1, 0, sizeof(int64_t), stream));
  const LoadSpace w(workspace, n_syms);
  const int st = launch_decode<true>(packed + lo_bytes, out, n_syms,
                                     ScanOut{w.bits, w.count, info}, stream);
  if (st != SSEQS_OK) return st;
  { tile_scan_kernel<<<1, kScanThreads, 0, stream>>>(w.count, decode_tiles(n_syms), w.off, info + 1);
    count_launches(1); }
  return status_of(cudaGetLastError());
}

extern "C" int sseqs_decode_scan_delims(int64_t n_syms, int64_t n_delims, int32_t* out_pos,
                                        const void* workspace, size_t ws_bytes,
                                        cudaStream_t stream) {
  if (n_syms < 0 || n_delims < 0 || n_delims > n_syms) return SSEQS_ERR_ARG;
  if (n_delims == 0) return SSEQS_OK;
  if (!out_pos) return SSEQS_ERR_ARG;
  if (!workspace || ws_bytes < sseqs_decode_scan_workspace_bytes(n_syms)) return SSEQS_ERR_WORKSPACE;
  const LoadSpace w(const_cast<void*>(workspace), n_syms);
  const int64_t tiles = decode_tiles(n_syms);
  const int grid = (int)std::min<int64_t>(tiles, (int64_t)device_sm_count() * 8);
  { delim_scatter_kernel<<<grid, kDecThreads, 0, stream>>>(w.bits, w.off, tiles, n_delims, out_pos);
    count_launches(1); }
  return status_of(cudaGetLastError());
}

extern "C" size_t sseqs_segments_workspace_bytes(int64_t max_segments) {
  return max_segments < 0 ? 0 : 2 * align256(8 * (size_t)seg_tiles(max_segments));
}

extern "C" int sseqs_segments(int64_t n, const int32_t* delim, int64_t n_delims, int trailing,
                              int32_t* seg_index, int32_t* lengths, int64_t* offsets,
                              int64_t* info, void* workspace, size_t ws_bytes,
                              cudaStream_t stream) {
  const int64_t nseg = n_delims + (trailing ? 1 : 0);
  if (n < 0 || n_delims < 0 || (n_delims > 0 && !delim) || !info ||
      (nseg > 0 && (!seg_index || !lengths || !offsets)))
    return SSEQS_ERR_ARG;
  if (n > INT32_MAX) return SSEQS_ERR_UNSUPPORTED;   // positions are int32 per batch
  if (!workspace || ws_bytes < sseqs_segments_workspace_bytes(nseg)) return SSEQS_ERR_WORKSPACE;
  if (cudaMemsetAsync(info, 0, 3 * sizeof(int64_t), stream) != cudaSuccess) return SSEQS_ERR_CUDA;
  if (nseg == 0) return SSEQS_OK;
  const int64_t tiles = seg_tiles(nseg);
  int64_t* cnt = static_cast<int64_t*>(workspace);
  int64_t* sum = reinterpret_cast<int64_t*>(static_cast<char*>(workspace) + align256(8 * (size_t)tiles));
  const SegArgs a{delim, n_delims, nseg, n};
  const int grid = (int)std::min<int64_t>(tiles, (int64_t)device_sm_count() * 8);
  { seg_count_kernel<<<grid, kSegThreads, 0, stream>>>(a, tiles, cnt, sum, info); count_launches(1); }
  { seg_scan_kernel<<<1, kScanThreads, 0, stream>>>(cnt, sum, tiles, info); count_launches(1); }
  { seg_scatter_kernel<<<grid, kSegThreads, 0, stream>>>(a, tiles, cnt, sum, seg_index, lengths,
                                                         offsets); count_launches(1); }
  return status_of(cudaGetLastError());
}

extern "C" int sseqs_xbit_compress(const uint8_t* in, uint8_t* out, int64_t n_syms,
                                   cudaStream_t stream) {
  if (n_syms < 0) return SSEQS_ERR_ARG;
  if (n_syms == 0) return SSEQS_OK;
  if (!in || !out) return SSEQS_ERR_ARG;
  const int64_t n_groups = (n_syms + 7) / 8;
  const int grid = (int)std::min<int64_t>((n_groups + 255) / 256, (int64_t)device_sm_count() * 16);
  { xbit_encode_kernel<<<grid, 256, 0, stream>>>(in, out, n_syms); count_launches(1); }
  return status_of(cudaGetLastError());
}
