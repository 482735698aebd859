// Device-wide building blocks written for this library: exclusive scan and a
// stable LSD radix sort (8-bit digits, warp-match ranking).  Used by the BVH
// build, the query sort, octree compaction, the flood-fill extraction and
// the DMC edge sort.
#pragma once

#include "a3d_common.cuh"

namespace a3d {

// ---------------------------------------------------------------------------
// warp / block scans
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T warp_inclusive_scan(T v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T n = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += n;
  }
  return v;
}

template <typename T>
__device__ __forceinline__ T warp_reduce_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide exclusive scan for blockDim.x <= 1024 (multiple of 32).
// s_warp must hold kBlockScanSlots elements: one exclusive offset per warp
// and, in its own slot, the block total (with 32 warps the last warp's
// offset and the total would otherwise share a slot).  Returns the
// exclusive prefix; *total = block sum.
constexpr int kBlockScanSlots = 33;
template <typename T>
__device__ __forceinline__ T block_exclusive_scan(T v, T* s_warp, T* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  T inc = warp_inclusive_scan(v);
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    T w = lane < nwarps ? s_warp[lane] : T(0);
    T wi = warp_inclusive_scan(w);
    if (lane < nwarps) s_warp[lane] = wi - w;
    if (lane == nwarps - 1) s_warp[32] = wi;
  }
  __syncthreads();
  T res = inc - v + s_warp[warp];
  if (total) *total = s_warp[32];
  __syncthreads();
  return res;
}

// ---------------------------------------------------------------------------
// device-wide exclusive scan: reduce tiles -> scan tile sums -> scan tiles
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

template <typename TIn, typename T>
__global__ void scan_tile_reduce_kernel(const TIn* __restrict__ in, int64_t n, T* __restrict__ tile_sums) {
  pdl_wait();
  __shared__ T s_warp[kBlockScanSlots];
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  T acc = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    int64_t idx = base + (int64_t)i * kScanThreads + threadIdx.x;
    if (idx < n) acc += (T)in[idx];
  }
  T total;
  block_exclusive_scan<T>(acc, s_warp, &total);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// Single block: exclusive scan of tile sums in place, total -> *total.
template <typename T>
__global__ void scan_tile_sums_kernel(T* __restrict__ sums, int64_t nb, T* __restrict__ total) {
  pdl_wait();
  __shared__ T s_warp[kBlockScanSlots];
  const int64_t per = ceil_div(nb, (int64_t)blockDim.x);
  const int64_t lo = (int64_t)threadIdx.x * per;
  const int64_t hi = lo + per < nb ? lo + per : nb;
  T local = 0;
  for (int64_t i = lo; i < hi; ++i) local += sums[i];
  T tot;
  T run = block_exclusive_scan<T>(local, s_warp, &tot);
  for (int64_t i = lo; i < hi; ++i) {
    T v = sums[i];
    sums[i] = run;
    run += v;
  }
  if (threadIdx.x == 0 && total) *total = tot;
}

// The tile passes through shared memory: loaded and stored with consecutive
// threads on consecutive elements (coalesced), scanned with each thread
// owning kScanItems consecutive elements (one padding slot per 32 keeps the
// per-thread reads off a single bank).  out may alias in: a block reads its
// whole tile before writing it.
//
// kFused: tile_offsets holds the raw tile sums of scan_tile_reduce_kernel and
// each block adds up those before its own (at most kScanFuseTiles of them,
// read from L2), so the single-block scan of the tile sums is skipped; the
// last block writes the total.
__host__ __device__ constexpr int scan_pad(int i) { return i + (i >> 5); }
constexpr int64_t kScanFuseTiles = 2048;

template <typename TIn, typename T, bool kFused>
__global__ void scan_tile_down_kernel(const TIn* __restrict__ in, T* __restrict__ out, int64_t n,
                                      const T* __restrict__ tile_offsets, T* __restrict__ total) {
  pdl_wait();
  __shared__ T s_warp[kBlockScanSlots];
  __shared__ T s_tile[scan_pad(kScanTile)];
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  T offset;
  if constexpr (kFused) {
    T part = 0;
    for (int64_t b = threadIdx.x; b < (int64_t)blockIdx.x; b += kScanThreads) part += tile_offsets[b];
    block_exclusive_scan<T>(part, s_warp, &offset);
  } else {
    offset = tile_offsets[blockIdx.x];
  }
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    const int li = i * kScanThreads + threadIdx.x;
    const int64_t idx = base + li;
    s_tile[scan_pad(li)] = idx < n ? (T)in[idx] : T(0);
  }
  __syncthreads();
  // each thread owns kScanItems consecutive elements
  T vals[kScanItems];
  T acc = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    vals[i] = s_tile[scan_pad(threadIdx.x * kScanItems + i)];
    acc += vals[i];
  }
  T tile_total;
  T run = block_exclusive_scan<T>(acc, s_warp, &tile_total) + offset;
  if (kFused && total && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total = offset + tile_total;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    s_tile[scan_pad(threadIdx.x * kScanItems + i)] = run;
    run += vals[i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    const int li = i * kScanThreads + threadIdx.x;
    const int64_t idx = base + li;
    if (idx < n) out[idx] = s_tile[scan_pad(li)];
  }
}

inline size_t scan_workspace_elems(int64_t n) { return (size_t)ceil_div(n > 0 ? n : 1, kScanTile) + 1; }

// Exclusive scan of in[0..n) into out (may alias in).  tmp must hold
// scan_workspace_elems(n) elements of T; the total goes to total_dev on the
// device, or to tmp[num_tiles] when total_dev is null.  Up to
// kScanFuseTiles tiles (4M elements) the scan is two launches (tile sums,
// then the tiles with their offsets summed in each block), above it three
// (the tile sums scanned by one block in between).
template <typename TIn, typename T>
int device_exclusive_scan(const TIn* in, T* out, int64_t n, T* tmp, T* total_dev, cudaStream_t s) {
  if (n <= 0) {
    if (total_dev) A3D_CUDA_TRY(cudaMemsetAsync(total_dev, 0, sizeof(T), s));
    return A3D_OK;
  }
  const int64_t nb = ceil_div(n, kScanTile);
  // The down pass reads thread-contiguous items, the reduce pass strided
  // items: both cover the same tile so tile sums agree.
  // the passes back to back with programmatic dependent launch
  T* total = total_dev ? total_dev : tmp + nb;
  A3D_PDL(scan_tile_reduce_kernel<TIn, T>, dim3((unsigned)nb), dim3(kScanThreads), 0, s, in, n, tmp);
  if (nb <= kScanFuseTiles) {
    A3D_PDL((scan_tile_down_kernel<TIn, T, true>), dim3((unsigned)nb), dim3(kScanThreads), 0, s, in, out, n,
            (const T*)tmp, total);
  } else {
    A3D_PDL(scan_tile_sums_kernel<T>, dim3(1), dim3(1024), 0, s, tmp, nb, total);
    A3D_PDL((scan_tile_down_kernel<TIn, T, false>), dim3((unsigned)nb), dim3(kScanThreads), 0, s, in, out, n,
            (const T*)tmp, (T*)nullptr);
  }
  return A3D_OK;
}

// n copies of v at p, a grid-stride kernel launched with programmatic
// dependent launch (a memset between two kernels would break the chain)
template <typename T>
__global__ void fill_kernel(T* __restrict__ p, int64_t n, T v) {
  pdl_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = v;
}

template <typename T>
int fill_async(T* p, int64_t n, T v, cudaStream_t s) {
  if (n <= 0) return A3D_OK;
  const int64_t want = ceil_div(n, 256);
  const int64_t cap = (int64_t)num_sms() * 8;
  A3D_PDL(fill_kernel<T>, dim3((unsigned)(want < cap ? want : cap)), dim3(256), 0, s, p, n, v);
  return A3D_OK;
}

// ---------------------------------------------------------------------------
// stable LSD radix sort of (key, uint32 value) pairs, 8-bit digits
// ---------------------------------------------------------------------------
// Per digit an upsweep (the digit counts of each tile) and a downsweep.  The
// downsweep ranks a tile's keys warp by warp with ballots against counters
// of the warp's own, so it needs three block barriers a tile, then brings the
// tile into digit order in shared memory and writes it in runs of consecutive
// addresses.  (Ranking and scattering 256 keys at a time took 64 barriers a
// tile of 4,096 keys and one sector per key.)  Tiles are 4,096 keys, fewer
// while there would be less than two tiles an SM.
constexpr int kRsThreads = 256;
constexpr int kRsWarps = kRsThreads / 32;
constexpr int kRsMaxItems = 16;
// up to this many tiles a downsweep block adds up the tiles' counts itself
// (kRsFuseTiles x 1 KB from L2) instead of a scan launched in between
constexpr int64_t kRsFuseTiles = 128;

// the lanes whose 8-bit digit equals this lane's, by one ballot a bit (in a
// quarter of the time of match_any, whose rate falls with the distinct values)
__device__ __forceinline__ unsigned rs_peers(uint32_t d) {
  unsigned peers = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const unsigned ones = __ballot_sync(0xffffffffu, (d >> b) & 1u);
    peers &= (d >> b) & 1u ? ones : ~ones;
  }
  return peers;
}

// keys a thread of a sort of n keys: the fused form's tiles up to 131,072
// keys, above it two tiles an SM up to 16 (of 148: scratch sizes are asked for
// without a device)
inline int radix_items(int64_t n) {
  if (n <= kRsFuseTiles * 2 * kRsThreads) return 2;
  int items = kRsMaxItems;
  while (items > 4 && n < (int64_t)items * kRsThreads * 296) items >>= 1;
  return items;
}
inline int64_t radix_num_tiles(int64_t n) {
  return ceil_div(n > 0 ? n : 1, (int64_t)radix_items(n) * kRsThreads);
}
// uint32 elements of scratch needed by radix_sort_pairs, for n keys and for any
// smaller sort (just below a change of the keys a thread, fewer keys take more
// tiles), so that a workspace for n serves every smaller call
inline size_t radix_sort_scratch_elems(int64_t n) {
  int64_t tiles = radix_num_tiles(n);
  for (int items = 2; items < kRsMaxItems; items *= 2) {
    const int64_t below = items == 2 ? kRsFuseTiles * 2 * kRsThreads : (int64_t)items * kRsThreads * 296 - 1;
    const int64_t t = radix_num_tiles(below);
    if (n > below && tiles < t) tiles = t;
  }
  const int64_t h = 256 * tiles;
  return (size_t)h + scan_workspace_elems(h);
}

// hist: [digit][tile] for the scanned form, [tile][digit] for the fused one
template <typename K, int kItems, bool kFused>
__global__ void __launch_bounds__(kRsThreads)
    rs_upsweep_kernel(const K* __restrict__ keys, int64_t n, int shift, uint32_t* __restrict__ hist,
                      int64_t num_tiles) {
  pdl_wait();
  __shared__ uint32_t s_hist[256];
  s_hist[threadIdx.x] = 0;
  const int64_t base = (int64_t)blockIdx.x * (kItems * kRsThreads);
  const int lane = threadIdx.x & 31;
  uint32_t d[kItems];
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int64_t idx = base + (int64_t)i * kRsThreads + threadIdx.x;
    d[i] = idx < n ? (uint32_t)((keys[idx] >> shift) & 0xff) : 0x100u;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    // a warp of one digit (sorted or narrow keys) adds once
    const uint32_t d0 = __shfl_sync(0xffffffffu, d[i], 0);
    if (__all_sync(0xffffffffu, d[i] == d0)) {
      if (lane == 0 && d0 < 256u) atomicAdd(&s_hist[d0], 32u);
    } else if (d[i] < 256u) {
      atomicAdd(&s_hist[d[i]], 1u);
    }
  }
  __syncthreads();
  hist[kFused ? (int64_t)blockIdx.x * 256 + threadIdx.x : (int64_t)threadIdx.x * num_tiles + blockIdx.x] =
      s_hist[threadIdx.x];
}

template <typename K, int kItems>
struct RsSmem {
  uint32_t warp[kRsWarps][256];  // digit counts, then the warps' offsets in the digit
  uint32_t start[256];           // where a digit starts in the tile
  uint32_t out[256];             // where it goes, less that
  uint32_t scan[kBlockScanSlots];
  K buf[kItems * kRsThreads];    // the tile in digit order: keys, then values
};

// resident blocks an SM: more would spill the 16 keys a thread holds
template <typename K>
constexpr int kRsBlocks = sizeof(K) == 8 ? 3 : 4;

template <typename K, int kItems, bool kFused>
__global__ void __launch_bounds__(kRsThreads, kRsBlocks<K>)
    rs_downsweep_kernel(const K* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, K* __restrict__ keys_out,
                        uint32_t* __restrict__ vals_out, int64_t n, int shift, const uint32_t* __restrict__ hist,
                        int64_t num_tiles) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char rs_raw[];
  RsSmem<K, kItems>& S = *reinterpret_cast<RsSmem<K, kItems>*>(rs_raw);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll
  for (int w = 0; w < kRsWarps; ++w) S.warp[w][t] = 0;
  // a warp's keys are consecutive, 32 a step, so ranks follow the input order
  const int64_t base = (int64_t)blockIdx.x * (kItems * kRsThreads);
  const int64_t mine = base + (int64_t)warp * (kItems * 32) + lane;
  K key[kItems];
  uint32_t rank[kItems];
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int64_t idx = mine + i * 32;
    key[i] = idx < n ? keys_in[idx] : ~K(0);  // past the end: after every other key of digit 255
  }
  // this block's place in each digit's output
  uint32_t before = 0, total = 0;
  if constexpr (kFused) {
    for (int64_t j = 0; j < num_tiles; ++j) {
      const uint32_t c = hist[j * 256 + t];
      before += j < (int64_t)blockIdx.x ? c : 0u;
      total += c;
    }
  } else {
    before = hist[(int64_t)t * num_tiles + blockIdx.x];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const uint32_t d = (uint32_t)((key[i] >> shift) & 0xff);
    const unsigned peers = rs_peers(d);
    const uint32_t c = S.warp[warp][d];
    rank[i] = c + (uint32_t)__popc(peers & ((1u << lane) - 1u));
    __syncwarp();
    if (lane == __ffs(peers) - 1) S.warp[warp][d] = c + (uint32_t)__popc(peers);
    __syncwarp();
  }
  if constexpr (kFused) before += block_exclusive_scan<uint32_t>(total, S.scan, nullptr);
  __syncthreads();
  uint32_t run = 0;
#pragma unroll
  for (int w = 0; w < kRsWarps; ++w) {
    const uint32_t c = S.warp[w][t];
    S.warp[w][t] = run;
    run += c;
  }
  const uint32_t start = block_exclusive_scan<uint32_t>(run, S.scan, nullptr);
  S.start[t] = start;
  S.out[t] = before - start;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const uint32_t d = (uint32_t)((key[i] >> shift) & 0xff);
    rank[i] += S.start[d] + S.warp[warp][d];
    S.buf[rank[i]] = key[i];
  }
  __syncthreads();
  const int64_t left = n - base;
  const int count = left < kItems * kRsThreads ? (int)left : kItems * kRsThreads;
  uint32_t to[kItems];
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int at = i * kRsThreads + t;
    to[i] = 0;
    if (at < count) {
      const K k = S.buf[at];
      to[i] = S.out[(uint32_t)((k >> shift) & 0xff)] + (uint32_t)at;
      keys_out[to[i]] = k;
    }
  }
  __syncthreads();
  uint32_t* vbuf = reinterpret_cast<uint32_t*>(S.buf);
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int64_t idx = mine + i * 32;
    vbuf[rank[i]] = idx < n ? vals_in[idx] : 0u;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int at = i * kRsThreads + t;
    if (at < count) vals_out[to[i]] = vbuf[at];
  }
}

template <typename K, int kItems, bool kFused>
int radix_pass(const K* kin, const uint32_t* vin, K* kout, uint32_t* vout, int64_t n, int shift, uint32_t* hist,
               uint32_t* tmp, int64_t nt, cudaStream_t s) {
  constexpr size_t smem = sizeof(RsSmem<K, kItems>);
  static_assert(smem <= 48 * 1024, "above 48 KB the kernel needs an opt-in per device");
  A3D_PDL((rs_upsweep_kernel<K, kItems, kFused>), dim3((unsigned)nt), dim3(kRsThreads), 0, s, kin, n, shift, hist, nt);
  if (!kFused) A3D_TRY((device_exclusive_scan<uint32_t, uint32_t>(hist, hist, 256 * nt, tmp, (uint32_t*)nullptr, s)));
  A3D_PDL((rs_downsweep_kernel<K, kItems, kFused>), dim3((unsigned)nt), dim3(kRsThreads), smem, s, kin, vin, kout,
          vout, n, shift, (const uint32_t*)hist, nt);
  return A3D_OK;
}

// Sorts (keys, vals) by bits [begin_bit, end_bit) of the key.  Ping-pongs
// between (keys, vals) and (keys_alt, vals_alt); *result_in_alt tells the
// caller which pair holds the sorted data.  n must be < 2^32.
template <typename K>
int radix_sort_pairs(K* keys, uint32_t* vals, K* keys_alt, uint32_t* vals_alt, int64_t n, int begin_bit,
                     int end_bit, uint32_t* scratch, bool* result_in_alt, cudaStream_t s) {
  *result_in_alt = false;
  if (n <= 1) return A3D_OK;
  A3D_REQUIRE(n < (int64_t)0xffffffffll, A3D_ERR_ARGUMENT, "radix sort: too many elements");
  const int items = radix_items(n);
  const int64_t nt = radix_num_tiles(n);
  uint32_t* hist = scratch;
  uint32_t* tmp = scratch + 256 * nt;
  K *kin = keys, *kout = keys_alt;
  uint32_t *vin = vals, *vout = vals_alt;
  for (int shift = begin_bit; shift < end_bit; shift += 8) {
    switch (items) {
      case 16: A3D_TRY((radix_pass<K, 16, false>(kin, vin, kout, vout, n, shift, hist, tmp, nt, s))); break;
      case 8: A3D_TRY((radix_pass<K, 8, false>(kin, vin, kout, vout, n, shift, hist, tmp, nt, s))); break;
      case 4:
        A3D_TRY(nt <= kRsFuseTiles ? (radix_pass<K, 4, true>(kin, vin, kout, vout, n, shift, hist, tmp, nt, s))
                                   : (radix_pass<K, 4, false>(kin, vin, kout, vout, n, shift, hist, tmp, nt, s)));
        break;
      default: A3D_TRY((radix_pass<K, 2, true>(kin, vin, kout, vout, n, shift, hist, tmp, nt, s)));
    }
    K* tk = kin; kin = kout; kout = tk;
    uint32_t* tv = vin; vin = vout; vout = tv;
    *result_in_alt = !*result_in_alt;
  }
  return A3D_OK;
}

__global__ void iota_u32_kernel(uint32_t* out, int64_t n);

}  // namespace a3d
