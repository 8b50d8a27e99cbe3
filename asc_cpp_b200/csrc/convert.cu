// Device format conversions for sm_100a: CSR <-> CSC and coordinates ->
// CSR / CSC, and the transposed structure that deterministic transposed
// products run on.
//
// Each of them is one STABLE sort of entry positions by the entry's new outer
// index.  That is the order in which the reference's host conversions emit
// entries (CompressedSparseArray::FromCoordinate, compressed.h:1082-1131, and
// FromCompressed, :1151-1221, scan the source in stored order once per
// destination outer index), and the order in which the reference's standard
// transposed products accumulate (blas.h:1241-1256, outer then inner).
//
// The sort is a least-significant-digit radix sort over tiles of 4096 entries,
// ceil(bits(limit - 1) / 8) passes of equally wide digits (20 bits: 7 + 7 + 6;
// fewer bins than 8 + 8 + 4 give longer runs).  It is bound by memory traffic,
// so keys and positions travel as 32-bit words whenever the entry count and
// the key range allow (8 bytes per entry and direction; 64-bit words
// otherwise), and every tile is brought into digit order in shared memory
// before it is written, so that a pass stores runs of consecutive words.
// Per pass:
//   * count:   each tile histograms its digits in shared memory (the counts
//              do not depend on the order of the atomics);
//   * scan:    one block per digit scans that digit's counts over the tiles;
//   * scatter: each warp ranks its 256 entries 32 at a time, in stored order
//              (one ballot per digit bit finds the lanes of equal digit:
//              __match_any_sync measured 1.2 times slower in all); the
//              tile's warps are offset by a scan of their per-digit counts, so
//              equal digits keep their input order.
// The last pass writes the outputs themselves (permutation, new inner
// indices, values) in place of a key and a position.  The bucket offsets are
// read off the sorted keys: the first entry of each bucket writes its place,
// empty buckets search theirs.  Everything is integer work, so the results are
// exact by construction and independent of scheduling.
//
// Figures: at ascb_stable_sort.
#include "common.cuh"
#include "kernels.h"

namespace ascb {
namespace {

// (512 threads of 8 entries: a thread has its keys, indices and values all in
// flight at once in 64 registers, two blocks to an SM.  256 threads of 16, the
// values fetched after the ranking: 163 against 132 us for a middle pass over
// 16.9 M FP64 entries on a B200)
constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortPer = 8;                                  // entries per thread
constexpr int kSortTile = kSortThreads * kSortPer;           // 4096
constexpr int kWarpSpan = 32 * kSortPer;                     // 256 per warp
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;                      // digits are at most this wide
constexpr int kScanThreads = 1024;

std::size_t Round256(std::size_t v) { return (v + 255) / 256 * 256; }

template <typename U>
__device__ __forceinline__ int digit_of(U key, int shift, int mask) {
  return static_cast<int>(key >> shift) & mask;
}

// Exclusive scan of one value per thread over the block; *total receives the
// block's sum.  `sums` holds 32 entries of shared memory.
template <typename U>
__device__ __forceinline__ U block_exclusive(U v, U* sums, U* total) {
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  U inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const U t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) sums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const int nwarps = static_cast<int>(blockDim.x >> 5);
    U w = lane < nwarps ? sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const U t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += t;
    }
    sums[lane] = w;
  }
  __syncthreads();
  const U prefix = warp > 0 ? sums[warp - 1] : 0;
  *total = sums[31];
  __syncthreads();  // sums is reused by the caller's next round
  return prefix + inc - v;
}

// ---- radix passes ---------------------------------------------------------

// The keys of a pass: the caller's int64 array (first pass) or a key buffer.
template <typename U>
struct KeySource {
  const int64_t* first;  // not null: the first pass, entry e at first[e * stride]
  int64_t stride;
  const U* keys;
  __device__ __forceinline__ U at(int64_t e) const {
    return first != nullptr ? static_cast<U>(__ldg(first + e * stride)) : __ldg(keys + e);
  }
};

template <typename U>
__global__ void __launch_bounds__(kSortThreads)
radix_count(KeySource<U> src, int64_t n, int shift, int mask, U* __restrict__ table,
            int64_t tiles) {
  __shared__ int counts[kRadix];
  if (threadIdx.x < kRadix) counts[threadIdx.x] = 0;
  __syncthreads();
  const int64_t begin = static_cast<int64_t>(blockIdx.x) * kSortTile;
  U key[kSortPer];
#pragma unroll
  for (int j = 0; j < kSortPer; ++j) {
    const int64_t e = begin + j * kSortThreads + threadIdx.x;
    key[j] = e < n ? src.at(e) : 0;
  }
#pragma unroll
  for (int j = 0; j < kSortPer; ++j) {
    const int64_t e = begin + j * kSortThreads + threadIdx.x;
    if (e < n) atomicAdd(&counts[digit_of(key[j], shift, mask)], 1);
  }
  __syncthreads();
  const int d = threadIdx.x;
  if (d <= mask) table[d * tiles + blockIdx.x] = counts[d];
}

// Block d: exclusive scan of digit d's counts over the tiles, in place, and
// the digit's total.
template <typename U>
__global__ void __launch_bounds__(kScanThreads) radix_scan(U* __restrict__ table, int64_t tiles,
                                                           U* __restrict__ totals) {
  __shared__ U sums[32];
  constexpr int kPer = 4;
  U* row = table + static_cast<int64_t>(blockIdx.x) * tiles;
  U carry = 0;
  for (int64_t base = 0; base < tiles; base += kScanThreads * kPer) {
    const int64_t i = base + threadIdx.x * kPer;
    U v[kPer];
    U s = 0;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      v[u] = i + u < tiles ? row[i + u] : 0;
      s += v[u];
    }
    U total = 0;
    U run = carry + block_exclusive(s, sums, &total);
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      if (i + u < tiles) row[i + u] = run;
      run += v[u];
    }
    carry += total;
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

struct alignas(8) Bytes16 {
  uint64_t lo, hi;
};

// What travels with a key.  kPositions: the entry's position; the last pass
// writes it as the permutation and fetches the new inner index and the value
// through it.  kCarry: the new inner index and the value themselves, for
// callers that need no permutation: the random fetches at the end cost more
// than carrying 12 bytes through two more passes once values and indices
// outgrow L2 (16.9 M FP64 entries: 602 us for the fetching pass, DRAM 4.7 TB/s
// of 64-byte bursts for 12 bytes each).
enum class Payload { kPositions, kCarry };

template <typename U, typename V>
struct Side {
  // in (null pay in the first pass of kPositions: the entry's own position)
  const U* pay;
  const int64_t* other;  // first pass of kCarry without outer indices
  int64_t ostride;
  const V* val;
  // out of all but the last pass (kPositions has no values)
  U* pay_out;
  V* val_out;  // also out of the last pass, null: not written
  // out of the last pass
  int64_t* perm;     // null: not written
  int64_t* idx_out;  // null: not written
  const U* outer_of;  // kPositions: fetched through the position
};

template <typename U, typename V>
struct TileSmem {
  union {
    struct {
      U key[kSortTile];
      U pay[kSortTile];
    };
    V val[kSortTile];
  };
  unsigned short warp_count[kSortWarps][kRadix];  // at most 256 entries a warp
  unsigned short slot[kRadix];  // the digit's first slot in the tile
  U start[kRadix];  // output position of local slot 0 if it held digit d
  U sums[32];
};

// (Entries past the end of the last tile take the largest digit: they stand
// after every entry of the tile in any order and are not written.)
template <typename U, typename V, Payload P, bool FIRST, bool LAST>
__global__ void __launch_bounds__(kSortThreads, sizeof(U) == 4 ? 2 : 1)
radix_scatter(KeySource<U> src, Side<U, V> side, int64_t n, int shift, int digit_bits,
              const U* __restrict__ table, const U* __restrict__ totals, int64_t tiles,
              U* __restrict__ keys_out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TileSmem<U, V>& w = *reinterpret_cast<TileSmem<U, V>*>(smem_raw);
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int mask = (1 << digit_bits) - 1;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t tile0 = static_cast<int64_t>(blockIdx.x) * kSortTile;
  const int count = static_cast<int>(n - tile0 < kSortTile ? n - tile0 : kSortTile);
  const int d0 = threadIdx.x;  // this thread's digit
  const U digit_total = d0 <= mask ? __ldg(totals + d0) : U(0);
  const U digit_before = d0 <= mask ? __ldg(table + d0 * tiles + blockIdx.x) : U(0);
  const int own0 = warp * kWarpSpan + lane;  // entry j of the thread: own0 + 32 j
  U key[kSortPer];
#pragma unroll
  for (int j = 0; j < kSortPer; ++j) {
    const int i = own0 + j * 32;
    key[j] = ~U(0);
    if (i < count) {
      key[j] = FIRST ? static_cast<U>(__ldg(src.first + (tile0 + i) * src.stride))
                     : __ldg(src.keys + tile0 + i);
    }
  }
  // in flight while the keys are ranked (16-byte values: fetched afterwards,
  // for want of registers)
  constexpr bool kEarly = P == Payload::kCarry && sizeof(V) <= 8;
  U pay[kSortPer];
  V val[kEarly ? kSortPer : 1];
#pragma unroll
  for (int j = 0; j < kSortPer; ++j) {
    const int i = own0 + j * 32;
    pay[j] = 0;
    if (i >= count) continue;
    if constexpr (!FIRST) {
      pay[j] = __ldg(side.pay + tile0 + i);
    } else if constexpr (P == Payload::kPositions) {
      pay[j] = static_cast<U>(tile0 + i);
    } else {
      pay[j] = side.pay != nullptr
                   ? __ldg(side.pay + tile0 + i)
                   : static_cast<U>(__ldg(side.other + (tile0 + i) * side.ostride));
    }
  }
  if constexpr (kEarly) {
#pragma unroll
    for (int j = 0; j < kSortPer; ++j) {
      const int i = own0 + j * 32;
      val[j] = V{};
      if (i < count) val[j] = side.val[tile0 + i];
    }
  }
  for (int i = lane; i < kRadix / 2; i += 32) {
    reinterpret_cast<unsigned*>(w.warp_count[warp])[i] = 0u;
  }
  __syncwarp();
  unsigned short at[kSortPer];  // rank in the warp, then slot in the tile
#pragma unroll
  for (int j = 0; j < kSortPer; ++j) {
    const int d = digit_of(key[j], shift, mask);
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < kRadixBits; ++b) {  // bits past the digit are 0 in all lanes
      const bool bit = (d >> b) & 1;
      const unsigned m = __ballot_sync(0xffffffffu, bit);
      peers &= bit ? m : ~m;
    }
    const int before = w.warp_count[warp][d];
    at[j] = static_cast<unsigned short>(before + __popc(peers & lt));
    __syncwarp();
    if ((peers & lt) == 0u) {
      w.warp_count[warp][d] = static_cast<unsigned short>(before + __popc(peers));
    }
    __syncwarp();
  }
  __syncthreads();
  // thread d: the digit's entries of earlier warps, its first slot in the
  // tile (scan over digits) and in the output (scan of the digit totals)
  U in_tile = 0;
  if (d0 < kRadix) {
#pragma unroll
    for (int q = 0; q < kSortWarps; ++q) {
      const unsigned short c = w.warp_count[q][d0];
      w.warp_count[q][d0] = static_cast<unsigned short>(in_tile);
      in_tile += c;
    }
  }
  U all = 0;
  const U slot = block_exclusive(in_tile, w.sums, &all);
  const U out0 = block_exclusive(digit_total, w.sums, &all);
  if (d0 < kRadix) {
    w.slot[d0] = static_cast<unsigned short>(slot);
    w.start[d0] = out0 + digit_before - slot;
  }
  __syncthreads();
  // the tile in digit order, so that neighbouring threads write neighbouring
  // words: keys and indices first, then the values through the same memory
#pragma unroll
  for (int j = 0; j < kSortPer; ++j) {
    const int d = digit_of(key[j], shift, mask);
    at[j] = static_cast<unsigned short>(at[j] + w.warp_count[warp][d] + w.slot[d]);
    w.key[at[j]] = key[j];
    w.pay[at[j]] = pay[j];
  }
  __syncthreads();
  U out[kSortPer];
#pragma unroll
  for (int j = 0; j < kSortPer; ++j) {
    const int i = j * kSortThreads + threadIdx.x;
    const U k = w.key[i];
    const U p = w.pay[i];
    out[j] = w.start[digit_of(k, shift, mask)] + static_cast<U>(i);
    if (i >= count) continue;
    keys_out[out[j]] = k;
    if constexpr (!LAST) {
      side.pay_out[out[j]] = p;
    } else if constexpr (P == Payload::kCarry) {
      side.idx_out[out[j]] = static_cast<int64_t>(p);
    } else {
      if (side.perm != nullptr) side.perm[out[j]] = static_cast<int64_t>(p);
      if (side.idx_out != nullptr) {
        side.idx_out[out[j]] = static_cast<int64_t>(__ldg(side.outer_of + p));
      }
      if (side.val_out != nullptr) side.val_out[out[j]] = side.val[p];
    }
  }
  if constexpr (P == Payload::kCarry) {
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSortPer; ++j) {
      const int i = own0 + j * 32;
      if constexpr (kEarly) {
        w.val[at[j]] = val[j];
      } else if (i < count) {
        w.val[at[j]] = side.val[tile0 + i];
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSortPer; ++j) {
      const int i = j * kSortThreads + threadIdx.x;
      if (i < count) side.val_out[out[j]] = w.val[i];
    }
  }
}

// offsets[k] = q for the first entry q of every key k that occurs.
template <typename U>
__global__ void bucket_starts(const U* __restrict__ keys, int64_t n, int64_t limit,
                              int64_t* __restrict__ offsets) {
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t q = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; q < n; q += step) {
    const U k = __ldg(keys + q);
    if ((q == 0 || __ldg(keys + q - 1) != k) && static_cast<uint64_t>(k) < static_cast<uint64_t>(limit)) {
      offsets[k] = q;
    }
  }
}

// The other offsets (marked -1): the first entry whose key is not below k.
template <typename U>
__global__ void bucket_gaps(const U* __restrict__ keys, int64_t n, int64_t limit,
                            int64_t* __restrict__ offsets) {
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; k <= limit;
       k += step) {
    if (offsets[k] >= 0) continue;
    int64_t lo = 0, hi = n;
    while (lo < hi) {
      const int64_t mid = lo + ((hi - lo) >> 1);
      if (static_cast<int64_t>(__ldg(keys + mid)) < k) {
        lo = mid + 1;
      } else {
        hi = mid;
      }
    }
    offsets[k] = lo;
  }
}

// out[q] = outer index of entry q.  Tile t takes the items [4096 t, 4096
// (t + 1)) of the merged sequence in which outer index r stands at r + ptr[r],
// before its entries: as many entries as index starts whatever the lengths.
// Each start is marked at its entry's place (the largest of several, as empty
// ones share a place); an entry takes the mark of the last marked place up to
// its own, found in a bitmap of the places.
// (One warp per outer index took 105 us for 1 M rows of 16 entries on a B200,
// against a few microseconds of traffic.)
template <typename O>
__global__ void __launch_bounds__(kSortThreads)
expand_outer(const int64_t* __restrict__ ptr, int64_t outer, int64_t nnz, O* __restrict__ out) {
  constexpr int kWords = kSortTile / 32;
  __shared__ int mark[kSortTile];
  __shared__ unsigned bits[kWords];  // places that are marked
  __shared__ int last[kWords];       // the last marked place before a word, or -1
  __shared__ int64_t bound[2];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int64_t d0 = static_cast<int64_t>(blockIdx.x) * kSortTile;
  const int64_t d1 = d0 + kSortTile < outer + nnz ? d0 + kSortTile : outer + nnz;
  if (warp < 2) {
    const int64_t r = warp_first_row_at(ptr, outer, 1, warp == 0 ? d0 : d1, lane);
    if (lane == 0) bound[warp] = r;
  }
#pragma unroll
  for (int j = 0; j < kSortPer / 4; ++j) {
    reinterpret_cast<int4*>(mark)[j * kSortThreads + threadIdx.x] = make_int4(0, 0, 0, 0);
  }
  if (threadIdx.x < kWords) bits[threadIdx.x] = 0u;
  __syncthreads();
  const int64_t r0 = bound[0], r1 = bound[1];
  const int64_t q0 = d0 - r0;
  const int count = static_cast<int>((d1 - r1) - q0);
  for (int64_t r = r0 + threadIdx.x; r < r1; r += kSortThreads) {
    const int64_t at = __ldg(ptr + r) - q0;
    if (at < count) {
      atomicMax(&mark[at], static_cast<int>(r - r0) + 1);
      atomicOr(&bits[at >> 5], 1u << (at & 31));
    }
  }
  __syncthreads();
  if (warp == 0) {
    int seen = -1;
#pragma unroll
    for (int j = 0; j < kWords / 32; ++j) {
      const unsigned b = bits[32 * j + lane];
      int top = b != 0u ? 32 * (32 * j + lane) + 31 - __clz(b) : -1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, top, o);
        if (lane >= o && u > top) top = u;
      }
      const int before = __shfl_up_sync(0xffffffffu, top, 1);
      last[32 * j + lane] = lane > 0 && before > seen ? before : seen;
      const int end = __shfl_sync(0xffffffffu, top, 31);
      if (end > seen) seen = end;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSortPer; ++j) {
    const int i = j * kSortThreads + threadIdx.x;
    if (i < count) {
      const unsigned upto = bits[i >> 5] & (0xffffffffu >> (31 - lane));
      const int place = upto != 0u ? (i & ~31) + 31 - __clz(upto) : last[i >> 5];
      out[q0 + i] = static_cast<O>(r0 - 1 + (place >= 0 ? mark[place] : 0));
    }
  }
}

template <typename V>
__global__ void permute_values(const int64_t* __restrict__ perm, int64_t n,
                               const V* __restrict__ val_in, V* __restrict__ val_out) {
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < n;
       j += step) {
    val_out[j] = val_in[__ldg(perm + j)];
  }
}

unsigned GridFor(int64_t n, int threads, int sm_count) {
  const int64_t cap = static_cast<int64_t>(sm_count > 0 ? sm_count : 148) * 8;
  int64_t blocks = (n + threads - 1) / threads;
  if (blocks > cap) blocks = cap;
  return static_cast<unsigned>(blocks < 1 ? 1 : blocks);
}

int KeyBits(int64_t limit) {
  int bits = 0;
  for (uint64_t v = limit > 1 ? static_cast<uint64_t>(limit - 1) : 0; v != 0; v >>= 1) ++bits;
  return bits < 1 ? 1 : bits;
}

// 32-bit keys, positions and outer indices hold every value (all ones stays
// unused, so that limit and n themselves fit too).
bool Fits32(int64_t n, int64_t limit, int64_t outer) {
  constexpr int64_t kMost = 0xfffffffell;
  return n <= kMost && limit <= kMost && outer <= kMost;
}

// Where values travel with the keys (kCarry) there is one value buffer: the
// passes go to it and to the output array in turn, the last one to the output.
struct SortLayout {
  std::size_t keys[2], pay[2], val, table, totals, total;
};

SortLayout Layout(int64_t n, std::size_t word, std::size_t carried) {
  SortLayout l{};
  const int64_t tiles = (n + kSortTile - 1) / kSortTile;
  const std::size_t count = static_cast<std::size_t>(n > 0 ? n : 1);
  std::size_t at = 0;
  for (std::size_t* part : {l.keys, l.pay}) {
    for (int i = 0; i < 2; ++i) {
      part[i] = at;
      at += Round256(count * word);
    }
  }
  l.val = at;
  at += Round256(count * carried);
  l.table = at;
  at += Round256(static_cast<std::size_t>(kRadix) * static_cast<std::size_t>(tiles > 0 ? tiles : 1) *
                 word);
  l.totals = at;
  at += Round256(kRadix * word);
  l.total = at;
  return l;
}

template <typename U, typename V, Payload P, bool FIRST, bool LAST>
cudaError_t Scatter(cudaStream_t stream, KeySource<U> src, const Side<U, V>& side, int64_t n,
                    int shift, int bits, const U* table, const U* totals, int64_t tiles,
                    U* keys_out) {
  auto kernel = radix_scatter<U, V, P, FIRST, LAST>;
  constexpr std::size_t kBytes = sizeof(TileSmem<U, V>);
  if (kBytes > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(
        kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kBytes));
    if (e != cudaSuccess) return e;
  }
  kernel<<<static_cast<unsigned>(tiles), kSortThreads, kBytes, stream>>>(
      src, side, n, shift, bits, table, totals, tiles, keys_out);
  return cudaGetLastError();
}

template <typename U, typename V, Payload P>
cudaError_t Sort(cudaStream_t stream, const int64_t* keys, int64_t kstride, int64_t n,
                 int64_t limit, int64_t* offsets, int64_t* perm, unsigned char* ws,
                 const ascb_sort_emit& out) {
  constexpr bool kCarry = P == Payload::kCarry;
  const SortLayout l = Layout(n, sizeof(U), kCarry ? sizeof(V) : 0);
  const int64_t tiles = (n + kSortTile - 1) / kSortTile;
  U* kbuf[2] = {reinterpret_cast<U*>(ws + l.keys[0]), reinterpret_cast<U*>(ws + l.keys[1])};
  U* pbuf[2] = {reinterpret_cast<U*>(ws + l.pay[0]), reinterpret_cast<U*>(ws + l.pay[1])};
  V* val_out = static_cast<V*>(out.val_out);
  U* table = reinterpret_cast<U*>(ws + l.table);
  U* totals = reinterpret_cast<U*>(ws + l.totals);
  U* outer_of = static_cast<U*>(out.outer_of);
  if (out.ptr != nullptr) {
    const int64_t blocks = (out.outer + n + kSortTile - 1) / kSortTile;
    expand_outer<U><<<static_cast<unsigned>(blocks), kSortThreads, 0, stream>>>(out.ptr, out.outer,
                                                                              n, outer_of);
  }
  const int bits = KeyBits(limit);
  const int passes = (bits + kRadixBits - 1) / kRadixBits;
  // value buffer of pass p: vbuf[p & 1], the output for the last
  V* vbuf[2] = {val_out, val_out};
  if (kCarry) vbuf[passes & 1] = reinterpret_cast<V*>(ws + l.val);
  int shift = 0;
  U* sorted = nullptr;
  for (int p = 0; p < passes; ++p) {
    // the remaining bits split evenly over the remaining passes
    const int width = (bits - shift + passes - p - 1) / (passes - p);
    const int mask = (1 << width) - 1;
    const int from = (p - 1) & 1;
    KeySource<U> src{p == 0 ? keys : nullptr, kstride, p == 0 ? nullptr : kbuf[from]};
    Side<U, V> side{};
    if (p > 0) {
      side.pay = pbuf[from];
      if (kCarry) side.val = vbuf[from];
    } else if (kCarry) {
      if (out.ptr != nullptr) {
        side.pay = outer_of;
      } else {
        side.other = out.other;
        side.ostride = out.ostride;
      }
      side.val = static_cast<const V*>(out.val_in);
    }
    side.pay_out = pbuf[p & 1];
    side.val_out = vbuf[p & 1];
    if (p + 1 == passes) {
      side.perm = perm;
      side.idx_out = out.idx_out;
      side.outer_of = outer_of;
      if (!kCarry) side.val = static_cast<const V*>(out.val_in);
    }
    sorted = kbuf[p & 1];
    radix_count<U><<<static_cast<unsigned>(tiles), kSortThreads, 0, stream>>>(src, n, shift, mask,
                                                                             table, tiles);
    radix_scan<U><<<static_cast<unsigned>(mask + 1), kScanThreads, 0, stream>>>(table, tiles,
                                                                              totals);
    const bool last = p + 1 == passes;
    auto scatter = p == 0 ? (last ? Scatter<U, V, P, true, true> : Scatter<U, V, P, true, false>)
                          : (last ? Scatter<U, V, P, false, true> : Scatter<U, V, P, false, false>);
    const cudaError_t e =
        scatter(stream, src, side, n, shift, width, table, totals, tiles, sorted);
    if (e != cudaSuccess) return e;
    shift += width;
  }
  cudaError_t e =
      cudaMemsetAsync(offsets, 0xff, static_cast<std::size_t>(limit + 1) * 8, stream);  // -1
  if (e != cudaSuccess) return e;
  bucket_starts<U><<<GridFor(n, 256, 148), 256, 0, stream>>>(sorted, n, limit, offsets);
  bucket_gaps<U><<<GridFor(limit + 1, 256, 148), 256, 0, stream>>>(sorted, n, limit, offsets);
  return cudaGetLastError();
}

template <typename U>
cudaError_t SortAny(cudaStream_t stream, const int64_t* keys, int64_t kstride, int64_t n,
                    int64_t limit, int64_t* offsets, int64_t* perm, unsigned char* ws,
                    const ascb_sort_emit& out) {
  constexpr Payload kPos = Payload::kPositions, kCarry = Payload::kCarry;
  if (out.val_out == nullptr) {
    return Sort<U, uint32_t, kPos>(stream, keys, kstride, n, limit, offsets, perm, ws, out);
  }
  const bool carry = perm == nullptr;
  switch (out.elem_bytes) {
    case 4:
      return carry ? Sort<U, uint32_t, kCarry>(stream, keys, kstride, n, limit, offsets, perm, ws,
                                               out)
                   : Sort<U, uint32_t, kPos>(stream, keys, kstride, n, limit, offsets, perm, ws,
                                             out);
    case 8:
      return carry ? Sort<U, uint64_t, kCarry>(stream, keys, kstride, n, limit, offsets, perm, ws,
                                               out)
                   : Sort<U, uint64_t, kPos>(stream, keys, kstride, n, limit, offsets, perm, ws,
                                             out);
    case 16:
      return carry ? Sort<U, Bytes16, kCarry>(stream, keys, kstride, n, limit, offsets, perm, ws,
                                              out)
                   : Sort<U, Bytes16, kPos>(stream, keys, kstride, n, limit, offsets, perm, ws,
                                            out);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace
}  // namespace ascb

extern "C" size_t ascb_sort_workspace_bytes(int64_t n, int64_t limit, int64_t other_limit,
                                            int elem_bytes) {
  return ascb::Layout(n, ascb::Fits32(n, limit, other_limit) ? 4 : 8,
                      static_cast<std::size_t>(elem_bytes))
      .total;
}

// Measured on a B200, FP64 values: CSR -> CSC of 16.9 M entries and 1,048,576
// columns 575 us (2260 us with 64-bit words stored entry by entry, a histogram
// of the whole key by global atomics and a separate permutation); a
// transposed product that builds its structure of 8.4 M entries first, 381 us
// (1120).  Of the 575: scatters 144 + 133 + 132, counts 65, scans 19,
// expansion 33, offsets 36.
extern "C" int ascb_stable_sort(void* stream_ptr, const int64_t* keys, int64_t kstride, int64_t n,
                                int64_t limit, int64_t* offsets, int64_t* perm, void* workspace,
                                const ascb_sort_emit* emit) {
  using namespace ascb;
  auto stream = static_cast<cudaStream_t>(stream_ptr);
  if (n <= 0) {
    return static_cast<int>(
        cudaMemsetAsync(offsets, 0, static_cast<std::size_t>(limit + 1) * 8, stream));
  }
  const ascb_sort_emit out = emit != nullptr ? *emit : ascb_sort_emit{};
  auto* ws = static_cast<unsigned char*>(workspace);
  return static_cast<int>(
      Fits32(n, limit, out.other_limit)
          ? SortAny<uint32_t>(stream, keys, kstride, n, limit, offsets, perm, ws, out)
          : SortAny<uint64_t>(stream, keys, kstride, n, limit, offsets, perm, ws, out));
}

extern "C" int ascb_outer_of_entries(void* stream, const int64_t* ptr, int64_t outer, int64_t nnz,
                                     int64_t* out) {
  using namespace ascb;
  if (outer <= 0 || nnz <= 0) return 0;
  const int64_t blocks = (outer + nnz + kSortTile - 1) / kSortTile;
  expand_outer<int64_t><<<static_cast<unsigned>(blocks), kSortThreads, 0,
                          static_cast<cudaStream_t>(stream)>>>(ptr, outer, nnz, out);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int ascb_permute_values(void* stream_ptr, const int64_t* perm, int64_t n,
                                   const void* val_in, void* val_out, int elem_bytes,
                                   int sm_count) {
  using namespace ascb;
  if (n <= 0) return 0;
  auto stream = static_cast<cudaStream_t>(stream_ptr);
  const unsigned blocks = GridFor(n, 256, sm_count);
  switch (elem_bytes) {
    case 4:
      permute_values<uint32_t><<<blocks, 256, 0, stream>>>(
          perm, n, static_cast<const uint32_t*>(val_in), static_cast<uint32_t*>(val_out));
      break;
    case 8:
      permute_values<uint64_t><<<blocks, 256, 0, stream>>>(
          perm, n, static_cast<const uint64_t*>(val_in), static_cast<uint64_t*>(val_out));
      break;
    case 16:
      permute_values<Bytes16><<<blocks, 256, 0, stream>>>(
          perm, n, static_cast<const Bytes16*>(val_in), static_cast<Bytes16*>(val_out));
      break;
    default:
      return static_cast<int>(cudaErrorInvalidValue);
  }
  return static_cast<int>(cudaGetLastError());
}
