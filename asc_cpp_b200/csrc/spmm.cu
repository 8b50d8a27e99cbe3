// CSR x dense (SpMM) and the scatter (transpose) products, sm_100a.
//
// Row-major right-hand sides take the row kernel: G lanes share an output row and
// own whole chunks of 16, 8 or 4 bytes of it (the widest that the columns and
// strides allow), so a stored entry (o, c, v) costs one broadcast load of
// (c, v) and one vector load per lane and chunk of the row B(c, :).  EXACT
// adds the terms in stored order,
//     C(o, j) = C(o, j) + (alpha * v) * B(c, j),
// every product and sum rounded separately -- the per-entry update of
// asc::Spmm (include/asc/sparse/blas.h:1736-1748), bit for bit; FAST sums with
// FMA and applies alpha once.
//
// Rows far longer than the mean would each be one group's serial chain of
// loads while the chip idles (a power-law matrix of 262,144 rows and 4.2 M
// entries, FP32, B200: k = 50 950 us that way, 269 us with the rule below;
// k = 8 968 and 68, k = 32 bit-exact 2240 and 211).
// They are set aside and then taken by all groups of a warp or of their block
// together: FAST splits the entries and adds the groups' sums in a fixed order,
// EXACT (the block) forms the products in parallel and adds them in stored order
// from shared memory.
//
// Column-major right-hand sides: a lane per row, several columns at a time
// (spmm_columns_kernel), with the same rule for long rows.  One thread per
// output element, which this replaces, read every index and value once per
// column: 27-point stencil on 80^3, FP64, k = 5 540 us against 137 (B200; DRAM
// floor 43), k = 40 FP32 3560 against 529; power law, 100,000 rows, k = 5 1088
// against 165.  Packing the columns into rows first measured within 10% on the
// stencil and two to four times faster on the power law, but its scratch costs
// 18 us per MB to allocate and cannot be used under stream capture.
// Transposed products that have no transposed structure at hand scatter with
// atomics (BACKEND_DEFAULT only; order-dependent rounding within the bound).
#include "common.cuh"
#include "kernels.h"

namespace ascb {
namespace {

constexpr int kThreads = 256;
constexpr int kEntryUnroll = 4;

// N elements that are loaded at once: 16, 8 or 4 bytes.
template <typename T, int N>
struct Chunk;
template <typename T>
struct Chunk<T, 1> {
  using type = T;
  __device__ static void split(T v, T (&e)[1]) { e[0] = v; }
  __device__ static T join(const T (&e)[1]) { return e[0]; }
};
template <>
struct Chunk<float, 2> {
  using type = float2;
  __device__ static void split(const float2& v, float (&e)[2]) {
    e[0] = v.x; e[1] = v.y;
  }
  __device__ static float2 join(const float (&e)[2]) { return make_float2(e[0], e[1]); }
};
template <>
struct Chunk<float, 4> {
  using type = float4;
  __device__ static void split(const float4& v, float (&e)[4]) {
    e[0] = v.x; e[1] = v.y; e[2] = v.z; e[3] = v.w;
  }
  __device__ static float4 join(const float (&e)[4]) { return make_float4(e[0], e[1], e[2], e[3]); }
};
template <>
struct Chunk<double, 2> {
  using type = double2;
  __device__ static void split(const double2& v, double (&e)[2]) {
    e[0] = v.x; e[1] = v.y;
  }
  __device__ static double2 join(const double (&e)[2]) { return make_double2(e[0], e[1]); }
};

// One product C += alpha * A * B.
template <typename T>
struct RowArgs {
  int64_t rows;
  int64_t k;       // columns of C
  int64_t chunks;  // chunks of a row of B
  const int64_t* ptr;
  const int64_t* idx;
  const T* val;
  const T* b;
  int64_t ldb;    // B(c, j) = b[c * ldb + j], or b[c + j * ldb] (COLUMNS)
  T* c;
  int64_t c_row, c_col;  // C(o, j) = c[o * c_row + j * c_col]
  T alpha;
  int64_t long_row;  // rows with more entries are set aside
};

constexpr int kLongRows = 64;  // rows a block can list
// Entries per group up to which one warp takes a listed row, contracted form of up
// to 4 lanes a row: 8 rows go side by side without a barrier, a longer one keeps
// its warp too long.
// 1M-row power law, FP32, k = 1 / 16, us: 16 entries 144 / 400, 32 141 / 379, 64
// 143 / 376, 256 152 / 409.
constexpr int kWarpShare = 32;

// Shared memory comes out of L1, which serves B to neighbouring rows (10 KB a
// block cost the 27-point stencil 9% at k = 128), so long rows get little of
// it.  Entries per group and round of a long row, EXACT: a round of products
// fits 4 KB where it can.
template <typename T, int N, int G, int J>
__host__ __device__ constexpr int round_entries() {
  return 4096 / (kThreads * J * N * static_cast<int>(sizeof(T))) > 0
             ? 4096 / (kThreads * J * N * static_cast<int>(sizeof(T)))
             : 1;
}
// Shared memory for a long row: a round of products, or one sum per column.
template <typename T, int N, int G, int J, bool EXACT>
__host__ __device__ constexpr int long_bytes() {
  return EXACT ? kThreads * J * N * static_cast<int>(sizeof(T)) * round_entries<T, N, G, J>()
               : G * J * N * static_cast<int>(sizeof(T));
}

// Chunk t of B's row `col`; bl: the lane's first chunk of row 0.
template <int N, int G, bool COLUMNS, typename T>
__device__ __forceinline__ const T* chunk_at(const RowArgs<T>& a, const T* bl, int64_t col, int t) {
  return COLUMNS ? bl + col + t * G * a.ldb : bl + col * a.ldb + t * G * N;
}

// Entries [q, qe) of a row into acc (J chunks of N columns per lane).
template <typename T, int N, int G, int J, bool EXACT, bool COLUMNS = false>
__device__ __forceinline__ void add_entries(T (&acc)[J][N], const bool (&live)[J], int64_t q,
                                            int64_t qe, const RowArgs<T>& a, const T* bl) {
  using C = Chunk<T, N>;
  using V = typename C::type;
  for (; q + kEntryUnroll <= qe; q += kEntryUnroll) {
    int64_t col[kEntryUnroll];
    T av[kEntryUnroll];
#pragma unroll
    for (int u = 0; u < kEntryUnroll; ++u) {
      col[u] = __ldg(a.idx + q + u);
      av[u] = EXACT ? mul_rn(a.alpha, __ldg(a.val + q + u)) : __ldg(a.val + q + u);
    }
    V bv[kEntryUnroll][J];
#pragma unroll
    for (int u = 0; u < kEntryUnroll; ++u) {
#pragma unroll
      for (int t = 0; t < J; ++t) {
        bv[u][t] = live[t] ? __ldg(reinterpret_cast<const V*>(chunk_at<N, G, COLUMNS>(a, bl, col[u], t)))
                           : V{};
      }
    }
#pragma unroll
    for (int u = 0; u < kEntryUnroll; ++u) {
#pragma unroll
      for (int t = 0; t < J; ++t) {
        T e[N];
        C::split(bv[u][t], e);
#pragma unroll
        for (int i = 0; i < N; ++i) {
          acc[t][i] = EXACT ? add_rn(acc[t][i], mul_rn(av[u], e[i])) : fma(av[u], e[i], acc[t][i]);
        }
      }
    }
  }
  for (; q < qe; ++q) {
    const int64_t cq = __ldg(a.idx + q);
    const T av = EXACT ? mul_rn(a.alpha, __ldg(a.val + q)) : __ldg(a.val + q);
#pragma unroll
    for (int t = 0; t < J; ++t) {
      if (!live[t]) continue;
      T e[N];
      C::split(__ldg(reinterpret_cast<const V*>(chunk_at<N, G, COLUMNS>(a, bl, cq, t))), e);
#pragma unroll
      for (int i = 0; i < N; ++i) {
        acc[t][i] = EXACT ? add_rn(acc[t][i], mul_rn(av, e[i])) : fma(av, e[i], acc[t][i]);
      }
    }
  }
}

// WHOLE: a chunk of C is one aligned vector; otherwise element by element.
template <typename T, int N, bool WHOLE>
__device__ __forceinline__ void load_c(const RowArgs<T>& a, int64_t o, int64_t jv, T (&e)[N]) {
  using C = Chunk<T, N>;
  if constexpr (WHOLE) {
    C::split(*reinterpret_cast<const typename C::type*>(a.c + o * a.c_row + jv * N), e);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int64_t j = jv * N + i;
      e[i] = j < a.k ? a.c[o * a.c_row + j * a.c_col] : T(0);
    }
  }
}
template <typename T, int N, bool WHOLE>
__device__ __forceinline__ void store_c(const RowArgs<T>& a, int64_t o, int64_t jv,
                                        const T (&e)[N]) {
  using C = Chunk<T, N>;
  if constexpr (WHOLE) {
    *reinterpret_cast<typename C::type*>(a.c + o * a.c_row + jv * N) = C::join(e);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int64_t j = jv * N + i;
      if (j < a.k) a.c[o * a.c_row + j * a.c_col] = e[i];
    }
  }
}

// A row set aside, contracted: every group of the block (or warp) sums a share
// of the entries, shuffles join the groups of a warp, and the warps add to one
// sum in shared memory in turn.
template <typename T, int N, int G, int J, bool WHOLE, bool COLUMNS = false, bool BLOCK = true>
__device__ __forceinline__ void long_row_fast(const RowArgs<T>& a, int64_t o, int64_t pb,
                                              int64_t pe, T* smem) {
  constexpr int kGroups = (BLOCK ? kThreads : 32) / G;
  const int lane = threadIdx.x % G;
  const int group = threadIdx.x / G % kGroups;
  const int64_t share = (pe - pb + kGroups - 1) / kGroups;
  const int64_t q0 = pb + group * share < pe ? pb + group * share : pe;
  const int64_t q1 = q0 + share < pe ? q0 + share : pe;
  for (int64_t v0 = 0; v0 < a.chunks; v0 += int64_t{G} * J) {
    T acc[J][N];
    bool live[J];
#pragma unroll
    for (int t = 0; t < J; ++t) {
      live[t] = v0 + t * G + lane < a.chunks;
#pragma unroll
      for (int e = 0; e < N; ++e) acc[t][e] = T(0);
    }
    add_entries<T, N, G, J, false, COLUMNS>(acc, live, q0, q1, a,
                                            a.b + (v0 + lane) * (COLUMNS ? a.ldb : N));
#pragma unroll
    for (int t = 0; t < J; ++t) {
#pragma unroll
      for (int e = 0; e < N; ++e) {
#pragma unroll
        for (int m = G; m < 32; m <<= 1) acc[t][e] += shfl_xor(acc[t][e], m);
      }
    }
    if constexpr (!BLOCK) {
      if (threadIdx.x % 32 < G) {
#pragma unroll
        for (int t = 0; t < J; ++t) {
          if (!live[t]) continue;
          T old[N];
          load_c<T, N, WHOLE>(a, o, v0 + t * G + lane, old);
#pragma unroll
          for (int e = 0; e < N; ++e) acc[t][e] = fma(a.alpha, acc[t][e], old[e]);
          store_c<T, N, WHOLE>(a, o, v0 + t * G + lane, acc[t]);
        }
      }
      continue;
    }
    for (int w = 0; w < kThreads / 32; ++w) {
      if (static_cast<int>(threadIdx.x) / 32 == w && threadIdx.x % 32 < G) {
#pragma unroll
        for (int t = 0; t < J; ++t) {
#pragma unroll
          for (int e = 0; e < N; ++e) {
            T& sum = smem[(t * G + lane) * N + e];
            sum = w == 0 ? acc[t][e] : sum + acc[t][e];
          }
        }
      }
      __syncthreads();
    }
    if (threadIdx.x < G) {
#pragma unroll
      for (int t = 0; t < J; ++t) {
        if (!live[t]) continue;
        T sum[N], old[N];
        load_c<T, N, WHOLE>(a, o, v0 + t * G + lane, old);
#pragma unroll
        for (int e = 0; e < N; ++e) {
          sum[e] = fma(a.alpha, smem[(t * G + lane) * N + e], old[e]);
        }
        store_c<T, N, WHOLE>(a, o, v0 + t * G + lane, sum);
      }
    }
    __syncthreads();
  }
}

// The same in stored order: the groups form a round of products, one thread
// per column adds them while the next round's operands are on their way.
template <typename T, int N, int G, int J, bool COLUMNS = false>
__device__ __forceinline__ void long_row_exact(const RowArgs<T>& a, int64_t o, int64_t pb,
                                               int64_t pe, T* smem) {
  using C = Chunk<T, N>;
  using V = typename C::type;
  constexpr int kGroups = kThreads / G;
  constexpr int kWidth = G * J * N;  // columns of a pass
  constexpr int kPer = round_entries<T, N, G, J>();
  static_assert(kWidth <= kThreads, "a thread per column");
  constexpr int kRound = kGroups * kPer;  // entries
  const int lane = threadIdx.x % G;
  const int group = threadIdx.x / G;
  for (int64_t v0 = 0; v0 < a.chunks; v0 += int64_t{G} * J) {
    const T* bl = a.b + (v0 + lane) * (COLUMNS ? a.ldb : N);
    const int64_t j = v0 * N + threadIdx.x;  // this thread's column in the sums
    const bool mine = static_cast<int>(threadIdx.x) < kWidth && j < a.k;
    T sum = mine ? a.c[o * a.c_row + j * a.c_col] : T(0);
    V bv[kPer][J];
    T av[kPer];
    auto fetch = [&](int64_t base) {
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        const int64_t q = base + group * kPer + u;
        const bool ok = q < pe;
        av[u] = ok ? mul_rn(a.alpha, __ldg(a.val + q)) : T(0);
        const int64_t col = ok ? __ldg(a.idx + q) : 0;
#pragma unroll
        for (int t = 0; t < J; ++t) {
          bv[u][t] = ok && v0 + t * G + lane < a.chunks
                         ? __ldg(reinterpret_cast<const V*>(chunk_at<N, G, COLUMNS>(a, bl, col, t)))
                         : V{};
        }
      }
    };
    fetch(pb);
    for (int64_t base = pb; base < pe; base += kRound) {
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
#pragma unroll
        for (int t = 0; t < J; ++t) {
          T e[N];
          C::split(bv[u][t], e);
#pragma unroll
          for (int i = 0; i < N; ++i) e[i] = mul_rn(av[u], e[i]);
          *reinterpret_cast<V*>(smem + (group * kPer + u) * kWidth + (t * G + lane) * N) =
              C::join(e);
        }
      }
      __syncthreads();
      if (base + kRound < pe) fetch(base + kRound);
      if (mine) {
        const int n = static_cast<int>(pe - base < kRound ? pe - base : kRound);
#pragma unroll 8
        for (int e = 0; e < n; ++e) sum = add_rn(sum, smem[e * kWidth + threadIdx.x]);
      }
      __syncthreads();
    }
    if (mine) a.c[o * a.c_row + j * a.c_col] = sum;
  }
}

// CTAs per SM: at 5 the contracted narrow forms spill (27-point 64^3, FP64, k = 2
// 55 us, 36 at 4; 100,000 random rows of 64 entries want the warps: FP32, k = 8
// 79 us, 95 at 4).
template <typename T, int N, int G, int J, bool EXACT, bool WHOLE>
__global__ void __launch_bounds__(kThreads, J * N * sizeof(T) > 16 || J == 4 || !EXACT ? 4 : 5)
spmm_rows_kernel(RowArgs<T> a) {
  constexpr int kGroups = kThreads / G;
  __shared__ __align__(16) unsigned char buffer[long_bytes<T, N, G, J, EXACT>()];
  __shared__ int long_rows[kLongRows];  // (round, group) they came up in
  __shared__ int long_count;
  const int lane = threadIdx.x % G;
  const int64_t first = static_cast<int64_t>(blockIdx.x) * kGroups + threadIdx.x / G;
  const int64_t step = static_cast<int64_t>(gridDim.x) * kGroups;
  if (threadIdx.x == 0) long_count = 0;
  __syncthreads();
  for (int64_t o = first; o < a.rows; o += step) {
    const int64_t pb = __ldg(a.ptr + o);
    const int64_t pe = __ldg(a.ptr + o + 1);
    if (pb == pe) continue;  // C keeps its bits
    if (pe - pb > a.long_row) {
      int at = 0;
      if (lane == 0) at = atomicAdd(&long_count, 1);
      if constexpr (G > 1) {
        const unsigned group = (G == 32 ? 0xffffffffu : ((1u << (G % 32)) - 1u))
                               << (threadIdx.x % 32 / G * G);
        at = __shfl_sync(group, at, 0, G);
      }
      if (lane == 0 && at < kLongRows) {
        long_rows[at] = static_cast<int>((o - first) / step * kGroups + threadIdx.x / G);
      }
      // (stored order gives the same bits whoever adds)
      if (!EXACT || at < kLongRows) continue;
    }
    for (int64_t v0 = 0; v0 < a.chunks; v0 += int64_t{G} * J) {
      // C is read first where that costs few registers: one wait less at the end
      constexpr bool kEarlyC = !EXACT && J * N * sizeof(T) <= 16;
      T acc[J][N], old[J][N];
      bool live[J];
#pragma unroll
      for (int t = 0; t < J; ++t) {
        live[t] = v0 + t * G + lane < a.chunks;
        if (EXACT && live[t]) {
          load_c<T, N, WHOLE>(a, o, v0 + t * G + lane, acc[t]);
        } else {
#pragma unroll
          for (int e = 0; e < N; ++e) acc[t][e] = T(0);
        }
        if (kEarlyC && live[t]) load_c<T, N, WHOLE>(a, o, v0 + t * G + lane, old[t]);
      }
      add_entries<T, N, G, J, EXACT>(acc, live, pb, pe, a, a.b + (v0 + lane) * N);
#pragma unroll
      for (int t = 0; t < J; ++t) {
        if (!live[t]) continue;
        if (!EXACT) {
          if (!kEarlyC) load_c<T, N, WHOLE>(a, o, v0 + t * G + lane, old[t]);
#pragma unroll
          for (int i = 0; i < N; ++i) acc[t][i] = fma(a.alpha, acc[t][i], old[t][i]);
        }
        store_c<T, N, WHOLE>(a, o, v0 + t * G + lane, acc[t]);
      }
    }
  }
  __syncthreads();
  auto row_at = [&](int place) {
    return static_cast<int64_t>(blockIdx.x) * kGroups + place % kGroups + place / kGroups * step;
  };
  if constexpr (EXACT) {
    const int count = long_count < kLongRows ? long_count : kLongRows;
    for (int i = 0; i < count; ++i) {
      const int64_t o = row_at(long_rows[i]);
      long_row_exact<T, N, G, J>(a, o, __ldg(a.ptr + o), __ldg(a.ptr + o + 1),
                                 reinterpret_cast<T*>(buffer));
    }
    return;
  }
  // Contracted: who takes a row follows from its length and from how many there
  // are, never from the order in which they were listed, so that it is added up
  // the same way on every run.
  int count = long_count;
  if (count == 0) return;
  const bool listed = count <= kLongRows;
  const int places = listed ? count : static_cast<int>((a.rows + step - 1) / step) * kGroups;
  // rows of a range of places with more than `least` entries into the list
  auto list_again = [&](int begin, int end, int64_t least) {
    __syncthreads();
    if (threadIdx.x == 0) long_count = 0;
    __syncthreads();
    for (int i = begin + static_cast<int>(threadIdx.x); i < end; i += kThreads) {
      const int64_t o = row_at(i);
      if (o < a.rows && __ldg(a.ptr + o + 1) - __ldg(a.ptr + o) > least) {
        const int at = atomicAdd(&long_count, 1);
        if (at < kLongRows) long_rows[at] = i;
      }
    }
    __syncthreads();
    count = long_count;
  };
  if constexpr (G <= 4) {
    // rows of up to `most` entries to a warp each, the others to the whole block;
    // where there are too many of those for the list, `most` grows until they fit
    int64_t most = kWarpShare * (32 / G);
    while (!listed) {
      list_again(0, places, max(most, a.long_row));
      if (count <= kLongRows) break;
      most *= 4;
    }
    for (int i = threadIdx.x / 32; i < places; i += kThreads) {
      auto row_of = [&](int lane_of) {
        const int j = i + lane_of * (kThreads / 32);
        return j < places ? row_at(listed ? long_rows[j] : j) : a.rows;
      };
      unsigned mine;
      {
        const int64_t o = row_of(threadIdx.x % 32);
        const int64_t n = o < a.rows ? __ldg(a.ptr + o + 1) - __ldg(a.ptr + o) : 0;
        mine = __ballot_sync(0xffffffffu, n > a.long_row && n <= most);
      }
      for (; mine != 0u; mine &= mine - 1u) {
        const int64_t o = row_of(__ffs(mine) - 1);
        long_row_fast<T, N, G, J, WHOLE, false, false>(a, o, __ldg(a.ptr + o),
                                                       __ldg(a.ptr + o + 1), nullptr);
      }
    }
    for (int i = 0; i < count; ++i) {
      const int64_t o = row_at(long_rows[i]);
      const int64_t pb = __ldg(a.ptr + o);
      const int64_t pe = __ldg(a.ptr + o + 1);
      if (pe - pb > most) {
        long_row_fast<T, N, G, J, WHOLE>(a, o, pb, pe, reinterpret_cast<T*>(buffer));
      }
    }
  } else {
    // all to the whole block, as many places at a time as the list holds
    for (int begin = 0; begin < places; begin += kLongRows) {
      if (!listed) list_again(begin, min(begin + kLongRows, places), a.long_row);
      for (int i = 0; i < count; ++i) {
        const int64_t o = row_at(long_rows[i]);
        long_row_fast<T, N, G, J, WHOLE>(a, o, __ldg(a.ptr + o), __ldg(a.ptr + o + 1),
                                         reinterpret_cast<T*>(buffer));
      }
    }
  }
}

// Column-major right-hand sides: a lane owns a row and KC columns of it, so an
// entry's index and value are read once for KC columns and neighbouring rows,
// whose columns are mostly neighbours too, read neighbouring elements of B.
// Entries come four at a time in 32-byte loads from the aligned position at or
// before the row's first (VEC: both arrays on 32-byte boundaries); a lane has
// 4 KC elements of B in flight.  Rows above the limit are set aside for the
// whole block, lanes over columns.
template <typename T, int KC, bool EXACT, bool VEC>
__global__ void __launch_bounds__(kThreads) spmm_columns_kernel(RowArgs<T> a, int64_t nnz) {
  __shared__ __align__(16) unsigned char buffer[long_bytes<T, 1, 8, 1, EXACT>()];
  __shared__ int long_rows[kThreads];
  __shared__ int long_count;
  for (int64_t o0 = static_cast<int64_t>(blockIdx.x) * kThreads; o0 < a.rows;
       o0 += static_cast<int64_t>(gridDim.x) * kThreads) {
    const int64_t o = o0 + threadIdx.x;
    const int64_t pb = o < a.rows ? __ldg(a.ptr + o) : 0;
    const int64_t pe = o < a.rows ? __ldg(a.ptr + o + 1) : 0;
    if (threadIdx.x == 0) long_count = 0;
    __syncthreads();
    const bool set_aside = pe - pb > a.long_row;
    if (set_aside) long_rows[atomicAdd(&long_count, 1)] = static_cast<int>(threadIdx.x);
    int count = -1;  // known once every lane has been here
    for (int64_t j0 = int64_t{KC} * blockIdx.y; j0 < a.k; j0 += int64_t{KC} * gridDim.y) {
      RowArgs<T> part = a;  // this pass's columns
      part.k = a.k - j0 < KC ? a.k - j0 : KC;
      part.chunks = part.k;
      part.b = a.b + j0 * a.ldb;
      part.c = a.c + j0 * a.c_col;
      if (pb < pe && !set_aside) {
        T acc[KC];
        T* cp = part.c + o * a.c_row;
#pragma unroll
        for (int u = 0; u < KC; ++u) acc[u] = EXACT && u < part.k ? cp[u * a.c_col] : T(0);
        for (int64_t q = VEC ? pb & ~int64_t{3} : pb; q < pe; q += 4) {
          int64_t col[4];
          T av[4];
          if (VEC && q + 4 <= nnz) {
            ld_stream32(a.idx + q, col);
            if constexpr (sizeof(T) == 8) {
              ld_stream32(a.val + q, av);
            } else {
              const float4 v = __ldcs(reinterpret_cast<const float4*>(a.val + q));
              av[0] = v.x, av[1] = v.y, av[2] = v.z, av[3] = v.w;
            }
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const bool ok = q + e >= pb && q + e < pe;
              col[e] = ok ? __ldg(a.idx + q + e) : 0;
              av[e] = ok ? __ldg(a.val + q + e) : T(0);
            }
          }
          T bv[4][KC];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const bool ok = q + e >= pb && q + e < pe;
#pragma unroll
            for (int u = 0; u < KC; ++u) {
              bv[e][u] = ok && u < part.k ? __ldg(part.b + col[e] + u * a.ldb) : T(0);
            }
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (q + e < pb || q + e >= pe) continue;
            if (EXACT) av[e] = mul_rn(a.alpha, av[e]);
#pragma unroll
            for (int u = 0; u < KC; ++u) {
              acc[u] = EXACT ? add_rn(acc[u], mul_rn(av[e], bv[e][u])) : fma(av[e], bv[e][u], acc[u]);
            }
          }
        }
#pragma unroll
        for (int u = 0; u < KC; ++u) {
          if (u < part.k) cp[u * a.c_col] = EXACT ? acc[u] : fma(a.alpha, acc[u], cp[u * a.c_col]);
        }
      }
      if (count < 0) {
        __syncthreads();
        count = long_count;
      }
      for (int i = 0; i < count; ++i) {
        const int64_t r = o0 + long_rows[i];
        const int64_t rb = __ldg(a.ptr + r);
        const int64_t re = __ldg(a.ptr + r + 1);
        if constexpr (EXACT) {
          long_row_exact<T, 1, 8, 1, true>(part, r, rb, re, reinterpret_cast<T*>(buffer));
        } else {
          long_row_fast<T, 1, 8, 1, false, true>(part, r, rb, re, reinterpret_cast<T*>(buffer));
        }
      }
    }
    __syncthreads();  // the list is rewritten for the next rows
  }
}

__device__ __forceinline__ int64_t dense_at(int layout, int64_t ld, int64_t r,
                                            int64_t col) {
  return layout == ASCB_ROW_MAJOR ? r * ld + col : col * ld + r;
}

// Transposed product by scatter: C(c, j) += alpha * v * B(r, j) for every
// stored (r, c, v); one thread per (entry, column).
template <typename T>
__global__ void __launch_bounds__(kThreads)
spmm_scatter_kernel(int64_t rows, int64_t k, const int64_t* __restrict__ ptr,
                    const int64_t* __restrict__ idx, const T* __restrict__ val,
                    const T* __restrict__ b, int b_layout, int64_t ldb,
                    T* __restrict__ c, int c_layout, int64_t ldc, T alpha) {
  // one warp per source row, lanes over (entry, column) pairs
  const int lane = threadIdx.x & 31;
  const int64_t first = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t step = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t r = first; r < rows; r += step) {
    const int64_t pb = __ldg(ptr + r);
    const int64_t n = (__ldg(ptr + r + 1) - pb) * k;
    for (int64_t t = lane; t < n; t += 32) {
      const int64_t q = pb + t / k;
      const int64_t j = t % k;
      const T term = alpha * __ldg(val + q) * ld_gather(b + dense_at(b_layout, ldb, r, j));
      atomicAdd(c + dense_at(c_layout, ldc, __ldg(idx + q), j), term);
    }
  }
}

unsigned grid_for(int64_t work, int per_block, int sm_count) {
  const int64_t needed = (work + per_block - 1) / per_block;
  const int64_t resident = static_cast<int64_t>(sm_count > 0 ? sm_count : 148) * 8;
  return static_cast<unsigned>(needed < resident ? (needed > 0 ? needed : 1) : resident);
}

// Rows with more entries than this are taken by a whole block: eight times the
// mean, and at least 128 (shorter ones cost less than the block's barriers).
int64_t long_row_limit(const ascb_csr* a) {
  const int64_t mean = a->nnz / (a->rows > 0 ? a->rows : 1);
  return 8 * mean > 128 ? 8 * mean : 128;
}

template <typename T, int N, int G, int J>
int launch_rows(cudaStream_t s, bool exact, bool whole, const RowArgs<T>& a, int sm) {
  // Two wide chunks a lane run with the 4 CTAs per SM that are resident: more
  // consecutive rows share an L1 at a time.  Against 8 per SM (k = 128, FP32,
  // exact): 27-point 96^3 713 / 748 us, 5-point 700^2 167 / 173; a power law,
  // whose uneven rows want the smaller shares, 846 / 766.
  const unsigned grid = grid_for(a.rows, kThreads / G, J * N * sizeof(T) > 16 ? (sm + 1) / 2 : sm);
  if (exact) {
    if (whole) {
      spmm_rows_kernel<T, N, G, J, true, true><<<grid, kThreads, 0, s>>>(a);
    } else {
      spmm_rows_kernel<T, N, G, J, true, false><<<grid, kThreads, 0, s>>>(a);
    }
  } else if (whole) {
    spmm_rows_kernel<T, N, G, J, false, true><<<grid, kThreads, 0, s>>>(a);
  } else {
    spmm_rows_kernel<T, N, G, J, false, false><<<grid, kThreads, 0, s>>>(a);
  }
  return static_cast<int>(cudaGetLastError());
}

// Lanes and chunks per lane, measured on B200 with the 27-point stencil and
// the 16 x 16 block-sparse matrices: a row's chunks are spread over G lanes, J
// chunks per lane.  Up to two chunks per row take one lane each (more rows
// per warp); wider rows take two chunks per lane (more independent loads in
// flight, and a CTA covers more consecutive rows whose right-hand-side rows
// then hit in L1).  Single elements: up to four per lane, so that k = 128
// reads a row's entries once.  More than 32 chunks of 16 bytes take a warp per
// row where rows average 12 or more entries (`wide`), half a warp in passes
// where they are shorter: power law (16 a row), k = 200, FP32 exact 1156
// against 1513 us, contracted 781 / 961; 27-point 64^3, k = 128, FP64 396 / 467
// and 413 / 453; 5-point 500^2, k = 100, FP64 158 / 147 and 203 / 168.  Single
// elements for the exact form at 32 or more chunks, as was, took 3476 us on the
// 16 x 16 blocks (k = 128, FP32; 2141) and 1104 on the power law (k = 64, FP64;
// 794).
//
// Few long rows (`few`: 32 or more entries on average, and four lanes a row make no
// more CTAs than are resident) spread over four lanes whatever the width, even if
// some stay idle: an SM more is worth more than a lane, a second wave is not.
// FP32, k = 1 / 3, us, one and two lanes / four: 2,000 rows of 64 entries 20.6 / 10.3 and
// 14.4 / 10.3, 37,800 rows 22.7 / 24.7 and 26.8 / 24.9; 8,192 rows of 160 47 / 19 and
// 29 / 21, 24,576 rows of 496 128 / 101 and 132 / 104; in a second wave 49,152 rows of 976
// bit-exact 451 / 457 and 351 / 469.  A power law of 5,000 rows, 16 entries on average,
// 12.4 / 18.5.
template <typename T, int N>
int launch_by_width(cudaStream_t s, bool exact, bool whole, bool wide, bool few,
                    const RowArgs<T>& a, int sm) {
#define ASCB_ROWS(G, J) return launch_rows<T, N, G, J>(s, exact, whole, a, sm)
  if (few && a.chunks <= 4) ASCB_ROWS(4, 1);
  if (a.chunks <= 1) ASCB_ROWS(1, 1);
  if (a.chunks <= 2) ASCB_ROWS(2, 1);
  if (a.chunks <= 4) ASCB_ROWS(2, 2);
  if (a.chunks <= 8) ASCB_ROWS(4, 2);
  if (a.chunks <= 16) ASCB_ROWS(8, 2);
  if (a.chunks > 32 && (N * sizeof(T) < 16 || wide)) {
    if constexpr (N == 1) {
      if (a.chunks > 64) ASCB_ROWS(32, 4);
    }
    ASCB_ROWS(32, 2);
  }
  ASCB_ROWS(16, 2);
#undef ASCB_ROWS
}

// Row-major B.
template <typename T>
int spmm_rows(cudaStream_t s, bool exact, const ascb_csr* m, int64_t k, const void* b,
              int64_t ldb, void* c, int c_layout, int64_t ldc, T alpha, int sm) {
  constexpr int kMost = 16 / sizeof(T);
  RowArgs<T> a{m->rows, k, 0, m->ptr, m->idx, static_cast<const T*>(m->val),
               static_cast<const T*>(b), ldb, static_cast<T*>(c), 1, 1, alpha, long_row_limit(m)};
  (c_layout == ASCB_ROW_MAJOR ? a.c_row : a.c_col) = ldc;
  auto divides = [k](int64_t n, int64_t ld, const void* p) {
    return k % n == 0 && ld % n == 0 &&
           (reinterpret_cast<uintptr_t>(p) & (static_cast<uintptr_t>(n) * sizeof(T) - 1)) == 0;
  };
  int n = kMost;
  while (n > 1 && !divides(n, ldb, b)) n /= 2;
  const bool whole = c_layout == ASCB_ROW_MAJOR && divides(n, ldc, c);
  const bool wide = m->nnz >= 12 * m->rows;
  const int64_t wave = (sm > 0 ? sm : 148) * (exact ? 5 : 4) * int64_t{kThreads / 4};  // rows
  const bool few = m->nnz >= 32 * m->rows && m->rows <= wave;
  a.chunks = k / n;
  if (n == 4) {
    if constexpr (sizeof(T) == 4) return launch_by_width<T, 4>(s, exact, whole, wide, few, a, sm);
  }
  if (n == 2) return launch_by_width<T, 2>(s, exact, whole, wide, few, a, sm);
  return launch_by_width<T, 1>(s, exact, whole, wide, few, a, sm);
}

// Rows past four times the mean and 32 go to the whole block: a warp takes as
// long as its longest row.
int64_t long_column_limit(const ascb_csr* a) {
  const int64_t mean = a->nnz / (a->rows > 0 ? a->rows : 1);
  return 4 * mean > 32 ? 4 * mean : 32;
}

template <typename T, int KC>
int launch_columns(cudaStream_t s, bool exact, const RowArgs<T>& a, int64_t nnz, int sm) {
  // short rows straddle two or three aligned fours: single loads serve them better
  const bool vec =
      nnz >= 12 * a.rows &&
      ((reinterpret_cast<uintptr_t>(a.idx) | reinterpret_cast<uintptr_t>(a.val)) & 31u) == 0;
  // few rows: the passes over the columns spread over the grid too
  const unsigned blocks = grid_for(a.rows, kThreads, sm);
  const int64_t passes = (a.k + KC - 1) / KC;
  const int64_t room = static_cast<int64_t>(sm > 0 ? sm : 148) * 16 / blocks;
  const dim3 grid(blocks, static_cast<unsigned>(room < 1 ? 1 : (room < passes ? room : passes)));
  auto kernel = exact ? (vec ? spmm_columns_kernel<T, KC, true, true>
                             : spmm_columns_kernel<T, KC, true, false>)
                      : (vec ? spmm_columns_kernel<T, KC, false, true>
                             : spmm_columns_kernel<T, KC, false, false>);
  kernel<<<grid, kThreads, 0, s>>>(a, nnz);
  return static_cast<int>(cudaGetLastError());
}

template <typename T>
int spmm_columns(cudaStream_t s, bool exact, const ascb_csr* m, int64_t k, const void* b,
                 int64_t ldb, void* c, int c_layout, int64_t ldc, T alpha, int sm) {
  RowArgs<T> a{m->rows, k, k, m->ptr, m->idx, static_cast<const T*>(m->val),
               static_cast<const T*>(b), ldb, static_cast<T*>(c), 1, 1, alpha,
               long_column_limit(m)};
  (c_layout == ASCB_ROW_MAJOR ? a.c_row : a.c_col) = ldc;
  // passes of about equal width, at most 4 columns: 8 a lane (120 registers)
  // measured 10-20% slower, a block fewer warps having to hide the gathers
  const int64_t passes = (k + 3) / 4;
  const int64_t width = (k + passes - 1) / passes;
  if (width <= 1) return launch_columns<T, 1>(s, exact, a, m->nnz, sm);
  if (width <= 2) return launch_columns<T, 2>(s, exact, a, m->nnz, sm);
  return launch_columns<T, 4>(s, exact, a, m->nnz, sm);
}

template <typename T>
int spmm_typed(cudaStream_t s, int transpose, int exact, const ascb_csr* a, int64_t k,
               const void* b, int b_layout, int64_t ldb, void* c, int c_layout,
               int64_t ldc, double alpha_d, int sm) {
  const T alpha = static_cast<T>(alpha_d);
  if (transpose) {
    spmm_scatter_kernel<T><<<grid_for(a->rows, kThreads / 32, sm), kThreads, 0, s>>>(
        a->rows, k, a->ptr, a->idx, static_cast<const T*>(a->val),
        static_cast<const T*>(b), b_layout, ldb, static_cast<T*>(c), c_layout,
        ldc, alpha);
    return static_cast<int>(cudaGetLastError());
  }
  if (b_layout == ASCB_ROW_MAJOR) {
    return spmm_rows<T>(s, exact != 0, a, k, b, ldb, c, c_layout, ldc, alpha, sm);
  }
  return spmm_columns<T>(s, exact != 0, a, k, b, ldb, c, c_layout, ldc, alpha, sm);
}

template <typename T, int LANES>
__global__ void __launch_bounds__(kThreads)
spmv_scatter_kernel(int64_t rows, const int64_t* __restrict__ ptr,
                    const int64_t* __restrict__ idx, const T* __restrict__ val,
                    const T* __restrict__ x, int64_t incx, T* __restrict__ y,
                    int64_t incy, T alpha) {
  constexpr int kGroups = kThreads / LANES;
  const int lane = threadIdx.x % LANES;
  const int64_t first = static_cast<int64_t>(blockIdx.x) * kGroups + threadIdx.x / LANES;
  const int64_t step = static_cast<int64_t>(gridDim.x) * kGroups;
  for (int64_t r = first; r < rows; r += step) {
    const T ax = alpha * ld_gather(x + r * incx);
    for (int64_t q = __ldg(ptr + r) + lane; q < __ldg(ptr + r + 1); q += LANES) {
      atomicAdd(y + ld_stream(idx + q) * incy, ld_stream(val + q) * ax);
    }
  }
}

}  // namespace
}  // namespace ascb

extern "C" {

int ascb_spmm(void* stream, int dtype, int transpose, int exact, const ascb_csr* a,
              int64_t k, const void* b, int b_layout, int64_t ldb, void* c,
              int c_layout, int64_t ldc, double alpha, int sm_count) {
  if (a->rows <= 0 || k <= 0) return 0;
  auto s = static_cast<cudaStream_t>(stream);
  return dtype == ASCB_F64
             ? ascb::spmm_typed<double>(s, transpose, exact, a, k, b, b_layout, ldb, c,
                                        c_layout, ldc, alpha, sm_count)
             : ascb::spmm_typed<float>(s, transpose, exact, a, k, b, b_layout, ldb, c,
                                       c_layout, ldc, alpha, sm_count);
}

int ascb_spmv_scatter(void* stream, int dtype, const ascb_csr* a, double alpha,
                      const ascb_vec* x, const ascb_vec* y, int sm_count) {
  if (a->rows <= 0 || a->nnz == 0) return 0;
  auto s = static_cast<cudaStream_t>(stream);
  const unsigned blocks = ascb::grid_for(a->rows, ascb::kThreads / 8, sm_count);
  if (dtype == ASCB_F64) {
    ascb::spmv_scatter_kernel<double, 8><<<blocks, ascb::kThreads, 0, s>>>(
        a->rows, a->ptr, a->idx, static_cast<const double*>(a->val),
        static_cast<const double*>(x->data), x->stride,
        static_cast<double*>(y->data), y->stride, alpha);
  } else {
    ascb::spmv_scatter_kernel<float, 8><<<blocks, ascb::kThreads, 0, s>>>(
        a->rows, a->ptr, a->idx, static_cast<const float*>(a->val),
        static_cast<const float*>(x->data), x->stride,
        static_cast<float*>(y->data), y->stride, static_cast<float>(alpha));
  }
  return static_cast<int>(cudaGetLastError());
}

}  // extern "C"
