// Complex (C and Z) standard SpMV and SpMM for sm_100a.
//
// Every stored entry does out += (alpha * v') * in, v' = conj(v) for the
// conjugate transpose (include/asc/sparse/blas.h:1653-1665 and 1739-1748,
// MaybeConjugate).  Arrays hold (re, im) pairs, the layout of std::complex<R>,
// aligned to R only; where the arrays happen to start on whole elements a pair is
// one load.  A complex product
// (a, b)(c, d) is (ac - bd, ad + bc); in EXACT mode every product, difference
// and sum is rounded separately (the value std::complex<R> gives under GCC
// without -march for every product that is not NaN + NaN i).
//   * row products: the CSR arrays handed in are the rows of op(A) (for a
//     transposed product, the transposed structure of a plan).  A warp takes up
//     to 32 consecutive rows, whose entries lie one behind the other: all lanes
//     form 128 products at a time in shared memory while the next 128 entries
//     are on their way, and each row's lane adds its own in stored order (EXACT
//     to y, FAST to a sum that y gets once, lanes to spare sharing a row and
//     rounds inside one row by warp trees).  With a warp per row and the products
//     handed to one sum by shuffles, rows of 27 entries left lanes idle and
//     cost 4 x 27 dependent steps: 27-point stencil on 63^3, Z, bit-exact, B200:
//     167 us, now 44 (DRAM floor 26).
//   * scatter: FAST transposed products without a plan, one warp per stored
//     row, atomic adds of both components.
//   * SpMM: one thread per (row, right-hand side) in stored order, or the
//     scatter form for FAST transposed products without a plan.
#include "common.cuh"
#include "kernels.h"
#include "round_part.h"

namespace ascb {
namespace {

constexpr int kThreads = 256;

template <typename R>
struct Cx {
  R re, im;
};

template <bool EXACT, typename R>
__device__ __forceinline__ Cx<R> cmul(Cx<R> a, Cx<R> b) {
  if (EXACT) {
    return {sub_rn(mul_rn(a.re, b.re), mul_rn(a.im, b.im)),
            add_rn(mul_rn(a.re, b.im), mul_rn(a.im, b.re))};
  }
  return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}

template <bool EXACT, typename R>
__device__ __forceinline__ Cx<R> cadd(Cx<R> a, Cx<R> b) {
  if (EXACT) return {add_rn(a.re, b.re), add_rn(a.im, b.im)};
  return {a.re + b.re, a.im + b.im};
}

template <typename R>
__device__ __forceinline__ Cx<R> load(const Cx<R>* p) {
  return {__ldg(&p->re), __ldg(&p->im)};
}

template <bool CONJ, typename R>
__device__ __forceinline__ Cx<R> stored(const Cx<R>* val, int64_t q) {
  Cx<R> v = load(val + q);
  if (CONJ) v.im = -v.im;
  return v;
}

// A whole element at a time (PAIR: on whole-element boundaries).
template <bool PAIR>
__device__ __forceinline__ Cx<double> fetch(const Cx<double>* p) {
  if (!PAIR) return load(p);
  const double2 v = __ldg(reinterpret_cast<const double2*>(p));
  return {v.x, v.y};
}
template <bool PAIR>
__device__ __forceinline__ Cx<float> fetch(const Cx<float>* p) {
  if (!PAIR) return load(p);
  const float2 v = __ldg(reinterpret_cast<const float2*>(p));
  return {v.x, v.y};
}

constexpr int kPer = 4;             // products per lane and round
constexpr int kRound = 32 * kPer;   // 128

template <typename R, bool EXACT, bool CONJ, bool UNIT, bool PAIR>
__global__ void __launch_bounds__(kThreads)
complex_rows(const int64_t* __restrict__ ptr, const int64_t* __restrict__ idx,
             const Cx<R>* __restrict__ val, const Cx<R>* __restrict__ x, int64_t incx,
             Cx<R>* __restrict__ y, int64_t incy, Cx<R> alpha, int64_t rows, int per_warp,
             int log_share) {
  __shared__ Cx<R> staged[kThreads / 32][kRound];
  Cx<R>* prod = staged[threadIdx.x / 32];
  const int lane = threadIdx.x & 31;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (kThreads / 32);
  for (int64_t r0 = (static_cast<int64_t>(blockIdx.x) * (kThreads / 32) + threadIdx.x / 32) *
                    per_warp;
       r0 < rows; r0 += warps * per_warp) {
    const int64_t last = r0 + per_warp < rows ? r0 + per_warp : rows;
    const int share = EXACT ? 1 : 1 << log_share;  // lanes of a row
    const int64_t r = r0 + (EXACT ? lane : lane >> log_share);
    const bool mine = r < last;
    const int64_t end = __ldg(ptr + last);
    const int64_t b = mine ? __ldg(ptr + r) : end;
    const int64_t e = mine ? __ldg(ptr + r + 1) : end;
    const int64_t begin = __shfl_sync(0xffffffffu, b, 0);
    Cx<R> s{R(0), R(0)};
    if (EXACT && b < e) s = at<UNIT>(y, r, incy);
    int64_t col[kPer];
    Cx<R> v[kPer];
    auto entries = [&](int64_t w) {
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        const int64_t q = w + u * 32 + lane;
        if (q < end) {
          col[u] = __ldg(idx + q);
          v[u] = fetch<PAIR>(val + q);
          if (CONJ) v[u].im = -v[u].im;
        }
      }
    };
    Cx<R> wide{R(0), R(0)};  // FAST: this lane's share of a long row, and that row's lane
    int owner = -1;
    auto join = [&]() {
      if (owner < 0) return;
#pragma unroll
      for (int m = 16; m > 0; m >>= 1) {
        wide.re += __shfl_xor_sync(0xffffffffu, wide.re, m);
        wide.im += __shfl_xor_sync(0xffffffffu, wide.im, m);
      }
      if (lane == owner) s = cadd<false>(s, wide);
      wide = {R(0), R(0)};
      owner = -1;
    };
    entries(begin);
    for (int64_t w = begin; w < end; w += kRound) {
      Cx<R> xv[kPer];
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        if (w + u * 32 + lane < end) xv[u] = fetch<PAIR>(&at<UNIT>(x, col[u], incx));
      }
      if constexpr (!EXACT) {
        // a round wholly inside one row: every lane keeps its own sum
        const unsigned whole = __ballot_sync(0xffffffffu, b <= w && e - w >= kRound);
        if (whole != 0u) {
          if (owner >= 0 && owner != __ffs(whole) - 1) join();
#pragma unroll
          for (int u = 0; u < kPer; ++u) {
            wide = cadd<false>(wide, cmul<false>(cmul<false>(alpha, v[u]), xv[u]));
          }
          owner = __ffs(whole) - 1;
          if (w + kRound < end) entries(w + kRound);
          continue;
        }
        join();
      }
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        if (w + u * 32 + lane < end) {
          prod[u * 32 + lane] = cmul<EXACT>(cmul<EXACT>(alpha, v[u]), xv[u]);
        }
      }
      if (w + kRound < end) entries(w + kRound);
      __syncwarp();
      const RoundPart part = round_part(b, e, w, kRound);
      // (loads 16 at a time ahead of the chain of sums; 4 at a time, power law of 262,144
      // rows, bit-exact, C / Z: 87 / 139 us against 77 / 105)
#pragma unroll 16
      for (int q = part.from + (lane & (share - 1)); q < part.to; q += share) {
        s = cadd<EXACT>(s, prod[q]);
      }
      __syncwarp();  // the products are replaced
    }
    if constexpr (!EXACT) {
      join();
      for (int m = share >> 1; m > 0; m >>= 1) {
        s.re += __shfl_xor_sync(0xffffffffu, s.re, m);
        s.im += __shfl_xor_sync(0xffffffffu, s.im, m);
      }
    }
    if (b < e && (lane & (share - 1)) == 0) {  // (without entries y keeps its bits)
      Cx<R>* yp = &at<UNIT>(y, r, incy);
      *yp = EXACT ? s : cadd<false>(*yp, s);
    }
  }
}

template <typename R, bool CONJ, bool UNIT>
__global__ void __launch_bounds__(kThreads)
complex_scatter(const int64_t* __restrict__ ptr, const int64_t* __restrict__ idx,
                const Cx<R>* __restrict__ val, const Cx<R>* __restrict__ x, int64_t incx,
                Cx<R>* __restrict__ y, int64_t incy, Cx<R> alpha, int64_t rows) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (kThreads / 32);
  for (int64_t r = (static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x) >> 5; r < rows;
       r += warps) {
    const int64_t b = __ldg(ptr + r);
    const int64_t e = __ldg(ptr + r + 1);
    if (b == e) continue;
    const Cx<R> xr = load(&at<UNIT>(x, r, incx));
    for (int64_t q = b + lane; q < e; q += 32) {
      const Cx<R> p = cmul<false>(cmul<false>(alpha, stored<CONJ>(val, q)), xr);
      Cx<R>* yp = &at<UNIT>(y, __ldg(idx + q), incy);
      atomicAdd(&yp->re, p.re);
      atomicAdd(&yp->im, p.im);
    }
  }
}

__device__ __forceinline__ int64_t dense_at(int layout, int64_t ld, int64_t r, int64_t c) {
  return layout == ASCB_ROW_MAJOR ? r * ld + c : c * ld + r;
}

// One thread per (row of op(A), right-hand side j), j fastest.
template <typename R, bool EXACT, bool CONJ>
__global__ void __launch_bounds__(kThreads)
complex_spmm_rows(const int64_t* __restrict__ ptr, const int64_t* __restrict__ idx,
                  const Cx<R>* __restrict__ val, const Cx<R>* __restrict__ bm, int b_layout,
                  int64_t ldb, Cx<R>* __restrict__ cm, int c_layout, int64_t ldc, int64_t k,
                  Cx<R> alpha, int64_t rows) {
  const int64_t total = rows * k;
  const int64_t step = static_cast<int64_t>(gridDim.x) * kThreads;
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x; t < total;
       t += step) {
    const int64_t r = t / k;
    const int64_t j = t - r * k;
    const int64_t b = __ldg(ptr + r);
    const int64_t e = __ldg(ptr + r + 1);
    if (b == e) continue;
    Cx<R>* cp = cm + dense_at(c_layout, ldc, r, j);
    Cx<R> s = EXACT ? *cp : Cx<R>{R(0), R(0)};
    for (int64_t q = b; q < e; ++q) {
      const Cx<R> bv = load(bm + dense_at(b_layout, ldb, __ldg(idx + q), j));
      s = cadd<EXACT>(s, cmul<EXACT>(cmul<EXACT>(alpha, stored<CONJ>(val, q)), bv));
    }
    *cp = EXACT ? s : cadd<false>(*cp, s);
  }
}

// Transposed SpMM by scatter: one thread per (stored row r, rhs j).
template <typename R, bool CONJ>
__global__ void __launch_bounds__(kThreads)
complex_spmm_scatter(const int64_t* __restrict__ ptr, const int64_t* __restrict__ idx,
                     const Cx<R>* __restrict__ val, const Cx<R>* __restrict__ bm, int b_layout,
                     int64_t ldb, Cx<R>* __restrict__ cm, int c_layout, int64_t ldc, int64_t k,
                     Cx<R> alpha, int64_t rows) {
  const int64_t total = rows * k;
  const int64_t step = static_cast<int64_t>(gridDim.x) * kThreads;
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x; t < total;
       t += step) {
    const int64_t r = t / k;
    const int64_t j = t - r * k;
    const Cx<R> bv = load(bm + dense_at(b_layout, ldb, r, j));
    for (int64_t q = __ldg(ptr + r); q < __ldg(ptr + r + 1); ++q) {
      const Cx<R> p = cmul<false>(cmul<false>(alpha, stored<CONJ>(val, q)), bv);
      Cx<R>* cp = cm + dense_at(c_layout, ldc, __ldg(idx + q), j);
      atomicAdd(&cp->re, p.re);
      atomicAdd(&cp->im, p.im);
    }
  }
}

unsigned Blocks(int64_t threads_needed, int sm_count) {
  const int64_t cap = static_cast<int64_t>(sm_count > 0 ? sm_count : 148) * 8;
  int64_t b = (threads_needed + kThreads - 1) / kThreads;
  if (b > cap) b = cap;
  return static_cast<unsigned>(b < 1 ? 1 : b);
}

template <typename R, bool CONJ, bool UNIT>
int spmv_typed(cudaStream_t s, int mode, const ascb_csr* a, Cx<R> alpha, const ascb_vec* x,
               const ascb_vec* y, int sm) {
  const auto* ptr = a->ptr;
  const auto* idx = a->idx;
  const auto* val = static_cast<const Cx<R>*>(a->val);
  const auto* xd = static_cast<const Cx<R>*>(x->data);
  auto* yd = static_cast<Cx<R>*>(y->data);
  if (mode == 2) {
    complex_scatter<R, CONJ, UNIT><<<Blocks(a->rows * 32, sm), kThreads, 0, s>>>(
        ptr, idx, val, xd, x->stride, yd, y->stride, alpha, a->rows);
    return static_cast<int>(cudaGetLastError());
  }
  const bool pair = ((reinterpret_cast<uintptr_t>(val) | reinterpret_cast<uintptr_t>(xd)) &
                     (sizeof(Cx<R>) - 1)) == 0;
  // as many rows a warp as still leave every SM 16 warps, but no more entries
  // than four rounds' worth on average, nor a little more than one
  const int64_t mean = a->nnz / a->rows + 1;
  int64_t per_warp = a->rows / (static_cast<int64_t>(sm > 0 ? sm : 148) * 16);
  if (per_warp * mean > 4 * kRound) per_warp = 4 * kRound / mean;
  if (per_warp * mean > kRound && per_warp * mean < 2 * kRound) per_warp = kRound / mean;
  per_warp = per_warp < 1 ? 1 : (per_warp > 32 ? 32 : per_warp);
  // FAST: the lanes that this leaves over share the rows (100,000 rows of 64 entries,
  // one lane each / 4, C and Z, us: 52 / 38 and 69 / 51)
  int log_share = 0;
  while ((per_warp << (log_share + 1)) <= 32) ++log_share;
  const unsigned blocks = Blocks((a->rows + per_warp - 1) / per_warp * 32, sm);
  auto kernel = mode == 1 ? (pair ? complex_rows<R, true, CONJ, UNIT, true>
                                  : complex_rows<R, true, CONJ, UNIT, false>)
                          : (pair ? complex_rows<R, false, CONJ, UNIT, true>
                                  : complex_rows<R, false, CONJ, UNIT, false>);
  kernel<<<blocks, kThreads, 0, s>>>(ptr, idx, val, xd, x->stride, yd, y->stride, alpha, a->rows,
                                     static_cast<int>(per_warp), log_share);
  return static_cast<int>(cudaGetLastError());
}

template <typename R>
int spmv_dispatch(cudaStream_t s, int mode, int conj, const ascb_csr* a, double ar, double ai,
                  const ascb_vec* x, const ascb_vec* y, int sm) {
  const Cx<R> alpha{static_cast<R>(ar), static_cast<R>(ai)};
  const bool unit = x->stride == 1 && y->stride == 1;
  if (conj) {
    return unit ? spmv_typed<R, true, true>(s, mode, a, alpha, x, y, sm)
                : spmv_typed<R, true, false>(s, mode, a, alpha, x, y, sm);
  }
  return unit ? spmv_typed<R, false, true>(s, mode, a, alpha, x, y, sm)
              : spmv_typed<R, false, false>(s, mode, a, alpha, x, y, sm);
}

template <typename R, bool CONJ>
int spmm_typed(cudaStream_t s, int mode, const ascb_csr* a, int64_t k, const void* b,
               int b_layout, int64_t ldb, void* c, int c_layout, int64_t ldc, Cx<R> alpha,
               int sm) {
  const auto* val = static_cast<const Cx<R>*>(a->val);
  const auto* bm = static_cast<const Cx<R>*>(b);
  auto* cm = static_cast<Cx<R>*>(c);
  const unsigned blocks = Blocks(a->rows * k, sm);
  if (mode == 2) {
    complex_spmm_scatter<R, CONJ><<<blocks, kThreads, 0, s>>>(a->ptr, a->idx, val, bm, b_layout,
                                                              ldb, cm, c_layout, ldc, k, alpha,
                                                              a->rows);
  } else if (mode == 1) {
    complex_spmm_rows<R, true, CONJ><<<blocks, kThreads, 0, s>>>(
        a->ptr, a->idx, val, bm, b_layout, ldb, cm, c_layout, ldc, k, alpha, a->rows);
  } else {
    complex_spmm_rows<R, false, CONJ><<<blocks, kThreads, 0, s>>>(
        a->ptr, a->idx, val, bm, b_layout, ldb, cm, c_layout, ldc, k, alpha, a->rows);
  }
  return static_cast<int>(cudaGetLastError());
}

}  // namespace
}  // namespace ascb

extern "C" int ascb_complex_spmv(void* stream, int dtype, int mode, int conj, const ascb_csr* a,
                                 double alpha_re, double alpha_im, const ascb_vec* x,
                                 const ascb_vec* y, int sm_count) {
  if (a->rows <= 0) return 0;
  auto s = static_cast<cudaStream_t>(stream);
  if (dtype == ASCB_C128) {
    return ascb::spmv_dispatch<double>(s, mode, conj, a, alpha_re, alpha_im, x, y, sm_count);
  }
  if (dtype == ASCB_C64) {
    return ascb::spmv_dispatch<float>(s, mode, conj, a, alpha_re, alpha_im, x, y, sm_count);
  }
  return static_cast<int>(cudaErrorInvalidValue);
}

extern "C" int ascb_complex_spmm(void* stream, int dtype, int mode, int conj, const ascb_csr* a,
                                 int64_t k, const void* b, int b_layout, int64_t ldb, void* c,
                                 int c_layout, int64_t ldc, double alpha_re, double alpha_im,
                                 int sm_count) {
  if (a->rows <= 0 || k <= 0) return 0;
  auto s = static_cast<cudaStream_t>(stream);
  if (dtype == ASCB_C128) {
    const ascb::Cx<double> al{alpha_re, alpha_im};
    return conj ? ascb::spmm_typed<double, true>(s, mode, a, k, b, b_layout, ldb, c, c_layout,
                                                 ldc, al, sm_count)
                : ascb::spmm_typed<double, false>(s, mode, a, k, b, b_layout, ldb, c, c_layout,
                                                  ldc, al, sm_count);
  }
  if (dtype == ASCB_C64) {
    const ascb::Cx<float> al{static_cast<float>(alpha_re), static_cast<float>(alpha_im)};
    return conj ? ascb::spmm_typed<float, true>(s, mode, a, k, b, b_layout, ldb, c, c_layout,
                                                ldc, al, sm_count)
                : ascb::spmm_typed<float, false>(s, mode, a, k, b, b_layout, ldb, c, c_layout,
                                                 ldc, al, sm_count);
  }
  return static_cast<int>(cudaErrorInvalidValue);
}
