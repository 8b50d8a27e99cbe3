// Vector-CSR SpMV for sm_100a: a group of LANES threads (1..32) owns a row,
// strides through its nonzeros (one by one, or in aligned fours of 32-byte loads)
// with fused multiply-adds and combines the lane
// partials with a butterfly of warp shuffles.  Persistent grid-stride CTAs
// (a whole number of waves over the 148 SMs).  Numerics: each lane's partial is
// a contracted running sum and the butterfly reorders it, so results satisfy
// |y - y_ref| <= gamma_{n+2} (|alpha||A||x| + |beta||y|) rather than being
// bit-identical to the serial order.
#include "common.cuh"
#include "kernels.h"

namespace ascb {
namespace {

constexpr int kThreads = 256;
constexpr int kUnroll = 4;

__device__ __forceinline__ void load_four(const double* p, double (&v)[4]) { ld_stream32(p, v); }
__device__ __forceinline__ void load_four(const float* p, float (&v)[4]) {
  const float4 f = __ldcs(reinterpret_cast<const float4*>(p));
  v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
}

template <typename T, int LANES, bool STANDARD, bool UNIT, bool WIDE>
__global__ void __launch_bounds__(kThreads)
vector_kernel(int64_t rows, int64_t nnz, const int64_t* __restrict__ ptr,
              const int64_t* __restrict__ idx, const T* __restrict__ val,
              const T* __restrict__ x, int64_t incx, T* __restrict__ y,
              int64_t incy, T alpha, T beta) {
  constexpr int kGroups = kThreads / LANES;
  const int lane = threadIdx.x % LANES;
  const int64_t first =
      static_cast<int64_t>(blockIdx.x) * kGroups + threadIdx.x / LANES;
  const int64_t step = static_cast<int64_t>(gridDim.x) * kGroups;
  for (int64_t row = first; row < rows; row += step) {
    const int64_t b = __ldg(ptr + row);
    const int64_t e = __ldg(ptr + row + 1);
    T acc[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) acc[u] = T(0);
    if constexpr (WIDE) {
      // aligned fours from the one that holds the row's first entry
      constexpr int kFours = 2;  // of each lane in flight
      for (int64_t q = (b & ~int64_t{3}) + 4 * lane; q < e; q += kFours * 4 * LANES) {
        int64_t col[kFours][4];
        T v[kFours][4];
#pragma unroll
        for (int f = 0; f < kFours; ++f) {
          const int64_t p = q + f * 4 * LANES;
          if (p + 4 <= nnz && p < e) {
            ld_stream32(idx + p, col[f]);
            load_four(val + p, v[f]);
          } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const bool ok = p + u >= b && p + u < e;
              col[f][u] = ok ? ld_stream(idx + p + u) : 0;
              v[f][u] = ok ? ld_stream(val + p + u) : T(0);
            }
          }
        }
        T xv[kFours][4];
#pragma unroll
        for (int f = 0; f < kFours; ++f) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int64_t p = q + f * 4 * LANES + u;
            xv[f][u] = p >= b && p < e ? ld_gather(&at<UNIT>(x, col[f][u], incx)) : T(0);
          }
        }
#pragma unroll
        for (int f = 0; f < kFours; ++f) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int64_t p = q + f * 4 * LANES + u;
            if (p >= b && p < e) acc[u] = fma(v[f][u], xv[f][u], acc[u]);
          }
        }
      }
    } else {
      int64_t q = b + lane;
      for (; q + (kUnroll - 1) * LANES < e; q += kUnroll * LANES) {
        int64_t col[kUnroll];
        T v[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
          col[u] = ld_stream(idx + q + u * LANES);
          v[u] = ld_stream(val + q + u * LANES);
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
          acc[u] = fma(v[u], ld_gather(&at<UNIT>(x, col[u], incx)), acc[u]);
        }
      }
      for (; q < e; q += LANES) {
        acc[0] = fma(ld_stream(val + q),
                     ld_gather(&at<UNIT>(x, ld_stream(idx + q), incx)), acc[0]);
      }
    }
    T s = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
    for (int m = LANES / 2; m > 0; m >>= 1) s += shfl_xor(s, m, LANES);
    if (lane == 0) {
      T* yp = &at<UNIT>(y, row, incy);
      if (STANDARD) {
        *yp = fma(alpha, s, *yp);
      } else {
        *yp = beta != T(0) ? fma(alpha, s, beta * *yp) : alpha * s;
      }
    }
  }
}

template <typename T, int LANES, bool STANDARD, bool UNIT>
int launch(cudaStream_t stream, const ascb_csr* a, T alpha, T beta,
           const ascb_vec* x, const ascb_vec* y, int sm_count) {
  constexpr int kGroups = kThreads / LANES;
  const int64_t needed = (a->rows + kGroups - 1) / kGroups;
  const int64_t resident = static_cast<int64_t>(sm_count > 0 ? sm_count : 148) * 8;
  const unsigned blocks =
      static_cast<unsigned>(needed < resident ? needed : resident);
  // Aligned fours where a lane has at least four FP64 or twelve FP32 entries of an
  // average row: then they use every sector whole, which single loads leave to
  // an L1 that the rows of all resident warps do not fit.  On a B200, us, single
  // loads / fours: 27-point stencil 120^3 FP64, 1 lane 603 / 151, 2 lanes 267 /
  // 147, 4 lanes 145 / 145, 8 lanes 169 / 231; FP32, 2 lanes 130 / 121, 4 lanes 102
  // / 123; 5-point 2000^2 FP64, 1 lane 116 / 95, 2 lanes 99 / 148; FP32, 1 lane 64 /
  // 82; power law 300,000 rows FP64, 4 lanes 330 / 185.
  constexpr int kFewest = sizeof(T) == 8 ? 4 : 12;
  auto kernel = vector_kernel<T, LANES, STANDARD, UNIT, false>;
  if constexpr (LANES <= 4) {
    if (a->nnz >= kFewest * LANES * a->rows &&
        ((reinterpret_cast<uintptr_t>(a->idx) | reinterpret_cast<uintptr_t>(a->val)) & 31u) == 0) {
      kernel = vector_kernel<T, LANES, STANDARD, UNIT, true>;
    }
  }
  kernel<<<blocks, kThreads, 0, stream>>>(
      a->rows, a->nnz, a->ptr, a->idx, static_cast<const T*>(a->val),
      static_cast<const T*>(x->data), x->stride, static_cast<T*>(y->data),
      y->stride, alpha, beta);
  return static_cast<int>(cudaGetLastError());
}

template <typename T, int LANES>
int by_form(cudaStream_t s, int form, const ascb_csr* a, T al, T be,
            const ascb_vec* x, const ascb_vec* y, int sm) {
  const bool unit = x->stride == 1 && y->stride == 1;
  if (form == ASCB_STANDARD) {
    return unit ? launch<T, LANES, true, true>(s, a, al, be, x, y, sm)
                : launch<T, LANES, true, false>(s, a, al, be, x, y, sm);
  }
  return unit ? launch<T, LANES, false, true>(s, a, al, be, x, y, sm)
              : launch<T, LANES, false, false>(s, a, al, be, x, y, sm);
}

template <typename T>
int by_lanes(cudaStream_t s, int form, int lanes, const ascb_csr* a,
             double alpha, double beta, const ascb_vec* x, const ascb_vec* y,
             int sm) {
  const T al = static_cast<T>(alpha);
  const T be = static_cast<T>(beta);
  switch (lanes) {
    case 1: return by_form<T, 1>(s, form, a, al, be, x, y, sm);
    case 2: return by_form<T, 2>(s, form, a, al, be, x, y, sm);
    case 4: return by_form<T, 4>(s, form, a, al, be, x, y, sm);
    case 8: return by_form<T, 8>(s, form, a, al, be, x, y, sm);
    case 16: return by_form<T, 16>(s, form, a, al, be, x, y, sm);
    case 32: return by_form<T, 32>(s, form, a, al, be, x, y, sm);
    default: return static_cast<int>(cudaErrorInvalidValue);
  }
}

}  // namespace
}  // namespace ascb

extern "C" int ascb_spmv_vector(void* stream, int dtype, int form, int lanes,
                                const ascb_csr* a, double alpha, double beta,
                                const ascb_vec* x, const ascb_vec* y,
                                int sm_count) {
  if (a->rows <= 0) return 0;
  auto s = static_cast<cudaStream_t>(stream);
  return dtype == ASCB_F64
             ? ascb::by_lanes<double>(s, form, lanes, a, alpha, beta, x, y,
                                      sm_count)
             : ascb::by_lanes<float>(s, form, lanes, a, alpha, beta, x, y,
                                     sm_count);
}
