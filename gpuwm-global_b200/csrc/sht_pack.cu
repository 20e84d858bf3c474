// Spectral-side layout kernels.
//
// pack:   coefficients (planes, T+1, T+1) [n, m] -> the synthesis operand
//         Cfold, rows (m, q, i) with n = m + q + 2i and the (plane, field,
//         re/im) columns innermost; optional per-degree factor (the inverse
//         Laplacian of the vector synthesis, transform.py:1804-1811).
// unpack: the analysis output Cfold -> coefficients, zero above the
//         triangle and Imag(c[n,0]) = 0 (transform.py:1435-1452); the vector
//         mode combines the rotational and shear contractions into
//         (vorticity, divergence) with the i*m factor and projects
//         (vector.py:113-134).
// Both go through a 32 x 32 shared tile so the [n, m] side is read/written
// along m and the folded side along the plane index.
#include "sht_plan.h"

namespace sht {
namespace {

template <typename T> using V2 = typename Vec2<T>::type;

// Row base of order m in the folded operand Cfold (orders below m fill
// sum_{m' < m} (T + 1 - m') rows); with size0 the size of its parity-0
// block, row(m, q, i) = base + (q ? size0 : 0) + i.
__device__ __forceinline__ int64_t cf_base(int T, int m) {
  return (int64_t)m * (T + 1) - (int64_t)m * (m - 1) / 2;
}

template <typename T>
__device__ __forceinline__ void copy_async(V2<T>* dst, const V2<T>* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

// (n, m) coefficients -> folded rows.  One CTA: 32 orders x NB degrees x 32
// columns (c = plane F + field, so two fields' columns are stored side by
// side: one field a CTA left every other column to another CTA and 40 planes
// took four blocks of columns instead of three; T511 x 2 x 40 planes 74 us,
// 47).  Every load of the CTA is issued before its one barrier, FP32 by
// cp.async without a register, and the row maxima are merged over the whole
// block before one atomic per column.  INVLAP: divide by the Laplacian
// eigenvalue -n(n+1)/a^2 (zero at degree 0, Imag = 0 at m = 0).
template <typename T> struct PackCfg { static constexpr int NB = sizeof(T) == 4 ? 4 : 2; };

template <typename T, bool INVLAP>
__global__ void __launch_bounds__(256) pack_kernel(int Tn, double radius,
                                                   const V2<T>* __restrict__ c0,
                                                   const V2<T>* __restrict__ c1, int64_t ncols,
                                                   int64_t Rc, int F, V2<T>* __restrict__ cf,
                                                   float* __restrict__ rowmax) {
  constexpr int NB = PackCfg<T>::NB;
  __shared__ V2<T> tile[NB][32][33];
  __shared__ float red[2][8][32];
  // The eigenvalues of the block's degrees, divided out in FP64 once per CTA
  // (T511 x 2 x 40 planes: 84 us with the division per thread, 71 us without,
  // both with one field a CTA).
  __shared__ T eigs[NB];
  const int m0 = blockIdx.x * 32;
  const int n0 = blockIdx.y * NB;
  if (m0 > n0 + NB - 1 || n0 > Tn) return;  // the whole block is above the triangle
  if (INVLAP && threadIdx.y == 0 && threadIdx.x < NB) {
    const int n = n0 + threadIdx.x;
    eigs[threadIdx.x] = T(-((double)n * ((double)n + 1.0)) / (radius * radius));
  }
  const int64_t q0 = (int64_t)blockIdx.z * 32;  // first column p * F + f
  const int fsh = F >> 1;                       // log2 of the field count
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int64_t t1 = Tn + 1;
  if constexpr (sizeof(T) == 4) {
    const int m = m0 + tx;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const int n = n0 + nb;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int64_t col = q0 + ty + 8 * k;
        const V2<T>* src = (col & (F - 1)) ? c1 : c0;
        if (col < ncols && n <= Tn && m <= n)
          copy_async<T>(&tile[nb][ty + 8 * k][tx], src + ((col >> fsh) * t1 + n) * t1 + m);
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    const int m = m0 + tx;
    V2<T> v[NB][4];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const int n = n0 + nb;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int64_t col = q0 + ty + 8 * k;
        const V2<T>* src = (col & (F - 1)) ? c1 : c0;
        v[nb][k] = mk2<T>(T(0), T(0));
        if (col < ncols && n <= Tn && m <= n)
          v[nb][k] = __ldcs(src + ((col >> fsh) * t1 + n) * t1 + m);
      }
    }
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int k = 0; k < 4; ++k) tile[nb][ty + 8 * k][tx] = v[nb][k];
  }
  __syncthreads();
  const int64_t q = q0 + tx;
  float mre = 0.f, mim = 0.f;
  if (q < ncols) {
    V2<T>* col = cf + q;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int m = m0 + ty + 8 * k;
      if (m > Tn) break;
      const int64_t base = cf_base(Tn, m);
      const int size0 = parity_count(Tn, m, 0);
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        const int n = n0 + nb;
        if (n > Tn || m > n) continue;
        const int par = (n - m) & 1, i = (n - m) >> 1;
        V2<T> v = tile[nb][tx][ty + 8 * k];
        if constexpr (INVLAP) {
          const T eig = eigs[nb];
          // c / eig (complex by real), zero at degree 0
          v = n == 0 ? mk2<T>(T(0), T(0)) : mk2<T>(v.x / eig, v.y / eig);
          if (m == 0) v.y = T(0);  // project() inside inverse_laplacian
        }
        col[(base + (par ? size0 : 0) + i) * Rc] = v;
        mre = fmaxf(mre, (float)fabs(v.x));
        mim = fmaxf(mim, (float)fabs(v.y));
      }
    }
  }
  if (rowmax != nullptr) {
    // Row maxima of this CTA's 32 columns: reduce the 8 ty groups, publish once.
    red[0][ty][tx] = mre;
    red[1][ty][tx] = mim;
    __syncthreads();
    if (ty == 0 && q < ncols) {
      float ra = 0.f, rb = 0.f;
      for (int k = 0; k < 8; ++k) {
        ra = fmaxf(ra, red[0][k][tx]);
        rb = fmaxf(rb, red[1][k][tx]);
      }
      atomicMax(reinterpret_cast<int*>(rowmax + 2 * q), __float_as_int(ra));
      atomicMax(reinterpret_cast<int*>(rowmax + 2 * q + 1), __float_as_int(rb));
    }
  }
}

// Folded rows -> (n, m) coefficients.  One CTA: 32 orders x NB degrees x 32
// columns (c = plane, or 2 plane + field for vorticity / divergence), raw
// columns of the one or two row sets in shared memory, combined as they are
// stored.  FP32 columns arrive by cp.async: every load of the CTA is then in
// flight without a register (T511 x 200 planes: 140 us through registers, 113;
// two fields of 40 planes 78, 68).  FP64 stays in registers (T62 x 161 planes
// 8.9 us, 10.6 by cp.async).  A CTA wholly above the triangle writes zeros only.
template <typename T, int MODE> struct UnpackCfg {
  static constexpr int NO = MODE == kUnpackVorDiv ? 2 : 1;  // output fields
  static constexpr int NT = MODE == kUnpackScalar ? 1 : 2;  // row sets
  static constexpr int NB = sizeof(T) == 4 && NT == 1 ? 2 : 1;
};


template <typename T, int MODE>
__global__ void __launch_bounds__(256) unpack_kernel(int Tn, const V2<T>* __restrict__ cf0,
                                                     const V2<T>* __restrict__ cf1, int64_t ncols,
                                                     int64_t Rc, V2<T>* __restrict__ o0, V2<T>* __restrict__ o1) {
  using Cfg = UnpackCfg<T, MODE>;
  constexpr int NB = Cfg::NB, NT = Cfg::NT;
  __shared__ V2<T> tile[NT][NB][32][33];
  const int m0 = blockIdx.x * 32;
  const int n0 = blockIdx.y * NB;
  const int64_t q0 = (int64_t)blockIdx.z * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int64_t t1 = Tn + 1;
  const V2<T> zero = mk2<T>(T(0), T(0));
  // Column col of the output, degree n.
  auto row_of = [&](int64_t col, int n) -> V2<T>* {
    if constexpr (Cfg::NO == 2)
      return ((col & 1) ? o1 : o0) + ((col >> 1) * t1 + n) * t1;
    else
      return o0 + (col * t1 + n) * t1;
  };
  const bool above = m0 > n0 + NB - 1;
  if (!above) {
    const int64_t col = q0 + tx;
    V2<T> v[NT][NB][4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int m = m0 + ty + 8 * k;
      const int64_t base = m <= Tn ? cf_base(Tn, m) : 0;
      const int size0 = m <= Tn ? parity_count(Tn, m, 0) : 0;
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        const int n = n0 + nb;
        const bool in = n <= Tn && m <= n && col < ncols;
        const int64_t off = (base + (((n - m) & 1) ? size0 : 0) + ((n - m) >> 1)) * Rc + col;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const V2<T>* src = (t ? cf1 : cf0) + off;
          if constexpr (sizeof(T) == 4) {
            if (in) copy_async<T>(&tile[t][nb][tx][ty + 8 * k], src);
          } else {
            v[t][nb][k] = in ? __ldcs(src) : zero;
          }
        }
      }
    }
    if constexpr (sizeof(T) == 4) {
      asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
          for (int k = 0; k < 4; ++k) tile[t][nb][tx][ty + 8 * k] = v[t][nb][k];
    }
    __syncthreads();
  }
  const int m = m0 + tx;
  if (m > Tn) return;
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    const int n = n0 + nb;
    if (n > Tn) break;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = ty + 8 * k;
      if (q0 + c >= ncols) continue;
      V2<T> val = zero;
      if (m <= n) {
        if constexpr (MODE == kUnpackScalar) {
          val = tile[0][nb][c][tx];
        } else {
          const T mf = T(m);
          if (MODE == kUnpackDiv || (c & 1)) {
            // D = i m rot[u] - shear[v]: rows of the own plane's u and v
            const V2<T> ru = tile[0][nb][MODE == kUnpackDiv ? c : c - 1][tx], sv = tile[NT - 1][nb][c][tx];
            val = mk2<T>(-mf * ru.y - sv.x, mf * ru.x - sv.y);
          } else {
            // zeta = i m rot[v] + shear[u]
            const V2<T> rv = tile[0][nb][c + 1][tx], su = tile[NT - 1][nb][c][tx];
            val = mk2<T>(-mf * rv.y + su.x, mf * rv.x + su.y);
          }
        }
        if (m == 0) val.y = T(0);
      }
      row_of(q0 + c, n)[m] = val;
    }
  }
}

template <typename T>
__global__ void elementwise_kernel(int Tn, double radius, int mode, const V2<T>* __restrict__ in,
                                   int64_t total, V2<T>* __restrict__ out) {
  const int64_t t1 = Tn + 1;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    int m = (int)(idx % t1);
    int n = (int)((idx / t1) % t1);
    V2<T> v = in[idx];
    T eig = T(-((double)n * ((double)n + 1.0)) / (radius * radius));
    if (mode == kElemLaplacian) {
      v = mk2<T>(v.x * eig, v.y * eig);
    } else {
      if (mode == kElemInvLaplacian) v = n == 0 ? mk2<T>(T(0), T(0)) : mk2<T>(v.x / eig, v.y / eig);
      if (m > n) v = mk2<T>(T(0), T(0));
      if (m == 0) v.y = T(0);
    }
    out[idx] = v;
  }
}

}  // namespace

template <typename T>
void launch_pack(const sht_plan* p, const T* coeff0, const T* coeff1, int64_t planes, int64_t ldc, int mode,
                 T* cfold, cudaStream_t s, float* rowmax) {
  if (planes == 0) return;
  int F = coeff1 ? 2 : 1;
  dim3 grid((unsigned)div_up(p->T + 1, 32), (unsigned)div_up(p->T + 1, PackCfg<T>::NB),
            (unsigned)div_up(planes * F, 32));
  SHT_REQUIRE(div_up(planes, 32) * F <= 65535, "too many planes for one pack launch");
  if (mode == kPackInvLap)
    pack_kernel<T, true><<<grid, dim3(32, 8), 0, s>>>(p->T, p->radius, (const V2<T>*)coeff0,
                                                      (const V2<T>*)coeff1, planes * F, ldc, F,
                                                      (V2<T>*)cfold, rowmax);
  else
    pack_kernel<T, false><<<grid, dim3(32, 8), 0, s>>>(p->T, p->radius, (const V2<T>*)coeff0,
                                                       (const V2<T>*)coeff1, planes * F, ldc, F,
                                                       (V2<T>*)cfold, rowmax);
  SHT_CUDA_OR_THROW(cudaGetLastError());
}

template <typename T, int MODE>
void launch_unpack_mode(const sht_plan* p, const T* cf0, const T* cf1, int64_t planes,
                        int64_t ldc, T* out0, T* out1, cudaStream_t s) {
  using Cfg = UnpackCfg<T, MODE>;
  SHT_REQUIRE(div_up(planes, 32) <= 65535, "too many planes for one unpack launch");
  const int64_t ncols = planes * Cfg::NO, t2 = (int64_t)(p->T + 1) * (p->T + 1);
  // at most 65535 blocks of columns a launch
  for (int64_t c = 0; c < ncols; c += 65535 * 32) {
    dim3 grid((unsigned)div_up(p->T + 1, 32), (unsigned)div_up(p->T + 1, Cfg::NB),
              (unsigned)std::min<int64_t>(65535, div_up(ncols - c, 32)));
    const int64_t o = c / Cfg::NO * t2;
    unpack_kernel<T, MODE><<<grid, dim3(32, 8), 0, s>>>(
        p->T, (const V2<T>*)cf0 + c, Cfg::NT == 2 ? (const V2<T>*)cf1 + c : nullptr, ncols - c, ldc,
        (V2<T>*)out0 + o, Cfg::NO == 2 ? (V2<T>*)out1 + o : nullptr);
  }
  SHT_CUDA_OR_THROW(cudaGetLastError());
}

template <typename T>
void launch_unpack(const sht_plan* p, int mode, const T* cf0, const T* cf1, int64_t planes,
                   int64_t ldc, T* out0, T* out1, cudaStream_t s) {
  if (planes == 0) return;
  if (mode == kUnpackVorDiv)
    launch_unpack_mode<T, kUnpackVorDiv>(p, cf0, cf1, planes, ldc, out0, out1, s);
  else if (mode == kUnpackDiv)
    launch_unpack_mode<T, kUnpackDiv>(p, cf0, cf1, planes, ldc, out0, out1, s);
  else
    launch_unpack_mode<T, kUnpackScalar>(p, cf0, cf1, planes, ldc, out0, out1, s);
}

template <typename T>
void launch_elementwise(const sht_plan* p, int mode, const T* in, int64_t planes, T* out,
                        cudaStream_t s) {
  int64_t total = planes * (int64_t)(p->T + 1) * (p->T + 1);
  if (total == 0) return;
  int blocks = (int)std::min<int64_t>(div_up(total, 256), 148 * 16);
  elementwise_kernel<T><<<blocks, 256, 0, s>>>(p->T, p->radius, mode, (const V2<T>*)in, total,
                                               (V2<T>*)out);
  SHT_CUDA_OR_THROW(cudaGetLastError());
}

#define INST(T)                                                                                  \
  template void launch_pack<T>(const sht_plan*, const T*, const T*, int64_t, int64_t, int, T*,          \
                               cudaStream_t, float*);                                           \
  template void launch_unpack<T>(const sht_plan*, int, const T*, const T*, int64_t, int64_t, T*, T*,    \
                                 cudaStream_t);                                                 \
  template void launch_elementwise<T>(const sht_plan*, int, const T*, int64_t, T*, cudaStream_t);
INST(float)
INST(double)
#undef INST

}  // namespace sht
