// Longitude real FFTs that write and read the equator-folded Fourier waist.
//
// Forward (grid -> waist): rows of nlon reals are transformed as complex
// sequences of L = nlon/2 (z_k = x_2k + i x_2k+1) by a shared-memory Stockham
// FFT, untangled into the real-input spectrum X_m, scaled by 1/nlon and cut
// to m <= T (the reference's rfft(f)/nlon[..., :T+1], transform.py:1386-1390),
// then folded across the equator: S = X(row h) + X(mirror row), D = X(h) -
// X(mirror).  The waist layout is [m][s][h][r] with the row index r = 2*plane
// + (re, im) innermost, which is the operand layout of the per-order Legendre
// contraction, so no separate transpose kernel exists.
//
// Inverse (waist -> grid): the folded synthesis output is unfolded (X(h) = S
// + D, X(mirror) = S - D), optionally combined (zonal i*m factor, gradient
// metric factors, the (u, v) combination of the vector synthesis), entangled
// into a length-L complex sequence and inverted; the result equals
// irfft(nlon * W) of the reference (transform.py:1654-1702), which discards
// Imag(W_0) and has no Nyquist term because T < nlon/2.
//
// Any even nlon in FP32 and FP64 (the register kernels of sht_fft_fast.cu
// take nlon = 64 F in FP32).  A CTA transforms 2^lr rows of one latitude pair
// together, held row-innermost in shared memory ([k][row]): every thread
// keeps one row through all passes, so no pass divides an index by a run-time
// row or butterfly count, shared accesses are consecutive, and the threads of
// one butterfly column read their twiddles as broadcasts.  What bounds it is
// the chain of passes, a barrier apart, so the radix plan takes the fewest
// passes, radices up to 16, and three CTAs (two in FP64) share an SM.  Against
// a kernel that held rows one after another, divided indices in every pass and
// had 24 of 256 threads busy in a radix-16 pass (forward / inverse): T62 x 161
// planes in FP64 on 94 x 192, 94 / 58 -> 19 / 19 us; T300 x 41 planes in FP32
// on 452 x 960, 162 / 171 -> 73 / 67 us (1.6 TB/s); T21, one plane, 12.8 /
// 13.6 -> 3.4 / 3.8 us.
#include <algorithm>

#include "sht_plan.h"

namespace sht {
namespace {

template <typename T> using V2 = typename Vec2<T>::type;

template <typename T>
__device__ __forceinline__ V2<T> cmul(V2<T> a, V2<T> b) {
  return mk2<T>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename T>
__device__ __forceinline__ V2<T> cadd(V2<T> a, V2<T> b) { return mk2<T>(a.x + b.x, a.y + b.y); }
template <typename T>
__device__ __forceinline__ V2<T> csub(V2<T> a, V2<T> b) { return mk2<T>(a.x - b.x, a.y - b.y); }
template <typename T>
__device__ __forceinline__ V2<T> cconj(V2<T> a) { return mk2<T>(a.x, -a.y); }
// multiply by -i (forward) or +i (inverse)
template <typename T, bool INV>
__device__ __forceinline__ V2<T> rot90(V2<T> a) {
  return INV ? mk2<T>(-a.y, a.x) : mk2<T>(a.y, -a.x);
}
// multiply by (c, -s) forward, (c, s) inverse
template <typename T, bool INV>
__device__ __forceinline__ V2<T> turn(V2<T> a, double c, double s) {
  return cmul<T>(a, mk2<T>(T(c), INV ? T(s) : T(-s)));
}

// In-register DFTs, forward with exp(-2 pi i rs / R), natural order in and out.
template <typename T, bool INV>
__device__ __forceinline__ void dft2(V2<T>& a, V2<T>& b) {
  const V2<T> t = a;
  a = cadd<T>(t, b);
  b = csub<T>(t, b);
}
template <typename T, bool INV>
__device__ __forceinline__ void dft4(V2<T>* v) {
  const V2<T> a0 = cadd<T>(v[0], v[2]), a1 = csub<T>(v[0], v[2]);
  const V2<T> b0 = cadd<T>(v[1], v[3]), b1 = rot90<T, INV>(csub<T>(v[1], v[3]));
  v[0] = cadd<T>(a0, b0);
  v[2] = csub<T>(a0, b0);
  v[1] = cadd<T>(a1, b1);
  v[3] = csub<T>(a1, b1);
}
template <typename T, bool INV>
__device__ __forceinline__ void dft8(V2<T>* v) {
  V2<T> e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
  dft4<T, INV>(e);
  dft4<T, INV>(o);
  constexpr double r = 0.70710678118654752440;
  o[1] = turn<T, INV>(o[1], r, r);
  o[2] = rot90<T, INV>(o[2]);
  o[3] = turn<T, INV>(o[3], -r, r);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = cadd<T>(e[k], o[k]);
    v[k + 4] = csub<T>(e[k], o[k]);
  }
}

// cos and sin of 2 pi k / R, k <= R / 2, of the odd prime radices.
template <int R> struct OddTrig;
template <> struct OddTrig<3> {
  static __device__ __forceinline__ double c(int k) { const double t[] = {1.0, -0.5}; return t[k]; }
  static __device__ __forceinline__ double s(int k) { const double t[] = {0.0, 0.866025403784438646764}; return t[k]; }
};
template <> struct OddTrig<5> {
  static __device__ __forceinline__ double c(int k) {
    const double t[] = {1.0, 0.309016994374947424102, -0.809016994374947424102};
    return t[k];
  }
  static __device__ __forceinline__ double s(int k) {
    const double t[] = {0.0, 0.951056516295153572116, 0.587785252292473129169};
    return t[k];
  }
};
template <> struct OddTrig<7> {
  static __device__ __forceinline__ double c(int k) {
    const double t[] = {1.0, 0.623489801858733530525, -0.222520933956314404289, -0.900968867902419126236};
    return t[k];
  }
  static __device__ __forceinline__ double s(int k) {
    const double t[] = {0.0, 0.781831482468029808708, 0.974927912181823607018, 0.433883739117558120476};
    return t[k];
  }
};
template <> struct OddTrig<11> {
  static __device__ __forceinline__ double c(int k) {
    const double t[] = {1.0, 0.841253532831181168862, 0.415415013001886425529,
                        -0.142314838273285140444, -0.654860733945285064057, -0.95949297361449738989};
    return t[k];
  }
  static __device__ __forceinline__ double s(int k) {
    const double t[] = {0.0, 0.540640817455597582108, 0.909631995354518371412,
                        0.989821441880932732376, 0.755749574354258283774, 0.281732556841429697711};
    return t[k];
  }
};
template <> struct OddTrig<13> {
  static __device__ __forceinline__ double c(int k) {
    const double t[] = {1.0, 0.8854560256532098959, 0.568064746731155802512, 0.120536680255323053349,
                        -0.35460488704253562597, -0.748510748171101098635, -0.970941817426052027157};
    return t[k];
  }
  static __device__ __forceinline__ double s(int k) {
    const double t[] = {0.0, 0.464723172043768545656, 0.82298386589365639458, 0.992708874098053992801,
                        0.93501624268541482344, 0.663122658240795202377, 0.239315664287557767149};
    return t[k];
  }
};
// Odd prime R by pairs: with t_i = v_i + v_{R-i} and u_i = v_i - v_{R-i},
// X_k, X_{R-k} = v_0 + sum_i cos(ik) t_i -+ i sum_i sin(ik) u_i.
template <typename T, bool INV, int R>
__device__ __forceinline__ void dft_odd(V2<T>* v) {
  constexpr int H = R / 2;
  V2<T> t[H], u[H];
  V2<T> sum = v[0];
#pragma unroll
  for (int i = 1; i <= H; ++i) {
    t[i - 1] = cadd<T>(v[i], v[R - i]);
    u[i - 1] = csub<T>(v[i], v[R - i]);
    sum = cadd<T>(sum, t[i - 1]);
  }
  const V2<T> v0 = v[0];
  v[0] = sum;
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    V2<T> a = v0, b = mk2<T>(T(0), T(0));
#pragma unroll
    for (int i = 1; i <= H; ++i) {
      const int e = (i * k) % R;
      const T c = T(OddTrig<R>::c(e <= H ? e : R - e));
      const T s = T(e <= H ? OddTrig<R>::s(e) : -OddTrig<R>::s(R - e));
      a.x += c * t[i - 1].x;
      a.y += c * t[i - 1].y;
      if constexpr (R == 3) {  // the product rounds with the sum it goes into
        const T t = INV ? -s : s;
        v[1] = mk2<T>(fma(t, u[0].y, a.x), fma(-t, u[0].x, a.y));
        v[2] = mk2<T>(fma(-t, u[0].y, a.x), fma(t, u[0].x, a.y));
        return;
      }
      b.x += s * u[i - 1].x;
      b.y += s * u[i - 1].y;
    }
    const V2<T> ib = rot90<T, INV>(b);
    v[k] = cadd<T>(a, ib);
    v[R - k] = csub<T>(a, ib);
  }
}

template <typename T, bool INV, int R>
__device__ __forceinline__ void dft(V2<T>* v);

// R = A B with A and B coprime (Good-Thomas): no twiddles; element
// (B a + A b) mod R in, (B Bi k1 + A Ai k2) mod R out, Bi = B^-1 mod A.
constexpr int inverse_mod(int x, int n) {
  for (int i = 1; i < n; ++i)
    if ((x * i) % n == 1) return i;
  return 1;
}
template <typename T, bool INV, int A, int B>
__device__ __forceinline__ void dft_coprime(V2<T>* v) {
  constexpr int R = A * B, EB = B * inverse_mod(B % A, A), EA = A * inverse_mod(A % B, B);
  V2<T> w[A][B];
#pragma unroll
  for (int a = 0; a < A; ++a) {
#pragma unroll
    for (int b = 0; b < B; ++b) w[a][b] = v[(B * a + A * b) % R];
    dft<T, INV, B>(w[a]);
  }
#pragma unroll
  for (int b = 0; b < B; ++b) {
    V2<T> c[A];
#pragma unroll
    for (int a = 0; a < A; ++a) c[a] = w[a][b];
    dft<T, INV, A>(c);
#pragma unroll
    for (int a = 0; a < A; ++a) v[(EB * a + EA * b) % R] = c[a];
  }
}
// R = A x A: columns, twiddles exp(-2 pi i ij / R), rows.
template <typename T, bool INV, int A>
__device__ __forceinline__ void dft_square(V2<T>* v) {
  V2<T> w[A][A];
#pragma unroll
  for (int i = 0; i < A; ++i) {
#pragma unroll
    for (int j = 0; j < A; ++j) w[i][j] = v[j * A + i];
    dft<T, INV, A>(w[i]);
  }
  if constexpr (A == 3) {
    w[1][1] = turn<T, INV>(w[1][1], 0.766044443118978035202, 0.642787609686539326323);
    w[1][2] = turn<T, INV>(w[1][2], 0.173648177666930348852, 0.984807753012208059367);
    w[2][1] = turn<T, INV>(w[2][1], 0.173648177666930348852, 0.984807753012208059367);
    w[2][2] = turn<T, INV>(w[2][2], -0.939692620785908384054, 0.342020143325668733044);
  } else {
    constexpr double c1 = 0.923879532511286756128, s1 = 0.382683432365089771728;
    constexpr double r = 0.70710678118654752440;
    w[1][1] = turn<T, INV>(w[1][1], c1, s1);
    w[1][2] = turn<T, INV>(w[1][2], r, r);
    w[1][3] = turn<T, INV>(w[1][3], s1, c1);
    w[2][1] = turn<T, INV>(w[2][1], r, r);
    w[2][2] = rot90<T, INV>(w[2][2]);
    w[2][3] = turn<T, INV>(w[2][3], -r, r);
    w[3][1] = turn<T, INV>(w[3][1], s1, c1);
    w[3][2] = turn<T, INV>(w[3][2], -r, r);
    w[3][3] = turn<T, INV>(w[3][3], -c1, -s1);
  }
#pragma unroll
  for (int j = 0; j < A; ++j) {
    V2<T> c[A];
#pragma unroll
    for (int i = 0; i < A; ++i) c[i] = w[i][j];
    dft<T, INV, A>(c);
#pragma unroll
    for (int i = 0; i < A; ++i) v[i * A + j] = c[i];
  }
}
template <typename T, bool INV, int R>
__device__ __forceinline__ void dft(V2<T>* v) {
  if constexpr (R == 2) dft2<T, INV>(v[0], v[1]);
  else if constexpr (R == 4) dft4<T, INV>(v);
  else if constexpr (R == 8) dft8<T, INV>(v);
  else if constexpr (R == 6) dft_coprime<T, INV, 2, 3>(v);
  else if constexpr (R == 10) dft_coprime<T, INV, 2, 5>(v);
  else if constexpr (R == 12) dft_coprime<T, INV, 4, 3>(v);
  else if constexpr (R == 15) dft_coprime<T, INV, 3, 5>(v);
  else if constexpr (R == 9) dft_square<T, INV, 3>(v);
  else if constexpr (R == 16) dft_square<T, INV, 4>(v);
  else dft_odd<T, INV, R>(v);
}

// ------------------------------------------------------------------ passes
constexpr int kMaxPass = 24;
struct FftPass {
  int R;           // radix
  int Ns;          // product of the earlier radices
  int nb;          // butterflies per row, L / R
  int stride;      // twiddle stride, L / (Ns R)
  unsigned magic;  // ceil(2^32 / Ns): j / Ns = umulhi(j, magic) for j < 2^16, Ns > 1
};
struct FftShape {
  int L;     // complex length nlon / 2
  int lc;    // log2 of the waist columns (plane, field) of a CTA
  int rs;    // shared row stride: entry k of row g lies at k * rs + g
  int npass;
  int tw_shared;  // 1: the twiddle table is staged in shared memory
  FftPass pass[kMaxPass];
};

// One Stockham pass; thread -> row g = tid % rows (fixed), butterflies
// j = tid / rows, + blockDim / rows, ...
template <typename T, bool INV, int R>
__device__ __forceinline__ void pass_fixed(const V2<T>* in, V2<T>* out, const FftShape& f,
                                           const FftPass& p, int lr, const V2<T>* tw) {
  const int row = threadIdx.x & ((1 << lr) - 1), step = blockDim.x >> lr;
  const int nb = p.nb, Ns = p.Ns, rs = f.rs;
  for (int j = threadIdx.x >> lr; j < nb; j += step) {
    const V2<T>* src = in + j * rs + row;
    V2<T> v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = src[r * nb * rs];
    const int q = Ns > 1 ? (int)__umulhi((unsigned)j, p.magic) : j;
    const int k = j - q * Ns;
    if (Ns > 1) {
      const V2<T>* w = tw + k * p.stride;
#pragma unroll
      for (int r = 1; r < R; ++r) {
        const V2<T> t = w[k * (r - 1) * p.stride];
        v[r] = cmul<T>(v[r], INV ? cconj<T>(t) : t);
      }
    }
    dft<T, INV, R>(v);
    V2<T>* dst = out + (q * Ns * R + k) * rs + row;
#pragma unroll
    for (int r = 0; r < R; ++r) dst[r * Ns * rs] = v[r];
  }
}

// Any other prime radix: direct DFT of the twiddled inputs.
template <typename T, bool INV>
__device__ __noinline__ void pass_generic(const V2<T>* in, V2<T>* out, const FftShape& f,
                                          const FftPass& p, int lr, const V2<T>* tw) {
  const int row = threadIdx.x & ((1 << lr) - 1), step = blockDim.x >> lr;
  const int nb = p.nb, Ns = p.Ns, R = p.R, rs = f.rs;
  for (int e = threadIdx.x >> lr; e < f.L; e += step) {
    const int s = e / nb, j = e - s * nb;  // output s of butterfly j
    const int q = Ns > 1 ? (int)__umulhi((unsigned)j, p.magic) : j;
    const int k = j - q * Ns;
    const int inc = (k * p.stride + s * nb) % f.L;  // twiddle and DFT phase per input
    V2<T> acc = mk2<T>(T(0), T(0));
    for (int r = 0, idx = 0; r < R; ++r) {
      const V2<T> w = tw[idx];
      acc = cadd<T>(acc, cmul<T>(in[(j + r * nb) * rs + row], INV ? cconj<T>(w) : w));
      idx += inc;
      if (idx >= f.L) idx -= f.L;
    }
    out[(q * Ns * R + k + s * Ns) * rs + row] = acc;
  }
}

// Runs the passes (a barrier after each); returns the buffer with the result.
template <typename T, bool INV>
__device__ __forceinline__ V2<T>* run_passes(V2<T>* a, V2<T>* b, const FftShape& f, int lr,
                                             const V2<T>* tw) {
  for (int i = 0; i < f.npass; ++i) {
    const FftPass& p = f.pass[i];
    switch (p.R) {
      case 2: pass_fixed<T, INV, 2>(a, b, f, p, lr, tw); break;
      case 3: pass_fixed<T, INV, 3>(a, b, f, p, lr, tw); break;
      case 4: pass_fixed<T, INV, 4>(a, b, f, p, lr, tw); break;
      case 5: pass_fixed<T, INV, 5>(a, b, f, p, lr, tw); break;
      case 6: pass_fixed<T, INV, 6>(a, b, f, p, lr, tw); break;
      case 7: pass_fixed<T, INV, 7>(a, b, f, p, lr, tw); break;
      case 8: pass_fixed<T, INV, 8>(a, b, f, p, lr, tw); break;
      case 9: pass_fixed<T, INV, 9>(a, b, f, p, lr, tw); break;
      case 10: pass_fixed<T, INV, 10>(a, b, f, p, lr, tw); break;
      case 11: pass_fixed<T, INV, 11>(a, b, f, p, lr, tw); break;
      case 12: pass_fixed<T, INV, 12>(a, b, f, p, lr, tw); break;
      case 13: pass_fixed<T, INV, 13>(a, b, f, p, lr, tw); break;
      case 15: pass_fixed<T, INV, 15>(a, b, f, p, lr, tw); break;
      case 16: pass_fixed<T, INV, 16>(a, b, f, p, lr, tw); break;
      default: pass_generic<T, INV>(a, b, f, p, lr, tw); break;
    }
    __syncthreads();
    V2<T>* t = a;
    a = b;
    b = t;
  }
  return a;
}

// The twiddle table exp(-2 pi i k / L): its shared copy (filled here; the
// caller's next barrier publishes it) or the table in global memory.
template <typename T>
__device__ __forceinline__ const V2<T>* stage_twiddles(const FftShape& f, V2<T>* room,
                                                       const V2<T>* __restrict__ tw_l) {
  if (!f.tw_shared) return tw_l;
  for (int k = threadIdx.x; k < f.L; k += blockDim.x) room[k] = tw_l[k];
  return room;
}

// ----------------------------------------------------------------- forward
struct FoldArgs {
  FftShape f;
  int nlat, nlon, T, H, nlat_odd;
  int F;         // fields stacked per plane (1 scalar, 2 for (u, v))
  int64_t cols;  // waist columns, planes * F
  int64_t ldc;   // their stride
};

// grid (planes, nlat, nlon) per field -> waist [m][s][h][r], r = (p*F + f)*2 + c.
// Row g of a CTA: side g >> lc (the latitude, its mirror) of column g % 2^lc.
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) forward_fold_kernel(
    const __grid_constant__ FoldArgs a, const T* __restrict__ g0, const T* __restrict__ g1,
    const V2<T>* __restrict__ tw_l, const V2<T>* __restrict__ tw_n, T* __restrict__ wfold,
    float* __restrict__ rowmax) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int L = a.f.L, lc = a.f.lc, lr = lc + 1, rs = a.f.rs;
  V2<T>* bufA = reinterpret_cast<V2<T>*>(smem_raw);
  V2<T>* bufB = bufA + L * rs;
  const int h = blockIdx.y;
  const int64_t c0 = (int64_t)blockIdx.x << lc;
  const bool eq = a.nlat_odd && h == a.H - 1;
  const int fsh = a.F - 1;  // log2 of the field count (1 or 2)
  const V2<T>* tw = stage_twiddles<T>(a.f, bufB + L * rs, tw_l);
  // Loads: four neighbouring k of a row per quad of lanes (one 32-byte
  // sector in FP32), rows across the quads; each thread stays on one row.
  {
    const int row = (threadIdx.x >> 2) & ((1 << lr) - 1);
    const int64_t col = min(c0 + (row & ((1 << lc) - 1)), a.cols - 1);  // past the end: any live column
    const int j = (row >> lc) && !eq ? a.nlat - 1 - h : h;
    const V2<T>* src = reinterpret_cast<const V2<T>*>(
        ((col & fsh) ? g1 : g0) + ((col >> fsh) * a.nlat + j) * (int64_t)a.nlon);
    const int kstep = blockDim.x >> lr;
#pragma unroll 4
    for (int k = ((threadIdx.x >> (2 + lr)) << 2) + (threadIdx.x & 3); k < L; k += kstep)
      bufA[k * rs + row] = src[k];
  }
  __syncthreads();
  const V2<T>* Z = run_passes<T, false>(bufA, bufB, a.f, lr, tw);

  // Untangle, scale, fold, write.  Thread -> (m, column), columns fastest.
  const int q = threadIdx.x & ((1 << lc) - 1), mstep = blockDim.x >> lc;
  const T half_inv_n = T(0.5) / T(a.nlon);
  V2<T>* out = reinterpret_cast<V2<T>*>(wfold);
  const V2<T>*z0 = Z + q, *z1 = Z + q + (1 << lc);
  const bool live = c0 + q < a.cols;
  float mre = 0.f, mim = 0.f;  // this thread's column maxima
  if (live) {
    const int64_t dsd = (int64_t)a.H * a.ldc;  // S row -> D row of the same order
    V2<T>* dst = out + ((int64_t)(2 * (threadIdx.x >> lc)) * a.H + h) * a.ldc + c0 + q;
    for (int m = threadIdx.x >> lc; m <= a.T; m += mstep, dst += 2 * mstep * dsd) {
      const V2<T> w = tw_n[m];
      const int mc = m == 0 ? 0 : L - m;
      V2<T> X[2];
#pragma unroll
      for (int sd = 0; sd < 2; ++sd) {
        const V2<T>* z = sd ? z1 : z0;
        const V2<T> zk = z[m * rs], zc = cconj<T>(z[mc * rs]);
        const V2<T> ev = cadd<T>(zk, zc);  // 2 * even part
        const V2<T> od = csub<T>(zk, zc);  // 2 * i * odd part
        const V2<T> t = cmul<T>(w, od);    // X = (ev - i w od) / 2
        X[sd] = mk2<T>((ev.x + t.y) * half_inv_n, (ev.y - t.x) * half_inv_n);
      }
      const V2<T> S = eq ? X[0] : cadd<T>(X[0], X[1]);
      const V2<T> D = eq ? mk2<T>(T(0), T(0)) : csub<T>(X[0], X[1]);
      dst[0] = S;
      dst[dsd] = D;
      mre = fmaxf(mre, (float)fmax(fabs(S.x), fabs(D.x)));
      mim = fmaxf(mim, (float)fmax(fabs(S.y), fabs(D.y)));
    }
  }
  if (rowmax != nullptr) rowmax_merge(rowmax, c0 + q, live, mre, mim, 1 << lc);
}

// ----------------------------------------------------------------- inverse
struct UnfoldArgs {
  FftShape f;  // 2^lc planes per CTA
  int nlat, nlon, T, H, nlat_odd;
  int zonal;   // NF = 1: multiply by i m
  int64_t planes;
  int64_t ldc;  // waist column stride
  double radius;
};

// waist(s) -> grid rows.  NF waist columns per plane: 1 (scalar, zonal,
// meridional), 2 (gradient: the P and dP syntheses of one field), 4 (wind: P
// and dP of psi and chi, stored (psi, chi) per plane).  Row g of a CTA:
// output field g >> (lc + 1), side (g >> lc) & 1, plane g % 2^lc.
template <typename T, int NF>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) inverse_unfold_kernel(
    const __grid_constant__ UnfoldArgs a, const T* __restrict__ wP, const T* __restrict__ wD,
    const double* __restrict__ coslat, const V2<T>* __restrict__ tw_l,
    const V2<T>* __restrict__ tw_n, T* __restrict__ out0, T* __restrict__ out1) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NO = NF == 1 ? 1 : 2;  // output fields
  constexpr int FW = NF == 4 ? 2 : 1;  // waist columns per plane and buffer
  const int L = a.f.L, lc = a.f.lc, lr = lc + NO, rs = a.f.rs;
  V2<T>* bufA = reinterpret_cast<V2<T>*>(smem_raw);
  V2<T>* bufB = bufA + L * rs;
  const int h = blockIdx.y;
  const int64_t p0 = (int64_t)blockIdx.x << lc;
  const bool eq = a.nlat_odd && h == a.H - 1;
  const V2<T>* tw = stage_twiddles<T>(a.f, bufB + L * rs, tw_l);

  // Unfold, combine and entangle: thread -> (k <= L / 2, plane), which reads
  // the waist at orders k and L - k and forms Z[k] and Z[L - k] of every
  // output row: Z[k] = A + conj(C) + i conj(w_k) (A - conj(C)) with A = X[k],
  // C = X[L - k], and Z[L - k] from the same three (w_{L-k} = -conj(w_k)).
  {
    const int q = threadIdx.x & ((1 << lc) - 1), kstep = blockDim.x >> lc;
    const int64_t plane = min(p0 + q, a.planes - 1);  // past the end: transformed, not stored
    const V2<T>* P2 = reinterpret_cast<const V2<T>*>(wP) + (int64_t)h * a.ldc + plane * FW;
    const V2<T>* D2 = reinterpret_cast<const V2<T>*>(wD) + (int64_t)h * a.ldc + plane * FW;
    const int64_t dsd = (int64_t)a.H * a.ldc;  // S row -> D row of the same order
    const T inv_a = T(1.0 / a.radius);
    Reciprocal<T> over_a{}, ie[2]{};  // 1 / a, and 1 / (a cos phi) of the two sides
    if constexpr (NF == 2) over_a = reciprocal(T(a.radius));
    if constexpr (NF != 1) {
      ie[0] = reciprocal(T(a.radius) * T(coslat[h]));
      ie[1] = reciprocal(T(a.radius) * T(coslat[a.nlat - 1 - h]));
    }
    // x[o][sd]: order m of output field o on side sd
    auto order_values = [&](int m, V2<T>(&x)[NO][2]) {
      V2<T> S[NF], D[NF];
      const int64_t at = 2 * m * dsd;
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        const V2<T>* w = (NF == 1 || k < NF / 2 ? P2 : D2) + at + (NF == 4 ? (k & 1) : 0);
        S[k] = w[0];
        D[k] = w[dsd];
      }
      const T mf = T(m);
#pragma unroll
      for (int sd = 0; sd < 2; ++sd) {
        V2<T> v[NF];
#pragma unroll
        for (int k = 0; k < NF; ++k) v[k] = sd ? csub<T>(S[k], D[k]) : cadd<T>(S[k], D[k]);
        if constexpr (NF == 1) {
          x[0][sd] = a.zonal ? mk2<T>(-mf * v[0].y, mf * v[0].x) : v[0];
        } else if constexpr (NF == 2) {
          // east: i m P / (a cos phi); north: dP / a
          x[0][sd] = mk2<T>(times(-mf * v[0].y, ie[sd]), times(mf * v[0].x, ie[sd]));
          x[1][sd] = mk2<T>(times(v[1].x, over_a), times(v[1].y, over_a));
        } else {
          // v = {P psi, P chi, dP psi, dP chi}: u = -dpsi/a + i m chi/(a cos),
          // v = i m psi/(a cos) + dchi/a
          const T im = times(mf, ie[sd]);
          x[0][sd] = mk2<T>(-v[2].x * inv_a - im * v[1].y, -v[2].y * inv_a + im * v[1].x);
          x[1][sd] = mk2<T>(-im * v[0].y + v[3].x * inv_a, im * v[0].x + v[3].y * inv_a);
        }
      }
    };
    for (int k = threadIdx.x >> lc; 2 * k <= L; k += kstep) {
      const int kc = L - k;
      V2<T> A[NO][2], C[NO][2];
#pragma unroll
      for (int o = 0; o < NO; ++o)
        A[o][0] = A[o][1] = C[o][0] = C[o][1] = mk2<T>(T(0), T(0));
      if (k <= a.T) order_values(k, A);
      if (k > 0 && kc <= a.T) order_values(kc, C);
      if (k == 0) {  // irfft reads only the real part of order 0
#pragma unroll
        for (int o = 0; o < NO; ++o) A[o][0].y = A[o][1].y = T(0);
      }
      const V2<T> w = cconj<T>(tw_n[k]);  // exp(+2 pi i k / N)
#pragma unroll
      for (int o = 0; o < NO; ++o)
#pragma unroll
        for (int sd = 0; sd < 2; ++sd) {
          V2<T>* row = bufA + (((o * 2 + sd) << lc) + q);
          const V2<T> p = A[o][sd], c = C[o][sd];
          const V2<T> sm = mk2<T>(p.x + c.x, p.y - c.y), df = mk2<T>(p.x - c.x, p.y + c.y);
          const V2<T> t = cmul<T>(w, df);
          row[k * rs] = mk2<T>(sm.x - t.y, sm.y + t.x);
          if (k > 0 && kc != k) row[kc * rs] = mk2<T>(sm.x + t.y, t.x - sm.y);
        }
    }
  }
  __syncthreads();
  const V2<T>* Z = run_passes<T, true>(bufA, bufB, a.f, lr, tw);

  // Store: four neighbouring k of a row per quad of lanes, as the forward's loads.
  const int row = (threadIdx.x >> 2) & ((1 << lr) - 1);
  const int64_t plane = p0 + (row & ((1 << lc) - 1));
  const int side = (row >> lc) & 1, o = row >> (lc + 1);
  if (plane >= a.planes || (eq && side)) return;
  V2<T>* dst = reinterpret_cast<V2<T>*>(
      (o ? out1 : out0) + (plane * a.nlat + (side ? a.nlat - 1 - h : h)) * (int64_t)a.nlon);
  const int kstep = blockDim.x >> lr;
#pragma unroll 4
  for (int k = ((threadIdx.x >> (2 + lr)) << 2) + (threadIdx.x & 3); k < L; k += kstep)
    dst[k] = Z[k * rs + row];
}

__global__ void twiddle_kernel(int L, int N, double2* tl, double2* tn) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < L) {
    double s, c;
    sincospi(-2.0 * (double)k / (double)L, &s, &c);
    tl[k] = make_double2(c, s);
  }
  if (k <= L) {
    double s, c;
    sincospi(-2.0 * (double)k / (double)N, &s, &c);
    tn[k] = make_double2(c, s);
  }
}

__global__ void twiddle_cast_kernel(const double2* in, float2* out, int n) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) out[k] = make_float2((float)in[k].x, (float)in[k].y);
}

// [k1][lane] twiddles of the register kernels: exp(-2 pi i lane k1 / L), L = 32 F.
__global__ void lane_twiddle_kernel(const double2* tl, float2* out, int F) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < 32 * F) {
    const double2 w = tl[(e & 31) * (e >> 5) % (32 * F)];
    out[e] = make_float2((float)w.x, (float)w.y);
  }
}

// The radix sequence of length L: the fewest passes of radices 2 .. 16 (13
// and below the prime ones), and among those the smallest sum of radices
// (the widest passes); other primes by the direct pass.
std::vector<int> radix_plan(int L) {
  std::vector<int> rest;
  int r = L;
  for (int q = 2; r > 1 && q <= 13; ++q)
    while (r % q == 0) r /= q;
  const int smooth = L / r;
  for (int q = 17; r > 1; q += 2)
    while (r % q == 0) { rest.push_back(q); r /= q; }
  constexpr int kRadix[] = {16, 15, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};
  std::vector<int> best, now;
  auto sum = [](const std::vector<int>& v) { int s = 0; for (int x : v) s += x; return s; };
  auto walk = [&](auto&& self, int n, int most) -> void {
    if (n == 1) {
      if (best.empty() || now.size() < best.size() || (now.size() == best.size() && sum(now) < sum(best))) best = now;
      return;
    }
    if (!best.empty() && now.size() + 1 > best.size()) return;
    for (int q : kRadix)
      if (q <= most && n % q == 0) {
        now.push_back(q);
        self(self, n / q, q);
        now.pop_back();
      }
  };
  walk(walk, smooth, 16);
  best.insert(best.end(), rest.begin(), rest.end());
  return best;
}

// Columns of a CTA: as many as leave room for three CTAs per SM (two in FP64;
// two buffers of 2 no columns rows each), at most 8 (in FP32 64-byte pieces of
// every waist row) and no more than the call has; fewer when the launch would
// leave SMs without a CTA.
template <typename T>
FftShape make_shape(const sht_plan* p, int64_t cols, int no, size_t* smem, int* threads) {
  constexpr size_t kTarget = (sizeof(T) == 4 ? 74 : 100) * 1024, kMost = 227 * 1024;
  FftShape f{};
  f.L = p->L;
  f.npass = (int)p->radices.size();
  int Ns = 1;
  for (int i = 0; i < f.npass; ++i) {
    const int R = p->radices[i];
    f.pass[i] = {R, Ns, p->L / R, p->L / (Ns * R),
                 Ns > 1 ? (unsigned)(((uint64_t)1 << 32) / Ns + 1) : 0u};
    Ns *= R;
  }
  // FP32 rows of 16 (FP64: 8) and more fill a whole bank sweep per k: the
  // quad's four k of the load and store phases then fall on the same banks
  // unless the row stride is padded.
  constexpr int kSlots = sizeof(T) == 4 ? 16 : 8;
  auto stride = [&](int lc) {
    const int rows = (2 * no) << lc;
    return rows >= kSlots ? rows + kSlots / 4 : rows;
  };
  auto bytes = [&](int lc) { return (size_t)2 * stride(lc) * p->L * sizeof(V2<T>); };
  const size_t table = (size_t)p->L * sizeof(V2<T>);
  int lc = 0;
  while (lc < 3 && ((int64_t)1 << lc) < cols && bytes(lc + 1) + table <= kTarget) ++lc;
  while (lc > 0 && p->H * div_up(cols, (int64_t)1 << lc) < 2 * 148) --lc;  // two to an SM
  f.lc = lc;
  f.rs = stride(lc);
  f.tw_shared = bytes(lc) + table <= kMost ? 1 : 0;
  *smem = bytes(lc) + (f.tw_shared ? table : 0);
  // About eight elements per thread and pass; in FP64 (128 registers a thread:
  // 16 warps an SM) 256 threads only where shared memory leaves two CTAs (T62,
  // forward: 256 threads 25 us, 128 threads 20; T159 x 39 planes: 41 against 49).
  const int work = ((2 * no) << lc) * p->L;
  const int wide = sizeof(T) == 8 && 3 * (*smem + 1024) <= kMost ? 3072 : 1536;
  *threads = std::max(work >= wide ? 256 : (work >= 768 ? 128 : 64), 4 * ((2 * no) << lc));
  return f;
}

}  // namespace

void build_fft(sht_plan* p, cudaStream_t s) {
  const int L = p->L;
  p->radices = radix_plan(L);
  SHT_REQUIRE(p->radices.size() <= kMaxPass, "nlon has too many prime factors");
  p->fast_fft = fast_fft_supported(p) && !p->force_generic_fft;
  if (p->fast_fft) fast_fft_init_constants(s);

  double2 *tl = nullptr, *tn = nullptr;
  SHT_CUDA_OR_THROW(cudaMalloc(&tl, sizeof(double2) * L));
  SHT_CUDA_OR_THROW(cudaMalloc(&tn, sizeof(double2) * (L + 1)));
  twiddle_kernel<<<(L + 256) / 256, 256, 0, s>>>(L, p->nlon, tl, tn);
  SHT_CUDA_OR_THROW(cudaGetLastError());
  if (p->prec == SHT_PREC_F64) {
    p->tw_l = tl;
    p->tw_n = tn;
  } else {
    float2 *fl = nullptr, *fn = nullptr;
    SHT_CUDA_OR_THROW(cudaMalloc(&fl, sizeof(float2) * L));
    SHT_CUDA_OR_THROW(cudaMalloc(&fn, sizeof(float2) * (L + 1)));
    twiddle_cast_kernel<<<(L + 255) / 256, 256, 0, s>>>(tl, fl, L);
    twiddle_cast_kernel<<<(L + 256) / 256, 256, 0, s>>>(tn, fn, L + 1);
    if (fast_fft_supported(p)) {
      float2* lanes = nullptr;
      SHT_CUDA_OR_THROW(cudaMalloc(&lanes, sizeof(float2) * L));
      p->tw_lane = lanes;
      lane_twiddle_kernel<<<(L + 255) / 256, 256, 0, s>>>(tl, lanes, L / 32);
      SHT_CUDA_OR_THROW(cudaGetLastError());
    }
    SHT_CUDA_OR_THROW(cudaStreamSynchronize(s));
    cudaFree(tl);
    cudaFree(tn);
    p->tw_l = fl;
    p->tw_n = fn;
  }
}

template <typename T>
void launch_forward_fold(const sht_plan* p, const T* g0, const T* g1, int64_t planes,
                         int64_t ldc, T* wfold, cudaStream_t s, float* rowmax) {
  if constexpr (sizeof(T) == 4) {
    if (p->fast_fft) {
      fast_forward_fold(p, g0, g1, planes, ldc, wfold, s, rowmax);
      return;
    }
  }
  // g0 (and g1 for a stacked (u, v) pair) are (planes, nlat, nlon) grids.
  const int fields = g1 ? 2 : 1;
  size_t sm = 0;
  int threads = 0;
  const FftShape f = make_shape<T>(p, planes * fields, 1, &sm, &threads);
  const FoldArgs a{f, p->nlat, p->nlon, p->T, p->H, p->nlat_odd ? 1 : 0, fields, planes * fields, ldc};
  allow_shared((const void*)forward_fold_kernel<T>, sm);
  const dim3 grid((unsigned)div_up(a.cols, (int64_t)1 << f.lc), (unsigned)p->H);
  forward_fold_kernel<T><<<grid, threads, sm, s>>>(a, g0, g1 ? g1 : g0, (const V2<T>*)p->tw_l,
                                                   (const V2<T>*)p->tw_n, wfold, rowmax);
  SHT_CUDA_OR_THROW(cudaGetLastError());
}

template <typename T, int NF>
void launch_unfold(const sht_plan* p, int mode, const T* wP, const T* wD, int64_t planes,
                   int64_t ldc, T* out0, T* out1, cudaStream_t s) {
  size_t sm = 0;
  int threads = 0;
  const FftShape f = make_shape<T>(p, planes, NF == 1 ? 1 : 2, &sm, &threads);
  const UnfoldArgs a{f, p->nlat, p->nlon, p->T, p->H, p->nlat_odd ? 1 : 0,
                     mode == kUnfoldZonal ? 1 : 0, planes, ldc, p->radius};
  allow_shared((const void*)inverse_unfold_kernel<T, NF>, sm);
  const dim3 grid((unsigned)div_up(planes, (int64_t)1 << f.lc), (unsigned)p->H);
  inverse_unfold_kernel<T, NF><<<grid, threads, sm, s>>>(
      a, wP, wD ? wD : wP, p->d_coslat, (const V2<T>*)p->tw_l, (const V2<T>*)p->tw_n, out0,
      out1 ? out1 : out0);
  SHT_CUDA_OR_THROW(cudaGetLastError());
}

template <typename T>
void launch_inverse_unfold(const sht_plan* p, int mode, const T* wP, const T* wD,
                           int64_t planes, int64_t ldc, T* out0, T* out1, cudaStream_t s) {
  if constexpr (sizeof(T) == 4) {
    if (p->fast_fft) {
      fast_inverse_unfold(p, mode, wP, wD, planes, ldc, out0, out1, s);
      return;
    }
  }
  if (mode == kUnfoldWind)
    launch_unfold<T, 4>(p, mode, wP, wD, planes, ldc, out0, out1, s);
  else if (mode == kUnfoldGradient)
    launch_unfold<T, 2>(p, mode, wP, wD, planes, ldc, out0, out1, s);
  else
    launch_unfold<T, 1>(p, mode, wP, wD, planes, ldc, out0, out1, s);
}

template void launch_forward_fold<float>(const sht_plan*, const float*, const float*, int64_t, int64_t,
                                         float*, cudaStream_t, float*);
template void launch_forward_fold<double>(const sht_plan*, const double*, const double*, int64_t, int64_t,
                                          double*, cudaStream_t, float*);
template void launch_inverse_unfold<float>(const sht_plan*, int, const float*, const float*,
                                           int64_t, int64_t, float*, float*, cudaStream_t);
template void launch_inverse_unfold<double>(const sht_plan*, int, const double*, const double*,
                                            int64_t, int64_t, double*, double*, cudaStream_t);

}  // namespace sht
