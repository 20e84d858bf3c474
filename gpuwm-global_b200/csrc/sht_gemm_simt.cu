// Plain SIMT Legendre contraction (the FP32 FFMA path and the FP64 parity
// path): for every (order m, degree parity q) block, C[x][r] = sum_k
// Tab[k][x] * D[k][r], with the plane/component rows r innermost in both the
// data and the output.  One launch covers the whole triangle: the work list
// holds (block, x-tile) items sorted by descending cost, so the large low-m
// blocks start first and the ragged high-m tail fills in behind them; the row
// blocks (and the tables of a two-table call) of one item are neighbours in
// the grid, so its table and data tiles come from L2 after the first.  This
// replaces the reference's per-band dense strided-batched GEMMs
// (transform.py:1178-1274), which multiply the zeros above the triangle too.
#include <algorithm>
#include <type_traits>

#include "sht_plan.h"

namespace sht {
namespace {

// Tiles in units of V, the elements of 16 bytes (4 floats, 2 doubles).  A
// thread holds 2 V columns of the table x GN V data rows, a warp 4 x 8 such
// threads (8 V columns x 8 GN V rows), a CTA WX warps side by side.  The 16-byte
// pieces a thread owns are interleaved across its warp (piece g of lane l at
// (g * lanes + l) * V), so every shared load of a warp is one contiguous
// stretch.  Bound by the FMA pipe (62 / 70 % busy at T511, analysis /
// synthesis) and the shared loads that feed it (65 %): FP32 issues packed pairs
// (fma.rn.f32x2), which halves the issue slots of the multiply-adds, and 8 x 8
// outputs per thread leave 16 warps on an SM; 8 x 16 with 8 warps measured the
// same at T511 and 10 to 25 % slower at T255 and T126, where the chain per tile
// is short.  (The 128-wide FP32 tile spills 56 bytes a thread at its 128
// registers, the 64-wide one 24.)  Analysis + synthesis against one element per
// instruction in 128 x 128 tiles of 256 threads loaded through registers, by
// events around the launches: T511 x 200 planes 2716 -> 2002 us (40 TF/s), T255 x
// 161 planes 444 -> 278 us, T126 x 200 planes 103 -> 73 us.  Each output element is one chain of fused multiply-adds over
// ascending k from zero, whatever the tile, so every tile shape returns the
// same bits.
template <typename T> struct SimtCfg {
  static constexpr int V = 16 / (int)sizeof(T);
  static constexpr int BK = 16;  // contraction rows per stage
  static constexpr int S = 3;    // stages
  static constexpr int G = 2;    // row pieces per thread of a whole row block
};
// Columns of a CTA (WX = 2 or 4 warps) and rows of a row block (GN pieces).
template <typename T> constexpr int tile_x(int wx) { return 8 * SimtCfg<T>::V * wx; }
template <typename T> constexpr int tile_r(int gn) { return 8 * SimtCfg<T>::V * gn; }

// One table of a launch; the groups of a launch share the item list and R.
template <typename T> struct SimtGroup {
  const ShtGemmDesc* descs;
  const T* table;
  const T* data;
  T* out;
};
template <typename T> struct SimtArgs {
  SimtGroup<T> g[2];
  const ShtGemmItem* items;
  int ng;      // groups (1 or 2)
  int nrb;     // row blocks of tile_r(G)
  bool half;   // the last one holds at most tile_r(1) rows
  int64_t R;
  int Tn;          // truncation and planes of a spectral side taken in place
  int64_t planes;
};

template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, bool live) {
  const uint32_t n = live ? BYTES : 0;  // the rest of the piece is zero-filled
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// One CTA tile.  DB: bytes of a data-row copy, 16 where every data row starts
// on a 16-byte boundary and 8 otherwise (FP32 with an odd plane count, which only
// the static-scratch forward has: its fixed buffer holds the exact columns, and a
// padded one would refuse calls that fit).
template <typename T, int WX, int GN, int DB>
__device__ __forceinline__ void simt_tile(const SimtGroup<T>& G, const ShtGemmDesc& d, int x0,
                                          int64_t r0, int64_t R, T* smem) {
  constexpr int V = SimtCfg<T>::V, BK = SimtCfg<T>::BK, S = SimtCfg<T>::S;
  constexpr int BX = tile_x<T>(WX), BR = tile_r<T>(GN), NT = 32 * WX;
  const T* __restrict__ Tb = G.table + d.t_off;
  const T* __restrict__ Db = G.data + d.d_row * R;
  T* sA = smem;                // [S][BK][BX]
  T* sB = smem + S * BK * BX;  // [S][BK][BR]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lx = lane >> 3, lr = lane & 7;
  // A warp whose columns lie wholly past the problem (the ragged x tail of an
  // analysis block) skips its arithmetic.
  const bool busy = x0 + warp * 8 * V < d.X;

  auto load_stage = [&](int kt) {
    const int buf = kt % S, k0 = kt * BK;
    constexpr int AP = BX / V;  // pieces per table row
#pragma unroll
    for (int e = tid; e < BK * AP; e += NT) {
      const int k = e / AP, x = (e % AP) * V;
      const bool live = k0 + k < d.K && x0 + x < d.ldt;
      cp_async<16>((uint32_t)__cvta_generic_to_shared(sA + (buf * BK + k) * BX + x),
                   live ? Tb + (int64_t)(k0 + k) * d.ldt + x0 + x : Tb, live);
    }
    constexpr int DV = DB / (int)sizeof(T), BP = BR / DV;
#pragma unroll
    for (int e = tid; e < BK * BP; e += NT) {
      const int k = e / BP, r = (e % BP) * DV;
      const bool live = k0 + k < d.K && r0 + r < R;
      cp_async<DB>((uint32_t)__cvta_generic_to_shared(sB + (buf * BK + k) * BR + r),
                   live ? Db + (int64_t)(k0 + k) * R + r0 + r : Db, live);
    }
  };

  // FP32: acc[i][j] holds the pair of rows (2j, 2j + 1) of column i.
  using Acc = std::conditional_t<sizeof(T) == 4, float2, double>;
  constexpr int NJ = sizeof(T) == 4 ? GN * V / 2 : GN * V;
  Acc acc[2 * V][NJ];
#pragma unroll
  for (int i = 0; i < 2 * V; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      if constexpr (sizeof(T) == 4) acc[i][j] = make_float2(0.f, 0.f);
      else acc[i][j] = 0.0;
    }

  const int nk = (d.K + BK - 1) / BK;
#pragma unroll
  for (int kt = 0; kt < S - 1; ++kt) {
    if (kt < nk) load_stage(kt);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
    __syncthreads();  // stage kt has landed; every warp is done with stage kt - 1
    if (kt + S - 1 < nk) load_stage(kt + S - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (!busy) continue;
    const T* pa = sA + (kt % S) * BK * BX + warp * 8 * V + lx * V;
    const T* pb = sB + (kt % S) * BK * BR + lr * V;
#pragma unroll 8
    for (int kk = 0; kk < BK; ++kk) {
      if constexpr (sizeof(T) == 4) {
        float a[8];
        float2 b[NJ];
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const float4 v = *reinterpret_cast<const float4*>(pa + kk * BX + g * 4 * V);
          a[4 * g] = v.x; a[4 * g + 1] = v.y; a[4 * g + 2] = v.z; a[4 * g + 3] = v.w;
        }
#pragma unroll
        for (int g = 0; g < GN; ++g) {
          const float4 v = *reinterpret_cast<const float4*>(pb + kk * BR + g * 8 * V);
          b[2 * g] = make_float2(v.x, v.y);
          b[2 * g + 1] = make_float2(v.z, v.w);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < NJ; ++j) acc[i][j] = __ffma2_rn(make_float2(a[i], a[i]), b[j], acc[i][j]);
      } else {
        double a[4], b[NJ];
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const double2 v = *reinterpret_cast<const double2*>(pa + kk * BX + g * 4 * V);
          a[2 * g] = v.x; a[2 * g + 1] = v.y;
        }
#pragma unroll
        for (int g = 0; g < GN; ++g) {
          const double2 v = *reinterpret_cast<const double2*>(pb + kk * BR + g * 8 * V);
          b[2 * g] = v.x; b[2 * g + 1] = v.y;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < NJ; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");

  // Epilogue: C[x][r], r innermost, in pieces of 16 (or 8) bytes.
  if (!busy) return;
  T* __restrict__ Cb = G.out + d.c_row * R;
#pragma unroll
  for (int i = 0; i < 2 * V; ++i) {
    const int x = x0 + warp * 8 * V + (i / V) * 4 * V + lx * V + i % V;
    if (x >= d.X) continue;
    T* crow = Cb + (int64_t)x * R;
#pragma unroll
    for (int g = 0; g < GN; ++g) {
      const int64_t r = r0 + g * 8 * V + lr * V;
      if constexpr (sizeof(T) == 4) {
        const float2 u = acc[i][2 * g], w = acc[i][2 * g + 1];
        if constexpr (DB == 16) {
          if (r < R) *reinterpret_cast<float4*>(crow + r) = make_float4(u.x, u.y, w.x, w.y);
        } else {
          if (r < R) *reinterpret_cast<float2*>(crow + r) = u;
          if (r + 2 < R) *reinterpret_cast<float2*>(crow + r + 2) = w;
        }
      } else {
        if (r < R) *reinterpret_cast<double2*>(crow + r) = make_double2(acc[i][2 * g], acc[i][2 * g + 1]);
      }
    }
  }
}

// Block -> (item, row block, group), groups fastest.  A last row block at most
// half full runs with half the rows per thread.
template <typename T, int WX, int DB>
__global__ void __launch_bounds__(32 * WX, 16 / WX) gemm_simt_kernel(const __grid_constant__ SimtArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* smem = reinterpret_cast<T*>(smem_raw);
  constexpr int G = SimtCfg<T>::G;
  unsigned b = blockIdx.x;
  const SimtGroup<T>& grp = a.g[a.ng == 2 ? (b & 1) : 0];
  if (a.ng == 2) b >>= 1;
  const int rb = (int)(b % (unsigned)a.nrb);
  const ShtGemmItem it = a.items[b / (unsigned)a.nrb];
  const ShtGemmDesc d = grp.descs[it.problem];
  const int64_t r0 = (int64_t)rb * tile_r<T>(G);
  if (a.half && rb == a.nrb - 1)
    simt_tile<T, WX, 1, DB>(grp, d, it.x0, r0, a.R, smem);
  else
    simt_tile<T, WX, G, DB>(grp, d, it.x0, r0, a.R, smem);
}

// At most 8 data rows (one to four planes): bound by reading the table once and
// by the latency of the chain over k, so every lane takes one column (the most
// warps in flight) with U table rows on their way; the data values are one
// address for the whole warp.  The same chain of fused multiply-adds per output
// as the tiles, which keep more table rows in flight once a lane holds more than
// four FP32 sums; skinny_folded and simt_takes_coefficients draw the lines.
//
// The transforms' own calls take the spectral side in place, too: with CPACK the
// data rows are read from the coefficients [plane][n][m] (the pack pass's
// layout change is nothing for values that a whole warp shares), with CUNPACK
// the outputs go to them, real at m = 0, and the block of parity 0 zeroes its
// order above the triangle.  T21 x 1 plane FP32, the pair: 36.3 us with the two
// layout passes, 32.2 us without.
enum SkinnySpectral { kFolded = 0, kCPack = 1, kCUnpack = 2 };
template <typename T, int RR, int SPEC>
__global__ void __launch_bounds__(128) gemm_skinny_kernel(const __grid_constant__ SimtArgs<T> a) {
  constexpr int U = 16 * 4 / (RR * (int)sizeof(T) / 4);
  unsigned b = blockIdx.x;
  const SimtGroup<T>& grp = a.g[a.ng == 2 ? (b & 1) : 0];
  if (a.ng == 2) b >>= 1;
  const ShtGemmItem it = a.items[b];
  const ShtGemmDesc d = grp.descs[it.problem];
  const int R = (int)a.R;
  const int x = it.x0 + (int)threadIdx.x;
  using Q = std::conditional_t<sizeof(T) == 4, float2, double2>;  // two rows
  const int64_t t1 = a.Tn + 1;
  const int n0 = d.m + (it.problem & 1);  // degree of the problem's first coefficient
  if constexpr (SPEC == kCUnpack) {
    if ((it.problem & 1) == 0 && it.x0 == 0)
      for (int64_t p = 0; p < a.planes; ++p)
        for (int n = threadIdx.x; n < d.m; n += blockDim.x)
          reinterpret_cast<Q*>(grp.out)[(p * t1 + n) * t1 + d.m] = Q{};
  }
  if (x >= d.X) return;
  const T* tab = grp.table + d.t_off + x;
  const T* dat = grp.data + d.d_row * a.R;
  T acc[RR];
#pragma unroll
  for (int r = 0; r < RR; ++r) acc[r] = T(0);
  auto step = [&](int k, T t) {
    const Q* p = SPEC == kCPack
                     ? reinterpret_cast<const Q*>(grp.data) + (n0 + 2 * k) * t1 + d.m
                     : reinterpret_cast<const Q*>(dat + (int64_t)k * R);
    const int64_t ld = SPEC == kCPack ? t1 * t1 : 1;
#pragma unroll
    for (int r = 0; r < RR; r += 2)
      if (SPEC == kCPack ? r < 2 * a.planes : r < R) {
        const Q q = __ldg(p + r / 2 * ld);
        acc[r] = fma(t, q.x, acc[r]);
        acc[r + 1] = fma(t, q.y, acc[r + 1]);
      }
  };
  int k = 0;
  for (; k + U <= d.K; k += U) {
    T t[U];
#pragma unroll
    for (int u = 0; u < U; ++u) t[u] = __ldg(tab + (int64_t)(k + u) * d.ldt);
#pragma unroll
    for (int u = 0; u < U; ++u) step(k + u, t[u]);
  }
  for (; k < d.K; ++k) step(k, __ldg(tab + (int64_t)k * d.ldt));
#pragma unroll
  for (int r = 0; r < RR; r += 2) {
    Q q;
    q.x = acc[r];
    q.y = acc[r + 1];
    if constexpr (SPEC == kCUnpack) {
      if (d.m == 0) q.y = T(0);
      if (r < 2 * a.planes)
        reinterpret_cast<Q*>(grp.out)[(r / 2 * t1 + n0 + 2 * x) * t1 + d.m] = q;
    } else if (r < R) {
      *reinterpret_cast<Q*>(grp.out + (d.c_row + x) * a.R + r) = q;
    }
  }
}

}  // namespace

void build_gemm_items(sht_plan* p) {
  const int T = p->T;
  const int bx = p->prec == SHT_PREC_F64 ? tile_x<double>(4) : tile_x<float>(4);
  p->gemm_bx = bx;
  // Every (m, q) is a problem, including the empty parity-1 block of m = T:
  // its synthesis item has K = 0 and writes the zeros the inverse FFT reads
  // from that waist slot (nothing else writes it).  Empty analysis blocks
  // have X = 0 and produce no items.
  std::vector<int> probs;
  for (int m = 0; m <= T; ++m)
    for (int q = 0; q < 2; ++q) probs.push_back(m * 2 + q);
  p->n_problems = (int)probs.size();
  for (int f = 0; f < 2; ++f) {
    auto& syn = p->h_desc[0][f];
    auto& ana = p->h_desc[1][f];
    syn.clear();
    ana.clear();
    for (int idx : probs) {
      int m = idx / 2, q = idx % 2, s = q ^ f;
      ShtGemmDesc a{};
      a.t_off = p->syn_off[idx];
      a.ldt = p->Hx;
      a.X = p->H;
      a.K = p->e[idx];
      a.d_row = p->cf_row[idx];
      a.c_row = (int64_t)(m * 2 + s) * p->H;
      a.m = m;
      syn.push_back(a);
      ShtGemmDesc b{};
      b.t_off = p->ana_off[idx];
      b.ldt = p->ex[idx];
      b.X = p->e[idx];
      b.K = p->H;
      b.d_row = (int64_t)(m * 2 + s) * p->H;
      b.c_row = p->cf_row[idx];
      b.m = m;
      ana.push_back(b);
    }
  }
  // Item lists: (problem, x-tile) pairs sorted by descending cost, for the
  // plan's tile width and, on FP32 plans, for the narrow variant's.
  auto item_list = [&](int dir, int width, ShtGemmItem** dst, int* count) {
    std::vector<std::pair<int64_t, ShtGemmItem>> items;
    const auto& descs = p->h_desc[dir][0];
    for (int i = 0; i < (int)descs.size(); ++i) {
      const auto& d = descs[i];
      for (int x0 = 0; x0 < d.X; x0 += width) {
        int64_t cost = (int64_t)d.K * std::min(width, d.X - x0);
        items.push_back({cost, ShtGemmItem{i, x0}});
      }
    }
    std::stable_sort(items.begin(), items.end(),
                     [](const auto& a, const auto& b) { return a.first > b.first; });
    std::vector<ShtGemmItem> flat;
    for (auto& it : items) flat.push_back(it.second);
    *count = (int)flat.size();
    SHT_CUDA_OR_THROW(cudaMalloc(dst, sizeof(ShtGemmItem) * std::max<size_t>(flat.size(), 1)));
    upload_now(*dst, flat.data(), sizeof(ShtGemmItem) * flat.size());
  };
  for (int dir = 0; dir < 2; ++dir) {
    item_list(dir, bx, &p->d_items[dir], &p->n_items[dir]);
    if (p->prec != SHT_PREC_F64)
      item_list(dir, tile_x<float>(2), &p->d_items_narrow[dir], &p->n_items_narrow[dir]);
    for (int f = 0; f < 2; ++f) {
      auto& v = p->h_desc[dir][f];
      SHT_CUDA_OR_THROW(cudaMalloc(&p->d_desc[dir][f], sizeof(ShtGemmDesc) * std::max<size_t>(v.size(), 1)));
      upload_now(p->d_desc[dir][f], v.data(), sizeof(ShtGemmDesc) * v.size());
    }
  }
}

namespace {

template <typename T, int WX, int DB>
void launch_simt(const SimtArgs<T>& a, int n_items, cudaStream_t s) {
  using C = SimtCfg<T>;
  const size_t sm = sizeof(T) * C::S * C::BK * (tile_x<T>(WX) + tile_r<T>(C::G));
  const int64_t blocks = (int64_t)n_items * a.nrb * a.ng;
  SHT_REQUIRE(blocks < ((int64_t)1 << 31), "too many planes for one launch");
  allow_shared((const void*)gemm_simt_kernel<T, WX, DB>, sm);
  gemm_simt_kernel<T, WX, DB><<<(unsigned)blocks, 32 * WX, sm, s>>>(a);
  SHT_CUDA_OR_THROW(cudaGetLastError());
}

}  // namespace

namespace {

// Folded operands by the streaming kernel: four FP32 rows (one or two planes;
// one of a wind).  Forward and gradient of two planes, streaming and in tiles:
// T170 24.9 / 22.8 and 24.8 / 26.4 us, T255 34.9 / 37.1 and 35.9 / 45.5, T511
// 97 / 136 and 132 / 197.  Eight rows: T255 46 / 38 and 45 / 46, T511 215 / 138
// and 213 / 207; FP64 four rows: T126 (wind of one plane) 29.7 / 24.7, T255
// (forward of two planes) 58.8 / 42.5.
template <typename T>
constexpr bool skinny_folded(int64_t R) { return sizeof(T) == 4 && R <= 4; }

template <typename T, int SPEC>
void launch_skinny(const SimtArgs<T>& a, int n_items, cudaStream_t s) {
  const unsigned blocks = (unsigned)n_items * (unsigned)a.ng, threads = tile_x<T>(4);
  if (SPEC == kFolded || a.R <= 4)
    gemm_skinny_kernel<T, 4, SPEC><<<blocks, threads, 0, s>>>(a);
  else if constexpr (SPEC != kFolded)
    gemm_skinny_kernel<T, 8, SPEC><<<blocks, threads, 0, s>>>(a);
  SHT_CUDA_OR_THROW(cudaGetLastError());
}

}  // namespace

// In place while the chain is short: past these truncations the tiles with their
// layout passes are faster, for the two tables of a gradient a little later.
// Microseconds in place and in tiles, forward, inverse and gradient: FP32 two
// planes T126 19.6 / 19.6, 18.5 / 20.6 and 19.4 / 22.8; four planes T53 17.5 /
// 18.7, 16.4 / 17.7 and 18.6 / 21.9, T75 22.7 / 18.6, 18.5 / 17.6 and 21.4 / 21.7;
// FP64 two planes T75 18.5 / 18.4, 16.5 / 17.6 and 18.7 / 21.9, T106 21.6 / 18.6,
// 19.6 / 18.5 and 22.3 / 21.9; four planes T30 15.7 / 18.6, 16.4 / 17.7 and 18.8 /
// 21.9, T53 20.6 / 18.8, 20.6 / 17.9 and 20.6 / 22.0, T62 gradient 22.7 / 22.0.
bool simt_takes_coefficients(const sht_plan* p, int64_t R, int tables) {
  const bool f64 = p->prec == SHT_PREC_F64, two = tables == 2;
  if (R <= 4) return p->T < (f64 ? (two ? 100 : 80) : 128);
  return R <= 8 && p->T < (f64 ? (two ? 60 : 43) : (two ? 76 : 56));
}

template <typename T>
void launch_simt_from_coefficients(const sht_plan* p, int ngroups, const int* flip,
                                   const T* const* table, const T* coeff, int64_t planes,
                                   T* const* wfold, int64_t R, cudaStream_t s) {
  SimtArgs<T> a{};
  for (int g = 0; g < ngroups; ++g) a.g[g] = {p->d_desc[0][flip[g]], table[g], coeff, wfold[g]};
  a.items = p->d_items[0];
  a.ng = ngroups;
  a.R = R;
  a.Tn = p->T;
  a.planes = planes;
  launch_skinny<T, kCPack>(a, p->n_items[0], s);
}

template <typename T>
void launch_simt_to_coefficients(const sht_plan* p, const T* table, const T* wfold, T* coeff,
                                 int64_t planes, int64_t R, cudaStream_t s) {
  SimtArgs<T> a{};
  a.g[0] = {p->d_desc[1][0], table, wfold, coeff};
  a.items = p->d_items[1];
  a.ng = 1;
  a.R = R;
  a.Tn = p->T;
  a.planes = planes;
  launch_skinny<T, kCUnpack>(a, p->n_items[1], s);
}

template <typename T>
void launch_gemm_simt_groups(const sht_plan* p, int direction, int ngroups, const int* flip,
                             const T* const* table, const T* const* data, T* const* out,
                             int64_t R, cudaStream_t s) {
  // 64-wide tiles waste less of the ragged analysis blocks and hold twice as
  // many CTAs; from 256 latitude pairs on the 128-wide ones' fewer table and
  // data reloads make up for it (128 and 64 wide, us: T511 x 200 planes 2002 and
  // 2023, T341 x 100 planes 438 and 443; T255 x 161 planes 302 and 278, T126 x 200
  // planes 77 and 73).
  const bool narrow = std::is_same<T, float>::value &&
                      (p->tune_simt_tile == 1 || (p->tune_simt_tile == 0 && p->H < 256));
  const bool skinny = skinny_folded<T>(R);
  const int n_items = narrow && !skinny ? p->n_items_narrow[direction] : p->n_items[direction];
  if (n_items == 0 || R == 0) return;
  SHT_REQUIRE(ngroups == 1 || ngroups == 2, "one or two tables per SIMT launch");
  SHT_REQUIRE(p->gemm_bx == tile_x<T>(4), "SIMT work list built for another tile width");
  SimtArgs<T> a{};
  for (int g = 0; g < ngroups; ++g)
    a.g[g] = {p->d_desc[direction][flip[g]], table[g], data[g], out[g]};
  a.items = narrow && !skinny ? p->d_items_narrow[direction] : p->d_items[direction];
  SHT_REQUIRE(a.items != nullptr, "SIMT work list not built");
  a.ng = ngroups;
  a.R = R;
  if constexpr (sizeof(T) == 4) {
    if (skinny) {
      launch_skinny<T, kFolded>(a, n_items, s);
      return;
    }
  }
  const int whole = tile_r<T>(SimtCfg<T>::G);
  a.nrb = (int)div_up(R, whole);
  a.half = R % whole != 0 && R % whole <= whole / 2;
  if constexpr (std::is_same<T, float>::value) {
    const bool aligned = R % 4 == 0;
    if (narrow && aligned) launch_simt<T, 2, 16>(a, n_items, s);
    else if (narrow) launch_simt<T, 2, 8>(a, n_items, s);
    else if (aligned) launch_simt<T, 4, 16>(a, n_items, s);
    else launch_simt<T, 4, 8>(a, n_items, s);
  } else {
    launch_simt<T, 4, 16>(a, n_items, s);  // R is even: every data row is 16-byte aligned
  }
}

template <typename T>
void launch_gemm_simt(const sht_plan* p, int direction, int flip, const T* table, const T* data,
                      T* out, int64_t R, cudaStream_t s) {
  launch_gemm_simt_groups<T>(p, direction, 1, &flip, &table, &data, &out, R, s);
}

template void launch_gemm_simt<float>(const sht_plan*, int, int, const float*, const float*,
                                      float*, int64_t, cudaStream_t);
template void launch_gemm_simt<double>(const sht_plan*, int, int, const double*, const double*,
                                       double*, int64_t, cudaStream_t);
#define INST(T)                                                                                  \
  template void launch_simt_from_coefficients<T>(const sht_plan*, int, const int*,              \
                                                 const T* const*, const T*, int64_t, T* const*, \
                                                 int64_t, cudaStream_t);                        \
  template void launch_simt_to_coefficients<T>(const sht_plan*, const T*, const T*, T*, int64_t, \
                                               int64_t, cudaStream_t);
INST(float)
INST(double)
#undef INST
template void launch_gemm_simt_groups<float>(const sht_plan*, int, int, const int*,
                                             const float* const*, const float* const*,
                                             float* const*, int64_t, cudaStream_t);
template void launch_gemm_simt_groups<double>(const sht_plan*, int, int, const int*,
                                              const double* const*, const double* const*,
                                              double* const*, int64_t, cudaStream_t);

}  // namespace sht
