// Definitions shared by the MGPCG translation units: levels, boundary flags, level storage, the
// 7- (5-) point stencil, compensated sums and the stopping rule.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "pfm_internal.cuh"

namespace pfm {

struct Lvl {
  int n0, n1, n2;
  int64_t count;
  Div32 d1, d2;  // divisors n1, n2
  Div32 dh;      // divisor (last extent + 1) / 2: the cell pairs of a smoothing sweep
};

static inline Lvl make_lvl(int n0, int n1, int n2, int D) {
  const int last = (D == 3) ? n2 : n1;
  return Lvl{n0, n1, n2, (int64_t)n0 * n1 * n2, make_div32((unsigned)n1), make_div32((unsigned)n2),
             make_div32((unsigned)((last + 1) >> 1))};
}

struct BC {
  int lo[3], hi[3];  // 2 = Neumann
};

static inline Lvl lvl_of(const pfm_handle* h, int l) {
  return make_lvl(h->lv[l].n[0], h->lv[l].n[1], h->lv[l].n[2], h->cfg.dim);
}

// Multigrid level storage: FP32 (the reference), or FP16 / BF16 in the mixed-precision solve;
// values are widened to FP32 on load and rounded to nearest on store.
__device__ __forceinline__ float ldv(const float* p) { return *p; }
__device__ __forceinline__ float ldv(const __half* p) { return __half2float(*p); }
__device__ __forceinline__ float ldv(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void stv(float* p, float v) { *p = v; }
__device__ __forceinline__ void stv(__half* p, float v) { *p = __float2half_rn(v); }
__device__ __forceinline__ void stv(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

// neighbor_sum / num_fluid_neighbors (3D/mgpcg.py:92-115)
template <int D, typename S>
__device__ __forceinline__ void stencil(const S* __restrict__ f, const Lvl& L, const BC& bc, int i, int j,
                                        int k, int64_t e, float& nb, float& mult) {
  float ret = 0.f;
  float num = 2.f * D;
  const int64_t sx = (int64_t)L.n1 * L.n2, sy = L.n2;
  if (i < L.n0 - 1) ret += ldv(f + e + sx);
  if (i > 0) ret += ldv(f + e - sx);
  if (D == 3) {
    if (j < L.n1 - 1) ret += ldv(f + e + sy);
    if (j > 0) ret += ldv(f + e - sy);
    if (k < L.n2 - 1) ret += ldv(f + e + 1);
    if (k > 0) ret += ldv(f + e - 1);
  } else {
    if (j < L.n1 - 1) ret += ldv(f + e + sy);
    if (j > 0) ret += ldv(f + e - sy);
  }
  if (i <= 0 && bc.lo[0] == 2) num -= 1.f;
  if (i >= L.n0 - 1 && bc.hi[0] == 2) num -= 1.f;
  if (j <= 0 && bc.lo[1] == 2) num -= 1.f;
  if (j >= L.n1 - 1 && bc.hi[1] == 2) num -= 1.f;
  if (D == 3) {
    if (k <= 0 && bc.lo[2] == 2) num -= 1.f;
    if (k >= L.n2 - 1 && bc.hi[2] == 2) num -= 1.f;
  }
  nb = ret;
  mult = num;
}

// num_fluid_neighbors alone (the mult of stencil<D>, no loads)
template <int D>
__device__ __forceinline__ float stencil_mult(const Lvl& L, const BC& bc, int i, int j, int k) {
  float num = 2.f * D;
  if (i <= 0 && bc.lo[0] == 2) num -= 1.f;
  if (i >= L.n0 - 1 && bc.hi[0] == 2) num -= 1.f;
  if (j <= 0 && bc.lo[1] == 2) num -= 1.f;
  if (j >= L.n1 - 1 && bc.hi[1] == 2) num -= 1.f;
  if (D == 3) {
    if (k <= 0 && bc.lo[2] == 2) num -= 1.f;
    if (k >= L.n2 - 1 && bc.hi[2] == 2) num -= 1.f;
  }
  return num;
}

__device__ __forceinline__ void decode(const Lvl& L, int64_t e, int& i, int& j, int& k) {
  split3((unsigned)e, L.d1, L.d2, i, j, k);
}

// GB300 issues one FP64 warp instruction per 16 cycles and SM, with 63 cycles of latency for an addition
// and 670 for a division, so the sums of f32 products in a cluster solve, a serial chain, are trees of f32 pairs
// (Knuth's TwoSum, about 48 bits; in FP64 an iteration took 26.3 us instead of 23.2 at 128 x 128, 35.5 instead of
// 31.0 at 256 x 256).  A sum of 1,024 to 262,144 squares differs from the FP64 sum by at most 5e-15 of itself; its
// error against 64 bits is the rounding of the f32 terms, 5e-10 to 8e-9, the same to three digits either way.
struct Pair {
  float s, c;
};

// s is the chain of plain additions, c collects their exact errors
__device__ __forceinline__ Pair pair_add(Pair a, Pair b) {
  const float t = a.s + b.s;
  const float bb = t - a.s;
  return Pair{t, ((a.s - (t - bb)) + (b.s - bb)) + (a.c + b.c)};
}

__device__ __forceinline__ double pair_value(Pair a) { return (double)a.s + (double)a.c; }
__device__ __forceinline__ Pair to_pair(double x) {
  const float s = (float)x;
  return Pair{s, (float)(x - (double)s)};
}

template <int WIDTH>
__device__ __forceinline__ Pair pair_reduce(Pair v) {
#pragma unroll
  for (int o = WIDTH / 2; o > 0; o >>= 1) {
    const Pair w{__shfl_xor_sync(0xffffffffu, v.s, o), __shfl_xor_sync(0xffffffffu, v.c, o)};
    v = pair_add(v, w);
  }
  return v;
}

// the stopping rule of k_update_xr / k_true_residual; the relative rules accept an exactly zero
// residual, so a zero right-hand side (a fluid at rest) ends at the first check
// (ref: the r.r or b.b that tol_mode 1 or 2 compares with)
__device__ __forceinline__ bool converged(double rTr, double ref, double tol, int tol_mode) {
  if (tol_mode == 0) return rTr < tol;
  return rTr == 0.0 || sqrt(rTr) < tol * sqrt(ref);
}
__device__ __forceinline__ bool converged(double rTr, const SolveState* st, double tol, int tol_mode) {
  return converged(rTr, tol_mode == 1 ? st->rTr0 : st->bTb, tol, tol_mode);
}

static inline BC bc_of(const pfm_handle* h) {
  BC b;
  for (int d = 0; d < 3; ++d) {
    b.lo[d] = (d < h->cfg.dim) ? h->cfg.boundary[d][0] : 2;
    b.hi[d] = (d < h->cfg.dim) ? h->cfg.boundary[d][1] : 2;
  }
  return b;
}

}  // namespace pfm
