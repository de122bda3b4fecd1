// The cluster-resident MGPCG (pfm_mgcluster.cu): plan types and host entry points.
#pragma once

#include "pfm_mg.cuh"

namespace pfm {

constexpr int kClusterThreads = 512;
// A cluster grows until its CTAs hold at most this many cells of the finest level (a vector of
// four cells of a colour for every fourth thread).  An iteration with 512 / 1024 / 2048 / 4096 cells per CTA takes
// 20.4 / 20.0 / 20.5 / 22.1 us at 64^2, 24.6 / 24.5 / 25.0 / 27.8 at 128^2, 20.1 / 21.3 / 21.6 / 24.6 at 16^3 and 30.1 /
// 30.0 / 29.9 / 32.9 at 32^3; larger grids fill 16 CTAs either way.
constexpr int kCellsPerCta = 1024;
// Levels of at most this many cells run on one CTA of a whole solve: with 1024 / 4096 / 16384 an iteration takes 33.5 /
// 33.4 / 44.6 us at 256^2, 57.0 / 56.6 / 91.2 at 512^2, 90.0 / 61.6 / 62.6 at 64^3 and 83.3 / 83.4 / 78.7 at 48^3.
constexpr int kSoloCells = 4096;

struct CLev {
  int n0, n1, nk;    // rows, middle extent (1 in 2D), last extent
  int half, hs;      // (nk + 1) / 2, and rounded up to a multiple of four: the stride of a row's colour
  int plane;         // n1 * hs: one colour of a row
  int rmax, shift;   // rows of the largest share; share boundaries are (c nbase / nc) << shift
  int cz, cr;        // elements per colour of z (a ghost row on either side, a zero pad) and of r
  Div32 dh, dhv, dh2, d1;  // divisors half, hs / 4, half / 2, n1
  unsigned z, r;     // byte offsets in shared memory
};

struct CPlan {
  int nc, L, l0, lg;  // CTAs; levels l0 .. lg-1 distributed, lg .. L-1 solo
  int ld, nbase;      // the level whose rows define the shares (the first solo level, else the last), its rows
  int pre_post, bottom;
  unsigned wait_ns;   // limit of a wait for other CTAs
  BC bc;
  CLev lv[kMaxLevels];
};

struct CSolve {
  const float* rhs;
  float *x, *p, *Ap, *b;
  SolveState* st;
  double tol, inv_n;
  float eps_s, eps_c, inv_n_s, inv_n_c;  // eps and 1 / cells as sums of two floats
  int tol_mode, max_iters, warm, true_every, keep_b, neu;
  unsigned rf;  // byte offset of the FP32 residual
};

// Whether a solve of this handle and these options runs as one cluster launch, and that launch: from
// the right-hand side in r_0 (and x, warm-started) of the workspace to x and the solve state.
bool cluster_solve_fits(const pfm_handle* h, const pfm_solve_opts& o);
[[nodiscard]] int cluster_solve_launch(pfm_handle* h, const pfm_solve_opts& o, cudaStream_t s);

// The first level (at least 1) from which a V-cycle runs as one cluster launch, or h->L; the launch.
int cluster_tail_level(const pfm_handle* h, int precision);
[[nodiscard]] int cluster_tail_launch(pfm_handle* h, int precision, int l0, void* z, const void* r,
                                      const SolveState* st, cudaStream_t s);

}  // namespace pfm
