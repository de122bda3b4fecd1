// MGPCG on one thread-block cluster: small pressure solves whole, and the coarse part of large
// ones' V-cycles, in one launch.
//
// A solve of a few hundred thousand cells is a serial chain: at 256 x 256 one PCG iteration is 27
// kernels, 16 of them half-sweeps of 2-8 us of launch, drain and memory latency for well under 1 us
// of work.  Here the multigrid vectors of every level live in the shared memory of one cluster of up to
// 16 CTAs, a half-sweep ends with its edge rows' arrival in the neighbour's memory instead of a launch,
// and the iteration's scalars never leave the cluster.
//
//  * Rows (the first axis) of the distributed levels l0 .. lg-1 are split into contiguous shares, one
//    per CTA, nested so that a coarse row and its two fine rows have the same owner.  A share holds a
//    ghost row on either side; the owner of a boundary row stores it into its neighbour's ghost row
//    as well (distributed shared memory), so every stencil reads local memory.
//  * The levels from lg on (at most tail_cells cells) are solo: the first CTA runs them alone, FP32;
//    the rows it restricts from and prolongs to travel by st.async, and the others wait for theirs.
//  * A level's vectors are split by colour ([colour][row][middle][half of the last axis, rounded up to
//    four]): a thread updates four consecutive cells of a colour with 16-byte (8-byte) accesses, free of
//    bank conflicts.  The cells beyond the last axis stay zero.
//  * The division by the 1..6 fluid neighbours is the correctly rounded two-operation form for a
//    divisor known in advance (Brisebarre, Muller and Raina, "Accelerating correctly rounded
//    floating-point division when the divisor is known in advance", IEEE Trans. Computers 53(8),
//    2004): q = fma(x, zh, x zl) with zh = RN(1/m), zl = RN(1/m - zh).  For m = 1..6 it equals the
//    IEEE quotient for every significand (tests/test_mg_cluster.py checks all 2^23 on the CPU), so
//    every cell update is bitwise the grid-wide kernels' (below some 1e-30 the last bit may differ).
//
// The waits for other CTAs' rows and totals are mbarrier waits bounded in time; the others are hardware
// cluster or block barriers that all threads reach the same number of times.  A wait that gives up says so in
// every CTA's shared memory (Exchange::lost).  From then on totals, and what is decided on them, may differ
// between CTAs, so a CTA acts on a decision to end only behind one more cluster barrier: whatever each of them
// decided, they meet at that barrier, and behind it all see that a wait gave up before it and end together
// (pass_barrier).  A thread that has seen it neither pushes nor expects rows any more, and no CTA returns its
// shared memory before the rows in flight have landed (leave).
//
// Measured (one PCG iteration, FP32, GB300; against the grid-wide kernels of now): 128^2 89 -> 24 us, 256^2
// 111 -> 33 us, 512^2 141 -> 56 us, 32^3 91 -> 31 us, 64^3 125 -> 62 us; the coarse levels of 128^3 and 1024^2 as one
// launch: 190 -> 157 and 182 -> 132 us per iteration.  What bounds it: the chain of half-sweeps -- about 850 cycles each on the
// distributed levels (a row's flight through the cluster is some 400 of them), 60 to 200 on the solo ones.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "pfm_mg.cuh"
#include "pfm_mgcluster.cuh"
#include "pfm_tma.cuh"

namespace cg = cooperative_groups;

namespace pfm {

namespace {

constexpr int kT = kClusterThreads;

// ---------------------------------------------------------------------------------------------
// cluster barrier
// ---------------------------------------------------------------------------------------------
// cg::cluster_group::sync() releases in every warp, 600 cycles with 1024 threads and 475 with 512 on
// GB300; a block barrier, one releasing warp (its release covers what the block barrier ordered before it)
// and relaxed arrivals from the others do the same in less.
__device__ __forceinline__ void cluster_barrier() {
  __syncthreads();
  if (threadIdx.x < 32)
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  else
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <class T>
__device__ __forceinline__ T* remote(T* p, int rank) {
  return cg::this_cluster().map_shared_rank(p, rank);
}

// This CTA of the cluster: its share of the base rows (those of level ld, so that every distributed
// level restricts and prolongs within a share) is [b0, b1), the share above begins at up0.
struct Me {
  int rank, up0, b0, b1;
  unsigned limit;  // of a wait, in ns; 0: every wait gives up at once
  int passed;   // cluster barriers so far
  bool gone;    // this thread has seen that a wait gave up: it pushes and expects nothing any more
};

__device__ __forceinline__ Me who_am_i(const CPlan& P) {
  const int rank = (int)cg::this_cluster().block_rank();
  return Me{rank, (rank - 1) * P.nbase / P.nc, rank * P.nbase / P.nc, (rank + 1) * P.nbase / P.nc, P.wait_ns, 0, false};
}

struct Share {  // this CTA's rows of a level
  int lo, rows;
};

__device__ __forceinline__ Share share_of(const CLev& v, const Me& me) {
  return Share{me.b0 << v.shift, (me.b1 - me.b0) << v.shift};
}

// ---------------------------------------------------------------------------------------------
// vectors of V consecutive cells of one colour
// ---------------------------------------------------------------------------------------------
template <int V, typename F>
struct alignas(V * sizeof(F)) Vec {
  F e[V];
};

template <int V, typename F>
__device__ __forceinline__ void ldvec(const F* p, float (&f)[V]) {
  const Vec<V, F> u = *reinterpret_cast<const Vec<V, F>*>(p);
#pragma unroll
  for (int q = 0; q < V; ++q) f[q] = ldv(u.e + q);
}

template <int V, typename F>
__device__ __forceinline__ Vec<V, F> pack(const float (&f)[V]) {
  Vec<V, F> u;
#pragma unroll
  for (int q = 0; q < V; ++q) stv(u.e + q, f[q]);
  return u;
}

// x rounded to level storage R: what passes between a distributed and a solo level is stored in R by the
// grid-wide V-cycle, whose one-block tail is FP32 within
template <typename R>
__device__ __forceinline__ float through(float x) {
  R s;
  stv(&s, x);
  return ldv(&s);
}

// x / m for m = 1 .. 6 fluid neighbours (inv = (zh, zl); m = 0 gives x / 0)
__device__ __forceinline__ float div_n(float x, float2 inv) { return fmaf(x, inv.x, x * inv.y); }

// Fluid neighbours of a cell of row (i, j), the last axis aside.
template <int D>
__device__ __forceinline__ int row_neighbours(const CLev& v, const BC& bc, int i, int j) {
  int n = 2 * D;
  if (i == 0 && bc.lo[0] == 2) --n;
  if (i == v.n0 - 1 && bc.hi[0] == 2) --n;
  if (D == 3) {
    if (j == 0 && bc.lo[1] == 2) --n;
    if (j == v.n1 - 1 && bc.hi[1] == 2) --n;
  }
  return n;
}

template <int D>
__device__ __forceinline__ int cell_neighbours(const CLev& v, const BC& bc, int row_n, int k) {
  return row_n - ((k == 0 && bc.lo[D - 1] == 2) ? 1 : 0) - ((k == v.nk - 1 && bc.hi[D - 1] == 2) ? 1 : 0);
}

// Vector t of a colour's rows -> (row, middle, first half index); returns its first element.
template <int D>
__device__ __forceinline__ int split_vec(const CLev& v, int t, int& il, int& j, int& h) {
  const unsigned q = udiv((unsigned)t, v.dhv);
  h = (t - (int)q * (v.hs >> 2)) << 2;
  if (D == 3) {
    const unsigned i = udiv(q, v.d1);
    j = (int)(q - i * (unsigned)v.n1);
    il = (int)i;
  } else {
    j = 0;
    il = (int)q;
  }
  return (int)q * v.hs + h;
}

// Where a vector of four cells lies in a level, the same for both colours: its element and, in fl, the
// parity of i + j (bit 0), whether the middle axis goes on (1, 2: next, previous) and the row (3: after,
// 4: before the vector), the valid cells of the even (5-7) and of the odd colour (8-10), whether the
// row's last cell ends the grid in this vector (11), and the fluid neighbours of the row (12-).
struct Place {
  int e;
  unsigned fl;
};

template <int D>
__device__ __forceinline__ Place make_place(const CLev& v, const BC& bc, int lo, int t) {
  int il, j, h;
  Place x;
  x.e = split_vec<D>(v, t, il, j, h);
  const int i = lo + il;
  const int n0 = min(4, max(0, (v.nk - 2 * h + 1) >> 1)), n1 = min(4, max(0, (v.nk - 2 * h) >> 1));
  x.fl = ((unsigned)(i + j) & 1u) | (h + 4 < v.half ? 8u : 0u) | (h > 0 ? 16u : 0u) | ((unsigned)n0 << 5) |
         ((unsigned)n1 << 8) | (h + 4 >= v.half && h < v.half ? 2048u : 0u) |
         ((unsigned)row_neighbours<D>(v, bc, i, j) << 12);
  if (D == 3) x.fl |= (j < v.n1 - 1 ? 2u : 0u) | (j > 0 ? 4u : 0u);
  return x;
}

// The same unpacked: the elements of the neighbours across the middle axis and along the row (a missing
// one is the level's zero pad; the rows above and below always exist, as ghost rows that are zero
// outside the grid) and the reciprocals of the cells' fluid neighbours.
struct Spot {
  int e, jn, jp, left, right;
  unsigned fl;
  float2 inner, begin, end;
};

template <int D>
__device__ __forceinline__ Spot unpack(const CLev& v, const BC& bc, const float2* inv, Place x) {
  const int pad = (v.rmax + 1) * v.plane, n = (int)(x.fl >> 12);
  Spot s;
  s.e = x.e;
  s.fl = x.fl;
  s.jn = D == 3 && (x.fl & 2u) ? x.e + v.hs : pad;
  s.jp = D == 3 && (x.fl & 4u) ? x.e - v.hs : pad;
  s.right = x.fl & 8u ? x.e + 4 : pad;
  s.left = x.fl & 16u ? x.e - 1 : pad;
  s.inner = inv[n];
  s.begin = inv[n - (!(x.fl & 16u) && bc.lo[D - 1] == 2)];
  s.end = inv[n - (bc.hi[D - 1] == 2)];
  return s;
}

// Neighbour sums of the four cells of a spot whose last indices have parity a, from the other colour's
// array zo, in stencil<D>'s order (a missing neighbour adds zero).
template <int D, typename F>
__device__ __forceinline__ void neighbour_sums(const F* __restrict__ zo, int plane, const Spot& x, int a,
                                               float (&acc)[4]) {
  float f[4], g[4], k[4], m[4];
  ldvec<4>(zo + x.e + plane, acc);
  ldvec<4>(zo + x.e - plane, f);
  if (D == 3) {
    ldvec<4>(zo + x.jn, g);
    ldvec<4>(zo + x.jp, k);
  }
  ldvec<4>(zo + x.e, m);
  const float s = ldv(zo + (a ? x.right : x.left));
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    acc[q] += f[q];
    if (D == 3) {
      acc[q] += g[q];
      acc[q] += k[q];
    }
    acc[q] += a ? (q < 3 ? m[(q + 1) & 3] : s) : m[q];
    acc[q] += a ? m[q] : (q > 0 ? m[(q - 1) & 3] : s);
  }
}

// The new values of a spot's cells of colour `col`: (r + neighbour sum) / fluid neighbours; `fresh`: z is
// zero, no neighbour is read.
template <int D, typename F>
__device__ __forceinline__ void update_spot(const F* __restrict__ zo, const F* __restrict__ r, const CLev& v,
                                            const Spot& x, int col, bool fresh, float (&f)[4]) {
  const int a = (int)((x.fl ^ (unsigned)col) & 1u);
  const int valid = (int)(x.fl >> (a ? 8 : 5)) & 7;
  // the grid's last cell along the axis is the last valid one of its colour
  const int ends = (x.fl & 2048u) && a == 1 - (v.nk & 1) ? valid - 1 : -1;
  const bool begins = !(x.fl & 16u) && a == 0;
  float rr[4];
  ldvec<4>(r + x.e, rr);
  if (fresh) {
#pragma unroll
    for (int q = 0; q < 4; ++q) f[q] = 0.f;
  } else {
    neighbour_sums<D>(zo, v.plane, x, a, f);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float2 iv = q == 0 && begins ? x.begin : (q == ends ? x.end : x.inner);
    f[q] = q < valid ? div_n(rr[q] + f[q], iv) : 0.f;
  }
}

// ---------------------------------------------------------------------------------------------
// distributed half-sweeps
// ---------------------------------------------------------------------------------------------
// A boundary row goes into the neighbour's ghost row by st.async, whose bytes complete a transaction on
// the neighbour's mbarrier: a half-sweep waits for its two neighbours' rows only (a cluster barrier behind
// plain remote stores costs 700 cycles, mostly the release waiting for their acknowledgement).  Two
// mbarriers alternate: a neighbour can be at most one half-sweep ahead, since each needs the other's row.
// Ghost cells are read by the thread that then pushes the cell beside them, so a row that arrives a
// half-sweep early overwrites nothing that is still to be read: it has the colour not read.
struct Exchange {
  uint64_t full[2];  // in shared memory, one arrival (the expected bytes) per half-sweep
  uint64_t up, down;  // per V-cycle: the solo level's r is complete (rank 0); its z rows are here (the others)
  int lost;          // 0, or once a wait gave up 1 + the cluster barriers passed by then: later waits return at once
};

__device__ __forceinline__ uint32_t remote_addr(uint32_t local, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}

template <int BYTES>
__device__ __forceinline__ void push_async(uint32_t dst, const void* src, uint32_t bar) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(src);
  if constexpr (BYTES == 16)
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                     dst),
                 "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(bar)
                 : "memory");
  else if constexpr (BYTES == 8)
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "r"(w[0]), "r"(w[1]), "r"(bar)
                 : "memory");
  else
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst), "r"(w[0]),
                 "r"(bar)
                 : "memory");
}

// Waits for the phase of `bar` with the given parity; false (and me.gone) once a wait has given up.  This one does
// after me.limit and says so in every CTA's `lost`, which ends their waits and the solve.
__device__ __forceinline__ bool wait_rows(Exchange* x, uint64_t* bar, unsigned parity, Me& me) {
  if (me.gone) return false;
  if (me.limit && mbar_try_wait_cluster(bar, parity)) return true;
  const unsigned long long t0 = now_ns();
  while (!(me.limit && mbar_try_wait_cluster(bar, parity))) {
    me.gone = *(volatile int*)&x->lost != 0;
    if (!me.gone && (!me.limit || now_ns() - t0 > me.limit)) {
      const int n = (int)cg::this_cluster().num_blocks();
      for (int c = 0; c < n; ++c) *(volatile int*)remote(&x->lost, c) = me.passed + 1;
      me.gone = true;
    }
    if (me.gone) return false;
  }
  return true;
}

// A cluster barrier; true if a wait gave up before it -- the same answer in every thread of the cluster: what was
// written before the barrier is seen by all, and a wait that gives up behind it writes a larger number.
__device__ __forceinline__ bool pass_barrier(const Exchange* x, Me& me) {
  cluster_barrier();
  ++me.passed;
  const int lost = *(const volatile int*)&x->lost;
  return lost != 0 && lost <= me.passed;
}

// The end of a cluster in which a wait gave up, behind the barrier that said so: nobody pushes any more, and rows
// in flight land (in well under a microsecond) before any CTA gives its shared memory back.
__device__ __forceinline__ void leave() {
  const unsigned long long t0 = now_ns();
  while (now_ns() - t0 < 1000000) {
  }
  cluster_barrier();
}

// `half_sweeps` half-sweeps of a distributed level, colours `first`, 1 - first, ..; `fresh`: z starts at
// zero, so the first reads no neighbour.  `count` numbers the cluster's half-sweeps.  A thread with up to
// four vectors keeps their places in registers (64^3 on 16 CTAs has four).
template <int D, typename S>
__device__ __forceinline__ void sweeps_dist(const CPlan& P, const CLev& v, unsigned char* sm, const float2* inv,
                                            Exchange* ex, Me& me, int half_sweeps, int first, bool fresh,
                                            unsigned& count) {
  using VS = Vec<4, S>;
  const int lo = me.b0 << v.shift, rows = (me.b1 - me.b0) << v.shift;
  const int plane = v.plane, T = rows * plane / 4;
  S* z = reinterpret_cast<S*>(sm + v.z) + plane;  // this share's row 0 of colour 0
  const S* r = reinterpret_cast<const S*>(sm + v.r);
  if (*(volatile int*)&ex->lost) me.gone = true;
  bool up = me.rank > 0 && !me.gone, down = me.rank + 1 < P.nc && !me.gone;
  // element e of this share in the neighbours' ghost rows, of colour 0: its first row above, its last below
  const uint32_t zs = su32(z - plane);
  const uint32_t up_z =
      up ? remote_addr(zs, me.rank - 1) + (uint32_t)((((me.b0 - me.up0) << v.shift) + 1) * plane * (int)sizeof(S)) : 0u;
  const uint32_t dn_z = down ? remote_addr(zs, me.rank + 1) - (uint32_t)((rows - 1) * plane * (int)sizeof(S)) : 0u;
  const uint32_t bs = su32(&ex->full[0]);
  const uint32_t up_b = up ? remote_addr(bs, me.rank - 1) : 0u, dn_b = down ? remote_addr(bs, me.rank + 1) : 0u;
  unsigned expect = (unsigned)((up + down) * plane * (int)sizeof(S));
  const bool one = T <= kT, four = T <= 4 * kT;
  Spot mine{};
  Place at[4] = {};
  if (one) {
    if ((int)threadIdx.x < T) mine = unpack<D>(v, P.bc, inv, make_place<D>(v, P.bc, lo, threadIdx.x));
  } else if (four) {
#pragma unroll
    for (int m = 0; m < 4; ++m)
      if ((int)threadIdx.x + m * kT < T) at[m] = make_place<D>(v, P.bc, lo, threadIdx.x + m * kT);
  }
#pragma unroll 1
  for (int hs = 0; hs < half_sweeps; ++hs) {
    const int col = first ^ (hs & 1), which = (int)(count & 1u);
    const S* zo = z + (1 - col) * v.cz;
    S* zc = z + col * v.cz;
    const S* rc = r + col * v.cr;
    const uint32_t coff = (uint32_t)(col * v.cz * (int)sizeof(S));
    if (expect && threadIdx.x == 0) mbar_expect_tx(&ex->full[which], expect);
    auto update = [&](const Spot& x) {
      float f[4];
      update_spot<D>(zo, rc, v, x, col, fresh && hs == 0, f);
      const VS out = pack<4, S>(f);
      *reinterpret_cast<VS*>(zc + x.e) = out;
      const uint32_t off = coff + (uint32_t)(x.e * (int)sizeof(S));
      if (up && x.e < plane) push_async<sizeof(VS)>(up_z + off, &out, up_b + 8u * which);
      if (down && x.e >= (rows - 1) * plane) push_async<sizeof(VS)>(dn_z + off, &out, dn_b + 8u * which);
    };
    if (one) {
      if ((int)threadIdx.x < T) update(mine);
    } else if (four) {
#pragma unroll
      for (int m = 0; m < 4; ++m)
        if ((int)threadIdx.x + m * kT < T) update(unpack<D>(v, P.bc, inv, at[m]));
    } else {
#pragma unroll 1
      for (int t = threadIdx.x; t < T; t += kT) update(unpack<D>(v, P.bc, inv, make_place<D>(v, P.bc, lo, t)));
    }
    __syncthreads();
    if (expect && !wait_rows(ex, &ex->full[which], (count >> 1) & 1u, me)) {
      up = down = false;
      expect = 0;
    }
    ++count;
  }
}

// The half-sweeps of a solo level, on one CTA.  A level of at most one vector of a colour per thread is
// swept by just as many warps, so that the barrier between half-sweeps joins few of them.
template <int D>
__device__ __forceinline__ void sweeps_solo(const CLev& v, const BC& bc, float* z, const float* r, const float2* inv,
                                            int half_sweeps, int first, bool fresh) {
  const int T = v.n0 * v.plane / 4;
  float* z0 = z + v.plane;
  if (T <= kT) {
    const int nthr = (T + 31) & ~31;
    if ((int)threadIdx.x < nthr) {
      const bool have = (int)threadIdx.x < T;
      Spot x{};
      if (have) x = unpack<D>(v, bc, inv, make_place<D>(v, bc, 0, threadIdx.x));
#pragma unroll 1
      for (int hs = 0; hs < half_sweeps; hs += 2)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int col = first ^ c;
          if (have) {
            float f[4];
            update_spot<D>(z0 + (1 - col) * v.cz, r + col * v.cr, v, x, col, fresh && hs == 0 && c == 0, f);
            *reinterpret_cast<Vec<4, float>*>(z0 + col * v.cz + x.e) = pack<4, float>(f);
          }
          if (nthr == 32)
            __syncwarp();
          else
            asm volatile("bar.sync 1, %0;" ::"r"(nthr) : "memory");
        }
    }
    __syncthreads();
    return;
  }
#pragma unroll 1
  for (int hs = 0; hs < half_sweeps; ++hs) {
    const int col = first ^ (hs & 1);
#pragma unroll 1
    for (int t = threadIdx.x; t < T; t += kT) {
      const Spot x = unpack<D>(v, bc, inv, make_place<D>(v, bc, 0, t));
      float f[4];
      update_spot<D>(z0 + (1 - col) * v.cz, r + col * v.cr, v, x, col, fresh && hs == 0, f);
      *reinterpret_cast<Vec<4, float>*>(z0 + col * v.cz + x.e) = pack<4, float>(f);
    }
    __syncthreads();
  }
}

// The bottom's sweeps (from z = 0, colour 0 first) where a plane of cell pairs fits a warp -- in 2D the
// whole level, in 3D one i-plane per warp: the usual 8 x 8 and 8^3.  A lane holds the pair (2h, 2h + 1) of its
// row, one cell of either colour, in registers; the neighbours in the plane are its own other cell and three
// shuffles, those of the planes on either side come from z with one barrier of n0 warps per half-sweep.  A
// half-sweep is a chain of a shuffle (or load), the additions, the division and the barrier.
template <int D>
__device__ __forceinline__ bool fits_planes(const CLev& v) {
  return D == 3 ? v.n1 * v.half <= 32 && v.n0 * 32 <= kT : v.n0 * v.half <= 32;
}

template <int D>
__device__ __forceinline__ void sweeps_planes(const CLev& v, const BC& bc, float* z, const float* r, const float2* inv,
                                              int half_sweeps) {
  const int warps = D == 3 ? v.n0 : 1, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (w < warps) {
    const int rows = D == 3 ? v.n1 : v.n0;
    const bool have = lane < rows * v.half;
    const int y = have ? lane / v.half : 0, h = have ? lane - y * v.half : 0;
    const int i = D == 3 ? w : y, j = D == 3 ? y : 0;
    const int e = (D == 3 ? (i * v.n1 + j) : i) * v.hs + h;  // within a colour's rows
    const bool yn = have && y < rows - 1, yp = have && y > 0;
    float val[2] = {0.f, 0.f}, rr[2];
    float2 iv[2];
    bool cell[2], side[2];
    int src[2], par[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int a = (i + j + c) & 1, k = 2 * h + a;
      par[c] = a;
      cell[c] = have && k < v.nk;
      side[c] = cell[c] && (a ? k + 1 < v.nk : k > 0);
      src[c] = side[c] ? (a ? lane + 1 : lane - 1) : lane;
      rr[c] = cell[c] ? r[c * v.cr + e] : 0.f;
      iv[c] = cell[c] ? inv[cell_neighbours<D>(v, bc, row_neighbours<D>(v, bc, i, j), k)] : make_float2(1.f, 0.f);
    }
    float* z0 = z + v.plane;
#pragma unroll 1
    for (int hs = 0; hs < half_sweeps; hs += 2)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float o = val[1 - c];
        float above = 0.f, below = 0.f;
        if (D == 3 && !(hs == 0 && c == 0)) {
          const float* zo = z0 + (1 - c) * v.cz + e;
          above = zo[v.plane];
          below = zo[-v.plane];
        }
        float yn_ = __shfl_sync(0xffffffffu, o, lane + v.half), yp_ = __shfl_sync(0xffffffffu, o, lane - v.half);
        float sd = __shfl_sync(0xffffffffu, o, src[c]);
        yn_ = yn ? yn_ : 0.f;
        yp_ = yp ? yp_ : 0.f;
        sd = side[c] ? sd : 0.f;
        float s = 0.f;
        if (D == 3) {
          s += above;
          s += below;
        }
        s += yn_;
        s += yp_;
        s += par[c] ? sd : o;
        s += par[c] ? o : sd;
        val[c] = cell[c] ? div_n(rr[c] + s, iv[c]) : 0.f;
        if (D == 3) {
          if (have) z0[c * v.cz + e] = val[c];
          asm volatile("bar.sync 1, %0;" ::"r"(warps * 32) : "memory");
        }
      }
    if (D == 2 && have) {
      z0[e] = val[0];
      z0[v.cz + e] = val[1];
    }
  }
  __syncthreads();
}

// The restriction of the fine rows under the coarse rows [c_lo, c_lo + c_rows) into rc (its row 0 the
// coarse row c_base): restrict_blk's sums in its order, four coarse cells along the last axis at a time
// (the four cells of either colour of the fine rows under them).  zf, rf: the fine level's vectors with
// the fine row f_lo first (zf past its ghost row).  With `push` rc is that shared address of another CTA, and the
// cells go there by st.async on its `bar` (16 bytes per vector, the cells beyond the last axis included).
template <int D, typename R, typename F, typename C>
__device__ __forceinline__ void restrict_rows(const CLev& vf, const CLev& vc, const BC& bc, const F* __restrict__ zf,
                                              const F* __restrict__ rf, int f_lo, C* __restrict__ rc, int c_base,
                                              int c_lo, int c_rows, uint32_t push = 0, uint32_t bar = 0) {
  const int hv = vf.hs >> 2, T = c_rows * vc.n1 * hv, pad = (vf.rmax + 1) * vf.plane;
#pragma unroll 1
  for (int t = threadIdx.x; t < T; t += kT) {
    const unsigned q_ = udiv((unsigned)t, vf.dhv);
    const int K = (t - (int)q_ * hv) * 4;
    int il = (int)q_, J = 0;
    if (D == 3) {
      il = (int)udiv(q_, vc.d1);
      J = (int)q_ - il * vc.n1;
    }
    const int I = c_lo + il;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll(D == 3 ? 1 : 2)
    for (int ab = 0; ab < (D == 3 ? 4 : 2); ++ab) {
      const int i = 2 * I + (D == 3 ? ab >> 1 : ab), j = D == 3 ? 2 * J + (ab & 1) : 0;
      const int fc = (i + j) & 1;  // colour of the even cells (a = 0); the odd ones have the other
      const int rn = row_neighbours<D>(vf, bc, i, j);
      Spot x;
      x.e = (i - f_lo) * vf.plane + j * vf.hs + K;
      x.jn = D == 3 && j < vf.n1 - 1 ? x.e + vf.hs : pad;
      x.jp = D == 3 && j > 0 ? x.e - vf.hs : pad;
      x.left = K > 0 ? x.e - 1 : pad;
      x.right = K + 4 < vf.half ? x.e + 4 : pad;
      float n0[4], n1[4], z0[4], z1[4], r0[4], r1[4];
      neighbour_sums<D>(zf + (1 - fc) * vf.cz, vf.plane, x, 0, n0);
      neighbour_sums<D>(zf + fc * vf.cz, vf.plane, x, 1, n1);
      ldvec<4>(zf + fc * vf.cz + x.e, z0);
      ldvec<4>(zf + (1 - fc) * vf.cz + x.e, z1);
      ldvec<4>(rf + fc * vf.cr + x.e, r0);
      ldvec<4>(rf + (1 - fc) * vf.cr + x.e, r1);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int k = 2 * (K + q);
        const float m0 = (float)cell_neighbours<D>(vf, bc, rn, k), m1 = (float)cell_neighbours<D>(vf, bc, rn, k + 1);
        const float e0 = r0[q] - (m0 * z0[q] - n0[q]);
        acc[q] += e0 * 1.0f / ((float)D - 1.0f);
        const float e1 = r1[q] - (m1 * z1[q] - n1[q]);
        acc[q] += e1 * 1.0f / ((float)D - 1.0f);
      }
    }
    const int at = (I - c_base) * vc.plane + J * vc.hs;
    if (sizeof(C) == 4 && push) {
      const float even[2] = {through<R>(acc[0]), through<R>(acc[2])}, odd[2] = {through<R>(acc[1]), through<R>(acc[3])};
      const int c0 = (I + J) & 1;  // K is a multiple of 4
      push_async<8>(push + 4u * (uint32_t)(c0 * vc.cr + at + (K >> 1)), even, bar);
      push_async<8>(push + 4u * (uint32_t)((1 - c0) * vc.cr + at + (K >> 1)), odd, bar);
      continue;
    }
    C* dst = rc + at;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (K + q < vc.nk) stv(dst + ((I + J + K + q) & 1) * vc.cr + ((K + q) >> 1), through<R>(acc[q]));
  }
}

// z_l += z_{l+1}[I//2] on the fine rows [i0, i1) (row f_lo first in zf); zc holds the coarse row
// c_lo first.  Both cells of a pair (2h, 2h + 1) lie under the coarse cell h.  Of the rows outside [o0, o1), the
// ghost rows, only colour 0 is updated.
template <int D, typename R, typename F, typename C>
__device__ __forceinline__ void prolong_rows(const CLev& vf, const CLev& vc, F* __restrict__ zf, int f_lo, int i0,
                                             int i1, int o0, int o1, const C* __restrict__ zc, int c_lo) {
  const int T = (i1 - i0) * vf.plane / 4;
#pragma unroll 1
  for (int t = threadIdx.x; t < T; t += kT) {
    int il, j, h;
    split_vec<D>(vf, t, il, j, h);
    const int i = i0 + il, I = i >> 1, J = j >> 1;
    const C* src = zc + (I - c_lo) * vc.plane + J * vc.hs + (h >> 1);
    const int even = ((I + J) & 1) * vc.cz, odd = vc.cz - even;  // h is a multiple of 4
    float p[2], s[2];
    ldvec<2>(src + even, p);
    ldvec<2>(src + odd, s);
    const float add[4] = {p[0], s[0], p[1], s[1]};
    float f[4], g[4] = {0.f, 0.f, 0.f, 0.f};
    F* a = zf + (i - f_lo) * vf.plane + j * vf.hs + h;
    const bool own = i >= o0 && i < o1;
    ldvec<4>(a, f);
    if (own) ldvec<4>(a + vf.cz, g);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (h + q < vf.half) {
        f[q] += through<R>(add[q]);
        g[q] += through<R>(add[q]);
      }
    *reinterpret_cast<Vec<4, F>*>(a) = pack<4, F>(f);
    if (own) *reinterpret_cast<Vec<4, F>*>(a + vf.cz) = pack<4, F>(g);
  }
}

// The solo levels: one CTA, from r of level lg to its z.
template <int D>
__device__ __forceinline__ void solo_vcycle(const CPlan& P, unsigned char* sm, const float2* inv) {
  auto Z = [&](int l) { return reinterpret_cast<float*>(sm + P.lv[l].z); };
  auto R = [&](int l) { return reinterpret_cast<float*>(sm + P.lv[l].r); };
  // t = 0 .. n-1 pre-smooth and restrict, n the bottom, then up: one body for all three, so that the
  // sweeps are compiled once
  const int n = P.L - 1 - P.lg;
#pragma unroll 1
  for (int t = 0; t <= 2 * n; ++t) {
    const int l = P.lg + (t <= n ? t : 2 * n - t);
    const CLev v = P.lv[l];
    if (t > n) {
      const CLev c = P.lv[l + 1];
      prolong_rows<D, float, float, float>(v, c, Z(l) + v.plane, 0, 0, v.n0, 0, v.n0, Z(l + 1) + c.plane, 0);
      __syncthreads();
    }
    if (t == n && fits_planes<D>(v))
      sweeps_planes<D>(v, P.bc, Z(l), R(l), inv, 2 * P.bottom);
    else
      sweeps_solo<D>(v, P.bc, Z(l), R(l), inv, 2 * (t == n ? P.bottom : P.pre_post), t > n ? 1 : 0, t <= n);
    if (t < n) {
      const CLev c = P.lv[l + 1];
      restrict_rows<D, float, float, float>(v, c, P.bc, Z(l) + v.plane, R(l), 0, R(l + 1), 0, 0, c.n0);
      __syncthreads();
    }
  }
}

// The coarse rows under the fine rows [lo - 1, lo + rows] of a share (its own and the ghost rows inside the grid).
struct Under {
  int first, rows;
};
__device__ __forceinline__ Under rows_under(const CLev& v, int lo, int rows) {
  const int i0 = lo > 0 ? lo - 1 : 0, i1 = lo + rows < v.n0 ? lo + rows + 1 : v.n0;
  return Under{i0 >> 1, ((i1 - 1) >> 1) - (i0 >> 1) + 1};
}

// Rank 0's z of the solo level into the other CTAs, each the rows under its share, at their place in its own
// (otherwise unused) memory of that level: a warp per CTA.
__device__ __forceinline__ void push_solo(const CPlan& P, const CLev& v, const CLev& c, unsigned char* sm, Exchange* ex) {
  const int rank = (int)threadIdx.x >> 5;
  if (rank == 0 || rank >= P.nc) return;
  const int b0 = rank * P.nbase / P.nc, b1 = (rank + 1) * P.nbase / P.nc;
  const Under u = rows_under(v, b0 << v.shift, (b1 - b0) << v.shift);
  const float* z = reinterpret_cast<const float*>(sm + c.z);
  const uint32_t dst = remote_addr(su32(z), rank), bar = remote_addr(su32(&ex->down), rank);
  const int n = u.rows * c.plane, base = (u.first + 1) * c.plane;
  for (int e = (int)(threadIdx.x & 31) * 4; e < 2 * n; e += 128) {
    const int at = base + (e < n ? e : e - n + c.cz);
    const float4 q = *reinterpret_cast<const float4*>(z + at);
    push_async<16>(dst + 4u * (uint32_t)at, &q, bar);
  }
}

// apply_preconditioner (3D/mgpcg.py:182-200) from r of level l0 to its z.  Every thread of the
// cluster calls it; r of level l0 must be visible to its own CTA.  `cycles` numbers the calls.
// Between the distributed levels and the solo ones the rows travel by st.async, and a CTA waits for what it
// reads only (remote stores and loads between cluster barriers took 4400 cycles down and 5000 up at 64^2 solo
// cells; an iteration at 128^2 went from 26.0 to 23.1 us, at 32^3 from 32 to 28.4).  A ghost row takes its coarse rows in colour 0 only (the other is pushed by
// the first half-sweep up before anything reads it), so that no barrier parts the prolongation from that push.
template <int D, typename S>
__device__ __forceinline__ void cluster_vcycle(const CPlan& P, unsigned char* sm, const float2* inv, Exchange* ex,
                                               Me& me, unsigned& count, unsigned& cycles) {
  const int bottom = P.L - 1, n = (P.lg < P.L ? P.lg : bottom) - P.l0;  // distributed levels that restrict
  const unsigned parity = cycles++ & 1u;
  // down: t = 0 .. n-1; the solo levels or the distributed bottom: t = n; up: t = n+1 .. 2n
#pragma unroll 1
  for (int t = 0; t <= 2 * n; ++t) {
    if (t == n && P.lg < P.L) {
      if (me.rank == 0) {
        const CLev v = P.lv[P.lg - 1], c = P.lv[P.lg];
        if (threadIdx.x == 0 && !me.gone) mbar_expect_tx(&ex->up, (unsigned)(c.n0 * c.n1 * (v.hs >> 2) * 16));
        wait_rows(ex, &ex->up, parity, me);
        solo_vcycle<D>(P, sm, inv);
        if (!me.gone) push_solo(P, v, c, sm, ex);
      }
      continue;
    }
    const int l = P.l0 + (t <= n ? t : 2 * n - t);
    const CLev v = P.lv[l];  // in registers: an indexed parameter is a dependent load at every use
    const Share s = share_of(v, me);
    S* z = reinterpret_cast<S*>(sm + v.z) + v.plane;
    if (t > n) {
      const CLev c = P.lv[l + 1];
      const int i0 = s.lo > 0 ? s.lo - 1 : 0, i1 = s.lo + s.rows < v.n0 ? s.lo + s.rows + 1 : v.n0;
      if (l + 1 < P.lg) {
        prolong_rows<D, S, S, S>(v, c, z, s.lo, i0, i1, s.lo, s.lo + s.rows, reinterpret_cast<const S*>(sm + c.z) + c.plane,
                                 s.lo >> 1);
      } else {
        if (me.rank > 0) {
          if (threadIdx.x == 0 && !me.gone)
            mbar_expect_tx(&ex->down, (unsigned)(rows_under(v, s.lo, s.rows).rows * c.plane * 8));
          wait_rows(ex, &ex->down, parity, me);
        }
        prolong_rows<D, S, S, float>(v, c, z, s.lo, i0, i1, s.lo, s.lo + s.rows,
                                     reinterpret_cast<const float*>(sm + c.z) + c.plane, 0);
      }
      __syncthreads();
    }
    const int iters = t == n ? P.bottom : P.pre_post, first = t > n ? 1 : 0;
    sweeps_dist<D, S>(P, v, sm, inv, ex, me, 2 * iters, first, t <= n, count);
    if (t < n) {
      const CLev c = P.lv[l + 1];
      const S* r = reinterpret_cast<const S*>(sm + v.r);
      if (l + 1 < P.lg) {
        restrict_rows<D, S, S, S>(v, c, P.bc, z, r, s.lo, reinterpret_cast<S*>(sm + c.r), s.lo >> 1, s.lo >> 1,
                               s.rows >> 1);
        __syncthreads();
      } else {
        float* rc = reinterpret_cast<float*>(sm + c.r);
        // (a thread that pushes no more writes its own CTA's rows instead, which nothing reads)
        restrict_rows<D, S, S, float>(v, c, P.bc, z, r, s.lo, rc, 0, s.lo >> 1, s.rows >> 1,
                                   me.gone ? 0 : remote_addr(su32(rc), 0), remote_addr(su32(&ex->up), 0));
      }
    }
  }
}

__device__ __forceinline__ void fill_inverses(float2* inv) {
  if (threadIdx.x < 8) {
    const float m = (float)threadIdx.x;
    const float zh = threadIdx.x ? 1.f / m : __int_as_float(0x7f800000);
    // RN(1/m - zh): the residual 1 - m zh is exact in one FMA, and its quotient by m rounds once
    inv[threadIdx.x] = make_float2(zh, threadIdx.x ? fmaf(-m, zh, 1.f) / m : 0.f);
  }
}

__device__ __forceinline__ void init_exchange(Exchange* ex) {
  if (threadIdx.x == 0) {
    mbar_init(&ex->full[0], 1);
    mbar_init(&ex->full[1], 1);
    mbar_init(&ex->up, 1);
    mbar_init(&ex->down, 1);
    ex->lost = 0;
    fence_mbar_init();
  }
}

// What the sweeps rely on to be zero: the ghost rows outside the grid, the pad behind each colour, and
// the cells beyond the last axis.
template <typename S>
__device__ __forceinline__ void zero_z(const CPlan& P, const Me& me, unsigned char* sm) {
  for (int l = P.l0; l < P.L; ++l) {
    const CLev v = P.lv[l];
    const bool solo = l >= P.lg, all = 2 * v.hs != v.nk;
    const int rows = solo ? v.n0 : (me.b1 - me.b0) << v.shift;
    for (int e = threadIdx.x; e < 2 * v.cz; e += kT) {
      const int c = e >= v.cz ? 1 : 0, x = e - c * v.cz;
      const bool above = x < v.plane && (solo || me.rank == 0);
      const bool below = x >= (rows + 1) * v.plane && x < (rows + 2) * v.plane && (solo || me.rank + 1 == P.nc);
      if (!(all || above || below || x >= (v.rmax + 2) * v.plane)) continue;
      if (solo)
        reinterpret_cast<float*>(sm + v.z)[e] = 0.f;
      else
        stv(reinterpret_cast<S*>(sm + v.z) + e, 0.f);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// the coarse part of a large V-cycle: level l0's r from global memory, its z back
// ---------------------------------------------------------------------------------------------
template <int D, typename S>
__global__ void __launch_bounds__(kT, 1) k_cluster_tail(S* __restrict__ zg, const S* __restrict__ rg,
                                                        const __grid_constant__ CPlan P, SolveState* st) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ float2 inv[8];
  __shared__ Exchange ex;
  if (st && st->done) return;  // the same for the whole cluster
  Me me = who_am_i(P);
  unsigned count = 0, cycles = 0;
  init_exchange(&ex);
  fill_inverses(inv);
  zero_z<S>(P, me, sm);
  const CLev v = P.lv[P.l0];
  const Share s = share_of(v, me);
  S* r = reinterpret_cast<S*>(sm + v.r);
  const int T = s.rows * v.n1 * v.half;
  // pair t of this CTA's rows: its element, the global index of its even cell, that cell's colour
  auto pair_at = [&](int t, int& e, int64_t& g, int& c) {
    const unsigned q = udiv((unsigned)t, v.dh);
    const int h = t - (int)q * v.half, il = (int)udiv(q, v.d1), j = (int)q - il * v.n1;
    e = (int)q * v.hs + h;
    g = ((int64_t)(s.lo + il) * v.n1 + j) * v.nk + 2 * h;
    c = (s.lo + il + j) & 1;
    return 2 * h + 1 < v.nk;
  };
  for (int t = threadIdx.x; t < T; t += kT) {
    int e, c;
    int64_t g;
    const bool both = pair_at(t, e, g, c);
    r[c * v.cr + e] = rg[g];
    if (both) r[(1 - c) * v.cr + e] = rg[g + 1];
  }
  pass_barrier(&ex, me);  // every CTA of the cluster runs before the first remote store
  cluster_vcycle<D, S>(P, sm, inv, &ex, me, count, cycles);
  const S* z = reinterpret_cast<const S*>(sm + v.z) + v.plane;
  for (int t = threadIdx.x; t < T; t += kT) {
    int e, c;
    int64_t g;
    const bool both = pair_at(t, e, g, c);
    zg[g] = z[c * v.cz + e];
    if (both) zg[g + 1] = z[(1 - c) * v.cz + e];
  }
  if (pass_barrier(&ex, me)) {  // no CTA leaves while another may still write its shared memory
    if (threadIdx.x == 0 && st) atomicCAS(&st->done, 0, 4);
    leave();
  }
}

// ---------------------------------------------------------------------------------------------
// cluster-wide sums
// ---------------------------------------------------------------------------------------------
constexpr int kWarps = kT / 32;

struct ClusterRed {  // in shared memory
  Pair warp[2][kWarps];
  double part[kWarps * 8];
  Pair slot[2][2][16];  // [buffer][sum][rank]
  uint64_t full[2];     // the ranks' totals of a buffer have arrived
};

// The sum of r, for its mean: r's own mean was subtracted before, so the terms cancel to some 1e-11 of their
// magnitudes, and the 1e-15 that pairs lose would be 1e-4 of the mean.  A second compensation per thread and FP64
// above it keep what the grid-wide solve's FP64 sums keep.
struct WideSum {
  float s = 0.f, c = 0.f, d = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float t = s + x, e = (fabsf(s) >= fabsf(x)) ? ((s - t) + x) : ((x - t) + s);
    s = t;
    const float u = c + e;
    d += (fabsf(c) >= fabsf(e)) ? ((c - u) + e) : ((e - u) + c);
    c = u;
  }
  __device__ __forceinline__ double value() const { return (double)s + ((double)c + (double)d); }
};

__device__ __forceinline__ Pair bits_of(double x) {
  return Pair{__int_as_float(__double2loint(x)), __int_as_float(__double2hiint(x))};
}
__device__ __forceinline__ double of_bits(Pair p) {
  return __hiloint2double(__float_as_int(p.c), __float_as_int(p.s));
}

// The cluster's totals of the threads' sums: total[] of those in v times `unit` by trees of f32 pairs, and *mean of the wide one if
// there is one, in the calling CTA's first warp (the others' are undefined; the threads from `busy` on
// hold zero).  A non-finite term gives a non-finite total.  Every CTA sends its totals to every CTA with st.async;
// `uses` numbers the calls (two buffers alternate: a CTA is at most one call ahead).  The wide sum's tree stops at
// eight partial sums per warp, which the second warp adds up: an FP64 addition takes 16 cycles of the SM per warp.
template <int N>
__device__ __forceinline__ void cluster_sum(const CompSum (&v)[N], ClusterRed* red, Exchange* ex, int nc, Me& me,
                                            unsigned& uses, float unit, Pair (&total)[N], int busy = 0, const WideSum* wide = nullptr,
                                            double* mean = nullptr) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, buf = (int)(uses & 1u);
  const unsigned parity = (uses >> 1) & 1u;
  ++uses;
  auto push = [&](int n, Pair w) {
    if (lane < nc && !me.gone)
      push_async<8>(remote_addr(su32(&red->slot[buf][n][me.rank]), lane), &w, remote_addr(su32(&red->full[buf]), lane));
  };
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const Pair w = pair_reduce<32>(Pair{v[n].s * unit, v[n].c * unit});
    if (lane == 0) red->warp[n][wid] = w;
  }
  if (wide) {
    double w = 0.0;
    if (wid * 32 < busy) {
      w = wide->value();
      w += __shfl_xor_sync(0xffffffffu, w, 16);
      w += __shfl_xor_sync(0xffffffffu, w, 8);
    }
    if (lane < 8) red->part[wid * 8 + lane] = w;
  }
  __syncthreads();
  if (wide && wid == 1) {
    static_assert(kWarps == 16, "four partial sums per lane");
    const double* q = red->part + lane;
    double w = (q[0] + q[32]) + (q[64] + q[96]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    push(N, bits_of(w));
  }
  if (wid == 0) {
    if (lane == 0 && !me.gone) mbar_expect_tx(&red->full[buf], (unsigned)((N + (wide ? 1 : 0)) * nc * sizeof(Pair)));
#pragma unroll
    for (int n = 0; n < N; ++n) push(n, pair_reduce<kWarps>(red->warp[n][lane % kWarps]));
    wait_rows(ex, &red->full[buf], parity, me);
#pragma unroll
    for (int n = 0; n < N; ++n)
      total[n] = pair_reduce<16>((lane & 15) < nc ? red->slot[buf][n][lane & 15] : Pair{0.f, 0.f});
    if (wide) {
      double w = (lane & 15) < nc ? of_bits(red->slot[buf][N][lane & 15]) : 0.0;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
      *mean = w;
    }
  }
}

// a / (b + eps) in f32, from the pairs: the quotient of the leading parts corrected by its remainder
// (relative error about 2^-24, as the FP64 quotient rounded to f32; the FP64 division takes 670 cycles).
__device__ __forceinline__ float quotient(Pair a, Pair b, Pair eps) {
  const Pair d = pair_add(b, eps);
  const float ds = d.s + d.c, dc = d.c - (ds - d.s);
  const float q = a.s / ds;
  const float rem = fmaf(-q, ds, a.s) + fmaf(-q, dc, a.c);
  const float f = q + rem / ds;
  return isfinite(f) ? f : (float)(pair_value(a) / (pair_value(b) + pair_value(eps)));
}

struct Scalars {  // in shared memory: broadcast from thread 0 to its CTA, and thread 0's own
  float alpha, beta, mean, hscale, unit;
  int done, it, conv_it;
  Pair zTr_old, pAp, rTr, rTr0, bTb, rTr_true;
  float stop;  // a residual above this cannot meet the rule: `converged` is asked below it
};

// ---------------------------------------------------------------------------------------------
// the whole solve
// ---------------------------------------------------------------------------------------------
// The vectors x, p, A p and b stay in global memory (L2); four consecutive cells, two of either colour,
// are one 16-byte access.
template <int D, typename S>
__global__ void __launch_bounds__(kT, 1) k_cluster_solve(const __grid_constant__ CPlan P,
                                                         const __grid_constant__ CSolve A) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ float2 inv[8];
  __shared__ ClusterRed red;
  __shared__ Scalars sc;
  __shared__ Exchange ex;
  constexpr bool MIXED = sizeof(S) == 2;
  Me me = who_am_i(P);
  const int tid = threadIdx.x;
  unsigned count = 0, cycles = 0;
  init_exchange(&ex);
  fill_inverses(inv);
  zero_z<S>(P, me, sm);
  if (tid == 0) {
    mbar_init(&red.full[0], 1);
    mbar_init(&red.full[1], 1);
    fence_mbar_init();
    const Pair none{0.f, 0.f};
    sc = Scalars{0.f, 0.f, 0.f, 1.f, 1.f, 0, 0, 0, none, none, none, none, none, none, 0.f};
  }
  pass_barrier(&ex, me);  // every CTA of the cluster runs before the first remote store
  const CLev v = P.lv[0];
  const Share s = share_of(v, me);
  const int T = s.rows * v.n1 * (v.half / 2);  // groups of four cells (2h .. 2h + 3) of this CTA
  float* rf = reinterpret_cast<float*>(sm + A.rf);  // the FP32 residual, split by colour as r of level 0
  S* rl = reinterpret_cast<S*>(sm + v.r);
  const S* zl = reinterpret_cast<const S*>(sm + v.z) + v.plane;
  const int sx = v.n1 * v.nk, sy = v.nk;
  unsigned uses = 0;
  // The sums of products are held in units of 1 / unit: 1, or 2^60 where they could leave f32's range before
  // the f32 products do (all of them are compared with each other only, and with the tolerance and eps)
  float unit = 1.f;
  double back = 1.0;

  // f(element of the first pair, global index of the first cell, i, j, h, colour of the even cells)
  auto for_groups = [&](auto&& f) {
#pragma unroll 1
    for (int t = tid; t < T; t += kT) {
      int il, j, h;
      const unsigned q = udiv((unsigned)t, v.dh2);
      h = (t - (int)q * (v.half / 2)) * 2;
      il = (int)q;
      j = 0;
      if (D == 3) {
        il = (int)udiv(q, v.d1);
        j = (int)q - il * v.n1;
      }
      const int i = s.lo + il;
      f((int)q * v.hs + h, (i * v.n1 + j) * v.nk + 2 * h, i, j, h, (i + j) & 1);
    }
  };
  auto ld4f = [](const float* p) { return *reinterpret_cast<const float4*>(p); };
  // the four cells' values of a vector split by colour (c: colour of the even cells)
  auto get4 = [&](const float* a, int stride, int e, int c) {
    const float2 p = *reinterpret_cast<const float2*>(a + c * stride + e);
    const float2 q = *reinterpret_cast<const float2*>(a + (1 - c) * stride + e);
    return make_float4(p.x, q.x, p.y, q.y);
  };
  auto put4 = [&](float* a, int stride, int e, int c, float4 x) {
    *reinterpret_cast<float2*>(a + c * stride + e) = make_float2(x.x, x.z);
    *reinterpret_cast<float2*>(a + (1 - c) * stride + e) = make_float2(x.y, x.w);
  };
  auto get_z = [&](int e, int c) {
    float p[2], q[2];
    ldvec<2>(zl + c * v.cz + e, p);
    ldvec<2>(zl + (1 - c) * v.cz + e, q);
    return make_float4(p[0], q[0], p[1], q[1]);
  };
  auto put_storage = [&](int e, int c, float4 x) {  // the level-storage copy the V-cycle smooths against
    const float p[2] = {x.x, x.z}, q[2] = {x.y, x.w};
    *reinterpret_cast<Vec<2, S>*>(rl + c * v.cr + e) = pack<2, S>(p);
    *reinterpret_cast<Vec<2, S>*>(rl + (1 - c) * v.cr + e) = pack<2, S>(q);
  };
  auto add4 = [](auto& q, float4 x) {
    q.add(x.x);
    q.add(x.y);
    q.add(x.z);
    q.add(x.w);
  };
  // (A f) at four cells of a global field whose rows may belong to other CTAs: the rows above and
  // below come from L2, the CTA's own row from L1
  auto apply_A = [&](const float* f, int g, int i, int j, int h, float4 c) {
    const int k = 2 * h;
    float n[4] = {0.f, 0.f, 0.f, 0.f};
    auto acc = [&](float4 q) {
      n[0] += q.x;
      n[1] += q.y;
      n[2] += q.z;
      n[3] += q.w;
    };
    const float right = k + 4 < v.nk ? f[g + 4] : 0.f, left = k > 0 ? f[g - 1] : 0.f;
    if (i < v.n0 - 1) acc(__ldcg(reinterpret_cast<const float4*>(f + g + sx)));
    if (i > 0) acc(__ldcg(reinterpret_cast<const float4*>(f + g - sx)));
    if (D == 3) {
      if (j < v.n1 - 1) acc(ld4f(f + g + sy));
      if (j > 0) acc(ld4f(f + g - sy));
    }
    acc(make_float4(c.y, c.z, c.w, right));
    acc(make_float4(left, c.x, c.y, c.z));
    const int rn = row_neighbours<D>(v, P.bc, i, j);
    const float m = (float)rn;
    return make_float4((float)cell_neighbours<D>(v, P.bc, rn, k) * c.x - n[0], m * c.y - n[1], m * c.z - n[2],
                       (float)cell_neighbours<D>(v, P.bc, rn, k + 3) * c.w - n[3]);
  };
  auto scale_of = [&](Pair t) {
    if (unit != 1.f && t.s > 0.f) return (float)(1.0 / sqrt(pair_value(t) * back * A.inv_n));
    const float m = t.s * A.inv_n_s, mc = fmaf(t.s, A.inv_n_s, -m) + fmaf(t.s, A.inv_n_c, t.c * A.inv_n_s);
    if (!(t.s > 0.f)) return 1.f;
    if (!(m > 1e-30f && m < 1e30f)) return (float)(1.0 / sqrt(pair_value(t) * ((double)A.inv_n_s + (double)A.inv_n_c)));
    const float y = rsqrtf(m);
    const float my = m * y, myc = fmaf(m, y, -my) + mc * y;  // m y as a pair
    const float e = fmaf(-my, y, 1.f) - myc * y;             // 1 - m y y
    return fmaf(0.5f * y, e, y);
  };
  // |b - A x|^2 of the current x into thread 0's rTr_true; true if a wait gave up before
  auto true_residual = [&]() {
    if (pass_barrier(&ex, me)) return true;  // x of the neighbouring rows
    CompSum q;
    for_groups([&](int, int g, int i, int j, int h, int) {
      const float4 b = ld4f(A.b + g), a = apply_A(A.x, g, i, j, h, ld4f(A.x + g));
      const float4 d = make_float4(b.x - a.x, b.y - a.y, b.z - a.z, b.w - a.w);
      add4(q, make_float4(d.x * d.x, d.y * d.y, d.z * d.z, d.w * d.w));
    });
    Pair t[1];
    cluster_sum<1>({q}, &red, &ex, P.nc, me, uses, unit, t);
    if (tid == 0) sc.rTr_true = t[0];
    return false;
  };

  // ---- setup: r0, recenter, b, the warm start's residual, r0.r0
  {
    WideSum q;
    for_groups([&](int e, int g, int, int, int, int c) {
      const float4 b = ld4f(A.rhs + g);
      put4(rf, v.cr, e, c, b);
      add4(q, b);
      if (!A.warm) *reinterpret_cast<float4*>(A.x + g) = make_float4(0.f, 0.f, 0.f, 0.f);
    });
    if (A.neu) {
      Pair t[1];
      double sum;
      cluster_sum<1>({CompSum{}}, &red, &ex, P.nc, me, uses, unit, t, T, &q, &sum);
      if (tid == 0) sc.mean = (float)(sum * A.inv_n);
    }
    __syncthreads();
    const float mean = sc.mean;
    CompSum qb, qr;
    for_groups([&](int e, int g, int i, int j, int h, int c) {
      float4 r = get4(rf, v.cr, e, c);
      if (A.neu) r = make_float4(r.x - mean, r.y - mean, r.z - mean, r.w - mean);
      if (A.keep_b) {
        *reinterpret_cast<float4*>(A.b + g) = r;
        add4(qb, make_float4(r.x * r.x, r.y * r.y, r.z * r.z, r.w * r.w));
      }
      if (A.warm) {
        const float4 a = apply_A(A.x, g, i, j, h, ld4f(A.x + g));
        r = make_float4(r.x - a.x, r.y - a.y, r.z - a.z, r.w - a.w);
      }
      put4(rf, v.cr, e, c, r);
      add4(qr, make_float4(r.x * r.x, r.y * r.y, r.z * r.z, r.w * r.w));
    });
    Pair t[2];
#pragma unroll 1
    for (bool again = true; again;) {
      cluster_sum<2>({qr, qb}, &red, &ex, P.nc, me, uses, unit, t);
      if (tid == 0) sc.unit = unit == 1.f && !(t[0].s < 1e25f && t[1].s < 1e25f) ? 0x1p-60f : unit;
      __syncthreads();
      again = sc.unit != unit;
      unit = sc.unit;
    }
    back = unit == 1.f ? 1.0 : 0x1p60;
    if (tid == 0) {
      sc.rTr = sc.rTr0 = t[0];
      sc.bTb = A.keep_b ? t[1] : Pair{0.f, 0.f};
      sc.hscale = scale_of(t[0]);
      sc.stop = (float)(1.0001 * (A.tol_mode == 0 ? A.tol * unit
                                                  : A.tol * A.tol * pair_value(A.tol_mode == 1 ? sc.rTr0 : sc.bTb)));
    }
    __syncthreads();
    if (MIXED) {
      const float hs = sc.hscale;
      for_groups([&](int e, int, int, int, int, int c) {
        const float4 r = get4(rf, v.cr, e, c);
        put_storage(e, c, make_float4(r.x * hs, r.y * hs, r.z * hs, r.w * hs));
      });
      __syncthreads();
    }
  }

  bool first = true, lost = false;
#pragma unroll 1
  while (true) {
    // ---- V-cycle, z.r, beta, p
    cluster_vcycle<D, S>(P, sm, inv, &ex, me, count, cycles);
    {
      CompSum q;
      for_groups([&](int e, int, int, int, int, int c) {
        const float4 z = get_z(e, c), r = get4(rf, v.cr, e, c);
        add4(q, make_float4(z.x * r.x, z.y * r.y, z.z * r.z, z.w * r.w));
      });
      Pair t[1];
      cluster_sum<1>({q}, &red, &ex, P.nc, me, uses, unit, t);
      if (tid == 0) {
        // a 16-bit level vector answers the scaled residual
        Pair zTr = t[0];
        if (MIXED) {
          zTr.s = t[0].s / sc.hscale;
          zTr.c = (fmaf(-zTr.s, sc.hscale, t[0].s) + t[0].c) / sc.hscale;
        }
        if (first) {
          if (A.max_iters == 0) {
            sc.done = 2;
            sc.conv_it = 0;
          }
        } else {
          sc.beta = quotient(zTr, sc.zTr_old, Pair{A.eps_s * unit, A.eps_c * unit});
          sc.it += 1;
          if (sc.it >= A.max_iters) {
            sc.done = 2;
            sc.conv_it = sc.it;
          }
        }
        sc.zTr_old = zTr;
      }
      __syncthreads();
    }
    if (sc.done) break;
    {
      const float beta = sc.beta, us = MIXED ? 1.f / sc.hscale : 1.f;
      for_groups([&](int e, int g, int, int, int, int c) {
        float4 z = get_z(e, c);
        const float4 p = first ? make_float4(0.f, 0.f, 0.f, 0.f) : ld4f(A.p + g);
        auto step = [&](float zz, float pp) { return MIXED ? zz * us + beta * pp : zz + beta * pp; };
        z = make_float4(step(z.x, p.x), step(z.y, p.y), step(z.z, p.z), step(z.w, p.w));
        *reinterpret_cast<float4*>(A.p + g) = z;
      });
      first = false;
      lost = pass_barrier(&ex, me);  // p of the neighbouring rows
    }
    if (lost) break;
    // ---- A p, alpha, x and r, r.r, the stop test
    {
      CompSum q;
      for_groups([&](int, int g, int i, int j, int h, int) {
        const float4 p = ld4f(A.p + g), a = apply_A(A.p, g, i, j, h, p);
        *reinterpret_cast<float4*>(A.Ap + g) = a;
        add4(q, make_float4(p.x * a.x, p.y * a.y, p.z * a.z, p.w * a.w));
      });
      Pair t[1];
      cluster_sum<1>({q}, &red, &ex, P.nc, me, uses, unit, t);
      if (tid == 0) {
        sc.pAp = t[0];
        sc.alpha = quotient(sc.zTr_old, t[0], Pair{A.eps_s * unit, A.eps_c * unit});
      }
      __syncthreads();
    }
    {
      const float alpha = sc.alpha;
      CompSum qr;
      WideSum qm;
      for_groups([&](int e, int g, int, int, int, int c) {
        const float4 x = ld4f(A.x + g), p = ld4f(A.p + g), a = ld4f(A.Ap + g);
        float4 r = get4(rf, v.cr, e, c);
        *reinterpret_cast<float4*>(A.x + g) =
            make_float4(x.x + alpha * p.x, x.y + alpha * p.y, x.z + alpha * p.z, x.w + alpha * p.w);
        r = make_float4(r.x - alpha * a.x, r.y - alpha * a.y, r.z - alpha * a.z, r.w - alpha * a.w);
        put4(rf, v.cr, e, c, r);
        add4(qr, make_float4(r.x * r.x, r.y * r.y, r.z * r.z, r.w * r.w));
        add4(qm, r);
      });
      Pair t[1];
      double sum;
      cluster_sum<1>({qr}, &red, &ex, P.nc, me, uses, unit, t, T, &qm, &sum);
      if (tid == 0) {
        sc.rTr = t[0];
        if (A.neu) sc.mean = (float)(sum * A.inv_n);
        if (MIXED && t[0].s > 0.f) sc.hscale = scale_of(t[0]);
        if (!isfinite(t[0].s + t[0].c)) {
          sc.done = 3;
          sc.conv_it = sc.it;
        } else if (!(t[0].s > sc.stop) &&
                   converged(pair_value(t[0]) * back, pair_value(A.tol_mode == 1 ? sc.rTr0 : sc.bTb) * back, A.tol, A.tol_mode)) {
          sc.done = 1;
          sc.conv_it = sc.it;
        }
      }
      __syncthreads();
    }
    if (A.true_every > 0 && !sc.done && (sc.it + 1) % A.true_every == 0) lost = true_residual();
    if (lost || sc.done) break;
    // ---- recenter, the level-storage copy
    if (A.neu || MIXED) {
      const float mean = sc.mean, hs = sc.hscale;
      for_groups([&](int e, int, int, int, int, int c) {
        float4 r = get4(rf, v.cr, e, c);
        if (A.neu) {
          r = make_float4(r.x - mean, r.y - mean, r.z - mean, r.w - mean);
          put4(rf, v.cr, e, c, r);
        }
        if (MIXED) put_storage(e, c, make_float4(r.x * hs, r.y * hs, r.z * hs, r.w * hs));
      });
      __syncthreads();
    }
  }
  // behind this barrier the end is agreed; then no CTA leaves while another may still write its shared memory
  if (!lost) lost = pass_barrier(&ex, me);
  if (!lost && A.true_every > 0) lost = true_residual() || pass_barrier(&ex, me);
  if (me.rank == 0 && tid == 0) {
    SolveState* st = A.st;
    st->zTr_old = pair_value(sc.zTr_old) * back;
    st->pAp = pair_value(sc.pAp) * back;
    st->rTr = pair_value(sc.rTr) * back;
    st->rTr0 = pair_value(sc.rTr0) * back;
    st->bTb = pair_value(sc.bTb) * back;
    st->rTr_true = pair_value(sc.rTr_true) * back;
    st->sum = 0.0;
    st->alpha = sc.alpha;
    st->beta = sc.beta;
    st->mean = sc.mean;
    st->hscale = sc.hscale;
    st->it = sc.it;
    st->done = lost ? 4 : sc.done;
    st->conv_it = sc.conv_it;
    st->ticket = 0u;
    st->it_stop = sc.it;
  }
  if (lost) leave();
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
constexpr size_t kMaxSmem = 227 * 1024 - 4096;  // dynamic; the static part is under 4 KB
constexpr int kMaxCluster = 16;

// Largest cluster (16 or 8 CTAs) that this device co-schedules with full shared memory.
template <class K>
int max_cluster(K* kernel, std::atomic<unsigned long long>& known16, std::atomic<unsigned long long>& known8) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (bit && (known16.load() & bit)) return 16;
  if (bit && (known8.load() & bit)) return 8;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem) != cudaSuccess ||
      cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  int found = 1;
  for (int nc = kMaxCluster; nc >= 8; nc /= 2) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(nc);
    cfg.blockDim = dim3(kT);
    cfg.dynamicSmemBytes = kMaxSmem;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = nc;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0) {
      found = nc;
      break;
    }
    cudaGetLastError();
  }
  if (bit && found == 16) known16.fetch_or(bit);
  if (bit && found == 8) known8.fetch_or(bit);
  return found;
}

template <class K, class... Args>
int launch_cluster(pfm_handle* h, K* kernel, int nc, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nc);
  cfg.blockDim = dim3(kT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = nc;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  h->launches++;
  return check_cuda(h, cudaLaunchKernelEx(&cfg, kernel, args...), "cluster launch");
}

size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }

// Lays the levels l0 .. L-1 out for clusters of nc CTAs with levels below lg distributed in elements
// of `esz` bytes (whole: with the FP32 residual of level 0 beside 16-bit levels).  Returns the shared memory.
size_t layout(const pfm_handle* h, CPlan& P, int esz, bool whole, unsigned* rf) {
  const int D = h->cfg.dim;
  size_t off = 0;
  for (int l = P.l0; l < P.L; ++l) {
    CLev& v = P.lv[l];
    v.n0 = h->lv[l].n[0];
    v.n1 = D == 3 ? h->lv[l].n[1] : 1;
    v.nk = D == 3 ? h->lv[l].n[2] : h->lv[l].n[1];
    v.half = (v.nk + 1) / 2;
    v.hs = (v.half + 3) / 4 * 4;
    v.plane = v.n1 * v.hs;
    v.dh = make_div32((unsigned)v.half);
    v.dhv = make_div32((unsigned)(v.hs / 4));
    v.dh2 = make_div32((unsigned)(v.half >= 2 ? v.half / 2 : 1));
    v.d1 = make_div32((unsigned)v.n1);
    const bool dist = l < P.lg;
    v.shift = dist ? P.ld - l : 0;
    const int share = (P.nbase + P.nc - 1) / P.nc;
    v.rmax = dist ? share << v.shift : v.n0;
    v.cz = (v.rmax + 2) * v.plane + 4;  // and a zero pad
    v.cr = v.rmax * v.plane;
    const size_t e = dist ? (size_t)esz : 4;
    v.z = (unsigned)off;
    off = align16(off + 2 * (size_t)v.cz * e);
    v.r = (unsigned)off;
    off = align16(off + 2 * (size_t)v.cr * e);
  }
  if (whole && rf) {
    if (esz == 4) {
      *rf = P.lv[0].r;
    } else {
      *rf = (unsigned)off;
      off = align16(off + 2 * (size_t)P.lv[0].cr * 4);
    }
  }
  return off;
}

// CTAs of a cluster for a finest level of `cells` cells, by size alone.
int cluster_size(int64_t cells) {
  int nc = 1;
  while (nc < kMaxCluster && (int64_t)nc * kCellsPerCta < cells) nc *= 2;
  return nc;
}

// Whether the levels from l0 on halve exactly, down to at least two cells along the last axis.
bool halves(const pfm_handle* h, int l0) {
  if (h->lv[h->L - 1].n[h->cfg.dim - 1] < 2) return false;
  for (int l = l0; l + 1 < h->L; ++l)
    for (int a = 0; a < h->cfg.dim; ++a)
      if (h->lv[l].n[a] != 2 * h->lv[l + 1].n[a]) return false;
  return true;
}

// The cluster plan of the levels from l0 on, or false where they do not fit or do not halve exactly.
// A whole solve's plan depends on the grid alone.
bool make_plan(const pfm_handle* h, int l0, int esz, bool whole, int max_nc, CPlan& P, unsigned* rf, size_t* smem) {
  const int D = h->cfg.dim, L = h->L;
  if (l0 >= L - 1 || !halves(h, l0)) return false;
  auto first_below = [&](int cells) {
    int l = l0;
    while (l < L - 1 && h->lv[l].count > cells) ++l;
    return l;
  };
  P = CPlan{};
  P.L = L;
  P.l0 = l0;
  P.bc = bc_of(h);
  P.pre_post = h->cfg.pre_post_smoothing;
  P.bottom = h->cfg.bottom_smoothing;
  P.wait_ns = (unsigned)h->cluster_wait_us * 1000u;
  if (whole) {
    if ((D == 3 ? h->lv[0].n[2] : h->lv[0].n[1]) % 4 != 0) return false;  // 16-byte groups of cells
    P.lg = std::max(l0 + 1, first_below(kSoloCells));
  } else {  // the solo levels are the tail levels of the grid-wide V-cycle (FP32 in both), if it has any
    P.lg = first_below(h->tail_cells);
    if (h->lv[P.lg].count > h->tail_cells) P.lg = L;
    if (P.lg <= l0) return false;
  }
  P.ld = std::min(P.lg, L - 1);
  P.nbase = h->lv[P.ld].n[0];
  // one CTA per kCellsPerCta cells of the finest level, as many as the rows allow
  int nc = std::min(cluster_size(h->lv[l0].count), max_nc);
  while (nc > P.nbase) nc /= 2;
  for (;; nc *= 2) {
    P.nc = nc;
    *smem = layout(h, P, esz, whole, rf);
    if (*smem <= kMaxSmem) return true;
    if (2 * nc > max_nc || 2 * nc > P.nbase) return false;
  }
}

template <int D, typename S>
int max_cluster_of(bool whole) {
  static std::atomic<unsigned long long> s16{0}, s8{0}, t16{0}, t8{0};
  return whole ? max_cluster(k_cluster_solve<D, S>, s16, s8) : max_cluster(k_cluster_tail<D, S>, t16, t8);
}

template <class F>
int by_type(const pfm_handle* h, int precision, F&& f) {
  if (h->cfg.dim == 3) {
    if (precision == 1) return f(std::integral_constant<int, 3>(), __half());
    if (precision == 2) return f(std::integral_constant<int, 3>(), __nv_bfloat16());
    return f(std::integral_constant<int, 3>(), float());
  }
  if (precision == 1) return f(std::integral_constant<int, 2>(), __half());
  if (precision == 2) return f(std::integral_constant<int, 2>(), __nv_bfloat16());
  return f(std::integral_constant<int, 2>(), float());
}

}  // namespace

bool cluster_solve_fits(const pfm_handle* h, const pfm_solve_opts& o) {
  if (!h->mg_cluster || o.max_iters < 0) return false;
  // a 16-bit level 0 that the one-block tail takes whole is FP32 there: left to it
  if (o.precision != 0 && h->lv[0].count <= kSoloCells) return false;
  if (o.precision != 0 && o.true_residual_every > 0 && o.true_residual_replace) return false;  // FP64 x
  CPlan P;
  unsigned rf;
  size_t smem;
  return by_type(h, o.precision, [&](auto dd, auto ss) -> int {
           constexpr int D = decltype(dd)::value;
           using S = decltype(ss);
           const int nc = max_cluster_of<D, S>(true);
           return nc >= 8 && make_plan(h, 0, sizeof(S), true, nc, P, &rf, &smem);
         }) != 0;
}

int cluster_solve_launch(pfm_handle* h, const pfm_solve_opts& o, cudaStream_t s) {
  return by_type(h, o.precision, [&](auto dd, auto ss) -> int {
    constexpr int D = decltype(dd)::value;
    using S = decltype(ss);
    CPlan P;
    CSolve A{};
    size_t smem = 0;
    if (!make_plan(h, 0, sizeof(S), true, max_cluster_of<D, S>(true), P, &A.rf, &smem))
      return set_error(h, PFM_ERR_ARG, "MGPCG: the cluster solve does not fit");
    A.rhs = ws_ptr<float>(h, h->o_r[0]);
    A.x = ws_ptr<float>(h, h->o_x);
    A.p = ws_ptr<float>(h, h->o_p);
    A.Ap = ws_ptr<float>(h, h->o_Ap);
    A.b = ws_ptr<float>(h, h->o_b);
    A.st = ws_ptr<SolveState>(h, h->o_state);
    auto split = [](double x, float& s, float& c) {
      s = (float)x;
      c = (float)(x - (double)s);
    };
    split(o.eps, A.eps_s, A.eps_c);
    A.inv_n = 1.0 / (double)h->cells;
    split(A.inv_n, A.inv_n_s, A.inv_n_c);
    A.tol = o.tol;
    A.tol_mode = o.tol_mode;
    A.max_iters = o.max_iters;
    A.warm = o.warm_start != 0;
    A.true_every = o.true_residual_every > 0 ? o.true_residual_every : 0;
    A.keep_b = A.warm || A.true_every > 0 || o.tol_mode == 2;
    A.neu = 1;
    for (int d = 0; d < h->cfg.dim; ++d)
      if (h->cfg.boundary[d][0] != 2 || h->cfg.boundary[d][1] != 2) A.neu = 0;
    return launch_cluster(h, k_cluster_solve<D, S>, P.nc, smem, s, P, A);
  });
}

int cluster_tail_level(const pfm_handle* h, int precision) {
  if (!h->mg_cluster) return h->L;
  return by_type(h, precision, [&](auto dd, auto ss) -> int {
    constexpr int D = decltype(dd)::value;
    using S = decltype(ss);
    const int nc = max_cluster_of<D, S>(false);
    if (nc < 8) return h->L;
    CPlan P;
    size_t smem;
    for (int l = 1; l < h->L; ++l)
      if (make_plan(h, l, sizeof(S), false, nc, P, nullptr, &smem)) return l;
    return h->L;
  });
}

int cluster_tail_launch(pfm_handle* h, int precision, int l0, void* z, const void* r, const SolveState* st,
                        cudaStream_t s) {
  return by_type(h, precision, [&](auto dd, auto ss) -> int {
    constexpr int D = decltype(dd)::value;
    using S = decltype(ss);
    CPlan P;
    size_t smem = 0;
    if (!make_plan(h, l0, sizeof(S), false, max_cluster_of<D, S>(false), P, nullptr, &smem))
      return set_error(h, PFM_ERR_ARG, "MGPCG: the cluster tail does not fit");
    return launch_cluster(h, k_cluster_tail<D, S>, P.nc, smem, s, (S*)z, (const S*)r, P, const_cast<SolveState*>(st));
  });
}

}  // namespace pfm
