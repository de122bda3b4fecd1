// Learned warm start for the pressure solve: the layers of a 3D convolutional U-Net in BF16 with
// FP32 accumulation, forward and backward, on the fifth-generation tensor cores.
//
// Activation layout ("channel-blocked"): a tensor with C channels on an n0 x n1 x n2 grid is
// [C/8][n0][n1][n2][8] bf16 -- eight channels (16 bytes) per voxel per block.  This makes every
// operand an MMA needs a canonical no-swizzle K-major tile in shared memory without any copy:
//
//  * Forward / data-gradient convolution (k_conv3_fwd): implicit GEMM D[voxel][cout] =
//    sum over 27 taps and cin of X[voxel + tap][ci] W[tap][co][ci].  A CTA sweeps tiles of 128 voxels
//    (16 rows of 8 along d2) along d0.  TMA tiled loads bring each input plane with its halo (zero fill
//    outside the grid is the convolution's padding) as [cin/8][18][10][8]: for a fixed 8-channel block,
//    8 consecutive voxels along d2 are 8 consecutive 16-byte rows, i.e. an 8x16B "core matrix"; the rows
//    of the tile are 160 bytes apart.  Each (b, c) tap is then just another start address of the same
//    shared-memory descriptor: no im2col in memory or in shared memory.  tcgen05.mma (M 128, K 16,
//    kind::f16 BF16 x BF16 -> F32) accumulates in TMEM; four warps read it back with tcgen05.ld for the
//    epilogue (bias, ReLU, BF16 or F32 store).  The data gradient is the same kernel on the output
//    gradient with the weights flipped and transposed (k_pack_w).
//  * Weight gradient (k_conv3_wgrad): D[(b, co)][(a, ci)] for each c = sum over voxels of
//    dY[v][co] X[v + tap][ci], K = voxels.  With channels along the 16-byte rows the same layout is an
//    MN-major operand, so TMA loads feed the MMAs here too; each CTA sums a run of voxel tiles for a group
//    of input channels and a deterministic reduction sums the CTAs.
//
// Every wait (TMA, MMA completion) is bounded by wall time; on expiry the kernel raises a flag in
// device memory, skips its remaining work, frees its TMEM and returns, and later CTAs see the flag
// and return at once.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>

#include "pfm_internal.cuh"
#include "pfm_tma.cuh"

namespace pfm {
namespace nn {

constexpr int kTileD1 = 16, kTileD2 = 8;  // 128 output voxels per CTA
constexpr int kBoxD2 = kTileD2 + 2;
constexpr int kRowBytes = kBoxD2 * 16;  // one row of a tile along d2 with its halo: 160 B
constexpr int kSms = 152;
constexpr int kMaxCin = 128, kMaxNpad = 128;
constexpr int kSmPerGpuSmem = 233472;                  // shared memory per SM (228 KB)
constexpr int kMaxDynSmem = 232448 - 64;               // per-CTA limit (227 KB) less the static flag

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(slot)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem]^T, M 128, BF16 inputs, F32 accumulator
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// true in one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred e;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, e;\n\t}\n"
      : "=r"(p));
  return p != 0;
}

// arrives on `bar` once every tcgen05.mma this thread issued before has completed
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(bar))
               : "memory");
}

// 16 consecutive 32-bit TMEM columns of this warp's 32 lanes (lane = thread)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// zeros into 16 consecutive 32-bit TMEM columns of this warp's 32 lanes
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};"
      ::"r"(taddr), "r"(0)
      : "memory");
}

// a + b of two groups of 16 columns into the second
__device__ __forceinline__ void tmem_add16(uint32_t ta, uint32_t tb) {
  float a[16], b[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=f"(a[0]), "=f"(a[1]), "=f"(a[2]), "=f"(a[3]), "=f"(a[4]), "=f"(a[5]), "=f"(a[6]), "=f"(a[7]), "=f"(a[8]), "=f"(a[9]), "=f"(a[10]), "=f"(a[11]), "=f"(a[12]), "=f"(a[13]), "=f"(a[14]), "=f"(a[15]),
        "=f"(b[0]), "=f"(b[1]), "=f"(b[2]), "=f"(b[3]), "=f"(b[4]), "=f"(b[5]), "=f"(b[6]), "=f"(b[7]), "=f"(b[8]), "=f"(b[9]), "=f"(b[10]), "=f"(b[11]), "=f"(b[12]), "=f"(b[13]), "=f"(b[14]), "=f"(b[15])
      : "r"(ta), "r"(tb)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) b[i] += a[i];
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(tb), "f"(b[0]), "f"(b[1]), "f"(b[2]), "f"(b[3]), "f"(b[4]), "f"(b[5]), "f"(b[6]), "f"(b[7]), "f"(b[8]), "f"(b[9]), "f"(b[10]), "f"(b[11]), "f"(b[12]), "f"(b[13]), "f"(b[14]), "f"(b[15])
      : "memory");
}

__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor, no swizzle: start address, leading-dimension byte offset (the
// stride between core matrices along K) and stride-dimension byte offset (between 8-row groups
// along M or N), all in 16-byte units; bit 46 is the descriptor version of this architecture.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: F32 accumulator (bits 4-5 = 1), BF16 A and B (bits 7-9,
// 10-12 = 1), both K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

constexpr int kFwdThreads = 192;  // warp 0: TMA, warp 1: MMA, warps 2-5: epilogue
constexpr int kMaxRing = 16;      // output planes a CTA keeps in TMEM
constexpr int kPlaneStages = 4, kTapStages = 9;

struct ConvFwdParams {
  int n0, n1, n2;
  int tiles2;          // tiles along d2 (8 voxels each); blockIdx.x = t1 * tiles2 + t2
  int mt;              // 128-voxel tiles per CTA, side by side along d1
  int seg;             // output planes per CTA (blockIdx.y)
  int ring;            // output planes with an accumulator at a time (per tile)
  int cin, c1;         // input channels (x1 holds the first c1)
  int npad, cout;      // columns of one output plane (multiple of 16) and real output channels
  int ncols;           // TMEM columns allocated
  int nstage;          // ring of input planes
  int wstage;          // 9: every tap's weights stay in shared memory; else a ring of (b, c) taps
  const float* bias;   // [cout] or null
  int relu;
  __nv_bfloat16* y1;  // channel-blocked output, channels [0, cy1)
  int cy1;
  __nv_bfloat16* y2;  // channels [cy1, cout), or null
  float* yf;          // if set: f32 planar output [cout][n0][n1][n2] instead of y1/y2
  const float* yf_scale;  // device scalar multiplying yf (or null)
  int* err;
};

// A CTA owns mt x 128 voxels of the (d1, d2) plane and sweeps `seg` output planes along d0.  Every input
// plane is loaded once and multiplied by the taps of all three d0 offsets at once: the N columns of one MMA
// are the three output planes the input plane reaches, side by side in TMEM (column groups of npad, newest
// plane first), so a plane takes 9 (b, c) taps x cin/16 MMAs of N = 3 npad instead of 27 x cin/16 of
// N = npad.  An MMA here takes some 34 + N/2 cycles (reading A, 128 x 16 values, is not hidden: 57 at N 48,
// 80 at 96, 125 at 192), so that halves the tensor core's time, and the input is read 1.4 (seg + 2) / seg
// times instead of 4.2 times.  The column groups form a ring that the epilogue frees, zeroed, plane by plane,
// so `seg` is not bound by TMEM; where three planes straddle the ring's end their MMAs come in two.  An output
// plane's terms arrive in the order of its 27 taps: the planes below, beside and above it in turn, each by
// (b, c) and channel block.  Three roles overlap: TMA (a ring of planes, the weights once or as a ring of
// taps), MMA (one lane), epilogue of finished planes.  Bound by the tensor core for 48 channels and more
// and for 16, at four CTAs per SM, where the issuing warp (some 600 cycles per plane beside its MMAs) is next.
// 16 -> 16 at 192^3 684 -> 117 us, 48 -> 16 at 192^3 2359 -> 296 us, 96 -> 32 at 96^3 1094 -> 157 us
// (one tile per CTA, all 27 taps in turn, before).
__global__ void __launch_bounds__(kFwdThreads) k_conv3_fwd(const __grid_constant__ CUtensorMap tm1,
                                                           const __grid_constant__ CUtensorMap tm2,
                                                           const __grid_constant__ CUtensorMap tmw,
                                                           const ConvFwdParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int kc = p.cin >> 3;
  const uint32_t chunk = (uint32_t)(p.mt * kTileD1 + 2) * kRowBytes;  // one 8-channel block of a plane
  const uint32_t plane_bytes = (uint32_t)kc * chunk;
  const uint32_t plane_pitch = (plane_bytes + 127) & ~127u;
  const uint32_t wtap_bytes = (uint32_t)kc * 3u * (uint32_t)p.npad * 16u;  // one (b, c): [cin/8][3][npad][8]
  unsigned char* wbuf = smem + (size_t)p.nstage * plane_pitch;
  uint64_t* full = (uint64_t*)(wbuf + (size_t)p.wstage * wtap_bytes);
  uint64_t *empty = full + kPlaneStages, *wfull = empty + kPlaneStages, *wempty = wfull + kTapStages,
           *pdone = wempty + kTapStages, *pfree = pdone + kMaxRing, *fin = pfree + kMaxRing;
  uint32_t* slot = (uint32_t*)(fin + 1);
  int* skip = (int*)(slot + 1);
  float* s_bias = (float*)(slot + 2);

  const int t1 = blockIdx.x / p.tiles2, t2 = blockIdx.x - t1 * p.tiles2;
  const int y0 = t1 * p.mt * kTileD1, x0 = t2 * kTileD2;
  const int zs = (int)blockIdx.y * p.seg, ze = min(zs + p.seg, p.n0);
  const int in0 = max(zs - 1, 0), in1 = min(ze, p.n0 - 1);  // input planes inside the grid
  const bool resident = p.wstage == 9;

  if (warp == 0) {  // each lane its barriers
    if (lane < kPlaneStages) {
      mbar_init(full + lane, 1);
      mbar_init(empty + lane, 1);
    } else if (lane < kPlaneStages + kTapStages) {
      mbar_init(wfull + (lane - kPlaneStages), 1);
      mbar_init(wempty + (lane - kPlaneStages), 1);
    } else if (lane == 31) {
      mbar_init(fin, 1);
      *skip = *(volatile int*)p.err;
    }
    if (lane < kMaxRing) {
      mbar_init(pdone + lane, 1);
      mbar_init(pfree + lane, 128);
    }
    fence_mbar_init();
  } else if (warp == 1) {
    tmem_alloc(slot, (uint32_t)p.ncols);
  } else {
    if (warp == 2 && lane == 0) {
      prefetch_map(&tm1);
      prefetch_map(&tmw);
      if (p.cin > p.c1) prefetch_map(&tm2);
    }
    for (int i = tid - 64; i < p.npad; i += 128) s_bias[i] = p.bias && i < p.cout ? p.bias[i] : 0.f;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *slot;
  if (*skip) {  // an earlier CTA gave up: do nothing (uniform over the CTA)
    if (warp == 1) tmem_dealloc(tmem, (uint32_t)p.ncols);
    return;
  }

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      // the weights of tap pair (b, c): rows [a = 0][a = 1][a = 2] of each channel block, so that the columns
      // of an MMA are the output planes z + 1, z, z - 1 of input plane z
      auto load_tap = [&](int bc, int s) {
        mbar_expect_tx(wfull + s, wtap_bytes);
        tma_load_4d(wbuf + (size_t)s * wtap_bytes, &tmw, 0, 0, 0, bc, wfull + s);
      };
      int wi = 0, i = 0;  // taps and planes asked for
      for (; i <= in1 - in0; ++i) {
        const int s = i % p.nstage;
        if (i >= p.nstage) ok = mbar_wait(empty + s, (unsigned)(i / p.nstage - 1) & 1u, p.err, 1);
        if (!ok) break;
        unsigned char* dst = smem + (size_t)s * plane_pitch;
        mbar_expect_tx(full + s, plane_bytes);
        tma_load_4d(dst, &tm1, 8 * (x0 - 1), y0 - 1, in0 + i, 0, full + s);
        if (p.cin > p.c1)
          tma_load_4d(dst + (size_t)(p.c1 >> 3) * chunk, &tm2, 8 * (x0 - 1), y0 - 1, in0 + i, 0, full + s);
        if (!resident || i == 0)
          for (int bc = 0; bc < 9; ++bc, ++wi) {
            const int ws = wi % p.wstage;
            if (wi >= p.wstage) ok = mbar_wait(wempty + ws, (unsigned)(wi / p.wstage - 1) & 1u, p.err, 2);
            if (!ok) break;
            load_tap(bc, ws);
          }
        if (!ok) {
          ++i;
          break;
        }
      }
      if (*(volatile int*)p.err != 0) {  // giving up: the copies in flight land before this memory is given back
        for (int q = max(0, i - p.nstage); q < i; ++q) mbar_drain(full + q % p.nstage, (unsigned)(q / p.nstage) & 1u);
        for (int q = max(0, wi - p.wstage); q < wi; ++q) mbar_drain(wfull + q % p.wstage, (unsigned)(q / p.wstage) & 1u);
      }
    }
  } else if (warp == 1) {
    // The whole warp runs the loop, so that descriptors stay in uniform registers, and one lane issues: with
    // the loop inside a one-lane branch each MMA took 500 to 700 cycles to issue, more than it takes to run.
    const bool lead = elect_one();
    bool ok = true;
    int s = 0, ws = 0;               // plane and tap stage
    unsigned phase = 0, wphase = 0;
    int at = zs == 0 && ze > 1 ? 1 : 0, done = 0;  // ring slots of the newest plane and of the next one to finish
    unsigned lap = 0;
    const int gmax = 256 / p.npad;  // output planes one MMA can hold (N <= 256)
    const int nj = p.cin >> 4;
    const uint32_t lbo_b = 3u * (uint32_t)p.npad * 16u;
    // descriptors advance by their address field (16-byte units): no carry leaves it
    const uint32_t a_step = 2 * chunk / 16, b_step = 2 * lbo_b / 16, w_step = wtap_bytes / 16;
    const uint32_t a_tile = kTileD1 * kBoxD2, d_tile = (uint32_t)(p.ring * p.npad);
    const uint64_t bd0 = smem_desc(su32(wbuf), lbo_b, 128);
    const uint64_t a_first = smem_desc(su32(smem), chunk, kRowBytes);
    if (resident)
      for (int bc = 0; bc < 9; ++bc) ok = ok && mbar_wait(wfull + bc, 0, p.err, 4);
    if (at == 1) ok = ok && mbar_wait(pfree, 0, p.err, 6);
    // a plane's input and its new accumulator are looked for while the plane before is issued
    bool has_in = false, has_acc = false;
    for (int z = in0; z <= in1; ++z) {
      if (!has_acc) ok = ok && mbar_wait(pfree + at, lap & 1u, p.err, 6);
      if (!has_in) ok = ok && mbar_wait(full + s, phase, p.err, 3);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const int s1 = s + 1 == p.nstage ? 0 : s + 1, at1 = z + 2 > ze - 1 ? at : at + 1 == p.ring ? 0 : at + 1;
      const unsigned phase1 = phase ^ (s1 == 0), lap1 = lap + (at1 < at);
      has_in = mbar_test(full + s1, phase1);
      has_acc = at1 == at || mbar_test(pfree + at1, lap1 & 1u);
      const uint64_t ad0 = a_first + (uint32_t)s * (plane_pitch / 16);
      const uint32_t d1 = tmem + (uint32_t)((p.ring - 1 - at) * p.npad);
      const int lo = max(z - 1, zs), hi = min(z + 1, ze - 1), n = hi - lo + 1;
      const uint64_t bdz = bd0 + (uint32_t)((z + 1 - hi) * p.npad);  // rows of the planes that are not there left out
      if (resident && n <= at + 1 && n <= gmax) {  // the planes' columns are one run
        const uint32_t id = idesc_bf16(128, n * p.npad);
        if (lead) {
          uint64_t adb = ad0, bdb = bdz;
#pragma unroll 1
          for (int b = 0; b < 3; ++b, adb += kBoxD2, bdb += 3 * w_step) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              const uint64_t ad = adb + (uint32_t)c, bd = bdb + (uint32_t)c * w_step;
              mma_bf16(d1, ad, bd, id, 1u);
              for (int j = 1; j < nj; ++j) mma_bf16(d1, ad + (uint32_t)j * a_step, bd + (uint32_t)j * b_step, id, 1u);
            }
          }
        }
      } else if (resident && n <= gmax) {  // two runs, cut at the ring's end
        const uint32_t id1 = idesc_bf16(128, (at + 1) * p.npad), id2 = idesc_bf16(128, (n - at - 1) * p.npad);
        const uint32_t b2 = (uint32_t)((at + 1) * p.npad);
        if (lead) {
          uint64_t adb = ad0, bdb = bdz;
#pragma unroll 1
          for (int b = 0; b < 3; ++b, adb += kBoxD2, bdb += 3 * w_step) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              const uint64_t ad = adb + (uint32_t)c, bd = bdb + (uint32_t)c * w_step;
              for (int j = 0; j < nj; ++j) {
                mma_bf16(d1, ad + (uint32_t)j * a_step, bd + (uint32_t)j * b_step, id1, 1u);
                mma_bf16(tmem, ad + (uint32_t)j * a_step, bd + b2 + (uint32_t)j * b_step, id2, 1u);
              }
            }
          }
        }
      } else {
        // runs of columns, cut at the ring's end and at N = 256
        const int r1 = min(min(n, at + 1), gmax);
        const int at2 = r1 > at ? p.ring - 1 : at - r1, r2 = min(min(n - r1, at2 + 1), gmax);
        const int at3 = r2 > at2 ? p.ring - 1 : at2 - r2, r3 = n - r1 - r2;
        const uint32_t id1 = idesc_bf16(128, r1 * p.npad);
        const uint32_t d2 = tmem + (uint32_t)((p.ring - 1 - at2) * p.npad), id2 = idesc_bf16(128, r2 * p.npad);
        const uint32_t d3 = tmem + (uint32_t)((p.ring - 1 - at3) * p.npad), id3 = idesc_bf16(128, r3 * p.npad);
        const uint32_t b2 = (uint32_t)(r1 * p.npad), b3 = (uint32_t)((r1 + r2) * p.npad);
        auto step = [&](uint64_t ad, uint64_t bd) {
          mma_bf16(d1, ad, bd, id1, 1u);
          if (r2) mma_bf16(d2, ad, bd + b2, id2, 1u);
          if (r3) mma_bf16(d3, ad, bd + b3, id3, 1u);
          if (p.mt == 2) {
            mma_bf16(d1 + d_tile, ad + a_tile, bd, id1, 1u);
            if (r2) mma_bf16(d2 + d_tile, ad + a_tile, bd + b2, id2, 1u);
            if (r3) mma_bf16(d3 + d_tile, ad + a_tile, bd + b3, id3, 1u);
          }
        };
        uint64_t adr = ad0;
        bool has_tap = false;
        for (int b = 0; b < 3 && ok; ++b, adr += kBoxD2) {
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const int ws1 = ws + 1 == p.wstage ? 0 : ws + 1;
            const unsigned wphase1 = wphase ^ (ws1 == 0);
            if (!resident) {
              if (!has_tap) ok = ok && mbar_wait(wfull + ws, wphase, p.err, 4);
              ok = __all_sync(0xffffffffu, ok);
              has_tap = mbar_test(wfull + ws1, wphase1);
            }
            if (ok && lead) {
              uint64_t ad = adr + c, bd = bdz + (uint32_t)ws * w_step;
              if (r2) {
                for (int j = 0; j < nj; ++j, ad += a_step, bd += b_step) step(ad, bd);
              } else if (p.mt == 2) {
                for (int j = 0; j < nj; ++j, ad += a_step, bd += b_step) {
                  mma_bf16(d1, ad, bd, id1, 1u);
                  mma_bf16(d1 + d_tile, ad + a_tile, bd, id1, 1u);
                }
              } else {
                for (int j = 0; j < nj; ++j, ad += a_step, bd += b_step) mma_bf16(d1, ad, bd, id1, 1u);
              }
              if (!resident) mma_commit(wempty + ws);
            }
            ws = ws1;
            wphase = wphase1;
          }
        }
        if (!ok) break;
      }
      if (lead) {
        mma_commit(empty + s);
        if (z > zs) mma_commit(pdone + done);
      }
      if (z > zs && ++done == p.ring) done = 0;
      s = s1;
      phase = phase1;
      at = at1;
      lap = lap1;
    }
    if (ok && lead && in1 == ze - 1) mma_commit(pdone + done);  // the grid ends with the segment
    if (*(volatile int*)p.err != 0) {  // giving up: what was issued ends before its operands and TMEM go
      if (lead) mma_commit(fin);
      mbar_drain(fin, 0);
    }
    __syncwarp();
  } else {
    // epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 = output voxels m = 32 (w % 4) + lane
    const int m = (warp & 3) * 32 + lane;
    const int xx = x0 + (m & 7);
    const size_t V = (size_t)p.n0 * p.n1 * p.n2;
    const float scale = (p.yf && p.yf_scale) ? *p.yf_scale : 1.f;
    const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    // accumulators start from zero: here, and again as each plane is read
    for (int c0 = 0; c0 < p.mt * p.ring * p.npad; c0 += 16) tmem_zero16(lanes + (uint32_t)c0);
    tmem_st_wait();
    tc_fence_before();
    for (int s = 0; s < p.ring; ++s) mbar_arrive(pfree + s);
    int r = 0;
    unsigned phase = 0;
    for (int z = zs; z < ze; ++z) {
      if (!mbar_wait(pdone + r, phase, p.err, 5)) break;
      tc_fence_after();
      for (int tile = 0; tile < p.mt; ++tile) {
        const int yy = y0 + tile * kTileD1 + (m >> 3);
        const bool inside = yy < p.n1 && xx < p.n2;
        const size_t vox = ((size_t)z * p.n1 + yy) * p.n2 + xx;
        const uint32_t col = (uint32_t)((tile * p.ring + p.ring - 1 - r) * p.npad);
        for (int c0 = 0; c0 < p.npad; c0 += 16) {
          float v[16];
          tmem_ld16(lanes + col + (uint32_t)c0, v);
          tmem_zero16(lanes + col + (uint32_t)c0);
          if (!inside) continue;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int nb = c0 + 8 * q;
            if (nb >= p.cout) break;
            float o[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              float u = v[8 * q + e];
              if (p.bias) u += s_bias[nb + e];
              if (p.relu) u = fmaxf(u, 0.f);
              o[e] = u;
            }
            if (p.yf) {
              for (int e = 0; e < 8 && nb + e < p.cout; ++e) p.yf[(size_t)(nb + e) * V + vox] = o[e] * scale;
            } else {
              uint4 pk;
              __nv_bfloat162 h0 = __floats2bfloat162_rn(o[0], o[1]), h1 = __floats2bfloat162_rn(o[2], o[3]);
              __nv_bfloat162 h2 = __floats2bfloat162_rn(o[4], o[5]), h3 = __floats2bfloat162_rn(o[6], o[7]);
              pk.x = *(uint32_t*)&h0;
              pk.y = *(uint32_t*)&h1;
              pk.z = *(uint32_t*)&h2;
              pk.w = *(uint32_t*)&h3;
              __nv_bfloat16* dst = nb < p.cy1 ? p.y1 + ((size_t)(nb >> 3) * V + vox) * 8
                                              : p.y2 + ((size_t)((nb - p.cy1) >> 3) * V + vox) * 8;
              *(uint4*)dst = pk;
            }
          }
        }
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(pfree + r);
      if (++r == p.ring) {
        r = 0;
        phase ^= 1u;
      }
    }
  }
  tc_fence_before();
  __syncthreads();  // every role is done: the epilogue has waited for the last MMAs
  if (warp == 1) tmem_dealloc(tmem, (uint32_t)p.ncols);
}

// ---------------------------------------------------------------------------------------------
// weight gradient

__device__ __forceinline__ void unpack8(uint4 u, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float2 t = __bfloat1622float2(h[q]);
    f[2 * q] = t.x;
    f[2 * q + 1] = t.y;
  }
}

constexpr int kWgThreads = 192;  // warp 0: TMA, warp 1: MMA, warps 2-5: epilogue
constexpr int kWgStages = 4;
constexpr int kXChunk = kTileD1 * kRowBytes;  // one 8-channel block of an X plane (16 rows of 10 voxels): 2,560 B

struct ConvWgradParams {
  int n0, n1, n2;
  int tiles1, tiles2, steps;  // voxel tiles of 16 x 8 along d1, d2; steps = tiles x groups of P G planes
  int kc, kc1, dc;            // 8-channel blocks of the input, of x1, and of dY
  int P, G;                   // d0 planes side by side in M; MMA groups per step
  int nb;                     // input blocks per CTA (even)
  int mtiles;                 // M tiles of 128; blockIdx.y = M tile + mtiles * input group
  int N;                      // (P + 2) nb 8 columns per c
  int rows;                   // rows of a column of `partial`
  int flush;                  // steps whose sum moves to a second accumulator at a time (0: all of them stay)
  int nstage, ncols;
  uint32_t stage_bytes, dy_pitch;
  float* partial;  // [split][blockIdx.y][c = 3][N][rows]
  float* bias;     // [split][16][8]: sums of dY over groups of eight voxels, by the CTAs of blockIdx.y = 0 (or null)
  int* err;
};

// D[(s, p, co)][(q, ci)] per c, K = voxels.  Both operands keep channels along their 16-byte rows and voxels
// as rows (MN-major), just as they lie in memory, so TMA's boxes are the MMA's operands: X as
// [plane][8-channel block][16 rows][10 voxels], and dY as [18 rows][P planes][block][8 voxels].  The row shift
// s = 2 - b is a shift of the M groups over dY's rows (a K step of two rows starts 2 P dc groups further), the
// d0 offset a = q - p comes from the planes side by side in N (and, where dY has few channels, in M), and c
// is a start address in X: a step of P planes of 128 voxels takes 3 c x 8 MMAs for all 27 taps.  X rows
// belong to one tile and dY's are loaded with a halo row on each side; X planes and columns the other way round.
// A CTA adds up a run of steps for one group of input channels; the splits are summed with compensation.
// The epilogue warps, idle until then, add up dY's channels for the bias gradient from the stages they find it in
// (its own pass and sum took 80 us of a 96^3 gradient).
// Bound by the tensor core's reading of A, some 34 + N/2 cycles per MMA.  With its reduction, 16 -> 16 at 96^3
// 423 -> 35 us, 48 -> 16 at 96^3 1054 -> 71, 96 -> 32 at 48^3 474 -> 57 (operands transposed into shared memory by
// eight warps before, 592 splits added up by one thread per weight).
__global__ void __launch_bounds__(kWgThreads) k_conv3_wgrad(const __grid_constant__ CUtensorMap tm1,
                                                          const __grid_constant__ CUtensorMap tm2,
                                                          const __grid_constant__ CUtensorMap tmdy,
                                                          const ConvWgradParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t x_plane = (uint32_t)p.nb * kXChunk;
  const int planes = p.P * p.G + 2;
  uint64_t* full = (uint64_t*)(smem + (size_t)p.nstage * p.stage_bytes);
  uint64_t *empty = full + kWgStages, *fin = empty + kWgStages, *moved = fin + 1;
  uint32_t* slot = (uint32_t*)(moved + 1);
  int* skip = (int*)(slot + 1);

  const int mtile = blockIdx.y % p.mtiles, cb = (int)(blockIdx.y / p.mtiles) * p.nb;
  const int nblk = min(p.nb, p.kc - cb);
  const bool bias = p.bias && blockIdx.y == 0;
  const int s0 = (int)((long long)blockIdx.x * p.steps / gridDim.x);
  const int s1 = (int)((long long)(blockIdx.x + 1) * p.steps / gridDim.x);

  if (warp == 0) {
    if (lane < kWgStages) {
      mbar_init(full + lane, 1);
      mbar_init(empty + lane, bias ? 5 : 1);
    } else if (lane == 31) {
      mbar_init(fin, 1);
      mbar_init(moved, 128);
      *skip = *(volatile int*)p.err;
    }
    fence_mbar_init();
  } else if (warp == 1) {
    tmem_alloc(slot, (uint32_t)p.ncols);
  } else if (warp == 2 && lane == 0) {
    prefetch_map(&tm1);
    prefetch_map(&tmdy);
    if (p.kc > p.kc1) prefetch_map(&tm2);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *slot;
  if (*skip) {  // an earlier CTA gave up: do nothing (uniform over the CTA)
    if (warp == 1) tmem_dealloc(tmem, (uint32_t)p.ncols);
    return;
  }

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      const uint32_t bytes = (uint32_t)planes * (uint32_t)nblk * kXChunk + (uint32_t)(p.G * p.P * p.dc) * 18u * 128u;
      const int tiles = p.tiles1 * p.tiles2;
      int i = 0;
      for (; i < s1 - s0; ++i) {
        const int s = i % p.nstage;
        if (i >= p.nstage) ok = mbar_wait(empty + s, (unsigned)(i / p.nstage - 1) & 1u, p.err, 11);
        if (!ok) break;
        // steps run along d0 within a tile, so that a CTA's X planes are read again while they are in L2
        const int zsteps = p.steps / tiles, tile = (s0 + i) / zsteps, z0 = (s0 + i - tile * zsteps) * p.P * p.G;
        const int t1 = tile / p.tiles2, y0 = t1 * kTileD1, x0 = (tile - t1 * p.tiles2) * kTileD2;
        unsigned char* dst = smem + (size_t)s * p.stage_bytes;
        mbar_expect_tx(full + s, bytes);
        for (int g = 0; g < p.G; ++g)
          tma_load_4d(dst + (size_t)g * p.dy_pitch, &tmdy, 8 * x0, 0, z0 + g * p.P, y0 - 1, full + s);
        dst += (size_t)p.G * p.dy_pitch;
        for (int q = 0; q < planes; ++q)
          for (int b = 0; b < nblk; b += 2) {
            const int k = cb + b;
            tma_load_4d(dst + (size_t)q * x_plane + (size_t)b * kXChunk, k < p.kc1 ? &tm1 : &tm2, 8 * (x0 - 1), y0,
                        k < p.kc1 ? k : k - p.kc1, z0 + q - 1, full + s);
          }
      }
      if (*(volatile int*)p.err != 0)  // giving up: the copies in flight land before this memory is given back
        for (int q = max(0, i - p.nstage); q < i; ++q) mbar_drain(full + q % p.nstage, (unsigned)(q / p.nstage) & 1u);
    }
  } else if (warp == 1) {
    const bool lead = elect_one();
    bool ok = true;
    int s = 0;
    unsigned phase = 0;
    const uint32_t group = (uint32_t)(p.P * p.dc) * 128u;  // one dY row
    const uint64_t a0 = smem_desc(su32(smem), group, 128) + (uint32_t)mtile * 128u;
    const uint64_t b0 = smem_desc(su32(smem) + (uint32_t)p.G * p.dy_pitch, kRowBytes, kXChunk);
    const uint32_t a_k = 2 * group / 16, b_k = 2 * kRowBytes / 16;
    const uint32_t id = idesc_bf16(128, p.N) | (1u << 15) | (1u << 16);  // both operands MN-major
    const uint32_t d1 = tmem + (uint32_t)p.N, d2 = d1 + (uint32_t)p.N;
    bool has = false;
    int run = 0;  // steps in the accumulator
    unsigned mphase = 0;
    for (int i = 0; i < s1 - s0; ++i) {
      if (!has) ok = mbar_wait(full + s, phase, p.err, 12);
      if (p.flush && run == p.flush) {
        if (lead) mma_commit(fin);
        ok = ok && mbar_wait(moved, mphase, p.err, 14);
        mphase ^= 1u;
        run = 0;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const int sn = s + 1 == p.nstage ? 0 : s + 1;
      const unsigned phase1 = phase ^ (sn == 0);
      has = mbar_test(full + sn, phase1);
      uint64_t ad = a0 + (uint32_t)s * (p.stage_bytes / 16), bd = b0 + (uint32_t)s * (p.stage_bytes / 16);
      for (int g = 0; g < p.G; ++g) {
        const uint32_t acc = run > 0 || g > 0;
        if (lead) {
          mma_bf16(tmem, ad, bd, id, acc);
          mma_bf16(d1, ad, bd + 1u, id, acc);
          mma_bf16(d2, ad, bd + 2u, id, acc);
#pragma unroll
          for (int k = 1; k < 8; ++k) {
            const uint64_t ak = ad + (uint32_t)k * a_k, bk = bd + (uint32_t)k * b_k;
            mma_bf16(tmem, ak, bk, id, 1u);
            mma_bf16(d1, ak, bk + 1u, id, 1u);
            mma_bf16(d2, ak, bk + 2u, id, 1u);
          }
        }
        ad += p.dy_pitch / 16;
        bd += (uint32_t)p.P * (x_plane / 16);
      }
      if (lead) mma_commit(empty + s);
      __syncwarp();
      ++run;
      s = sn;
      phase = phase1;
    }
    if (lead) mma_commit(fin);
    if (*(volatile int*)p.err != 0) mbar_drain(fin, mphase);  // giving up: what was issued ends before its operands go
    __syncwarp();
  } else {
    const int m = (warp & 3) * 32 + lane, grp = mtile * 16 + (m >> 3);
    const int pl = grp / p.dc % p.P;
    const bool used = grp < 3 * p.P * p.dc;
    const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    float* out = p.partial + ((size_t)blockIdx.x * gridDim.y + blockIdx.y) * 3 * p.N * p.rows + m;
    const int moves = p.flush ? (s1 - s0 - 1) / p.flush : 0;
    const uint32_t sums = moves ? 3u * (uint32_t)p.N : 0u;  // columns of the second accumulator
    bool ok = true;
    if (moves)
      for (int c0 = 0; c0 < 3 * p.N; c0 += 16) tmem_zero16(lanes + sums + (uint32_t)c0);
    int f = 0;
    auto move = [&]() {
      ok = mbar_wait(fin, (unsigned)f & 1u, p.err, 13);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return;
      tmem_st_wait();
      tc_fence_after();
      for (int c0 = 0; c0 < 3 * p.N; c0 += 16) tmem_add16(lanes + (uint32_t)c0, lanes + sums + (uint32_t)c0);
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(moved);
      ++f;
    };
    if (bias) {
      // thread t takes every 128th 16-byte row (8 channels of a voxel) of a stage's 16 inner rows of dY, always
      // of channel block (t / 8) % dc (dc divides 16); the sum of a stage's rows, at most 32, is plain f32, those
      // of the CTA's stages compensated (some 370 rows per thread of 16 channels at 192^3)
      const int t = (int)threadIdx.x - 64, group = p.P * p.dc * 8, n = 16 * group;
      CompSum acc[8];
      int s = 0, run = 0;
      unsigned phase = 0;
      for (int i = 0; i < s1 - s0 && ok; ++i) {
        ok = __all_sync(0xffffffffu, mbar_wait(full + s, phase, p.err, 15));
        if (!ok) break;
        float part[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int g = 0; g < p.G; ++g) {
          const uint4* rows = (const uint4*)(smem + (size_t)s * p.stage_bytes + (size_t)g * p.dy_pitch) + group;
          for (int e = t; e < n; e += 128) {
            float v[8];
            unpack8(rows[e], v);
#pragma unroll
            for (int q = 0; q < 8; ++q) part[q] += v[q];
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + s);
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q].add(part[q]);
        if (p.flush && ++run == p.flush && i + 1 < s1 - s0) {
          run = 0;
          move();
        }
        if (++s == p.nstage) {
          s = 0;
          phase ^= 1u;
        }
      }
#pragma unroll
      for (int q = 0; q < 8; ++q)
        for (int o = 1; o < 8; o *= 2) {
          const float hi = __shfl_xor_sync(0xffffffffu, acc[q].s, o), lo = __shfl_xor_sync(0xffffffffu, acc[q].c, o);
          acc[q].add(hi);
          acc[q].c += lo;
        }
      if ((lane & 7) == 0)
#pragma unroll
        for (int q = 0; q < 8; ++q) p.bias[((size_t)blockIdx.x * 16 + (t >> 3)) * 8 + q] = acc[q].value32();
    } else {
      while (f < moves && ok) move();
    }
    ok = ok && mbar_wait(fin, (unsigned)moves & 1u, p.err, 13);
    if (__all_sync(0xffffffffu, ok)) {
      tc_fence_after();
      for (int c0 = 0; c0 < 3 * p.N; c0 += 16) {
        float v[16];
        if (moves) {
          tmem_add16(lanes + (uint32_t)c0, lanes + sums + (uint32_t)c0);
          tmem_st_wait();
        }
        tmem_ld16(lanes + sums + (uint32_t)c0, v);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int blk = (c0 % p.N >> 3) + h, a = blk / p.nb - pl;
          if (used && a >= 0 && a <= 2 && blk % p.nb < nblk)
#pragma unroll
            for (int e = 0; e < 8; ++e) out[(size_t)(c0 + 8 * h + e) * p.rows] = v[8 * h + e];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, (uint32_t)p.ncols);
}

// dw[co][ci][(a, b, c)] = sum over splits and planes p of their partial sums, compensated and in a fixed order.
// A block holds 32 rows (s, co) of one (c, a, ci): 8 lanes of a warp four rows each, its quarters and the block's
// warps different splits, so that a warp's load is four lines of 128 bytes.
constexpr int kWrWarps = 8;

__global__ void __launch_bounds__(32 * kWrWarps) k_wgrad_reduce(const ConvWgradParams p, int splits, int gy, int cout,
                                                                float* __restrict__ dw, float* __restrict__ db) {
  __shared__ float sh[kWrWarps][8][8];
  if (blockIdx.z == 9) {  // the bias gradient: a warp per channel
    const int c = (blockIdx.x + gridDim.x * blockIdx.y) * (blockDim.x >> 5) + (threadIdx.x >> 5), l = threadIdx.x & 31;
    if (c >= cout) return;
    CompSum v;
    const int per = 16 / p.dc;  // groups of a split that hold the channel
    for (int k = l; k < splits * per; k += 32)
      v.add(p.bias[((size_t)(k / per) * 16 + (c >> 3) + (k % per) * p.dc) * 8 + (c & 7)]);
    for (int o = 16; o > 0; o >>= 1) {
      const float hi = __shfl_xor_sync(0xffffffffu, v.s, o), lo = __shfl_xor_sync(0xffffffffu, v.c, o);
      v.add(hi);
      v.c += lo;
    }
    if (l == 0) db[c] = v.value32();
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int cdy = p.dc * 8, i = blockIdx.x * 32 + (lane & 7) * 4;
  const bool in = i < 3 * cdy;
  const int s = i / cdy, co = i - s * cdy, ci = blockIdx.y, cin = gridDim.y;
  const int c = blockIdx.z / 3, a = blockIdx.z - 3 * c;
  CompSum sum[4];
  if (in && co < cout) {
    const int blk = ci >> 3, y0 = p.mtiles * (blk / p.nb);
    const size_t pitch = (size_t)gy * 3 * p.N * p.rows;
    for (int q = 0; q < p.P; ++q) {
      const int row = (s * p.P + q) * cdy + co, col = ((a + q) * p.nb + blk % p.nb) * 8 + (ci & 7);
      const float* src = p.partial + (((size_t)(y0 + (row >> 7)) * 3 + c) * p.N + col) * p.rows + (row & 127);
#pragma unroll 4
      for (int k = warp * 4 + (lane >> 3); k < splits; k += 4 * warps) {
        const float4 v = *(const float4*)(src + (size_t)k * pitch);
        sum[0].add(v.x);
        sum[1].add(v.y);
        sum[2].add(v.z);
        sum[3].add(v.w);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int o = 8; o <= 16; o *= 2) {
      const float hi = __shfl_xor_sync(0xffffffffu, sum[e].s, o), lo = __shfl_xor_sync(0xffffffffu, sum[e].c, o);
      sum[e].add(hi);
      sum[e].c += lo;
    }
  if (lane < 8)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      sh[warp][lane][2 * e] = sum[e].s;
      sh[warp][lane][2 * e + 1] = sum[e].c;
    }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int r = blockIdx.x * 32 + lane, sr = r / cdy, cr = r - sr * cdy;
    CompSum v;
    for (int k = 0; k < warps; ++k) {
      v.add(sh[k][lane >> 2][2 * (lane & 3)]);
      v.c += sh[k][lane >> 2][2 * (lane & 3) + 1];
    }
    if (r < 3 * cdy && cr < cout) dw[((size_t)cr * cin + ci) * 27 + a * 9 + (2 - sr) * 3 + c] = v.value32();
  }
}

// ---------------------------------------------------------------------------------------------
// weight packing, element-wise layers and the optimizer

// wp[t][kc][n][e] = W'[n][kc*8+e][t] with W' = W ([cout][cin][27]) or, for the data gradient,
// W'[n][ci'][t] = W[ci'][n][26 - t] (n over the layer's input channels, ci' over its outputs).
__global__ void k_pack_w(const float* __restrict__ W, int cout, int cin, int flip, int kin, int npad,
                         __nv_bfloat16* __restrict__ wp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int total = 27 * kin * npad;
  if (i >= total) return;
  const int e = i & 7, n = (i >> 3) % npad, kc = (i >> 3) / npad % (kin >> 3), t = (i >> 3) / npad / (kin >> 3);
  const int k = kc * 8 + e;
  float v = 0.f;
  if (!flip) {
    if (n < cout && k < cin) v = W[((size_t)n * cin + k) * 27 + t];
  } else {
    if (n < cin && k < cout) v = W[((size_t)k * cin + n) * 27 + (26 - t)];
  }
  wp[i] = __float2bfloat16_rn(v);
}

// x (16 channels): channel 0 = f * (*inv_scale), channels 1..15 = 0
__global__ void k_pack_scalar(const float* __restrict__ f, size_t V, const float* __restrict__ inv_scale,
                              __nv_bfloat16* __restrict__ x) {
  const size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= V) return;
  const float s = inv_scale ? *inv_scale : 1.f;
  __nv_bfloat162 h0 = __floats2bfloat162_rn(f[v] * s, 0.f);
  uint4 a = make_uint4(*(uint32_t*)&h0, 0, 0, 0), z = make_uint4(0, 0, 0, 0);
  ((uint4*)x)[v] = a;
  ((uint4*)x)[V + v] = z;
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  uint32_t* w = reinterpret_cast<uint32_t*>(&u);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * q], f[2 * q + 1]);
    w[q] = *(uint32_t*)&h;
  }
  return u;
}

// 2x2x2 average pool (mode 0), its backward (mode 1: dx[v] = dy[v / 2] / 8), nearest upsampling
// (mode 2: y[v] = x[v / 2]) and its backward (mode 3: dx[V] = sum of the 8 children), on 8-channel blocks:
// lanes along d2, of coarse voxels (modes 0, 3: eight loads) or of fine ones (modes 1, 2: one load and the
// stores of the 2 x 2 rows above it).  Bound by memory; the index of a thread comes from the grid (with 64-bit
// divisions per thread the eight of a 96^3 gradient took 72 us, now 44).
__global__ void __launch_bounds__(256) k_resample(const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out,
                                                  int chunks, int n0, int n1, int n2, int mode) {
  const int m0 = n0 >> 1, m1 = n1 >> 1, m2 = n2 >> 1;
  const size_t Vf = (size_t)n0 * n1 * n2, Vc = (size_t)m0 * m1 * m2;
  const bool coarse = mode == 0 || mode == 3;
  const int k = blockIdx.x * 32 + threadIdx.x;
  if (k >= (coarse ? m2 : n2)) return;
  for (int z = blockIdx.z; z < m0 * chunks; z += gridDim.z) {
    const int ch = z / m0, i = z - ch * m0;
    for (int j = blockIdx.y * 8 + threadIdx.y; j < m1; j += gridDim.y * 8) {
      const size_t vf = (size_t)ch * Vf + ((size_t)(2 * i) * n1 + 2 * j) * n2, vc = (size_t)ch * Vc + ((size_t)i * m1 + j) * m2;
      if (coarse) {
        const uint4* src = (const uint4*)in + vf + 2 * k;
        uint4 u[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) u[q] = src[((size_t)(q >> 2) * n1 + (q >> 1 & 1)) * n2 + (q & 1)];
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          float f[8];
          unpack8(u[q], f);
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] += f[e];
        }
        if (mode == 0)
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] *= 0.125f;
        ((uint4*)out)[vc + k] = pack8(acc);
      } else {
        uint4 u = ((const uint4*)in)[vc + (k >> 1)];
        if (mode == 1) {
          float f[8];
          unpack8(u, f);
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] *= 0.125f;
          u = pack8(f);
        }
        uint4* dst = (uint4*)out + vf + k;
#pragma unroll
        for (int q = 0; q < 4; ++q) dst[((size_t)(q >> 1) * n1 + (q & 1)) * n2] = u;
      }
    }
  }
}

// g = g * (y > 0) (mode 0, the ReLU backward) or a = a + b (mode 1), on 8-channel blocks
__global__ void k_elementwise(__nv_bfloat16* __restrict__ g, const __nv_bfloat16* __restrict__ y, size_t n8,
                              int mode) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n8) return;
  float a[8], b[8];
  unpack8(((const uint4*)g)[i], a);
  unpack8(((const uint4*)y)[i], b);
#pragma unroll
  for (int e = 0; e < 8; ++e) a[e] = mode == 0 ? (b[e] > 0.f ? a[e] : 0.f) : a[e] + b[e];
  ((uint4*)g)[i] = pack8(a);
}

constexpr int kRedBlocks = 296;  // 2 x 148: fixed partition of the deterministic reductions
constexpr int kRedThreads = 256;

__device__ __forceinline__ float block_sum(float v, float* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  v = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.f;
  if (w == 0)
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// bias gradient partials: part[block][c] = sum over this block's voxels of dy channel c; blockIdx.y is the
// 8-channel block
__global__ void __launch_bounds__(kRedThreads) k_bias_grad_part(const __nv_bfloat16* __restrict__ dy, int chunks,
                                                                size_t V, float* __restrict__ part) {
  __shared__ float sh[kRedThreads / 32][8];
  const uint4* src = (const uint4*)dy + (size_t)blockIdx.y * V;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const size_t step = (size_t)gridDim.x * kRedThreads;
  for (size_t v = (size_t)blockIdx.x * kRedThreads + threadIdx.x; v < V; v += 4 * step) {
    uint4 u[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) u[q] = v + q * step < V ? src[v + q * step] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float f[8];
      unpack8(u[q], f);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += f[e];
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e)
    for (int o = 16; o > 0; o >>= 1) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int e = 0; e < 8; ++e) sh[threadIdx.x >> 5][e] = acc[e];
  __syncthreads();
  if (threadIdx.x < 8) {
    float s = 0.f;
    for (int w = 0; w < kRedThreads / 32; ++w) s += sh[w][threadIdx.x];
    part[(size_t)blockIdx.x * chunks * 8 + blockIdx.y * 8 + threadIdx.x] = s;
  }
}

// out[c] = sum over parts of part[p][c], fixed order: a warp per c (one thread each took 11 us)
__global__ void __launch_bounds__(32) k_sum_parts(const float* __restrict__ part, int parts, int width,
                                                  float* __restrict__ out) {
  CompSum s;
  for (int k = threadIdx.x; k < parts; k += 32) s.add(part[(size_t)k * width + blockIdx.x]);
  for (int o = 16; o > 0; o >>= 1) {
    const float hi = __shfl_xor_sync(0xffffffffu, s.s, o), lo = __shfl_xor_sync(0xffffffffu, s.c, o);
    s.add(hi);
    s.c += lo;
  }
  if (threadIdx.x == 0) out[blockIdx.x] = s.value32();
}

// Reads of kLossAhead elements per thread are in flight (one at a time: 45 us for 7.1M elements, 14 now; 8.0 and 4.1 for
// 0.9M); the sums keep their order.
constexpr int kLossAhead = 8;
// partial sums of e = pred - target * (*inv_scale) and e^2; part[block] = (sum e, sum e^2)
__global__ void k_loss_part(const float* __restrict__ pred, const float* __restrict__ target,
                            const float* __restrict__ inv_scale, size_t V, float* __restrict__ part) {
  __shared__ float sh[32];
  const float s = inv_scale ? *inv_scale : 1.f;
  float a = 0.f, b = 0.f;
  const size_t step = (size_t)gridDim.x * blockDim.x;
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += kLossAhead * step) {
    float t[kLossAhead], p[kLossAhead];
#pragma unroll
    for (int q = 0; q < kLossAhead; ++q) {
      const bool in = v + q * step < V;
      t[q] = in ? target[v + q * step] : 0.f;
      p[q] = in && pred ? pred[v + q * step] : 0.f;
    }
#pragma unroll
    for (int q = 0; q < kLossAhead; ++q) {
      if (v + q * step >= V) break;
      const float e = p[q] - t[q] * s;
      a += e;
      b += e * e;
    }
  }
  a = block_sum(a, sh);
  b = block_sum(b, sh);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = a;
    part[2 * blockIdx.x + 1] = b;
  }
}

// the loss of a pressure guess up to a constant: out = {L, mean e, 1 / rms e, rms e} with
// L = mean(e^2) - mean(e)^2 (with pred = null, e = -target: out[2] is the inverse RMS of the
// target, the scale of a right-hand side); k_loss_grad writes dL/dpred = 2 (e - mean e) / V as
// channel 0 of a 16-channel block tensor.
__global__ void k_loss_final(const float* __restrict__ part, int parts, size_t V, float* __restrict__ out) {
  // one warp: a chain of 296 FP64 sums in one thread took 47 us
  double a = 0.0, b = 0.0;
  for (int k = threadIdx.x; k < parts; k += 32) {
    a += part[2 * k];
    b += part[2 * k + 1];
  }
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if (threadIdx.x != 0) return;
  const double me = a / (double)V, mse = b / (double)V;
  out[0] = (float)(mse - me * me);
  out[1] = (float)me;
  out[2] = (float)(mse > 0 ? 1.0 / sqrt(mse) : 1.0);
  out[3] = (float)(mse > 0 ? sqrt(mse) : 1.0);
}

__global__ void k_loss_grad(const float* __restrict__ pred, const float* __restrict__ target,
                            const float* __restrict__ inv_scale, const float* __restrict__ stats, size_t V,
                            __nv_bfloat16* __restrict__ g) {
  const size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= V) return;
  const float s = inv_scale ? *inv_scale : 1.f;
  const float e = pred[v] - target[v] * s - stats[1];
  __nv_bfloat162 h0 = __floats2bfloat162_rn(2.f * e / (float)V, 0.f);
  ((uint4*)g)[v] = make_uint4(*(uint32_t*)&h0, 0, 0, 0);
  ((uint4*)g)[V + v] = make_uint4(0, 0, 0, 0);
}

// Adam (Kingma and Ba, 2015) on f32 master parameters, gradient scaled by gscale
__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       size_t n, float lr, float b1, float b2, float eps, float c1, float c2, float gscale) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i] * gscale;
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// ---------------------------------------------------------------------------------------------
// host side

// tensor map of a channel-blocked bf16 tensor: dims (8 n2, n1, n0, C/8), box (8 b2, b1, b0, C/8).  The eight
// channels of consecutive voxels are one run of memory, so a box row of b2 voxels is one copy of 16 b2
// bytes (as five dimensions with an inner one of 8 channels the engine moved 16 bytes at a time).
bool make_map(CUtensorMap* tm, const void* base, int C, int n0, int n1, int n2, int b0, int b1, int b2) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)n2 * 8, (cuuint64_t)n1, (cuuint64_t)n0, (cuuint64_t)(C / 8)};
  const cuuint64_t strides[3] = {(cuuint64_t)n2 * 16, (cuuint64_t)n1 * n2 * 16, (cuuint64_t)n0 * n1 * n2 * 16};
  const cuuint32_t box[4] = {(cuuint32_t)b2 * 8, (cuuint32_t)b1, (cuuint32_t)b0, (cuuint32_t)(C / 8)};
  const cuuint32_t es[4] = {1, 1, 1, 1};
  return fn(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// tensor map of packed weights [27 = (a, b, c)][cin/8][npad][8]: a box is one (b, c) as [cin/8][a][npad][8],
// dims (npad rows of 16 bytes as 8-byte elements: at most 256 of a box side), a, cin/8, (b, c)
bool make_weight_map(CUtensorMap* tm, const void* base, int kc, int npad) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t block = (cuuint64_t)npad * 16, tap = block * kc;
  const cuuint64_t dims[4] = {(cuuint64_t)(npad * 2), 3, (cuuint64_t)kc, 9};
  const cuuint64_t strides[3] = {9 * tap, block, tap};
  const cuuint32_t box[4] = {(cuuint32_t)(npad * 2), 3, (cuuint32_t)kc, 1};
  const cuuint32_t es[4] = {1, 1, 1, 1};
  return fn(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<void*>(base), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int pow2_cols(int n) {
  int c = 32;
  while (c < n) c <<= 1;
  return c;
}

// dynamic shared memory that also keeps resident CTAs x TMEM columns within the SM's 512 columns:
// at most k = 512 / ncols CTAs may share an SM, so k + 1 CTAs (each with 1 KB reserved) must not fit
size_t occupancy_smem(size_t need, int ncols) {
  const size_t k = 512 / (size_t)ncols;
  const size_t floor_bytes = (size_t)kSmPerGpuSmem / (k + 1) - 1024 + 1;
  return need > floor_bytes ? need : floor_bytes;
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

struct WgradPlan {
  ConvWgradParams p;
  int gx, gy;
  size_t smem;
};

// Planes side by side in M until its 128 rows are used (16 channels: 3 s x 2 planes x 16), two MMA groups per
// step (X planes are then read (2 P + 2) / 2 P times instead of (P + 2) / P), and as many input channels per CTA
// as cost least: an MMA takes some 34 + N/2 cycles.  All are cut back until two stages fit.
bool wgrad_plan(const pfm_conv3_wgrad_args* a, WgradPlan* w) {
  ConvWgradParams& p = w->p;
  p = ConvWgradParams{};
  p.n0 = a->d0;
  p.n1 = a->d1;
  p.n2 = a->d2;
  p.tiles1 = (a->d1 + kTileD1 - 1) / kTileD1;
  p.tiles2 = (a->d2 + kTileD2 - 1) / kTileD2;
  p.kc = (a->c1 + a->c2) / 8;
  p.kc1 = a->c1 / 8;
  p.dc = a->cdy / 8;
  p.P = std::max(1, 4 / p.dc);
  const int groups = 3 * p.P * p.dc;
  p.mtiles = (groups + 15) / 16;
  p.rows = std::min(128, groups * 8);
  p.dy_pitch = (uint32_t)std::max(15 * p.P * p.dc + 16 * p.mtiles, 18 * p.P * p.dc) * 128u;
  const size_t fixed = 1024 + 8 * (2 * kWgStages + 2) + 8;
  double best = -1.;
  for (int nb = 2; nb <= 6; nb += 2) {
    const int N = (p.P + 2) * nb * 8;
    if (3 * N > 512) continue;
    int G = 2;
    size_t stage = 0;
    for (; G >= 1; --G) {
      stage = (size_t)G * p.dy_pitch + (size_t)(p.P * G + 2) * nb * kXChunk;
      if (fixed + 2 * stage <= (size_t)kMaxDynSmem) break;
    }
    if (G == 0) continue;
    // a tenth more where TMEM has no room for a second accumulator (below)
    const double cost = (p.kc + nb - 1) / nb * (34. + N / 2.) * (6 * N > 512 ? 1.1 : 1.);
    if (best < 0 || cost < best) {
      best = cost;
      p.nb = nb;
      p.N = N;
      p.G = G;
      p.stage_bytes = (uint32_t)stage;
    }
  }
  if (best < 0) return false;
  const long long steps = (long long)p.tiles1 * p.tiles2 * ((a->d0 + p.P * p.G - 1) / (p.P * p.G));
  if (steps > 0x7fffffff) return false;
  p.steps = (int)steps;
  w->gy = p.mtiles * ((p.kc + p.nb - 1) / p.nb);
  // The tensor core rounds its sums towards zero, so their error grows with the number of K steps (16 -> 16 at
  // 192^3: 7.0e-6 of dW after 736).  A sum is kept to a 640th of the grid's K steps (fewer parts of layers with
  // many weights), or 48: where TMEM has room its sum then moves to a second accumulator (16 -> 16 at 192^3:
  // 137 us against 169 with the partial sums of 608 CTAs), else more CTAs share the steps.
  const long long weights = 27ll * 8 * p.kc * a->cdy, share = 640 / ((weights + 32767) / 32768);
  const long long chain = std::max<long long>(48, (long long)a->d0 * a->d1 * a->d2 / 16 / share) / (8 * p.G);
  int per = 1;
  for (int two = 0; two < 2; ++two) {
    p.ncols = pow2_cols((two ? 6 : 3) * p.N);
    const int slots = std::max(1, std::min(512 / p.ncols, (int)((size_t)kSmPerGpuSmem / (fixed + 2 * p.stage_bytes + 1024))));
    // stages: up to four where they leave as many CTAs on an SM as TMEM allows
    p.nstage = 2;
    while (p.nstage < kWgStages && fixed + (p.nstage + 1) * (size_t)p.stage_bytes <= (size_t)kMaxDynSmem &&
           slots * (fixed + (p.nstage + 1) * (size_t)p.stage_bytes + 1024) <= (size_t)kSmPerGpuSmem)
      ++p.nstage;
    w->smem = occupancy_smem(fixed + p.nstage * (size_t)p.stage_bytes, p.ncols);
    if (w->smem > (size_t)kMaxDynSmem) return false;
    p.flush = two ? (int)chain : 0;
    for (int wave = 1;; ++wave) {
      const long long want = std::max(1, wave * kSms * slots / w->gy);
      per = (int)((steps + want - 1) / want);
      if (per == 1 || per <= chain || two) break;
      if (6 * p.N <= 512) break;
    }
    if (per <= chain || 6 * p.N > 512) break;
  }
  w->gx = (p.steps + per - 1) / per;
  return true;
}

// tensor maps of a channel-blocked bf16 tensor for the weight gradient: X with dims (8 n2, n1, C/8, n0), box one
// plane of 16 channels; dY with dims (8 n2, C/8, n0, n1), box P planes of 18 rows of 8 voxels
bool make_wgrad_map(CUtensorMap* tm, const void* base, int C, int n0, int n1, int n2, int P) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t row = (cuuint64_t)n2 * 16, plane = (cuuint64_t)n1 * row, chunk = (cuuint64_t)n0 * plane;
  const bool dy = P > 0;
  const cuuint64_t dims[4] = {(cuuint64_t)n2 * 8, (cuuint64_t)(dy ? C / 8 : n1), (cuuint64_t)(dy ? n0 : C / 8),
                              (cuuint64_t)(dy ? n1 : n0)};
  const cuuint64_t strides[3] = {dy ? chunk : row, dy ? plane : chunk, dy ? row : plane};
  const cuuint32_t box[4] = {(cuuint32_t)(dy ? 64 : 8 * kBoxD2), (cuuint32_t)(dy ? C / 8 : kTileD1),
                             (cuuint32_t)(dy ? P : 2), (cuuint32_t)(dy ? kTileD1 + 2 : 1)};
  const cuuint32_t es[4] = {1, 1, 1, 1};
  return fn(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool wgrad_shape_ok(const pfm_conv3_wgrad_args* a) {
  const int cin = a->c1 + a->c2;
  return a->c1 > 0 && a->c1 % 16 == 0 && a->c2 >= 0 && a->c2 % 16 == 0 && cin <= kMaxCin && a->cdy > 0 &&
         a->cdy % 8 == 0 && a->cdy <= kMaxNpad;
}

}  // namespace nn
}  // namespace pfm

using namespace pfm::nn;

static int grid_ok(int n0, int n1, int n2) {
  return n0 > 0 && n1 > 0 && n2 > 0 && (long long)n0 * n1 * n2 < (1ll << 31);
}

extern "C" int pfm_nn_conv3(const pfm_conv3_args* a, void* stream) {
  if (!a || !a->x1 || !a->w || !a->err || (!a->y1 && !a->yf)) return PFM_ERR_NULL;
  if (!grid_ok(a->d0, a->d1, a->d2)) return PFM_ERR_SHAPE;
  const int cin = a->c1 + a->c2;
  if (a->c1 <= 0 || a->c1 % 16 || a->c2 < 0 || a->c2 % 16 || cin > kMaxCin || (a->c2 > 0 && !a->x2)) return PFM_ERR_SHAPE;
  if (a->cout <= 0 || a->cout > kMaxNpad) return PFM_ERR_SHAPE;
  const int npad = (a->cout + 15) / 16 * 16;
  if (!a->yf) {
    if (a->cout % 8 || a->cy1 <= 0 || a->cy1 % 8 || a->cy1 > a->cout || (a->cy1 < a->cout && !a->y2))
      return PFM_ERR_SHAPE;
  }
  if (!aligned16(a->x1) || (a->x2 && !aligned16(a->x2)) || !aligned16(a->w) || (a->y1 && !aligned16(a->y1)) ||
      (a->y2 && !aligned16(a->y2)))
    return PFM_ERR_ARG;
  ConvFwdParams p{};
  p.n0 = a->d0;
  p.n1 = a->d1;
  p.n2 = a->d2;
  p.tiles2 = (a->d2 + kTileD2 - 1) / kTileD2;
  const int tiles1 = (a->d1 + kTileD1 - 1) / kTileD1;
  p.cin = cin;
  p.c1 = a->c1;
  p.npad = npad;
  p.cout = a->cout;
  p.bias = a->bias;
  p.relu = a->relu;
  p.y1 = (__nv_bfloat16*)a->y1;
  p.cy1 = a->yf ? a->cout : a->cy1;
  p.y2 = (__nv_bfloat16*)a->y2;
  p.yf = a->yf;
  p.yf_scale = a->yf_scale;
  p.err = a->err;
  const size_t wtap = (size_t)(cin / 8) * 3 * npad * 16;
  const size_t fixed = 1024 + 8 * (2 * kPlaneStages + 2 * kTapStages + 2 * kMaxRing + 1) + 8 + 4 * kMaxNpad;
  size_t need = 0;
  // Output planes per CTA, TMEM columns and tiles per CTA by the time they should take, in cycles.  An SM's
  // tensor core works through the seg + 2 input planes of each of its CTAs (34 + N/2 per MMA; two MMAs where
  // the planes' columns straddle the ring's end or exceed N = 256), a CTA's issuing warp needs some 600 +
  // 60 per MMA, and a CTA's start-up and drain of 9000 are hidden where others share its SM.  Weights that
  // do not fit beside two planes come from L2 once per plane, at some 19 bytes per cycle and SM; two tiles
  // share them then.  16 -> 16 at 192^3: 147 us with rings of 16 planes (two CTAs per SM), 117
  // with the 8 this picks; 96 -> 32 at 96^3: 250 us with one tile per CTA, 157 with two.
  double best = -1.;
  for (int mt = 1; mt <= 2; ++mt) {
    const size_t plane = ((size_t)(cin / 8) * (mt * kTileD1 + 2) * kRowBytes + 127) & ~(size_t)127;
    int nstage = kPlaneStages, wstage = 9;
    while (nstage > 2 && fixed + nstage * plane + 9 * wtap > (size_t)kMaxDynSmem) --nstage;
    if (fixed + nstage * plane + 9 * wtap > (size_t)kMaxDynSmem) {
      wstage = 8;
      while (wstage > 1 && fixed + nstage * plane + wstage * wtap > (size_t)kMaxDynSmem) --wstage;
    }
    const size_t bytes = fixed + nstage * plane + wstage * wtap;
    if (bytes > (size_t)kMaxDynSmem || (mt == 2 && (wstage == 9 || tiles1 < 2))) continue;
    const int per_sm = (int)std::max<size_t>(1, (size_t)kSmPerGpuSmem / (bytes + 1024));
    const long long tiles = (long long)((tiles1 + mt - 1) / mt) * p.tiles2;
    for (int cols = 512; cols >= 64; cols >>= 1) {
      const int fit = std::min(cols / (npad * mt), kMaxRing);
      const int slots = std::min(per_sm, 512 / cols);
      if (fit < 1) break;
      for (int ns = 1, last = 0; ns <= a->d0; ++ns) {
        const int seg = (a->d0 + ns - 1) / ns;
        if (seg == last) continue;
        last = seg;
        if (seg > fit && fit < 4) continue;
        const double mmas = 9. * (cin / 16) * mt * (3 * npad > 256 ? 2. : 1.) * (seg > fit ? 1. + 2. / fit : 1.);
        const double tensor = 34. * mmas + 9. * (cin / 16) * mt * 1.5 * npad;
        double issue = 600. + 60. * mmas;
        if (wstage != 9) issue = std::max(issue + 9. * 200., 9. * wtap / 19.);
        const double alone = (seg + 2) * std::max(issue, tensor) + 9000.;
        const double work = (seg + 2) * std::max(issue / slots, tensor);
        const long long ctas = tiles * ((a->d0 + seg - 1) / seg), waves = ctas / ((long long)kSms * slots);
        const long long rest = ctas - waves * kSms * slots, share = (rest + kSms - 1) / kSms;
        const double cost = waves * std::max(alone, slots * work + 1000.) +
                            (rest ? std::max(alone, share * (seg + 2) * tensor) : 0.);
        if (best < 0 || cost < best) {
          best = cost;
          need = bytes;
          p.mt = mt;
          p.nstage = nstage;
          p.wstage = wstage;
          p.seg = seg;
          p.ring = std::min(seg, fit);
          p.ncols = cols;
        }
        if (seg == 1) break;
      }
    }
  }
  if (best < 0) return PFM_ERR_SHAPE;
  CUtensorMap tm1, tm2, tmw;
  if (!make_map(&tm1, a->x1, a->c1, a->d0, a->d1, a->d2, 1, p.mt * kTileD1 + 2, kBoxD2)) return PFM_ERR_CUDA;
  if (a->c2 > 0) {
    if (!make_map(&tm2, a->x2, a->c2, a->d0, a->d1, a->d2, 1, p.mt * kTileD1 + 2, kBoxD2)) return PFM_ERR_CUDA;
  } else {
    tm2 = tm1;
  }
  if (!make_weight_map(&tmw, a->w, cin / 8, npad)) return PFM_ERR_CUDA;
  const size_t smem = occupancy_smem(need, p.ncols);
  if (smem > kMaxDynSmem) return PFM_ERR_SHAPE;
  static std::atomic<unsigned long long> attr{0};  // above the default 48 KB: opt in per device
  if (pfm::opt_in_smem(k_conv3_fwd, kMaxDynSmem, attr) != cudaSuccess) return PFM_ERR_CUDA;
  dim3 grid((unsigned)((tiles1 + p.mt - 1) / p.mt * p.tiles2), (unsigned)((a->d0 + p.seg - 1) / p.seg));
  if (grid.y > 65535) return PFM_ERR_SHAPE;
  k_conv3_fwd<<<grid, kFwdThreads, smem, (cudaStream_t)stream>>>(tm1, tm2, tmw, p);
  return cudaGetLastError() == cudaSuccess ? PFM_OK : PFM_ERR_CUDA;
}

extern "C" int pfm_nn_wgrad_workspace(const pfm_conv3_wgrad_args* a, size_t* bytes) {
  if (!a || !bytes) return PFM_ERR_NULL;
  WgradPlan w;
  *bytes = 0;  // of a shape that pfm_nn_conv3_wgrad refuses
  if (grid_ok(a->d0, a->d1, a->d2) && wgrad_shape_ok(a) && wgrad_plan(a, &w))
    *bytes = ((size_t)w.gx * w.gy * 3 * w.p.N * w.p.rows + (size_t)w.gx * 128) * sizeof(float);
  return PFM_OK;
}

static int conv3_wgrad(const pfm_conv3_wgrad_args* a, float* db, cudaStream_t st) {
  if (!a || !a->x1 || !a->dy || !a->dw || !a->partial || !a->err) return PFM_ERR_NULL;
  if (!grid_ok(a->d0, a->d1, a->d2)) return PFM_ERR_SHAPE;
  if (!wgrad_shape_ok(a) || (a->c2 > 0 && !a->x2)) return PFM_ERR_SHAPE;
  if (a->cout <= 0 || a->cout > a->cdy) return PFM_ERR_SHAPE;
  if (!aligned16(a->x1) || (a->x2 && !aligned16(a->x2)) || !aligned16(a->dy) || !aligned16(a->partial))
    return PFM_ERR_ARG;
  WgradPlan w;
  if (!wgrad_plan(a, &w)) return PFM_ERR_SHAPE;
  size_t ws = 0;
  pfm_nn_wgrad_workspace(a, &ws);
  if (a->partial_bytes < ws) return PFM_ERR_WORKSPACE;
  CUtensorMap tm1, tm2, tmdy;
  if (!make_wgrad_map(&tm1, a->x1, a->c1, a->d0, a->d1, a->d2, 0)) return PFM_ERR_CUDA;
  if (a->c2 > 0) {
    if (!make_wgrad_map(&tm2, a->x2, a->c2, a->d0, a->d1, a->d2, 0)) return PFM_ERR_CUDA;
  } else {
    tm2 = tm1;
  }
  if (!make_wgrad_map(&tmdy, a->dy, a->cdy, a->d0, a->d1, a->d2, w.p.P)) return PFM_ERR_CUDA;
  w.p.partial = a->partial;
  w.p.bias = db ? a->partial + (size_t)w.gx * w.gy * 3 * w.p.N * w.p.rows : nullptr;
  w.p.err = a->err;
  static std::atomic<unsigned long long> attr{0};  // above the default 48 KB: opt in per device
  if (pfm::opt_in_smem(k_conv3_wgrad, kMaxDynSmem, attr) != cudaSuccess) return PFM_ERR_CUDA;
  k_conv3_wgrad<<<dim3((unsigned)w.gx, (unsigned)w.gy), kWgThreads, w.smem, st>>>(tm1, tm2, tmdy, w.p);
  int warps = 1;  // some eight loads per thread
  while (warps < kWrWarps && warps * 32 < w.gx * w.p.P) warps *= 2;
  const dim3 rgrid((unsigned)(3 * a->cdy + 31) / 32, (unsigned)(a->c1 + a->c2), db ? 10 : 9);
  k_wgrad_reduce<<<rgrid, 32 * warps, 0, st>>>(w.p, w.gx, w.gy, a->cout, a->dw, db);
  return cudaGetLastError() == cudaSuccess ? PFM_OK : PFM_ERR_CUDA;
}

extern "C" int pfm_nn_conv3_wgrad(const pfm_conv3_wgrad_args* a, void* stream) {
  return conv3_wgrad(a, nullptr, (cudaStream_t)stream);
}

extern "C" int pfm_nn_conv3_wgrad_bias(const pfm_conv3_wgrad_args* a, float* db, float* scratch, void* stream) {
  if (!a || !db || !scratch) return PFM_ERR_NULL;
  if (a->cdy > 0 && 128 % a->cdy == 0) return conv3_wgrad(a, db, (cudaStream_t)stream);
  const int rc = conv3_wgrad(a, nullptr, (cudaStream_t)stream);  // the epilogue's threads would mix channel blocks
  return rc ? rc : pfm_nn_bias_grad(a->dy, a->cdy, a->d0, a->d1, a->d2, a->cout, db, scratch, stream);
}

extern "C" int pfm_nn_pack_weights(const float* W, int cout, int cin, int flip, int kin, int npad, void* wp,
                                   void* stream) {
  if (!W || !wp) return PFM_ERR_NULL;
  if (cout <= 0 || cin <= 0 || kin % 16 || npad % 16 || npad <= 0 || kin <= 0) return PFM_ERR_SHAPE;
  if (!flip && (kin < cin || npad < cout)) return PFM_ERR_SHAPE;
  if (flip && (kin < cout || npad < cin)) return PFM_ERR_SHAPE;
  const int total = 27 * kin * npad;
  k_pack_w<<<(total + 255) / 256, 256, 0, (cudaStream_t)stream>>>(W, cout, cin, flip, kin, npad, (__nv_bfloat16*)wp);
  return cudaGetLastError() == cudaSuccess ? PFM_OK : PFM_ERR_CUDA;
}

extern "C" int pfm_nn_pack_scalar(const float* f, int d0, int d1, int d2, const float* inv_scale, void* x,
                                  void* stream) {
  if (!f || !x) return PFM_ERR_NULL;
  if (!grid_ok(d0, d1, d2)) return PFM_ERR_SHAPE;
  const size_t V = (size_t)d0 * d1 * d2;
  k_pack_scalar<<<(unsigned)((V + 255) / 256), 256, 0, (cudaStream_t)stream>>>(f, V, inv_scale, (__nv_bfloat16*)x);
  return cudaGetLastError() == cudaSuccess ? PFM_OK : PFM_ERR_CUDA;
}

extern "C" int pfm_nn_resample(const void* in, void* out, int channels, int d0, int d1, int d2, int mode,
                               void* stream) {
  if (!in || !out) return PFM_ERR_NULL;
  if (!grid_ok(d0, d1, d2) || d0 % 2 || d1 % 2 || d2 % 2 || channels <= 0 || channels % 8 || mode < 0 || mode > 3)
    return PFM_ERR_SHAPE;
  const int last = (mode == 0 || mode == 3) ? d2 / 2 : d2;
  const long long planes = (long long)(d0 / 2) * (channels / 8);
  if (planes > 0x7fffffff) return PFM_ERR_SHAPE;
  const dim3 grid((unsigned)((last + 31) / 32), (unsigned)std::min((d1 / 2 + 7) / 8, 65535),
                  (unsigned)std::min<long long>(planes, 65535));
  k_resample<<<grid, dim3(32, 8), 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)in, (__nv_bfloat16*)out, channels / 8,
                                                             d0, d1, d2, mode);
  return cudaGetLastError() == cudaSuccess ? PFM_OK : PFM_ERR_CUDA;
}

extern "C" int pfm_nn_elementwise(void* g, const void* y, size_t elements, int mode, void* stream) {
  if (!g || !y) return PFM_ERR_NULL;
  if (elements % 8 || (mode != 0 && mode != 1)) return PFM_ERR_SHAPE;
  const size_t n8 = elements / 8;
  if (n8 == 0) return PFM_OK;
  k_elementwise<<<(unsigned)((n8 + 255) / 256), 256, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)g,
                                                                                 (const __nv_bfloat16*)y, n8, mode);
  return cudaGetLastError() == cudaSuccess ? PFM_OK : PFM_ERR_CUDA;
}

extern "C" size_t pfm_nn_scratch_floats(int channels) {
  return (size_t)kRedBlocks * (size_t)(channels > 2 ? channels : 2);
}

extern "C" int pfm_nn_bias_grad(const void* dy, int channels, int d0, int d1, int d2, int cout, float* db,
                                float* scratch, void* stream) {
  if (!dy || !db || !scratch) return PFM_ERR_NULL;
  if (!grid_ok(d0, d1, d2) || channels <= 0 || channels % 8 || cout <= 0 || cout > channels) return PFM_ERR_SHAPE;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t V = (size_t)d0 * d1 * d2;
  k_bias_grad_part<<<dim3(kRedBlocks, (unsigned)(channels / 8)), kRedThreads, 0, st>>>((const __nv_bfloat16*)dy, channels / 8, V, scratch);
  k_sum_parts<<<(unsigned)cout, 32, 0, st>>>(scratch, kRedBlocks, channels, db);
  return cudaGetLastError() == cudaSuccess ? PFM_OK : PFM_ERR_CUDA;
}

extern "C" int pfm_nn_loss(const float* pred, const float* target, const float* inv_scale, int d0, int d1, int d2,
                           float* out4, void* grad, float* scratch, void* stream) {
  if (!target || !out4 || !scratch || (grad && !pred)) return PFM_ERR_NULL;
  if (!grid_ok(d0, d1, d2)) return PFM_ERR_SHAPE;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t V = (size_t)d0 * d1 * d2;
  k_loss_part<<<kRedBlocks, kRedThreads, 0, st>>>(pred, target, inv_scale, V, scratch);
  k_loss_final<<<1, 32, 0, st>>>(scratch, kRedBlocks, V, out4);
  if (grad)
    k_loss_grad<<<(unsigned)((V + 255) / 256), 256, 0, st>>>(pred, target, inv_scale, out4, V, (__nv_bfloat16*)grad);
  return cudaGetLastError() == cudaSuccess ? PFM_OK : PFM_ERR_CUDA;
}

extern "C" int pfm_nn_adam(float* p, const float* g, float* m, float* v, size_t n, float lr, float beta1, float beta2,
                           float eps, int step, float gscale, void* stream) {
  if (!p || !g || !m || !v) return PFM_ERR_NULL;
  if (step < 1 || n == 0) return PFM_ERR_ARG;
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  k_adam<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(p, g, m, v, n, lr, beta1, beta2, eps, c1, c2,
                                                                         gscale);
  return cudaGetLastError() == cudaSuccess ? PFM_OK : PFM_ERR_CUDA;
}
