// unet3d.cu — kernels of the learned warm start (include/unet3d.h): 3x3x3 convolutions as
// implicit GEMMs on the BF16 tensor cores (FP32 accumulation), their data and weight gradients,
// 2x pooling / upsampling with skip concatenation, the masked MSE loss and Adam.
//
// Forward (and data-gradient) convolution: halo tiles on tcgen05 (conv_halo_kernel).  The
// warp tiles (conv_fwd_kernel, mma.sync) take tensors that are not 16-byte aligned and are an
// engine of their own: one warp computes 16 consecutive voxels along x by all output
// channels, K runs over the 27 taps and 16-channel slices, A fragments come straight from the
// channels-last activations, B fragments from the [tap][Cout][Cin] weights.  Taps whose row lies
// outside the box are skipped warp-uniformly; voxels outside the row read zero.
//
// Weight gradient: dW[tap] = dY^T X_shift is a GEMM whose reduction runs over the voxels:
// tcgen05 on slabs staged by TMA (conv_bwdw_tc_kernel).  conv_bwdw_kernel takes what a tensor
// map cannot describe: a block owns one tap, a 16-channel input slice and a chunk of voxels,
// stages 64-voxel slabs of dY and of the shifted input in shared memory and feeds mma.sync
// with transposing ldmatrix loads; partial sums go to the FP32 gradient with one atomic add
// per element and block.
#include <cuda.h>  // CUtensorMap and its enums (the encoder is fetched at run time)
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <stdint.h>

#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <mutex>
#include <string>
#include <type_traits>

#include "../../include/unet3d.h"
#include "chained.cuh"

using lbm::chain_begin;
using lbm::chain_trigger;
using lbm::chain_wait;
using lbm::launch_chained_smem;  // (kernel, grid, block, dynamic shared memory, stream, arguments...)

namespace {

thread_local std::string g_err;

int fail(const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_err = buf;
  return 1;
}

int launched(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail("%s: %s", what, cudaGetErrorString(e));
  return 0;
}

using bf16 = __nv_bfloat16;

struct Geo {
  int n, d, h, w;
};

__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, const uint32_t* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ void ldsm_x4_trans(uint32_t* r, const void* smem_row) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem_row);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// ---- forward convolution ------------------------------------------------------------
template <int NT>  // output channels / 8
__global__ void __launch_bounds__(128) conv_fwd_kernel(const bf16* in, const bf16* w,
                                                       const float* bias, bf16* __restrict__ out,
                                                       const Geo g, const int cin, const int relu,
                                                       const long long tiles) {
  chain_begin();
  const int lane = threadIdx.x & 31;
  const long long tile = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (tile >= tiles) return;  // whole warp
  const int tpr = g.w / 16;
  long long row = tile / tpr;
  const int x0 = (int)(tile - row * tpr) * 16;
  const int y = (int)(row % g.h);
  row /= g.h;
  const int z = (int)(row % g.d);
  const int n = (int)(row / g.d);
  const int gid = lane >> 2, tig = lane & 3;
  constexpr int COUT = NT * 8;
  const int cw = cin / 2;  // 32-bit words per voxel
  const uint32_t* in32 = reinterpret_cast<const uint32_t*>(in);
  const uint32_t* w32 = reinterpret_cast<const uint32_t*>(w);
  float acc[NT][4];
#pragma unroll
  for (int t = 0; t < NT; t++) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
  for (int dz = -1; dz <= 1; dz++) {
    const int zz = z + dz;
    if (zz < 0 || zz >= g.d) continue;
    for (int dy = -1; dy <= 1; dy++) {
      const int yy = y + dy;
      if (yy < 0 || yy >= g.h) continue;
      const long long rbase = (((long long)n * g.d + zz) * g.h + yy) * g.w;
#pragma unroll
      for (int dx = -1; dx <= 1; dx++) {
        const int tap = ((dz + 1) * 3 + (dy + 1)) * 3 + (dx + 1);
        const int xa = x0 + gid + dx, xb = xa + 8;
        const bool va = xa >= 0 && xa < g.w, vb = xb >= 0 && xb < g.w;
        const uint32_t* pa = in32 + (rbase + (va ? xa : 0)) * cw + tig;
        const uint32_t* pb = in32 + (rbase + (vb ? xb : 0)) * cw + tig;
        const uint32_t* wt = w32 + ((long long)tap * COUT + gid) * cw + tig;
        for (int k2 = 0; k2 < cw; k2 += 8) {
          uint32_t a[4];
          a[0] = va ? pa[k2] : 0u;
          a[1] = vb ? pb[k2] : 0u;
          a[2] = va ? pa[k2 + 4] : 0u;
          a[3] = vb ? pb[k2 + 4] : 0u;
#pragma unroll
          for (int t = 0; t < NT; t++) {
            const uint32_t* wb = wt + (long long)t * 8 * cw + k2;
            const uint32_t b[2] = {wb[0], wb[4]};
            mma_bf16(acc[t], a, b);
          }
        }
      }
    }
  }
  const long long vbase = (((long long)n * g.d + z) * g.h + y) * g.w + x0;
  uint32_t* o32 = reinterpret_cast<uint32_t*>(out);
#pragma unroll
  for (int t = 0; t < NT; t++) {
    const int co = t * 8 + 2 * tig;
    const float b0 = bias ? bias[co] : 0.f, b1 = bias ? bias[co + 1] : 0.f;
    float v0 = acc[t][0] + b0, v1 = acc[t][1] + b1, v2 = acc[t][2] + b0, v3 = acc[t][3] + b1;
    if (relu) {
      v0 = fmaxf(v0, 0.f);
      v1 = fmaxf(v1, 0.f);
      v2 = fmaxf(v2, 0.f);
      v3 = fmaxf(v3, 0.f);
    }
    o32[((vbase + gid) * COUT + co) / 2] = pack_bf16(v0, v1);
    o32[((vbase + gid + 8) * COUT + co) / 2] = pack_bf16(v2, v3);
  }
}

// ---- tcgen05: descriptors and bounded waits --------------------------------------------
// MMAs are issued by one thread and committed to an mbarrier; accumulators live in tensor
// memory (TMEM).  Every wait is bounded: a wait that gives up sets the error word and the
// block still frees its TMEM.
constexpr int TC_M = 128;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, K-major, no swizzle: start, leading-dimension byte
// offset (between the two 8-element K halves), stride byte offset (between 8-row
// groups), descriptor version 1.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}

// Instruction descriptor of kind::f16: BF16 A and B (K-major), FP32 accumulator, M x N.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// One lane of a converged warp.  MMA loops run under it rather than under `lane == 0`: the
// compiler then knows that one thread is active and keeps the descriptors in uniform
// registers (measured on B200 with N = 48: 45 cycles per MMA against 68 to 117).
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(e));
  return e != 0u;
}

__device__ __forceinline__ void tc_mbar_init(uint64_t* bar, uint32_t arrivals = 1) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(arrivals) : "memory");
}

// Bounded wait on an mbarrier phase: false after `polls` polls (each try_wait blocks for
// a hardware-defined interval; the default gives up after seconds).
constexpr int TC_WAIT_POLLS = 1 << 22;
__device__ __forceinline__ bool tc_mbar_wait(uint64_t* bar, uint32_t parity, int polls = TC_WAIT_POLLS) {
  const uint32_t a = smem_addr(bar);
  for (int it = 0; it < polls; it++) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// Probe of tc_mbar_wait: thread 0 initialises an mbarrier that expects one arrival, no
// MMA commits to it and nothing arrives, so the wait gives up after `polls` polls and
// the block sets the error word as a convolution CTA does.  Nothing is in flight.
__global__ void __launch_bounds__(32) tc_wait_probe_kernel(const int polls, int* err) {
  chain_begin();
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    tc_mbar_init(&bar);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const bool ok = tc_mbar_wait(&bar, 0u, polls);
  if (!__all_sync(0xffffffffu, ok) && threadIdx.x == 0) atomicExch(err, 1);
}

// ---- forward convolution on halo tiles (tcgen05) --------------------------------------
// The input of a tile is staged once in shared memory with its one-voxel halo, and the 27
// taps are 27 start addresses into it.  Axes: x, P (16 voxels per tile) and R (a run of
// `br` planes); P and R are y and z or, where that leaves fewer voxels of padding, z and y.
//   A operand: the slab keeps a 16-channel slice as two planes of 8 channels (16 bytes) per
//     voxel, so 8 x-neighbours are one 128-byte core matrix of the K-major interleaved
//     layout, the 16 rows along P are 8-row groups one slab row apart (stride byte offset),
//     and the channel halves are one plane apart (leading byte offset).  A tap only moves
//     the start address.  A matrix is 8 (x) by 16 (P) voxels, M = 128, no padding rows.
//   D accumulator: the planes along R of one x group lie side by side in tensor memory.  An
//     input plane contributes to three output planes, so one MMA with N = 3 Cout (the
//     three R taps of one (P, x) tap side by side in the B operand) adds to all three:
//     9 MMAs per input plane and slice instead of 27 per output plane.
// What bounds it: an MMA with M = 128 reads 4 KB of A and 32 N bytes of B from shared memory,
// 33 + N / 4 cycles, against N / 2 of arithmetic; with Cout = 16 an MMA of N = 16 costs 40
// cycles and one of N = 48, three times the work, 45.  The MMAs of 16 -> 16 are half of its time
// (tensor pipe 27 %, shared memory 54 % busy): the same eight warps load a slab and then drain an
// accumulator between two block-wide barriers.
// Loads (cp.async, zero fill outside the box), MMAs and the epilogue of successive tiles run
// side by side: two slabs, two accumulators, one barrier per slice.  One block per SM.
// Measured (B200, 4 x 64 x 64 x 128 voxels): 16 -> 16 channels 592 us with the warp tiles, 52
// here; 48 -> 16 about 1700 -> 136; 96 -> 32 at 4 x 32 x 32 x 64 225 us (threads gathering
// every tap of 128 voxels into shared memory) -> 60; 64 -> 64 at 4 x 16 x 16 x 32 94 -> 20.
constexpr int HT_LOADERS = 256;                // load and epilogue threads (8 warps)
constexpr int HT_THREADS = HT_LOADERS + 32;    // plus the warp that issues the MMAs
constexpr int HT_P = 16;                       // voxels of a tile along P
constexpr int HT_MAX_SMEM = 227 * 1024 - 1024; // dynamic part; the rest is static

// 16 accumulator columns of this warp's lanes: read (complete on return), or set to zero.
__device__ __forceinline__ void tc_load16(uint32_t taddr, uint32_t* q) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7]), "=r"(q[8]),
        "=r"(q[9]), "=r"(q[10]), "=r"(q[11]), "=r"(q[12]), "=r"(q[13]), "=r"(q[14]), "=r"(q[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_zero16(uint32_t taddr) {
  const uint32_t z = 0u;
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};"
      ::"r"(taddr),
      "r"(z)
      : "memory");
}

struct HaloArgs {
  int n, np, nr, w;              // box: batch, P, R, x
  long long sp, sr, sn;          // strides in voxels
  int tap_p, tap_r;              // strides of P and R in the tap index (3 or 9)
  int cin, kcs;                  // input channels and 16-channel slices
  // concatenated input (UP): the first kcu slices are `low`, nearest-upsampled by two, the rest
  // the skip tensor; nothing of it is written to memory
  const bf16* low;
  int kcu, cu, cs;               // slices and channels of low, channels of the skip tensor
  long long lp, lr, ln;          // strides of low in voxels
  int br;                        // output planes of a tile along R
  int tx, tp, tr;                // tiles per axis
  int tiles;
  int relu;
  uint32_t plane, slab;          // bytes of one 8-channel plane (64 mod 128: the two planes' stores
                                 // of one warp fall on different banks), of one slab
  uint32_t stage;                // bytes from one stage to the next (slab, streamed weights)
  int wres;                      // 1: the weights of every slice stay in shared memory
  int cols;                      // tensor memory columns of one accumulator
  int alloc;                     // columns allocated (a power of two)
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool in) {
  const int n = in ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// Weights of one slice: [P tap, x tap][channel half][R tap (descending), Cout] x 16 bytes.
template <int COUT>
__device__ __forceinline__ void halo_load_weights(uint32_t dst, const bf16* w, const HaloArgs& a, int kc,
                                                  int tid) {
  for (int i = tid; i < 27 * COUT * 2; i += HT_LOADERS) {
    const int half = i & 1, co = (i >> 1) % COUT, t = (i >> 1) / COUT;  // t = (p * 3 + r) * 3 + x
    const int x = t % 3, r = (t / 3) % 3, p = t / 9;
    const int tap = p * a.tap_p + r * a.tap_r + x;
    const bf16* src = w + ((long long)tap * COUT + co) * a.cin + kc * 16 + half * 8;
    cp_async16(dst + (p * 3 + x) * (96 * COUT) + half * (48 * COUT) + ((2 - r) * COUT + co) * 16, src, true);
  }
}

template <int BX, bool UP>
__device__ __forceinline__ void halo_load_slab(uint32_t dst, const bf16* in, const HaloArgs& a, int tile,
                                               int kc, int tid) {
  constexpr int PX = BX + 2, PP = HT_P + 2;
  int t = tile;
  const int x0 = (t % a.tx) * BX - 1;
  t /= a.tx;
  const int p0 = (t % a.tp) * HT_P - 1;
  t /= a.tp;
  const int r0 = (t % a.tr) * a.br - 1;
  const int n = t / a.tr;
  // Thread pairs take the two halves of a voxel (32 contiguous bytes); a thread's voxels lie
  // STEP apart, so its coordinates and source advance by constants and carries (a division
  // per voxel made the loads the longest part of an iteration).
  constexpr int STEP = HT_LOADERS / 2, DX = STEP % PX, DP = STEP / PX;
  static_assert(DP + 1 < PP, "one carry per axis and step");
  const int half = tid & 1;
  int v = tid >> 1;
  int x = v % PX, p = v / PX, r = 0;
  if (p >= PP) {
    p -= PP;
    r++;
  }
  dst += half * a.plane + v * 16;
  if (UP && kc < a.kcu) {  // eight fine voxels read one coarse voxel
    const bf16* low = a.low + (long long)n * a.ln * a.cu + kc * 16 + half * 8;
#pragma unroll 2
    for (const int end = (a.br + 2) * PP * PX; v < end; v += STEP) {
      const int gx = x0 + x, gp = p0 + p, gr = r0 + r;
      const bool ok = (unsigned)gx < (unsigned)a.w && (unsigned)gp < (unsigned)a.np && (unsigned)gr < (unsigned)a.nr;
      cp_async16(dst, low + (ok ? ((gr >> 1) * a.lr + (gp >> 1) * a.lp + (gx >> 1)) * a.cu : 0), ok);
      dst += STEP * 16;
      x += DX;
      p += DP;
      if (x >= PX) {
        x -= PX;
        p++;
      }
      if (p >= PP) {
        p -= PP;
        r++;
      }
    }
    return;
  }
  const int ci = UP ? a.cs : a.cin, ch = (UP ? kc - a.kcu : kc) * 16 + half * 8;
  const bf16* base = in + (long long)n * a.sn * ci + ch;
  long long off = (r0 + r) * a.sr + (p0 + p) * a.sp + x0 + x;
  const long long step = DX + DP * a.sp, carry_x = a.sp - PX, carry_p = a.sr - PP * a.sp;
#pragma unroll 2
  for (const int end = (a.br + 2) * PP * PX; v < end; v += STEP) {
    const bool ok = (unsigned)(x0 + x) < (unsigned)a.w && (unsigned)(p0 + p) < (unsigned)a.np &&
                    (unsigned)(r0 + r) < (unsigned)a.nr;
    cp_async16(dst, base + (ok ? off * ci : 0), ok);
    dst += STEP * 16;
    off += step;
    x += DX;
    p += DP;
    if (x >= PX) {
      x -= PX;
      p++;
      off += carry_x;
    }
    if (p >= PP) {
      p -= PP;
      r++;
      off += carry_p;
    }
  }
}

template <int COUT, int BX, bool UP>
__global__ void __launch_bounds__(HT_THREADS, 1)
    conv_halo_kernel(const bf16* in, const bf16* w, const float* bias,
                     bf16* __restrict__ out, const HaloArgs a, int* err) {
  constexpr int PX = BX + 2, PP = HT_P + 2, GX = BX / 8;
  constexpr int NJ = 256 / COUT < 3 ? 256 / COUT : 3;  // output planes one MMA can take (N <= 256)
  constexpr uint32_t WSLICE = 27 * COUT * 32;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ uint32_t tmem_base;
  __shared__ float sbias[COUT];
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t s0 = smem_addr(smem);
  const uint32_t wbase = s0 + 2 * a.stage;  // resident weights follow the stages
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base)),
                 "r"(a.alloc)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    tc_mbar_init(&bar[0]);
    tc_mbar_init(&bar[1]);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();  // the columns are ours
  chain_trigger();
  chain_wait();
  for (int c = tid; c < COUT; c += HT_THREADS) sbias[c] = bias ? bias[c] : 0.f;
  const int first = blockIdx.x, stride = gridDim.x;
  const int mine = (a.tiles - first + stride - 1) / stride;
  const int total = mine * a.kcs;
  if (warp < 8) {
    if (a.wres)
      for (int k = 0; k < a.kcs; k++) halo_load_weights<COUT>(wbase + k * WSLICE, w, a, k, tid);
    else
      halo_load_weights<COUT>(s0 + a.slab, w, a, 0, tid);
    halo_load_slab<BX, UP>(s0, in, a, first, 0, tid);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;
  const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
  if (warp < 8) {  // every MMA accumulates: both accumulators start from zero
    for (int c = (warp >> 2) * 16; c < 2 * a.cols; c += 32) tc_zero16(tmem + lane_off + c);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  }

  // accumulator -> bias, ReLU, BF16 -> global, accumulator zeroed for its next tile
  const auto epilogue = [&](int seq) {
    int t = first + seq * stride;
    const int x0 = (t % a.tx) * BX;
    t /= a.tx;
    const int p = (t % a.tp) * HT_P + (warp & 3) * 4 + (lane >> 3);
    t /= a.tp;
    const int r0 = (t % a.tr) * a.br;
    const long long vox = (long long)(t / a.tr) * a.sn + p * a.sp + x0 + (lane & 7);
    const uint32_t acc = tmem + lane_off + (uint32_t)((seq & 1) * a.cols);
    for (int u = warp >> 2; u < GX * a.br; u += 2) {
      const int g = u / a.br, r = r0 + u - g * a.br;
      bf16* o = out + (vox + g * 8 + r * a.sr) * COUT;
      const bool in_box = p < a.np && r < a.nr;
#pragma unroll
      for (int c0 = 0; c0 < COUT; c0 += 16) {
        uint32_t q[16];
        const uint32_t ta = acc + (uint32_t)(u * COUT + c0);
        tc_load16(ta, q);
        tc_zero16(ta);
        if (in_box) {
          float f[16];
#pragma unroll
          for (int k = 0; k < 16; k++) {
            f[k] = __uint_as_float(q[k]) + sbias[c0 + k];
            if (a.relu) f[k] = fmaxf(f[k], 0.f);
          }
#pragma unroll
          for (int k = 0; k < 16; k += 8)
            *reinterpret_cast<uint4*>(o + c0 + k) = make_uint4(pack_bf16(f[k], f[k + 1]), pack_bf16(f[k + 2], f[k + 3]),
                                                               pack_bf16(f[k + 4], f[k + 5]), pack_bf16(f[k + 6], f[k + 7]));
        }
      }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  };

  bool ok = true;
  int it = 0, seq = 0, kc = 0;  // iteration, tile (in this block's order) and slice
  for (; it < total; it++) {
    if (warp < 8) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor core reads through the async proxy
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (!__syncthreads_and(ok)) {  // a wait gave up: stop issuing (block-uniform)
      ok = false;
      break;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t slab = s0 + (it & 1) * a.stage;
    if (warp == 8) {
      if (elect_one()) {
        const uint32_t wt = a.wres ? wbase + kc * WSLICE : slab + a.slab;
        const uint32_t acc = tmem + (uint32_t)((seq & 1) * a.cols);
        const int r0 = ((first + seq * stride) / (a.tx * a.tp) % a.tr) * a.br;
        const int rout = a.nr - r0 < a.br ? a.nr - r0 : a.br;  // output planes inside the box
        const uint64_t alo = umma_desc(0, a.plane, PX * 16), blo = umma_desc(0, 48 * COUT, 128);
        for (int r = 0; r < rout + 2; r++) {
          if (r0 + r - 1 < 0 || r0 + r - 1 >= a.nr) continue;  // an input plane outside the box is zero
          const int j1 = rout + 1 - r < 2 ? rout + 1 - r : 2;
          for (int j0 = r < 2 ? 2 - r : 0; j0 <= j1; j0 += NJ) {
            const int nj = j1 - j0 + 1 < NJ ? j1 - j0 + 1 : NJ;
            const uint32_t idesc = umma_idesc_bf16(TC_M, nj * COUT);
            for (int g = 0; g < GX; g++) {
              const uint32_t d = acc + (uint32_t)((g * a.br + r - 2 + j0) * COUT);
              // start addresses in 16-byte units; they stay below 2^14 for every tap
              const uint64_t ad = alo | ((slab >> 4) + r * PP * PX + g * 8), bd = blo | ((wt >> 4) + j0 * COUT);
#pragma unroll
              for (int px = 0; px < 9; px++)
                asm volatile(
                    "{\n .reg .pred p;\n setp.ne.b32 p, 1, 0;\n"
                    " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
                    "l"(ad + px / 3 * PX + px % 3), "l"(bd + px * (6 * COUT)), "r"(idesc)
                    : "memory");
            }
          }
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_addr(&bar[it & 1]))
                     : "memory");
      }
      __syncwarp();
    } else {
      if (it > 0) {  // the MMAs of the previous iteration: they read the other stage
        ok = __all_sync(0xffffffffu, tc_mbar_wait(&bar[(it - 1) & 1], (uint32_t)(((it - 1) >> 1) & 1)));
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      if (ok && it + 1 < total) {
        const int nk = kc + 1 == a.kcs ? 0 : kc + 1, ns = nk ? seq : seq + 1;
        const uint32_t next = s0 + ((it + 1) & 1) * a.stage;
        if (!a.wres) halo_load_weights<COUT>(next + a.slab, w, a, nk, tid);
        halo_load_slab<BX, UP>(next, in, a, first + ns * stride, nk, tid);
      }
      if (ok && kc == 0 && seq > 0) epilogue(seq - 1);
    }
    if (++kc == a.kcs) {
      kc = 0;
      seq++;
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  // the last commit tracks every MMA before it
  if (it > 0) {
    const bool done = tc_mbar_wait(&bar[(it - 1) & 1], (uint32_t)(((it - 1) >> 1) & 1));
    ok = ok && done;
  }
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (__syncthreads_and(ok)) {
    if (warp < 8) epilogue(mine - 1);
  } else if (tid == 0) {
    atomicExch(err, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 8)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.alloc) : "memory");
}

// ---- tcgen05 convolution fed by TMA --------------------------------------------------
// A CTA owns 128 consecutive voxels (M = 128) and all output channels (N = Cout); the A tile
// of a tap is a TMA box of the activations: a 5-D tensor map over (C, W, H, D, N) with box {8, min(W,128),
// 128 / min(W,128), 1, 1} lands in shared memory as 128 rows of 16 bytes — exactly the
// K-major interleaved core-matrix layout (8-row groups 128 bytes apart) — and its
// out-of-range rows (the 1-voxel halo at the box faces) are filled with zeros by the
// copy engine.  Two boxes (channel halves) per tap and 16-channel slice, two more for the
// weights; one thread runs the whole pipeline (TMA issue into a ring of stages, MMA issue
// when a stage's bytes have landed, commit that frees the stage), so no CTA barrier sits
// in the K loop.  Every wait is bounded.
constexpr int TMA_STAGES = 4;

__device__ __forceinline__ void tc_mbar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void tma_load_5d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, "
      "%6}], [%7];" ::"r"(smem_addr(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(smem_addr(bar))
      : "memory");
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smem_addr(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_addr(bar))
      : "memory");
}

template <int COUT>
__global__ void __launch_bounds__(TC_M) conv_fwd_tma_kernel(const __grid_constant__ CUtensorMap xmap,
                                                            const __grid_constant__ CUtensorMap wmap,
                                                            const float* bias, bf16* __restrict__ out,
                                                            const Geo g, const int cin, const int relu, int* err) {
  constexpr int NCOL = COUT <= 32 ? 32 : (COUT <= 64 ? 64 : 128);
  constexpr uint32_t A_LBO = TC_M * 16, B_LBO = COUT * 16;
  constexpr uint32_t STAGE_BYTES = 2 * A_LBO + 2 * B_LBO;
  __shared__ __align__(128) uint8_t sbuf[TMA_STAGES][STAGE_BYTES];
  __shared__ __align__(8) uint64_t full[TMA_STAGES], empty[TMA_STAGES];
  __shared__ uint32_t tmem_base;
  __shared__ int ok_s;
  const int tid = threadIdx.x, warp = tid >> 5;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base)),
                 "r"(NCOL)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < TMA_STAGES; s++) {
      tc_mbar_init(&full[s]);
      tc_mbar_init(&empty[s]);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  chain_trigger();
  chain_wait();
  const uint32_t tmem = tmem_base;
  // tile -> (n, z, y0, x0): 128 voxels = part of one row (W >= 128) or 128/W whole rows
  const int bw = g.w < TC_M ? g.w : TC_M, bh = TC_M / bw;
  const int tiles_x = g.w / bw, tiles_y = g.h / bh;
  long long tile = blockIdx.x;
  const int tx = (int)(tile % tiles_x);
  tile /= tiles_x;
  const int ty = (int)(tile % tiles_y);
  tile /= tiles_y;
  const int z = (int)(tile % g.d), n = (int)(tile / g.d);
  const int x0 = tx * bw, y0 = ty * bh;
  const int kcs = cin / 16, iters = 27 * kcs;
  constexpr uint32_t IDESC = umma_idesc_bf16(TC_M, COUT);
  if (tid == 0) {
    bool ok = true;
    uint32_t fpar[TMA_STAGES] = {}, epar[TMA_STAGES] = {};
    int issued_mma = 0;
    for (int it = 0; it < iters + TMA_STAGES - 1 && ok; it++) {
      if (it < iters) {  // producer: stage it % S
        const int s = it % TMA_STAGES;
        if (it >= TMA_STAGES) {  // the MMA of it - S must have released the stage
          ok = tc_mbar_wait(&empty[s], epar[s]);
          epar[s] ^= 1u;
          if (!ok) break;
        }
        const int tap = it / kcs, kc = it - tap * kcs;
        const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
        uint8_t* st = sbuf[s];
        tc_mbar_expect(&full[s], STAGE_BYTES);
        tma_load_5d(st, &xmap, kc * 16, x0 + dx, y0 + dy, z + dz, n, &full[s]);
        tma_load_5d(st + A_LBO, &xmap, kc * 16 + 8, x0 + dx, y0 + dy, z + dz, n, &full[s]);
        tma_load_3d(st + 2 * A_LBO, &wmap, kc * 16, 0, tap, &full[s]);
        tma_load_3d(st + 2 * A_LBO + B_LBO, &wmap, kc * 16 + 8, 0, tap, &full[s]);
      }
      const int j = it - (TMA_STAGES - 1);
      if (j >= 0) {  // consumer: MMA of iteration j
        const int s = j % TMA_STAGES;
        ok = tc_mbar_wait(&full[s], fpar[s]);
        fpar[s] ^= 1u;
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t adesc = umma_desc(smem_addr(sbuf[s]), A_LBO, 128);
        const uint64_t bdesc = umma_desc(smem_addr(sbuf[s] + 2 * A_LBO), B_LBO, 128);
        const uint32_t acc = j > 0 ? 1u : 0u, mask0 = 0u;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}\n" ::"r"(tmem),
            "l"(adesc), "l"(bdesc), "r"(IDESC), "r"(acc), "r"(mask0)
            : "memory");
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_addr(&empty[s]))
                     : "memory");
        issued_mma = j + 1;
      }
    }
    // the last commit tracks every MMA before it; drain the ring (bounded) either way
    if (issued_mma > 0) {
      const int s = (issued_mma - 1) % TMA_STAGES;
      const bool done = tc_mbar_wait(&empty[s], epar[s]);
      ok = ok && done;
    }
    ok_s = ok && issued_mma == iters ? 1 : 0;
  }
  __syncthreads();
  const bool ok = ok_s != 0;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (ok) {
    const int r = tid;  // accumulator lane = tile row = voxel
    const int x = x0 + (r % bw), y = y0 + r / bw;
    const long long v = (((long long)n * g.d + z) * g.h + y) * g.w + x;
    uint32_t* o32 = reinterpret_cast<uint32_t*>(out + v * COUT);
#pragma unroll
    for (int c0 = 0; c0 < COUT; c0 += 8) {
      uint32_t q[8];
      asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7])
                   : "r"(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      float f[8];
#pragma unroll
      for (int k = 0; k < 8; k++) {
        f[k] = __uint_as_float(q[k]) + (bias ? bias[c0 + k] : 0.f);
        if (relu) f[k] = fmaxf(f[k], 0.f);
      }
      *reinterpret_cast<uint4*>(o32 + c0 / 2) =
          make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
    }
  } else if (tid == 0) {
    atomicExch(err, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOL) : "memory");
}

// wt[26 - tap][ci][co] = w[tap][co][ci]
__global__ void flip_kernel(const bf16* w, bf16* __restrict__ wt, int cin, int cout) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int total = 27 * cin * cout;
  if (i >= total) return;
  const int ci = i % cin, co = (i / cin) % cout, tap = i / (cin * cout);
  wt[((26 - tap) * cin + ci) * cout + co] = w[i];
}

// ---- weight gradient ----------------------------------------------------------------
constexpr int BW_KV = 64;  // voxels per shared-memory slab

template <int CB>  // output channels / 16 (1, 2 or 4)
__global__ void __launch_bounds__(128) conv_bwdw_kernel(const bf16* in, const bf16* dout,
                                                        float* __restrict__ dw, const Geo g, const int cin,
                                                        const long long vox, const long long chunk) {
  chain_begin();
  constexpr int COUT = CB * 16;
  constexpr int SA = COUT + 8, SB = 16 + 8;  // padded row lengths (16-byte multiples)
  __shared__ __align__(16) bf16 sA[BW_KV * SA];
  __shared__ __align__(16) bf16 sB[BW_KV * SB];
  const int tap = blockIdx.z;
  const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
  const int ci0 = blockIdx.y * 16;
  const long long m_begin = (long long)blockIdx.x * chunk;
  const long long m_end = m_begin + chunk < vox ? m_begin + chunk : vox;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int NWB = CB < 4 ? CB : 4;  // warps sharing the output-channel blocks
  const int cb = warp % NWB, phase = warp / NWB, nphase = 4 / NWB;
  float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  for (long long m0 = m_begin; m0 < m_end; m0 += BW_KV) {
    // dY slab: BW_KV voxels x COUT channels, 16-byte chunks
    for (int c = tid; c < BW_KV * (COUT / 8); c += 128) {
      const int i = c / (COUT / 8), part = c % (COUT / 8);
      const long long m = m0 + i;
      const uint4 v = m < m_end ? *reinterpret_cast<const uint4*>(dout + m * COUT + part * 8) : zero;
      *reinterpret_cast<uint4*>(sA + i * SA + part * 8) = v;
    }
    // shifted input slab: BW_KV voxels x 16 channels
    {
      const int i = tid >> 1, part = tid & 1;
      const long long m = m0 + i;
      uint4 v = zero;
      if (m < m_end) {
        long long t = m;
        const int x = (int)(t % g.w);
        t /= g.w;
        const int y = (int)(t % g.h);
        t /= g.h;
        const int z = (int)(t % g.d);
        const int xx = x + dx, yy = y + dy, zz = z + dz;
        if (xx >= 0 && xx < g.w && yy >= 0 && yy < g.h && zz >= 0 && zz < g.d) {
          const long long nb = m + dx + (long long)g.w * (dy + (long long)g.h * dz);
          v = *reinterpret_cast<const uint4*>(in + nb * cin + ci0 + part * 8);
        }
      }
      *reinterpret_cast<uint4*>(sB + i * SB + part * 8) = v;
    }
    __syncthreads();
    for (int k16 = phase; k16 < BW_KV / 16; k16 += nphase) {
      const int i = lane & 7, mat = lane >> 3;
      uint32_t a[4], b[4];
      ldsm_x4_trans(a, sA + (k16 * 16 + i + (mat >= 2 ? 8 : 0)) * SA + cb * 16 + ((mat & 1) ? 8 : 0));
      ldsm_x4_trans(b, sB + (k16 * 16 + i + ((mat & 1) ? 8 : 0)) * SB + (mat >> 1) * 8);
      mma_bf16(acc[0], a, b);
      mma_bf16(acc[1], a, b + 2);
    }
    __syncthreads();
  }
  const int gid = lane >> 2, tig = lane & 3;
#pragma unroll
  for (int t = 0; t < 2; t++) {
    const int co = cb * 16 + gid, ci = ci0 + t * 8 + 2 * tig;
    float* p = dw + ((long long)tap * COUT + co) * cin + ci;
    atomicAdd(p, acc[t][0]);
    atomicAdd(p + 1, acc[t][1]);
    atomicAdd(p + 8LL * cin, acc[t][2]);
    atomicAdd(p + 8LL * cin + 1, acc[t][3]);
  }
}

// ---- weight gradient on tcgen05 ---------------------------------------------------------
// dW[tap] = dY^T X_shift as MMAs whose K axis is 16 voxels along x.  Both operands are read as
// they lie in shared memory, channels contiguous (MN-major, no swizzle: 8 channels by 8
// x-neighbours are one 128-byte core matrix), so no transposition and no copy per tap:
//   A (M): rows of the input slab.  A slab row (z, y) is CI / 8 sub-rows of 8 channels by 18
//          voxels, so consecutive 8-channel groups and then consecutive y rows are one sub-row
//          apart: four y rows by CI channels are M = 4 CI (64 or 128) at a single group stride.
//          Three of the four are the y taps of one dY row; the fourth is not used.
//   B (N): dY planes [z][8-channel group][y][x], so the dY planes of the three z taps of one
//          input plane are consecutive groups: N = 3 CO.
//   the three x taps move the start address of A, each with an accumulator of its own.
// Slabs come by TMA (one box per plane, zero fill beyond the row and column ends; input planes
// and dY planes outside the sample are skipped with their MMAs) into two stages; a block keeps
// one (input slice, output block) pair and adds its sums to dW once, at its end.
// The tensor core truncates when it adds to an accumulator, so a long chain loses digits (334
// steps: 60 times the rounding error of the sums).  A tile is therefore at most BT_STEPS steps,
// after which its sums move to registers, are added there with rounding, and the accumulator
// starts again from zero; with CO = 16 a second accumulator hides this, with CO = 32 the
// columns do not suffice and the MMAs wait for the reads (about 5 % of a tile).
// Measured (B200): 16 -> 16 channels at 4 x 64 x 64 x 128 voxels 71 us, 937 with one tap per
// block of mma.sync tiles; 96 -> 32 at 4 x 32 x 32 x 64 65 against 769.
constexpr int BT_THREADS = 256;  // warp 3 copies, warp 7 multiplies, the others hold the sums
constexpr int BT_STEPS = 64;
constexpr int BT_MAX_SMEM = 227 * 1024 - 1024;

struct BwArgs {
  int n, d, h, w;
  int cin, cout;
  int bp, br;            // tile: 16 (x) by bp (y) by br (z)
  int tx, tp, tr, tiles; // tiles per axis, all
  int slices, units;     // input slices; slices times output blocks
  int per_unit;          // blocks that share a unit
  uint32_t xplane, yplane, stage;  // bytes
};

template <int CI, int CO>
__global__ void __launch_bounds__(BT_THREADS, 1)
    conv_bwdw_tc_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap ymap,
                        float* __restrict__ dw, const BwArgs a, int* err) {
  constexpr int G = CI / 8, M = 4 * CI;
  constexpr int COLS = 9 * CO, BUFS = CO == 16 ? 2 : 1, ALLOC = 512;
  constexpr int MINE = (COLS / 16 + 1) / 2 * 16;  // columns of a summing warp (two warps per TMEM quadrant)
  constexpr uint32_t IDESC = umma_idesc_bf16(M, 0) | (1u << 15) | (1u << 16);  // both operands MN-major
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(8) uint64_t full[2], empty[2], dfull[2], dempty[2], done;
  __shared__ uint32_t tmem_base;
  __shared__ int dead;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (warp == 7) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base)),
                 "r"(ALLOC)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    dead = 0;
    for (int s = 0; s < 2; s++) {
      tc_mbar_init(&full[s]);
      tc_mbar_init(&empty[s]);
      tc_mbar_init(&dfull[s]);
      tc_mbar_init(&dempty[s], 6);
    }
    tc_mbar_init(&done);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  chain_trigger();
  chain_wait();
  const uint32_t tmem = tmem_base;
  const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  for (int c = (warp >> 2) * 16; c < BUFS * COLS; c += 32) tc_zero16(lanes + c);  // every MMA accumulates
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  const int unit = blockIdx.x % a.units, first = blockIdx.x / a.units;
  const int ci0 = (unit % a.slices) * CI, co0 = (unit / a.slices) * CO;
  const int mine = first < a.tiles ? (a.tiles - first + a.per_unit - 1) / a.per_unit : 0;
  struct Tile {
    int x0, y0, z0, n, rout;
  };
  const auto tile_at = [&](int k) {
    int t = first + k * a.per_unit;
    Tile q;
    q.x0 = (t % a.tx) * 16;
    t /= a.tx;
    q.y0 = (t % a.tp) * a.bp;
    t /= a.tp;
    q.z0 = (t % a.tr) * a.br;
    q.n = t / a.tr;
    q.rout = a.d - q.z0 < a.br ? a.d - q.z0 : a.br;  // dY planes inside the sample
    return q;
  };
  int issued = 0;  // tiles whose copies were started
  float sum[MINE];
#pragma unroll
  for (int i = 0; i < MINE; i++) sum[i] = 0.f;
  if (warp == 3) {
    if (elect_one()) {
      for (int k = 0; k < mine; k++) {
        const int s = k & 1;
        if (k >= 2 && !tc_mbar_wait(&empty[s], (uint32_t)(((k >> 1) - 1) & 1))) {
          dead = 1;
          break;
        }
        const Tile q = tile_at(k);
        uint8_t* st = smem + s * a.stage;
        const int lo = q.z0 == 0 ? 1 : 0, hi = q.z0 + q.rout == a.d ? q.rout : q.rout + 1;  // input planes lo..hi
        tc_mbar_expect(&full[s], (uint32_t)((hi - lo + 1) * (16 * 18 * G * (a.bp + 3)) + q.rout * a.yplane));
        const long long zn = (long long)q.n * a.d + q.z0;
        for (int r = lo; r <= hi; r++)
          tma_load_5d(st + r * a.xplane, &xmap, 0, q.x0 - 1, ci0 / 8, q.y0 - 1, (int)(zn + r - 1), &full[s]);
        for (int r = 0; r < q.rout; r++)
          tma_load_5d(st + (a.br + 2) * a.xplane + r * a.yplane, &ymap, 0, q.x0, q.y0, co0 / 8, (int)(zn + r), &full[s]);
        issued = k + 1;
      }
    }
    issued = __reduce_max_sync(0xffffffffu, issued);
  } else if (warp == 7) {
    if (elect_one()) {
      const uint64_t alo = umma_desc(0, 128, 18 * 16), blo = umma_desc(0, 128, a.bp * 256);
      for (int k = 0; k < mine; k++) {
        const int s = k & 1;
        const int buf = k % BUFS, use = k / BUFS;  // accumulator, and how often it was used before
        if (!tc_mbar_wait(&full[s], (uint32_t)((k >> 1) & 1)) ||
            (use && !tc_mbar_wait(&dempty[buf], (uint32_t)((use - 1) & 1)))) {
          dead = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const Tile q = tile_at(k);
        const uint32_t xs = smem_addr(smem) + s * a.stage, ys = xs + (a.br + 2) * a.xplane;
        const int rows = a.h - q.y0 < a.bp ? a.h - q.y0 : a.bp;
        for (int r = 0; r < q.rout + 2; r++) {
          const int z = q.z0 + r - 1;
          if (z < 0 || z >= a.d) continue;
          // dY plane r - 2 + j meets input plane r at z tap 2 - j
          const int j0 = r < 2 ? 2 - r : 0, j1 = q.rout + 1 - r < 2 ? q.rout + 1 - r : 2;
          const uint32_t idesc = IDESC | ((uint32_t)((j1 - j0 + 1) * CO / 8) << 17);
          uint64_t ad = alo | ((xs + r * a.xplane) >> 4), bd = blo | ((ys + (r - 2 + j0) * a.yplane) >> 4);
          const uint32_t d = tmem + (uint32_t)(buf * COLS + j0 * CO);
          for (int p = 0; p < rows; p++) {
#pragma unroll
            for (int dx = 0; dx < 3; dx++)
              asm volatile(
                  "{\n .reg .pred p;\n setp.ne.b32 p, 1, 0;\n"
                  " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d + dx * 3 * CO),
                  "l"(ad + dx), "l"(bd), "r"(idesc)
                  : "memory");
            ad += 18 * G;
            bd += 16;
          }
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_addr(&empty[s]))
                     : "memory");
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_addr(&dfull[buf]))
                     : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_addr(&done))
                   : "memory");
    }
    __syncwarp();
  } else {
    for (int k = 0; k < mine; k++) {
      const int buf = k % BUFS, use = k / BUFS;
      if (!__all_sync(0xffffffffu, tc_mbar_wait(&dfull[buf], (uint32_t)(use & 1)))) {
        dead = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int i = 0; i < MINE; i += 16) {
        const int c = (warp >> 2) * MINE + i;
        if (c < COLS) {
          uint32_t q[16];
          tc_load16(lanes + buf * COLS + c, q);
          tc_zero16(lanes + buf * COLS + c);
#pragma unroll
          for (int e = 0; e < 16; e++) sum[i + e] += __uint_as_float(q[e]);
        }
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&dempty[buf])) : "memory");
      __syncwarp();
    }
  }
  bool ok = __all_sync(0xffffffffu, tc_mbar_wait(&done, 0u));
  if (warp == 3)  // copies of the last two tiles, in flight only if a wait gave up
    for (int k = issued > 2 ? issued - 2 : 0; k < issued; k++)
      ok = __all_sync(0xffffffffu, tc_mbar_wait(&full[k & 1], (uint32_t)((k >> 1) & 1))) && ok;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  ok = __syncthreads_and(ok && !dead) != 0;
  if (!ok && tid == 0) atomicExch(err, 1);
  // accumulator row (4 CI of them) -> y tap = TMEM quadrant, input channel = lane
  if (ok && mine > 0 && (warp & 3) < 3 && lane < CI) {
    float* o = dw + ((long long)((warp & 3) * 3) * a.cout + co0) * a.cin + ci0 + lane;
    const long long tap_stride = (long long)a.cout * a.cin;
    const auto add = [&](auto half) {  // column constants per half, no division at run time
#pragma unroll
      for (int i = 0; i < MINE; i++) {
        constexpr int base = decltype(half)::value * MINE;
        const int c = base + i, dx = c / (3 * CO), j = c / CO % 3, co = c % CO;
        if (c < COLS) atomicAdd(o + ((2 - j) * 9 + dx) * tap_stride + co * a.cin, sum[i]);
      }
    };
    if (warp < 4)
      add(std::integral_constant<int, 0>{});
    else
      add(std::integral_constant<int, 1>{});
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 7)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ALLOC) : "memory");
}

__global__ void bias_grad_kernel(const bf16* dout, float* __restrict__ db, long long voxels, int c) {
  chain_begin();
  extern __shared__ float sacc[];
  for (int k = threadIdx.x; k < c; k += blockDim.x) sacc[k] = 0.f;
  __syncthreads();
  const long long total = voxels * c;
  float s = 0.f;
  // the stride is a multiple of c, so each thread keeps one channel; threads past
  // the stride would repeat elements and stay idle
  const long long stride = (long long)gridDim.x * blockDim.x / c * c;
  const long long start = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (start < stride) {
    for (long long i = start; i < total; i += stride) s += __bfloat162float(dout[i]);
    atomicAdd(&sacc[start % c], s);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < c; k += blockDim.x) atomicAdd(db + k, sacc[k]);
}

// The elementwise kernels below come in two forms.  With channels in groups of 8 and 16-byte
// aligned tensors a thread moves whole groups (one 16-byte access each) and a block stays in one
// row of the box, so its coordinates cost a few divisions per block instead of four 64-bit ones
// per element; the one-element forms take everything else.  Values are the same in both, but for
// the bias gradient and the loss, whose sums are made in another order (FP32 and FP64 rounding).
// Measured on B200 at 4 x 64 x 64 x 128 voxels: upsampling with
// concatenation (48 channels) 654 -> 80 us, pooling 45 -> 14 and its gradient 209 -> 32, the
// gradient of the concatenation 197 -> 67, ReLU gradient 89 -> 25, bias gradient 63 -> 15,
// masked loss 192 -> 30.
struct Vec8 {
  float f[8];
};
__device__ __forceinline__ Vec8 load8(const bf16* p) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  Vec8 r;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    r.f[2 * k] = __uint_as_float(w[k] << 16);
    r.f[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
  }
  return r;
}
__device__ __forceinline__ void store8(bf16* p, const Vec8& r) {
  *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16(r.f[0], r.f[1]), pack_bf16(r.f[2], r.f[3]),
                                            pack_bf16(r.f[4], r.f[5]), pack_bf16(r.f[6], r.f[7]));
}

// blockIdx.x = row (n, z, y) of the box, threads over (x, group) of the row.
struct Row {
  long long n;
  int z, y;
};
__device__ __forceinline__ Row row_of(long long r, int d, int h) {
  Row q;
  q.y = (int)(r % h);
  r /= h;
  q.z = (int)(r % d);
  q.n = r / d;
  return q;
}

__global__ void bias_grad8_kernel(const bf16* dout, float* __restrict__ db, long long groups, int c) {
  chain_begin();
  extern __shared__ float sacc[];
  for (int k = threadIdx.x; k < c; k += blockDim.x) sacc[k] = 0.f;
  __syncthreads();
  // the stride is a multiple of c / 8 groups, so a thread keeps its eight channels
  const int gc = c / 8;
  const long long stride = (long long)gridDim.x * blockDim.x / gc * gc;
  const long long start = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (start < stride) {
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (long long i = start; i < groups; i += stride) {
      const Vec8 v = load8(dout + i * 8);
#pragma unroll
      for (int k = 0; k < 8; k++) s[k] += v.f[k];
    }
    const int c0 = (int)(start % gc) * 8;
    const bool whole = 32 % gc == 0;  // then whole warps are here and lanes gc apart hold the same channels
    if (whole) {
      for (int o = 16; o >= gc; o >>= 1)
#pragma unroll
        for (int k = 0; k < 8; k++) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
    }
    if (!whole || (threadIdx.x & 31) < gc)
#pragma unroll
      for (int k = 0; k < 8; k++) atomicAdd(&sacc[c0 + k], s[k]);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < c; k += blockDim.x) atomicAdd(db + k, sacc[k]);
}

__device__ __forceinline__ uint32_t relu_mask2(uint32_t dy, uint32_t y) {  // two packed values
  const float lo = __uint_as_float(y << 16), hi = __uint_as_float(y & 0xffff0000u);
  return (lo > 0.f ? dy & 0xffffu : 0u) | (hi > 0.f ? dy & 0xffff0000u : 0u);
}
__global__ void relu_bwd8_kernel(uint4* __restrict__ dy, const uint4* y, long long groups) {
  chain_begin();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= groups) return;
  const uint4 g = dy[i], v = y[i];
  dy[i] = make_uint4(relu_mask2(g.x, v.x), relu_mask2(g.y, v.y), relu_mask2(g.z, v.z), relu_mask2(g.w, v.w));
}

__global__ void pool2x8_kernel(const bf16* in, bf16* __restrict__ out, Geo f, int c) {
  chain_begin();
  const int W = f.w / 2, gc = c / 8;
  const Row q = row_of(blockIdx.x, f.d / 2, f.h / 2);
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < W * gc; i += gridDim.y * blockDim.x) {
    const int x = i / gc, ch = (i - x * gc) * 8;
    Vec8 s{};
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const long long v = ((q.n * f.d + 2 * q.z + (k >> 2)) * f.h + 2 * q.y + ((k >> 1) & 1)) * f.w + 2 * x + (k & 1);
      const Vec8 a = load8(in + v * c + ch);
#pragma unroll
      for (int e = 0; e < 8; e++) s.f[e] += a.f[e];
    }
#pragma unroll
    for (int e = 0; e < 8; e++) s.f[e] *= 0.125f;
    store8(out + ((long long)blockIdx.x * W + x) * c + ch, s);
  }
}

__global__ void pool2x8_bwd_kernel(const bf16* dout, bf16* __restrict__ din, Geo f, int c, int accumulate) {
  chain_begin();
  const int gc = c / 8;
  const Row q = row_of(blockIdx.x, f.d, f.h);
  const long long parent = ((q.n * (f.d / 2) + q.z / 2) * (f.h / 2) + q.y / 2) * (f.w / 2);
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < f.w * gc; i += gridDim.y * blockDim.x) {
    const int x = i / gc, ch = (i - x * gc) * 8;
    Vec8 v = load8(dout + (parent + x / 2) * c + ch);
    bf16* o = din + ((long long)blockIdx.x * f.w + x) * c + ch;
#pragma unroll
    for (int e = 0; e < 8; e++) v.f[e] *= 0.125f;
    if (accumulate) {
      const uint4 u = *reinterpret_cast<const uint4*>(o);
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        v.f[2 * k] += __uint_as_float(w[k] << 16);
        v.f[2 * k + 1] += __uint_as_float(w[k] & 0xffff0000u);
      }
    }
    store8(o, v);
  }
}

__global__ void up2_concat8_kernel(const uint4* low, const uint4* skip,
                                   uint4* __restrict__ out, Geo f, int gu, int gs) {
  chain_begin();
  const int gt = gu + gs;
  const Row q = row_of(blockIdx.x, f.d, f.h);
  const long long parent = ((q.n * (f.d / 2) + q.z / 2) * (f.h / 2) + q.y / 2) * (f.w / 2);
  const long long row = (long long)blockIdx.x * f.w;
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < f.w * gt; i += gridDim.y * blockDim.x) {
    const int x = i / gt, g = i - x * gt;
    out[row * gt + i] = g >= gu ? skip[(row + x) * gs + (g - gu)] : low[(parent + x / 2) * gu + g];
  }
}

__global__ void up2_concat8_bwd_kernel(const bf16* dcat, bf16* __restrict__ dlow, uint4* __restrict__ dskip,
                                       Geo f, int gu, int gs, unsigned coarse_rows) {
  chain_begin();
  const int ct = (gu + gs) * 8;
  if (blockIdx.x < coarse_rows) {  // dlow: the 8 children of a coarse voxel
    const int W = f.w / 2;
    const Row q = row_of(blockIdx.x, f.d / 2, f.h / 2);
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < W * gu; i += gridDim.y * blockDim.x) {
      const int x = i / gu, ch = (i - x * gu) * 8;
      Vec8 s{};
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const long long v =
            ((q.n * f.d + 2 * q.z + (k >> 2)) * f.h + 2 * q.y + ((k >> 1) & 1)) * f.w + 2 * x + (k & 1);
        const Vec8 a = load8(dcat + v * ct + ch);
#pragma unroll
        for (int e = 0; e < 8; e++) s.f[e] += a.f[e];
      }
      store8(dlow + ((long long)blockIdx.x * W + x) * gu * 8 + ch, s);
    }
    return;
  }
  const long long row = (long long)(blockIdx.x - coarse_rows) * f.w;
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < f.w * gs; i += gridDim.y * blockDim.x) {
    const int x = i / gs, g = i - x * gs;
    dskip[row * gs + i] = reinterpret_cast<const uint4*>(dcat + (row + x) * ct)[gu + g];
  }
}

__global__ void relu_bwd_kernel(bf16* __restrict__ dy, const bf16* y, long long count) {
  chain_begin();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count && !(__bfloat162float(y[i]) > 0.f)) dy[i] = __float2bfloat16(0.f);
}

// ---- pooling, upsampling, concatenation ---------------------------------------------
__global__ void pool2_kernel(const bf16* in, bf16* __restrict__ out, Geo f, int c, long long count) {
  chain_begin();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;  // count = coarse elements
  const int ch = (int)(i % c);
  long long t = i / c;
  const int W = f.w / 2, H = f.h / 2, D = f.d / 2;
  const int x = (int)(t % W);
  t /= W;
  const int y = (int)(t % H);
  t /= H;
  const int z = (int)(t % D);
  const int n = (int)(t / D);
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const long long v = (((long long)n * f.d + 2 * z + (k >> 2)) * f.h + 2 * y + ((k >> 1) & 1)) * f.w + 2 * x + (k & 1);
    s += __bfloat162float(in[v * c + ch]);
  }
  out[i] = __float2bfloat16(s * 0.125f);
}

__global__ void pool2_bwd_kernel(const bf16* dout, bf16* __restrict__ din, Geo f, int c, int accumulate,
                                 long long count) {
  chain_begin();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;  // count = fine elements
  const int ch = (int)(i % c);
  long long t = i / c;
  const int x = (int)(t % f.w);
  t /= f.w;
  const int y = (int)(t % f.h);
  t /= f.h;
  const int z = (int)(t % f.d);
  const int n = (int)(t / f.d);
  const long long p = (((long long)n * (f.d / 2) + z / 2) * (f.h / 2) + y / 2) * (f.w / 2) + x / 2;
  float v = __bfloat162float(dout[p * c + ch]) * 0.125f;
  if (accumulate) v += __bfloat162float(din[i]);
  din[i] = __float2bfloat16(v);
}

__global__ void up2_concat_kernel(const bf16* low, const bf16* skip, bf16* __restrict__ out,
                                  Geo f, int cu, int cs, long long count) {
  chain_begin();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;  // count = fine voxels * (cu + cs)
  const int ct = cu + cs;
  const int ch = (int)(i % ct);
  const long long v = i / ct;
  if (ch >= cu) {
    out[i] = skip[v * cs + (ch - cu)];
    return;
  }
  long long t = v;
  const int x = (int)(t % f.w);
  t /= f.w;
  const int y = (int)(t % f.h);
  t /= f.h;
  const int z = (int)(t % f.d);
  const int n = (int)(t / f.d);
  const long long p = (((long long)n * (f.d / 2) + z / 2) * (f.h / 2) + y / 2) * (f.w / 2) + x / 2;
  out[i] = low[p * cu + ch];
}

__global__ void up2_concat_bwd_low_kernel(const bf16* dcat, bf16* __restrict__ dlow, Geo f, int cu, int cs,
                                          long long count) {
  chain_begin();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;  // count = coarse voxels * cu
  const int ch = (int)(i % cu);
  long long t = i / cu;
  const int W = f.w / 2, H = f.h / 2, D = f.d / 2;
  const int x = (int)(t % W);
  t /= W;
  const int y = (int)(t % H);
  t /= H;
  const int z = (int)(t % D);
  const int n = (int)(t / D);
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const long long v = (((long long)n * f.d + 2 * z + (k >> 2)) * f.h + 2 * y + ((k >> 1) & 1)) * f.w + 2 * x + (k & 1);
    s += __bfloat162float(dcat[v * (cu + cs) + ch]);
  }
  dlow[i] = __float2bfloat16(s);
}

__global__ void up2_concat_bwd_skip_kernel(const bf16* dcat, bf16* __restrict__ dskip, int cu, int cs,
                                           long long count) {
  chain_begin();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;  // count = fine voxels * cs
  const long long v = i / cs;
  dskip[i] = dcat[v * (cu + cs) + cu + (int)(i % cs)];
}

// ---- loss and optimiser -------------------------------------------------------------
// Each block keeps its loss until it has covered its voxels: one atomic per block (one per warp
// of voxels serialised 65,536 of them on one address).  PACKED: 16 channels of which 4 have
// targets, 16-byte aligned.
template <bool PACKED>
__global__ void __launch_bounds__(256) mse_kernel(const bf16* out, const float* target,
                                                  const uint8_t* mask, const float* cw,
                                                  bf16* __restrict__ dout, double* loss, long long voxels, int cpad,
                                                  int ct, double count) {
  chain_begin();
  __shared__ double part[8];
  double l = 0.0;
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < voxels; v += (long long)gridDim.x * blockDim.x) {
    const bool on = mask[v] != 0;
    if (PACKED) {
      uint4 lo = make_uint4(0u, 0u, 0u, 0u);
      if (on) {
        const uint2 o = *reinterpret_cast<const uint2*>(out + v * 16);
        const float4 t = *reinterpret_cast<const float4*>(target + v * 4);
        const float d[4] = {__uint_as_float(o.x << 16) - t.x, __uint_as_float(o.x & 0xffff0000u) - t.y,
                            __uint_as_float(o.y << 16) - t.z, __uint_as_float(o.y & 0xffff0000u) - t.w};
        float gr[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
          l += (double)cw[c] * d[c] * d[c];
          gr[c] = (float)(2.0 * cw[c] * d[c] / count);
        }
        lo.x = pack_bf16(gr[0], gr[1]);
        lo.y = pack_bf16(gr[2], gr[3]);
      }
      uint4* o4 = reinterpret_cast<uint4*>(dout + v * 16);
      o4[0] = lo;
      o4[1] = make_uint4(0u, 0u, 0u, 0u);
    } else {
      for (int c = 0; c < cpad; c++) {
        float gr = 0.f;
        if (on && c < ct) {
          const float d = __bfloat162float(out[v * cpad + c]) - target[v * ct + c];
          l += (double)cw[c] * d * d;
          gr = (float)(2.0 * cw[c] * d / count);
        }
        dout[v * cpad + c] = __float2bfloat16(gr);
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = l;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < 8; k++) t += part[k];
    if (t != 0.0) atomicAdd(loss, t / count);
  }
}

__global__ void adam_kernel(float* __restrict__ w, const float* g, float* __restrict__ m,
                            float* __restrict__ v, bf16* __restrict__ wb, long long count, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
  chain_begin();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  w[i] = wi;
  if (wb) wb[i] = __float2bfloat16(wi);
}

__global__ void to_bf16_kernel(const float* x, bf16* __restrict__ y, long long count) {
  chain_begin();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) y[i] = __float2bfloat16(x[i]);
}

__global__ void from_bf16_kernel(const bf16* x, float* __restrict__ y, long long count) {
  chain_begin();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) y[i] = __bfloat162float(x[i]);
}

// out[0] += sum (a - b)^2, out[1] += sum a^2 (FP64), for steady-state tests.
__global__ void diff_norms_kernel(const float* a, const float* b, long long count,
                                  double* out) {
  chain_begin();
  double d2 = 0.0, a2 = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x) {
    const double x = a[i], y = b[i];
    d2 += (x - y) * (x - y);
    a2 += x * x;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    d2 += __shfl_down_sync(0xffffffffu, d2, o);
    a2 += __shfl_down_sync(0xffffffffu, a2, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(out, d2);
    atomicAdd(out + 1, a2);
  }
}

struct Ellipsoid {
  double center[3];
  double rot[9];  // row-major body -> world
  double semi[3];
};

// Inputs of one case: mask, approximate signed distance / 16 in [-1, 4], Re feature,
// node position; the mask uses the solver's rasteriser expression with unfused
// FP64 operations, so it matches the solver's solid flags.
__global__ void features_kernel(bf16* __restrict__ out, int nx, int ny, int nz, Ellipsoid e, float re_feature) {
  chain_begin();
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = (long long)nx * ny * nz;
  if (v >= n) return;
  const int x = (int)(v % nx), y = (int)((v / nx) % ny), z = (int)(v / ((long long)nx * ny));
  const double dx = __dadd_rn(x + 0.5, -e.center[0]);
  const double dy = __dadd_rn(y + 0.5, -e.center[1]);
  const double dz = __dadd_rn(z + 0.5, -e.center[2]);
  const double* r = e.rot;
  double b[3], q[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    b[k] = __dadd_rn(__dadd_rn(__dmul_rn(r[k], dx), __dmul_rn(r[3 + k], dy)), __dmul_rn(r[6 + k], dz));
    q[k] = __ddiv_rn(b[k], e.semi[k]);
  }
  const double e2 = __dadd_rn(__dadd_rn(__dmul_rn(q[0], q[0]), __dmul_rn(q[1], q[1])), __dmul_rn(q[2], q[2]));
  const double er = sqrt(e2);
  double g2 = 0.0;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double t = b[k] / (e.semi[k] * e.semi[k]);
    g2 += t * t;
  }
  const double grad = sqrt(g2) / fmax(er, 1e-12);
  const double sdf = (er - 1.0) / fmax(grad, 1e-12);
  float f[16];
#pragma unroll
  for (int c = 0; c < 16; c++) f[c] = 0.f;
  f[0] = e2 <= 1.0 ? 1.f : 0.f;
  f[1] = fminf(fmaxf((float)(sdf / 16.0), -1.f), 4.f);
  f[2] = re_feature;
  f[3] = (float)((x + 0.5) / nx);
  f[4] = (float)((y + 0.5) / ny);
  f[5] = (float)((z + 0.5) / nz);
  uint32_t* o = reinterpret_cast<uint32_t*>(out + v * 16);
#pragma unroll
  for (int c = 0; c < 8; c++) o[c] = pack_bf16(f[2 * c], f[2 * c + 1]);
}

// out (n, 4, d, h, w) FP32 (+)= weight * the first four channels of y (n, d, h, w, 16),
// read from the mirror image in y and/or z, with the mirrored velocity components
// (channel 2 = u_y, 3 = u_z) negated: undoes a reflection of the input.
__global__ void unpack_fields_kernel(const bf16* y, float* __restrict__ out, Geo g, int flip_y, int flip_z,
                                     float weight, int accumulate, long long count) {
  chain_begin();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;  // count = n * d * h * w
  long long t = i;
  const int x = (int)(t % g.w);
  t /= g.w;
  const int yy = (int)(t % g.h);
  t /= g.h;
  const int z = (int)(t % g.d);
  const int n = (int)(t / g.d);
  const int ys = flip_y ? g.h - 1 - yy : yy, zs = flip_z ? g.d - 1 - z : z;
  const long long src = (((long long)n * g.d + zs) * g.h + ys) * g.w + x;
  const long long plane = (long long)g.d * g.h * g.w;
  const long long v = ((long long)z * g.h + yy) * g.w + x;
#pragma unroll
  for (int c = 0; c < 4; c++) {
    float val = __bfloat162float(y[src * 16 + c]) * weight;
    if ((c == 2 && flip_y) || (c == 3 && flip_z)) val = -val;
    float* o = out + ((long long)n * 4 + c) * plane + v;
    *o = accumulate ? *o + val : val;
  }
}

// forward convolutions: 0 = mma.sync warp tiles, 1 and 2 = halo tiles, 3 = tcgen05 with one
// TMA box per tap where the shape allows (slower on B200 with these 16-byte-wide boxes: the
// copy engine issues one request per 16-byte row, and 27 times per voxel)
int g_engine = 2;

// cuTensorMapEncodeTiled from the driver (fetched once, no link against libcuda); threads that ask
// at the same time wait for the one that fetches it.
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    const bool found = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
                       q == cudaDriverEntryPointSuccess;
    return found ? (PFN_cuTensorMapEncodeTiled_v12000)p : nullptr;
  }();
  return fn;
}

// Tensor map of BF16 tiles (no swizzle, zero fill).  The encoder fails on a thread that has not
// used the device yet and so has no current context (the kernel launch that follows would give
// it one): such a thread gets the runtime's and tries once more.
bool encode_tiles(CUtensorMap& map, int rank, const void* p, const cuuint64_t* dim, const cuuint64_t* str,
                  const cuuint32_t* box) {
  const PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint32_t one[5] = {1, 1, 1, 1, 1};
  const auto encode = [&] {
    return enc(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(p), dim, str, box, one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  if (encode()) return true;
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess && encode();
}

// The TMA-fed kernel takes tiles of 128 voxels that are whole rows or part of one row.
bool tma_tiles_fit(int h, int w) {
  if (w >= TC_M) return w % TC_M == 0;
  return TC_M % w == 0 && h % (TC_M / w) == 0;
}
__device__ int g_tc_err;  // set by a tcgen05 kernel whose wait gave up

// Device address of g_tc_err, looked up once per device under a lock (host code cannot
// use the symbol itself as a device address).
int* tc_err_ptr() {
  static int* ptrs[64] = {nullptr};
  static std::mutex lock;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> guard(lock);
  if (!ptrs[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_tc_err) != cudaSuccess) return nullptr;
    ptrs[dev] = (int*)p;
  }
  return ptrs[dev];
}

unsigned blocks_for(long long count, int per) { return (unsigned)((count + per - 1) / per); }

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

int sm_count() {
  static std::atomic<int> counts[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  int c = counts[dev].load(std::memory_order_relaxed);
  if (!c) {
    if (cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || c <= 0) c = 148;
    counts[dev].store(c, std::memory_order_relaxed);
  }
  return c;
}

// Raises a kernel's dynamic shared memory limit once per device.
template <class K>
bool allow_smem(K kernel, int bytes, std::atomic<unsigned long long>& done) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if ((done.load(std::memory_order_acquire) >> dev) & 1ull) return true;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return false;
  done.fetch_or(1ull << dev, std::memory_order_release);
  return true;
}

// Tile of a halo convolution: x width (8 or 16), planes along R, which axis is P.  The
// model counts cycles of the longest block: MMAs (33 + N / 4 cycles of operand reads or N / 2
// of arithmetic, measured on B200) against staged bytes, and the fixed cost of an iteration.
struct HaloPlan {
  HaloArgs a;
  int bx;
  unsigned grid;
  uint32_t smem;
};

bool halo_plan(const Geo& g, int cin, int cout, int sms, HaloPlan& best) {
  const int kcs = cin / 16, nj = 256 / cout < 3 ? 256 / cout : 3;
  const uint32_t wslice = 27u * cout * 32u;
  double best_cost = 1e300;
  for (int bx = 8; bx <= 16; bx += 8)
    for (int swap = 0; swap < 2; swap++)
      for (int br = 1; 2 * (bx / 8) * br * cout <= 512; br++) {
        HaloArgs a{};
        a.n = g.n;
        a.w = g.w;
        a.np = swap ? g.d : g.h;
        a.nr = swap ? g.h : g.d;
        const long long sy = g.w, sz = (long long)g.w * g.h;
        a.sp = swap ? sz : sy;
        a.sr = swap ? sy : sz;
        a.sn = sz * g.d;
        a.tap_p = swap ? 9 : 3;
        a.tap_r = swap ? 3 : 9;
        a.cin = cin;
        a.kcs = kcs;
        a.br = br;
        a.tx = g.w / bx;
        a.tp = (a.np + HT_P - 1) / HT_P;
        a.tr = (a.nr + br - 1) / br;
        const long long tiles = (long long)a.tx * a.tp * a.tr * a.n;
        if (tiles > 0x7fffffffLL / (kcs + 1)) continue;
        a.tiles = (int)tiles;
        const uint32_t raw = (uint32_t)(br + 2) * (HT_P + 2) * (bx + 2) * 16u;
        a.plane = raw + (192u - raw % 128u) % 128u;
        a.slab = 2 * a.plane;
        a.wres = 2 * a.slab + kcs * wslice <= (uint32_t)HT_MAX_SMEM;
        a.stage = a.slab + (a.wres ? 0u : wslice);
        const uint32_t smem = 2 * a.stage + (a.wres ? kcs * wslice : 0u);
        if (smem > (uint32_t)HT_MAX_SMEM) break;
        a.cols = (bx / 8) * br * cout;
        a.alloc = 32;
        while (a.alloc < 2 * a.cols) a.alloc *= 2;
        double mma = 0;
        for (int r = 0; r < br + 2; r++)
          for (int j0 = r < 2 ? 2 - r : 0, j1 = br + 1 - r < 2 ? br + 1 - r : 2; j0 <= j1; j0 += nj) {
            const int n = (j1 - j0 + 1 < nj ? j1 - j0 + 1 : nj) * cout;
            mma += 9.0 * (bx / 8) * (n / 2 > 33 + n / 4 ? n / 2 : 33 + n / 4);
          }
        const double load = a.stage / 24.0;
        const double cost = (double)((tiles + sms - 1) / sms) * kcs * ((mma > load ? mma : load) + 800.0) +
                            (a.wres ? kcs * wslice / 24.0 : 0.0);
        if (cost < best_cost) {
          best_cost = cost;
          best.a = a;
          best.bx = bx;
          best.grid = (unsigned)(tiles < sms ? tiles : sms);
          best.smem = smem;
        }
      }
  return best_cost < 1e300;
}

template <int COUT, int BX, bool UP>
int halo_launch(const bf16* in, const bf16* w, const float* bias, bf16* out, const HaloPlan& p, int* err,
                cudaStream_t s) {
  static std::atomic<unsigned long long> done{0};
  if (!allow_smem(conv_halo_kernel<COUT, BX, UP>, HT_MAX_SMEM, done)) return launched("nn_conv3d_fwd (shared memory)");
  launch_chained_smem(conv_halo_kernel<COUT, BX, UP>, p.grid, HT_THREADS, p.smem, s, in, w, bias, out, p.a, err);
  return launched("nn_conv3d_fwd (tcgen05)");
}

// Convolution of `in`, or, with cu > 0, of the nearest-upsampled `low` (cu channels) beside it.
template <int COUT>
int halo_conv(const bf16* in, const bf16* w, const float* bias, bf16* out, const Geo& g, int cin, int relu, int* err,
              cudaStream_t s, const bf16* low = nullptr, int cu = 0) {
  HaloPlan p{};
  if (!halo_plan(g, cin + cu, COUT, sm_count(), p)) return fail("nn_conv3d_fwd: no tile for %d x %d x %d", g.d, g.h, g.w);
  p.a.relu = relu;
  if (cu) {
    const bool z_is_p = p.a.tap_p == 9;
    const long long ly = g.w / 2, lz = ly * (g.h / 2);
    p.a.low = low;
    p.a.kcu = cu / 16;
    p.a.cu = cu;
    p.a.cs = cin;
    p.a.lp = z_is_p ? lz : ly;
    p.a.lr = z_is_p ? ly : lz;
    p.a.ln = lz * (g.d / 2);
    return p.bx == 16 ? halo_launch<COUT, 16, true>(in, w, bias, out, p, err, s)
                      : halo_launch<COUT, 8, true>(in, w, bias, out, p, err, s);
  }
  return p.bx == 16 ? halo_launch<COUT, 16, false>(in, w, bias, out, p, err, s)
                    : halo_launch<COUT, 8, false>(in, w, bias, out, p, err, s);
}

// Tensor map over channels-last activations seen as (8 channels, x, ...): the 8-channel groups
// are an axis of their own, before (group_first) or after y, and z runs over the whole batch.
bool activation_map(CUtensorMap& map, const void* p, const Geo& g, int c, bool group_first, int bx, int by, int bg) {
  if ((long long)g.n * g.d > 0x7fffffffLL) return false;
  const cuuint64_t row = (cuuint64_t)g.w * c * 2;
  const cuuint64_t ng = (cuuint64_t)c / 8, nh = (cuuint64_t)g.h;
  const cuuint64_t dim[5] = {8, (cuuint64_t)g.w, group_first ? ng : nh, group_first ? nh : ng, (cuuint64_t)g.n * g.d};
  const cuuint64_t str[4] = {(cuuint64_t)c * 2, group_first ? 16 : row, group_first ? row : 16, row * nh};
  const cuuint32_t box[5] = {8, (cuuint32_t)bx, (cuuint32_t)(group_first ? bg : by), (cuuint32_t)(group_first ? by : bg), 1};
  return encode_tiles(map, 5, p, dim, str, box);
}

// Tile of the weight gradient: y rows and z planes of a block's slab.  The model counts cycles
// per voxel of MMAs (operand reads, or N / 2 of arithmetic) and of copied 16-byte rows.
struct BwPlan {
  BwArgs a;
  unsigned grid;
  uint32_t smem;
};

bool bw_plan(const Geo& g, int cin, int cout, int ci, int co, int sms, BwPlan& best) {
  double best_cost = 1e300;
  const double read = ci == 16 ? 16 : 32;
  for (int bp = 4; bp <= 16; bp += 4)
    for (int br = 1; bp * br <= BT_STEPS; br++) {
      BwArgs a{};
      a.n = g.n;
      a.d = g.d;
      a.h = g.h;
      a.w = g.w;
      a.cin = cin;
      a.cout = cout;
      a.bp = bp;
      a.br = br;
      a.tx = (g.w + 15) / 16;
      a.tp = (g.h + bp - 1) / bp;
      a.tr = (g.d + br - 1) / br;
      const long long tiles = (long long)a.tx * a.tp * a.tr * a.n;
      if (tiles > 0x3fffffffLL) continue;
      a.tiles = (int)tiles;
      a.slices = cin / ci;
      a.units = a.slices * (cout / co);
      a.per_unit = sms / a.units;
      if (a.per_unit < 1) a.per_unit = 1;
      if (a.per_unit > a.tiles) a.per_unit = a.tiles;
      a.xplane = (uint32_t)(16 * 18 * (ci / 8) * (bp + 3) + 127) / 128 * 128;
      a.yplane = (uint32_t)bp * 256 * (co / 8);
      a.stage = (br + 2) * a.xplane + br * a.yplane;
      if (2 * a.stage > (uint32_t)BT_MAX_SMEM) break;
      double mma = 0;
      for (int r = 0; r < br + 2; r++) {
        const int j0 = r < 2 ? 2 - r : 0, j1 = br + 1 - r < 2 ? br + 1 - r : 2;
        const double n = (j1 - j0 + 1) * co;
        mma += 3.0 * bp * (n / 2 > read + n / 4 ? n / 2 : read + n / 4 + 1);
      }
      const double rows = a.stage / 16.0;
      const double cost = (double)((tiles + a.per_unit - 1) / a.per_unit) * ((mma > rows ? mma : rows) + (co == 16 ? 500.0 : 1200.0));
      if (cost < best_cost) {
        best_cost = cost;
        best.a = a;
        best.grid = (unsigned)(a.units * a.per_unit);
        best.smem = 2 * a.stage;
      }
    }
  return best_cost < 1e300;
}

// 1: launched, 0: not this path (no tensor map), -1: error.
template <int CI, int CO>
int bw_launch(const bf16* in, const bf16* dout, float* dw, const Geo& g, int cin, int cout, cudaStream_t s) {
  static std::atomic<unsigned long long> allowed{0};
  BwPlan p{};
  CUtensorMap xmap, ymap;
  int* err = tc_err_ptr();
  if (!err || !bw_plan(g, cin, cout, CI, CO, sm_count(), p) ||
      !activation_map(xmap, in, g, cin, true, 18, p.a.bp + 3, CI / 8) ||
      !activation_map(ymap, dout, g, cout, false, 16, p.a.bp, CO / 8))
    return 0;
  if (!allow_smem(conv_bwdw_tc_kernel<CI, CO>, BT_MAX_SMEM, allowed)) return launched("nn_conv3d_bwd_weight") ? -1 : 0;
  launch_chained_smem(conv_bwdw_tc_kernel<CI, CO>, p.grid, BT_THREADS, p.smem, s, xmap, ymap, dw, p.a, err);
  return launched("nn_conv3d_bwd_weight (tcgen05)") ? -1 : 1;
}

// Whole groups of 8 channels on 16-byte boundaries, rows that fit the grid's x axis.
template <class... P>
bool grouped(int c, long long rows, const P*... p) {
  return c % 8 == 0 && rows <= 0x7fffffffLL && (aligned16(p) && ...);
}
// One block row per row of the box, up to four blocks of 256 threads along it.
dim3 row_grid(long long rows, int per_row) {
  return dim3((unsigned)rows, (unsigned)(per_row > 1024 ? 4 : (per_row + 255) / 256));
}

bool geo_ok(int n, int d, int h, int w) { return n > 0 && d > 0 && h > 0 && w > 0; }

}  // namespace

extern "C" {

int32_t nn_abi_version(void) { return UNET3D_ABI_VERSION; }

const char* nn_last_error(void) { return g_err.c_str(); }

int32_t nn_conv3d_fwd(const void* in, const void* w, const float* bias, void* out, int32_t n, int32_t d, int32_t h,
                      int32_t wd, int32_t cin, int32_t cout, int32_t relu, void* stream) {
  if (!in || !w || !out || !geo_ok(n, d, h, wd)) return fail("nn_conv3d_fwd: null pointer or empty shape");
  if (wd % 16 || cin % 16 || cin <= 0) return fail("nn_conv3d_fwd: W (%d) and Cin (%d) must be multiples of 16", wd, cin);
  const Geo g{n, d, h, wd};
  const long long tiles = (long long)n * d * h * (wd / 16);
  const unsigned grid = blocks_for(tiles, 4);
  cudaStream_t s = (cudaStream_t)stream;
  const bf16* I = (const bf16*)in;
  const bf16* W = (const bf16*)w;
  bf16* O = (bf16*)out;
  if (g_engine != 0) {
    int* err = tc_err_ptr();
    if (!err) return fail("nn_conv3d_fwd: no device address for the error word");
    const bool enc = g_engine == 3 && tensor_map_encoder();
    if (enc && tma_tiles_fit(h, wd) && cin % 16 == 0) {
      CUtensorMap xmap, wmap;
      const cuuint64_t xdim[5] = {(cuuint64_t)cin, (cuuint64_t)wd, (cuuint64_t)h, (cuuint64_t)d, (cuuint64_t)n};
      const cuuint64_t xstr[4] = {(cuuint64_t)cin * 2, (cuuint64_t)wd * cin * 2, (cuuint64_t)h * wd * cin * 2,
                                  (cuuint64_t)d * h * wd * cin * 2};
      const int bw = wd < TC_M ? wd : TC_M;
      const cuuint32_t xbox[5] = {8, (cuuint32_t)bw, (cuuint32_t)(TC_M / bw), 1, 1};
      const cuuint64_t wdim[3] = {(cuuint64_t)cin, (cuuint64_t)cout, 27};
      const cuuint64_t wstr[2] = {(cuuint64_t)cin * 2, (cuuint64_t)cout * cin * 2};
      const cuuint32_t wbox[3] = {8, (cuuint32_t)cout, 1};
      if (!encode_tiles(xmap, 5, in, xdim, xstr, xbox) || !encode_tiles(wmap, 3, w, wdim, wstr, wbox))
        return fail("nn_conv3d_fwd: tensor map encoding failed");
      const unsigned tgrid = (unsigned)((long long)n * d * (h / (TC_M / bw)) * (wd / bw));
      switch (cout) {
        case 16: launch_chained_smem(conv_fwd_tma_kernel<16>, tgrid, TC_M, 0, s, xmap, wmap, bias, O, g, cin, relu,
                                     err); break;
        case 32: launch_chained_smem(conv_fwd_tma_kernel<32>, tgrid, TC_M, 0, s, xmap, wmap, bias, O, g, cin, relu,
                                     err); break;
        case 48: launch_chained_smem(conv_fwd_tma_kernel<48>, tgrid, TC_M, 0, s, xmap, wmap, bias, O, g, cin, relu,
                                     err); break;
        case 64: launch_chained_smem(conv_fwd_tma_kernel<64>, tgrid, TC_M, 0, s, xmap, wmap, bias, O, g, cin, relu,
                                     err); break;
        case 96: launch_chained_smem(conv_fwd_tma_kernel<96>, tgrid, TC_M, 0, s, xmap, wmap, bias, O, g, cin, relu,
                                     err); break;
        default: return fail("nn_conv3d_fwd: Cout %d not in {16, 32, 48, 64, 96}", cout);
      }
      return launched("nn_conv3d_fwd (tcgen05, TMA)");
    }
    if (aligned16(in) && aligned16(w) && aligned16(out)) {
      switch (cout) {
        case 16: return halo_conv<16>(I, W, bias, O, g, cin, relu, err, s);
        case 32: return halo_conv<32>(I, W, bias, O, g, cin, relu, err, s);
        case 48: return halo_conv<48>(I, W, bias, O, g, cin, relu, err, s);
        case 64: return halo_conv<64>(I, W, bias, O, g, cin, relu, err, s);
        case 96: return halo_conv<96>(I, W, bias, O, g, cin, relu, err, s);
        default: return fail("nn_conv3d_fwd: Cout %d not in {16, 32, 48, 64, 96}", cout);
      }
    }
  }
  switch (cout) {
    case 16: launch_chained_smem(conv_fwd_kernel<2>, grid, 128, 0, s, I, W, bias, O, g, cin, relu, tiles); break;
    case 32: launch_chained_smem(conv_fwd_kernel<4>, grid, 128, 0, s, I, W, bias, O, g, cin, relu, tiles); break;
    case 48: launch_chained_smem(conv_fwd_kernel<6>, grid, 128, 0, s, I, W, bias, O, g, cin, relu, tiles); break;
    case 64: launch_chained_smem(conv_fwd_kernel<8>, grid, 128, 0, s, I, W, bias, O, g, cin, relu, tiles); break;
    case 96: launch_chained_smem(conv_fwd_kernel<12>, grid, 128, 0, s, I, W, bias, O, g, cin, relu, tiles); break;
    default: return fail("nn_conv3d_fwd: Cout %d not in {16, 32, 48, 64, 96}", cout);
  }
  return launched("nn_conv3d_fwd");
}

int32_t nn_conv3d_up2cat_fwd(const void* low, const void* skip, const void* w, const float* bias, void* out, int32_t n,
                             int32_t d, int32_t h, int32_t wd, int32_t cu, int32_t cs, int32_t cout, int32_t relu,
                             void* stream) {
  if (!low || !skip || !w || !out || !geo_ok(n, d, h, wd)) return fail("nn_conv3d_up2cat_fwd: null pointer or empty shape");
  if (wd % 16 || d % 2 || h % 2 || cu % 16 || cs % 16 || cu <= 0 || cs <= 0)
    return fail("nn_conv3d_up2cat_fwd: W and the channels must be multiples of 16, D and H even");
  if ((g_engine != 1 && g_engine != 2) || (cout != 16 && cout != 32) || !aligned16(low) || !aligned16(skip) ||
      !aligned16(w) || !aligned16(out))
    return -1;
  int* err = tc_err_ptr();
  if (!err) return fail("nn_conv3d_up2cat_fwd: no device address for the error word");
  const auto run = cout == 16 ? halo_conv<16> : halo_conv<32>;
  return run((const bf16*)skip, (const bf16*)w, bias, (bf16*)out, Geo{n, d, h, wd}, cs, relu, err, (cudaStream_t)stream,
             (const bf16*)low, cu);
}

int32_t nn_set_conv_engine(int32_t engine) {
  if (engine < 0 || engine > 3) {
    fail("nn_set_conv_engine: engine must be 0 (mma.sync), 1 (tcgen05), 2 (the default, tcgen05 as well) or 3 (tcgen05, TMA-fed)");
    return -1;
  }
  const int prev = g_engine;
  g_engine = engine;
  g_err.clear();
  return prev;
}

int32_t nn_conv_uses_tma(int32_t h, int32_t wd, int32_t cin, int32_t cout) {
  (void)cout;
  return (g_engine == 3 && tensor_map_encoder() && tma_tiles_fit(h, wd) && cin % 16 == 0) ? 1 : 0;
}

int32_t nn_tc_status(void* stream) {
  int* err = tc_err_ptr();
  if (!err) return fail("nn_tc_status: no device address for the error word");
  int h = 0;
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return launched("nn_tc_status");
  if (h) {
    cudaMemsetAsync(err, 0, sizeof(int), s);
    return fail("a tcgen05 convolution gave up waiting for its MMA (error word %d)", h);
  }
  return 0;
}

int32_t nn_wait_selftest(int32_t polls, void* stream) {
  if (polls < 1 || polls > TC_WAIT_POLLS) return fail("nn_wait_selftest: polls %d outside [1, %d]", polls, TC_WAIT_POLLS);
  int* err = tc_err_ptr();
  if (!err) return fail("nn_wait_selftest: no device address for the error word");
  launch_chained_smem(tc_wait_probe_kernel, 1, 32, 0, (cudaStream_t)stream, polls, err);
  const int rc = launched("nn_wait_selftest");
  if (rc) return rc;
  return nn_tc_status(stream);
}

int32_t nn_conv3d_flip(const void* w, void* wt, int32_t cin, int32_t cout, void* stream) {
  if (!w || !wt || cin <= 0 || cout <= 0) return fail("nn_conv3d_flip: bad arguments");
  const int total = 27 * cin * cout;
  launch_chained_smem(flip_kernel, blocks_for(total, 256), 256, 0, (cudaStream_t)stream, (const bf16*)w, (bf16*)wt,
                      cin, cout);
  return launched("nn_conv3d_flip");
}

int32_t nn_conv3d_bwd_weight(const void* in, const void* dout, float* dw, int32_t n, int32_t d, int32_t h, int32_t wd,
                             int32_t cin, int32_t cout, void* stream) {
  if (!in || !dout || !dw || !geo_ok(n, d, h, wd)) return fail("nn_conv3d_bwd_weight: null pointer or empty shape");
  if (cin % 16 || cin <= 0) return fail("nn_conv3d_bwd_weight: Cin %d must be a multiple of 16", cin);
  const long long vox = (long long)n * d * h * wd;
  const long long chunk = 4096;
  dim3 grid(blocks_for(vox, (int)chunk), (unsigned)(cin / 16), 27);
  const Geo g{n, d, h, wd};
  cudaStream_t s = (cudaStream_t)stream;
  const bf16* I = (const bf16*)in;
  const bf16* D = (const bf16*)dout;
  if (cout != 16 && cout != 32 && cout != 64) return fail("nn_conv3d_bwd_weight: Cout %d not in {16, 32, 64}", cout);
  if (aligned16(in) && aligned16(dout)) {
    const int rc = cin % 32 == 0 ? (cout == 16 ? bw_launch<32, 16>(I, D, dw, g, cin, cout, s)
                                               : bw_launch<32, 32>(I, D, dw, g, cin, cout, s))
                                 : (cout == 16 ? bw_launch<16, 16>(I, D, dw, g, cin, cout, s)
                                               : bw_launch<16, 32>(I, D, dw, g, cin, cout, s));
    if (rc) return rc < 0 ? 1 : 0;
  }
  switch (cout) {
    case 16: launch_chained_smem(conv_bwdw_kernel<1>, grid, 128, 0, s, I, D, dw, g, cin, vox, chunk); break;
    case 32: launch_chained_smem(conv_bwdw_kernel<2>, grid, 128, 0, s, I, D, dw, g, cin, vox, chunk); break;
    case 64: launch_chained_smem(conv_bwdw_kernel<4>, grid, 128, 0, s, I, D, dw, g, cin, vox, chunk); break;
    default: return fail("nn_conv3d_bwd_weight: Cout %d not in {16, 32, 64}", cout);
  }
  return launched("nn_conv3d_bwd_weight");
}

int32_t nn_bias_grad(const void* dout, float* db, int64_t voxels, int32_t c, void* stream) {
  if (!dout || !db || voxels <= 0 || c <= 0 || c > 256) return fail("nn_bias_grad: bad arguments");
  if (grouped(c, 0, dout)) {
    const long long groups = voxels * (c / 8);
    unsigned grid = blocks_for(groups, 256 * 4);
    if (grid > 1184u) grid = 1184u;  // eight blocks on each of 148 SMs: 14 groups a thread at 2 M voxels
    launch_chained_smem(bias_grad8_kernel, grid, 256, c * sizeof(float), (cudaStream_t)stream, (const bf16*)dout, db,
                        groups, c);
    return launched("nn_bias_grad");
  }
  const long long total = voxels * c;
  unsigned grid = blocks_for(total, 256 * 16);
  if (grid > 4096) grid = 4096;
  launch_chained_smem(bias_grad_kernel, grid, 256, c * sizeof(float), (cudaStream_t)stream, (const bf16*)dout, db,
                      voxels, c);
  return launched("nn_bias_grad");
}

int32_t nn_relu_bwd(void* dy, const void* y, int64_t count, void* stream) {
  if (!dy || !y || count < 0) return fail("nn_relu_bwd: bad arguments");
  if (count == 0) return 0;
  if (count % 8 == 0 && aligned16(dy) && aligned16(y)) {
    launch_chained_smem(relu_bwd8_kernel, blocks_for(count / 8, 256), 256, 0, (cudaStream_t)stream, (uint4*)dy,
                        (const uint4*)y, count / 8);
    return launched("nn_relu_bwd");
  }
  launch_chained_smem(relu_bwd_kernel, blocks_for(count, 256), 256, 0, (cudaStream_t)stream, (bf16*)dy,
                      (const bf16*)y, count);
  return launched("nn_relu_bwd");
}

int32_t nn_pool2(const void* in, void* out, int32_t n, int32_t d, int32_t h, int32_t wd, int32_t c, void* stream) {
  if (!in || !out || !geo_ok(n, d, h, wd) || c <= 0 || d % 2 || h % 2 || wd % 2) return fail("nn_pool2: bad shape");
  const long long rows = (long long)n * (d / 2) * (h / 2);
  if (grouped(c, rows, in, out)) {
    launch_chained_smem(pool2x8_kernel, row_grid(rows, wd / 2 * (c / 8)), 256, 0, (cudaStream_t)stream, (const bf16*)in,
                        (bf16*)out, Geo{n, d, h, wd}, c);
    return launched("nn_pool2");
  }
  const long long count = (long long)n * (d / 2) * (h / 2) * (wd / 2) * c;
  launch_chained_smem(pool2_kernel, blocks_for(count, 256), 256, 0, (cudaStream_t)stream, (const bf16*)in, (bf16*)out,
                      Geo{n, d, h, wd}, c, count);
  return launched("nn_pool2");
}

int32_t nn_pool2_bwd(const void* dout, void* din, int32_t n, int32_t d, int32_t h, int32_t wd, int32_t c,
                     int32_t accumulate, void* stream) {
  if (!dout || !din || !geo_ok(n, d, h, wd) || c <= 0 || d % 2 || h % 2 || wd % 2) return fail("nn_pool2_bwd: bad shape");
  const long long rows = (long long)n * d * h;
  if (grouped(c, rows, dout, din)) {
    launch_chained_smem(pool2x8_bwd_kernel, row_grid(rows, wd * (c / 8)), 256, 0, (cudaStream_t)stream,
                        (const bf16*)dout, (bf16*)din, Geo{n, d, h, wd}, c, accumulate);
    return launched("nn_pool2_bwd");
  }
  const long long count = (long long)n * d * h * wd * c;
  launch_chained_smem(pool2_bwd_kernel, blocks_for(count, 256), 256, 0, (cudaStream_t)stream, (const bf16*)dout,
                      (bf16*)din, Geo{n, d, h, wd}, c, accumulate, count);
  return launched("nn_pool2_bwd");
}

int32_t nn_up2_concat(const void* low, const void* skip, void* out, int32_t n, int32_t d, int32_t h, int32_t wd,
                      int32_t cu, int32_t cs, void* stream) {
  if (!low || !skip || !out || !geo_ok(n, d, h, wd) || cu <= 0 || cs <= 0 || d % 2 || h % 2 || wd % 2)
    return fail("nn_up2_concat: bad shape");
  const long long rows = (long long)n * d * h;
  if (cu % 8 == 0 && grouped(cs, rows, low, skip, out)) {
    launch_chained_smem(up2_concat8_kernel, row_grid(rows, wd * ((cu + cs) / 8)), 256, 0, (cudaStream_t)stream,
                        (const uint4*)low, (const uint4*)skip, (uint4*)out, Geo{n, d, h, wd}, cu / 8, cs / 8);
    return launched("nn_up2_concat");
  }
  const long long count = (long long)n * d * h * wd * (cu + cs);
  launch_chained_smem(up2_concat_kernel, blocks_for(count, 256), 256, 0, (cudaStream_t)stream, (const bf16*)low,
                      (const bf16*)skip, (bf16*)out, Geo{n, d, h, wd}, cu, cs, count);
  return launched("nn_up2_concat");
}

int32_t nn_up2_concat_bwd(const void* dcat, void* dlow, void* dskip, int32_t n, int32_t d, int32_t h, int32_t wd,
                          int32_t cu, int32_t cs, void* stream) {
  if (!dcat || !dlow || !dskip || !geo_ok(n, d, h, wd) || cu <= 0 || cs <= 0 || d % 2 || h % 2 || wd % 2)
    return fail("nn_up2_concat_bwd: bad shape");
  cudaStream_t s = (cudaStream_t)stream;
  const long long coarse = (long long)n * (d / 2) * (h / 2), rows = coarse + (long long)n * d * h;
  if (cu % 8 == 0 && grouped(cs, rows, dcat, dlow, dskip)) {
    const int per_row = wd / 2 * (cu / 8) > wd * (cs / 8) ? wd / 2 * (cu / 8) : wd * (cs / 8);
    launch_chained_smem(up2_concat8_bwd_kernel, row_grid(rows, per_row), 256, 0, s, (const bf16*)dcat, (bf16*)dlow,
                        (uint4*)dskip, Geo{n, d, h, wd}, cu / 8, cs / 8, (unsigned)coarse);
    return launched("nn_up2_concat_bwd");
  }
  const long long cl = (long long)n * (d / 2) * (h / 2) * (wd / 2) * cu;
  launch_chained_smem(up2_concat_bwd_low_kernel, blocks_for(cl, 256), 256, 0, s, (const bf16*)dcat, (bf16*)dlow,
                      Geo{n, d, h, wd}, cu, cs, cl);
  const long long cf = (long long)n * d * h * wd * cs;
  launch_chained_smem(up2_concat_bwd_skip_kernel, blocks_for(cf, 256), 256, 0, s, (const bf16*)dcat, (bf16*)dskip, cu,
                      cs, cf);
  return launched("nn_up2_concat_bwd");
}

int32_t nn_mse(const void* out, const float* target, const uint8_t* mask, const float* cw, void* dout, double* loss,
               int64_t voxels, int32_t cpad, int32_t ct, double count, void* stream) {
  if (!out || !target || !mask || !cw || !dout || !loss || voxels <= 0 || ct <= 0 || ct > cpad || !(count > 0))
    return fail("nn_mse: bad arguments");
  const unsigned grid = blocks_for(voxels, 256) < 1184u ? blocks_for(voxels, 256) : 1184u;
  const auto kernel = cpad == 16 && ct == 4 && aligned16(out) && aligned16(target) && aligned16(dout) ? mse_kernel<true>
                                                                                                     : mse_kernel<false>;
  launch_chained_smem(kernel, grid, 256, 0, (cudaStream_t)stream, (const bf16*)out, target, mask, cw, (bf16*)dout,
                      loss, voxels, cpad, ct, count);
  return launched("nn_mse");
}

int32_t nn_adam(float* w, const float* g, float* m, float* v, void* wb, int64_t count, float lr, float beta1,
                float beta2, float eps, int32_t t, void* stream) {
  if (!w || !g || !m || !v || count < 0 || t < 1) return fail("nn_adam: bad arguments");
  if (count == 0) return 0;
  const float c1 = 1.f - powf(beta1, (float)t), c2 = 1.f - powf(beta2, (float)t);
  launch_chained_smem(adam_kernel, blocks_for(count, 256), 256, 0, (cudaStream_t)stream, w, g, m, v, (bf16*)wb, count,
                      lr, beta1, beta2, eps, c1, c2);
  return launched("nn_adam");
}

int32_t nn_diff_norms(const float* a, const float* b, int64_t count, double* out, void* stream) {
  if (!a || !b || !out || count < 0) return fail("nn_diff_norms: bad arguments");
  if (count == 0) return 0;
  unsigned grid = blocks_for(count, 256 * 8);
  if (grid > 2048) grid = 2048;
  launch_chained_smem(diff_norms_kernel, grid, 256, 0, (cudaStream_t)stream, a, b, count, out);
  return launched("nn_diff_norms");
}

int32_t nn_features_ellipsoid(void* out, int32_t nx, int32_t ny, int32_t nz, const double* center,
                              const double* rot, const double* semi, float re_feature, void* stream) {
  if (!out || !center || !rot || !semi || nx <= 0 || ny <= 0 || nz <= 0) return fail("nn_features_ellipsoid: bad arguments");
  Ellipsoid e{};
  for (int k = 0; k < 3; k++) {
    e.center[k] = center[k];
    e.semi[k] = semi[k];
  }
  for (int k = 0; k < 9; k++) e.rot[k] = rot[k];
  const long long n = (long long)nx * ny * nz;
  launch_chained_smem(features_kernel, blocks_for(n, 256), 256, 0, (cudaStream_t)stream, (bf16*)out, nx, ny, nz, e,
                      re_feature);
  return launched("nn_features_ellipsoid");
}

int32_t nn_unpack_fields(const void* y, float* out, int32_t n, int32_t d, int32_t h, int32_t wd, int32_t flip_y,
                         int32_t flip_z, float weight, int32_t accumulate, void* stream) {
  if (!y || !out || !geo_ok(n, d, h, wd)) return fail("nn_unpack_fields: bad arguments");
  const long long count = (long long)n * d * h * wd;
  launch_chained_smem(unpack_fields_kernel, blocks_for(count, 256), 256, 0, (cudaStream_t)stream, (const bf16*)y, out,
                      Geo{n, d, h, wd}, flip_y, flip_z, weight, accumulate, count);
  return launched("nn_unpack_fields");
}

int32_t nn_to_bf16(const float* x, void* y, int64_t count, void* stream) {
  if (!x || !y || count < 0) return fail("nn_to_bf16: bad arguments");
  if (count == 0) return 0;
  launch_chained_smem(to_bf16_kernel, blocks_for(count, 256), 256, 0, (cudaStream_t)stream, x, (bf16*)y, count);
  return launched("nn_to_bf16");
}

int32_t nn_from_bf16(const void* x, float* y, int64_t count, void* stream) {
  if (!x || !y || count < 0) return fail("nn_from_bf16: bad arguments");
  if (count == 0) return 0;
  launch_chained_smem(from_bf16_kernel, blocks_for(count, 256), 256, 0, (cudaStream_t)stream, (const bf16*)x, y, count);
  return launched("nn_from_bf16");
}

}  // extern "C"
