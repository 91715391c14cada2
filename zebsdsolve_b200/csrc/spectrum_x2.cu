// (b, first stage) The FP32 form's spectrum GEMM on the tcgen05 tensor cores, at FP32 quality: every
// operand is the sum of two FP16 values.
//
//   U[b][j][m'][iq] = Σ_l conj(g_b[l,m']) · Y[pair(m',l)][j·nc + iq]
//
// as the real GEMM per order m' of spectrum_tc.cu (rows ν = 2(j·nc+iq) + (re|im), M = 128 a tile;
// patterns, N = 128 a tile; K = (l, re|im)), each operand scaled by a power of two into FP16's range
// (patterns 2^14: their coefficients have unit norm; the table by its largest value) and split
// x = hi + lo, 11 significant bits each (the table from its FP64 values). The product keeps lo·hi +
// hi·lo + hi·hi; what it drops is 2^-24 of a factor's size.
//
// Accuracy. The tensor cores add into their FP32 accumulator with truncation, so the error grows with
// the accumulator's size at each step: K runs from the highest degree down (a pattern's and a master's
// energy is in the low degrees, which then come last) and, within a block of 32 degrees, the small cross
// products come before hi·hi. Relative error of U against 64 bits (60 × 60 patterns, a 401² master of
// degree 96), this product / k_spectrum_f32's FP32 sums: L = 24 1.07e-7 / 1.25e-7, L = 32 1.13e-7 /
// 1.52e-7, L = 64 1.16e-7 / 2.43e-7, L = 128 1.18e-7 / 3.65e-7. At L = 16 it is 1.05e-7 / 0.84e-7 (too few
// terms for FP32's rounding to add up), so bandwidths below 24 keep k_spectrum_f32, as do those above 128
// (the patterns' operand then does not stay in shared memory).
//
// Bound by writing U (1.06 MB a pattern at L = 64, fold 4). One CTA per (128 patterns, order, group of
// row tiles), 10 warps: bulk copies (the patterns' operand once; the table's blocks through a ring), MMA
// issue into two accumulators of 128 columns, and two groups of four drain warps, one an accumulator.
// 3072 patterns at L = 64: 0.73 ms (4.5 TB/s of U; the shared memory's bandwidth, taken by the operands'
// reads and the drain, is what holds it there) against 3.73 ms of k_spectrum_f32.
#include <cuda_fp16.h>

#include "abi_util.cuh"
#include "tc_util.cuh"

namespace zeb {

constexpr int X2_KB = 64;                        // K-elements per block (one 128-byte swizzled row)
constexpr int X2_BLOCK = 128 * 128;              // bytes of one operand block (128 rows)
constexpr int X2_MAX_KB = 4;                     // K <= 256: L <= 128
constexpr int X2_MIN_L = 24;
constexpr int X2_MAX_STAGES = 7;
constexpr int X2_DRAIN = 8;                      // drain warps: two groups of four, one an accumulator
constexpr int X2_THREADS = 64 + 32 * X2_DRAIN;
constexpr float X2_PATTERN_SCALE = 16384.f;

__host__ __device__ inline int x2_kblocks(int L, int mp) { return (2 * (L - mp) + X2_KB - 1) / X2_KB; }
// blocks of the orders below mp (one operand, one tile, one slice)
__host__ __device__ inline long long x2_blocks_before(int L, int mp) {
  long long o = 0;
  for (int q = 0; q < mp; ++q) o += x2_kblocks(L, q);
  return o;
}
__host__ inline int x2_stages(int kbmax) { return kbmax <= 2 ? 7 : kbmax == 3 ? 6 : 4; }

__device__ __forceinline__ uint16_t f16_bits(float x) { return __half_as_ushort(__float2half_rn(x)); }
__device__ __forceinline__ uint4 pack8(const uint16_t (&v)[8]) {
  return make_uint4(v[0] | ((uint32_t)v[1] << 16), v[2] | ((uint32_t)v[3] << 16), v[4] | ((uint32_t)v[5] << 16),
                    v[6] | ((uint32_t)v[7] << 16));
}

// The table's blocks of order mp, [row tile][K-block][lo, hi], a thread per 16-byte chunk of both
__global__ void k_x2_pack_master(const double2* __restrict__ Y, int L, int ncols, int mtiles, int mp, double scale,
                                 uint8_t* __restrict__ A) {
  const int kb = x2_kblocks(L, mp);
  const long long chunks = (long long)mtiles * kb * 128 * 8;
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= chunks) return;
  const int c16 = (int)(e & 7), row = (int)((e >> 3) & 127);
  const long long blk = e >> 10;
  const int kblock = (int)(blk % kb), mtile = (int)(blk / kb);
  const int nu = mtile * 128 + row;
  const int p0 = mp * L - (mp * (mp - 1)) / 2;
  uint16_t hi[8], lo[8];
  for (int i = 0; i < 8; ++i) {
    const int k = kblock * X2_KB + c16 * 8 + i;
    const int l = L - 1 - (k >> 1);
    double v = 0.0;
    if (l >= mp && nu < 2 * ncols) {
      const double2 y = Y[(size_t)(p0 + l - mp) * ncols + (nu >> 1)];
      v = scale * ((nu & 1) == 0 ? ((k & 1) == 0 ? y.x : y.y) : ((k & 1) == 0 ? y.y : -y.x));
    }
    const __half h = __double2half(v);
    hi[i] = __half_as_ushort(h);
    lo[i] = __half_as_ushort(__double2half(v - (double)__half2float(h)));
  }
  uint8_t* p = A + (size_t)blk * 2 * X2_BLOCK + sw128(row, c16 * 8);
  *(uint4*)p = pack8(lo);
  *(uint4*)(p + X2_BLOCK) = pack8(hi);
}

// The patterns' blocks, [order][pattern tile][K-block][hi, lo]: a block per (K-block, pattern tile, order;
// `most` K-blocks or fewer an order), a thread per 16-byte chunk (four degrees' re and im) of four rows
__global__ void __launch_bounds__(256) k_x2_pack_patterns(const float2* __restrict__ alm, int n_items, int n_pairs, int L,
                                                          int ptiles, int most, uint8_t* __restrict__ B) {
  const int ptile = blockIdx.x / most, kblock = blockIdx.x - ptile * most, mp = blockIdx.y;
  const int kb = x2_kblocks(L, mp);
  if (kblock >= kb) return;
  int before = 0;  // the blocks of the lower orders: a lane sums every 32nd of them
  for (int q = threadIdx.x & 31; q < mp; q += 32) before += x2_kblocks(L, q);
  before = __reduce_add_sync(0xffffffffu, before);
  uint8_t* blk = B + ((size_t)before * ptiles + (size_t)ptile * kb + kblock) * 2 * X2_BLOCK;
  const int p0 = mp * L - (mp * (mp - 1)) / 2;
  const int c16 = threadIdx.x & 7;
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int row = (threadIdx.x >> 3) + 32 * it, b = ptile * 128 + row;
    uint16_t hi[8], lo[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int l = L - 1 - (kblock * (X2_KB / 2) + c16 * 4 + i);
      float2 g = make_float2(0.f, 0.f);
      if (l >= mp && b < n_items) g = __ldg(alm + (size_t)b * n_pairs + p0 + l - mp);
      const float v[2] = {g.x * X2_PATTERN_SCALE, g.y * X2_PATTERN_SCALE};
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const __half h = __float2half_rn(v[q]);
        hi[2 * i + q] = __half_as_ushort(h);
        lo[2 * i + q] = f16_bits(v[q] - __half2float(h));
      }
    }
    uint8_t* p = blk + sw128(row, c16 * 8);
    *(uint4*)p = pack8(hi);
    *(uint4*)(p + X2_BLOCK) = pack8(lo);
  }
}

struct X2Args {
  int L, nb, nc, mtiles, ptiles, n_items;
  const uint8_t *A, *B;
  float* U;
  int* status;      // nonzero after a timed-out wait (what the CTA was waiting on)
  long long limit;  // nanoseconds before a wait gives up
  long long stall;  // > 0: the failure test (the MMA thread first waits on `never`)
  int per;          // row tiles per CTA (blockIdx.z picks the group)
  int kbmax, stages;
  float inv;        // 1 / (the two operands' scales)
};

struct X2Control {
  uint64_t b_full, a_full[X2_MAX_STAGES], a_empty[X2_MAX_STAGES], acc_full[2], acc_empty[2], mma_done, never;
  long long blocks_before;
  uint32_t tmem;
};

__host__ inline size_t x2_smem(int kbmax) {
  return (size_t)(2 * kbmax + x2_stages(kbmax) + 2) * X2_BLOCK + sizeof(X2Control) + 1024;
}

__global__ void __launch_bounds__(X2_THREADS, 1) k_spectrum_x2(X2Args a) {
  extern __shared__ __align__(1024) uint8_t x2_smem_raw[];
  uint8_t* sb = (uint8_t*)(((uintptr_t)x2_smem_raw + 1023) & ~(uintptr_t)1023);  // [K-block][hi, lo]
  uint8_t* sa = sb + (size_t)2 * a.kbmax * X2_BLOCK;                              // the ring
  uint8_t* so = sa + (size_t)a.stages * X2_BLOCK;                                 // 4 KB a drain warp
  X2Control& s = *reinterpret_cast<X2Control*>(so + (size_t)2 * X2_BLOCK);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ptile = blockIdx.x, mp = blockIdx.y;
  const int kb = x2_kblocks(a.L, mp);
  const int mt0 = blockIdx.z * a.per;
  const int mtiles = max(0, min(a.mtiles - mt0, a.per));
  const int nst = a.stages;
  if (threadIdx.x == 0) {
    mbar_init(&s.b_full, 1);
    mbar_init(&s.mma_done, 1);
    mbar_init(&s.never, 1);  // nothing arrives: the failure test's wait
    s.blocks_before = x2_blocks_before(a.L, mp);
    for (int i = 0; i < nst; ++i) {
      mbar_init(&s.a_full[i], 1);
      mbar_init(&s.a_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s.acc_full[i], 1);
      mbar_init(&s.acc_empty[i], 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s.tmem)),
                 "r"(256));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s.tmem;
  const long long lim = a.limit;

  if (warp == 0) {
    if (lane == 0) {
      // the patterns' operand once, then the table block by block through the ring
      const uint8_t* bsrc = a.B + (size_t)(s.blocks_before * a.ptiles + (long long)ptile * kb) * 2 * X2_BLOCK;
      mbar_expect_tx(&s.b_full, kb * 2 * X2_BLOCK);
      for (int k = 0; k < 2 * kb; ++k) bulk_g2s(sb + k * X2_BLOCK, bsrc + (size_t)k * X2_BLOCK, X2_BLOCK, &s.b_full);
      const uint8_t* asrc = a.A + (size_t)(s.blocks_before * a.mtiles + (long long)mt0 * kb) * 2 * X2_BLOCK;
      const int total = mtiles * kb * 2;
      int it = 0, st = 0, ph = 0;
      for (; it < total; ++it) {
        if (!mbar_wait(&s.a_empty[st], ph ^ 1, lim)) break;
        mbar_expect_tx(&s.a_full[st], X2_BLOCK);
        bulk_g2s(sa + st * X2_BLOCK, asrc + (size_t)it * X2_BLOCK, X2_BLOCK, &s.a_full[st]);
        if (++st == nst) { st = 0; ph ^= 1; }
      }
      if (it < total) atomicOr(a.status, 1);
      // the copies still in flight land before the CTA may leave, whether or not the MMAs took them
      mbar_wait(&s.b_full, 0, kDrainNs);
      for (int i = (it > nst ? it - nst : 0); i < it; ++i) mbar_wait(&s.a_full[i % nst], (i / nst) & 1, kDrainNs);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // kind::f16: F32 accumulate, FP16 A and B, both K-major, N = 128, M = 128
      const uint32_t idesc = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
      bool ok = mbar_wait(&s.b_full, 0, lim);
      if (a.stall > 0 && !mbar_wait(&s.never, 0, a.stall)) ok = false;  // the failure test
      int st = 0, ph = 0;
      const uint32_t b0 = smem_addr(sb), a0 = smem_addr(sa);
      for (int mt = 0; mt < mtiles && ok; ++mt) {
        const int acc = mt & 1;
        ok = mbar_wait(&s.acc_empty[acc], ((mt >> 1) & 1) ^ 1, lim);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = tmem + (uint32_t)(acc * 128);
        for (int k = 0; k < 2 * kb; ++k) {  // (even: the table's lo block; odd: its hi block)
          ok = mbar_wait(&s.a_full[st], ph, lim);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t ab = a0 + st * X2_BLOCK, bh = b0 + (k >> 1) * 2 * X2_BLOCK, bl = bh + X2_BLOCK;
          const uint32_t first = (k & 1) ? bl : bh;
#pragma unroll
          for (int ks = 0; ks < X2_KB / 16; ++ks)
            umma_f16(d, umma_desc(ab + ks * 32), umma_desc(first + ks * 32), idesc, (k | ks) != 0);
          if (k & 1) {
#pragma unroll
            for (int ks = 0; ks < X2_KB / 16; ++ks)
              umma_f16(d, umma_desc(ab + ks * 32), umma_desc(bh + ks * 32), idesc, 1);
          }
          umma_commit(&s.a_empty[st]);  // the stage is free once these MMAs have read it
          if (++st == nst) { st = 0; ph ^= 1; }
        }
        if (!ok) break;
        umma_commit(&s.acc_full[acc]);
      }
      if (!ok) atomicOr(a.status, 2);
      // every MMA issued has finished before TMEM may be freed
      umma_commit(&s.mma_done);
      if (!mbar_wait(&s.mma_done, 0, kDrainNs)) atomicOr(a.status, 8);
    }
  } else {
    // drain: group g (warps 2-5, 6-9) takes the tiles of accumulator g; a warp may reach only its TMEM
    // lane quadrant, rows 32·(w mod 4) … of a tile, and works alone: 32 patterns at a time, TMEM →
    // registers × inv → its buffer → U
    const int ew = warp & 3, grp = (warp - 2) >> 2;
    const int two_nc = 2 * a.nc, rows = two_nc * a.nb;
    const size_t stride = (size_t)rows * a.L;  // floats of a pattern
    float* buf = (float*)(so + (size_t)(warp - 2) * 4096);
    for (int mt = grp; mt < mtiles; mt += 2) {
      int got = 1;
      if (lane == 0) got = mbar_wait(&s.acc_full[grp], (mt >> 1) & 1, lim);
      got = __shfl_sync(0xffffffffu, got, 0);
      if (!got) {
        if (lane == 0) atomicOr(a.status, 4);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int nu = (mt0 + mt) * 128 + ew * 32 + 4 * (lane & 7);  // the lane's first row of four
      const bool in = (mt0 + mt) * 128 + ew * 32 < rows;            // (rows end at a multiple of 32)
      const int j = nu / two_nc;
      float* dst = a.U + ((size_t)j * a.L + mp) * two_nc + (nu - j * two_nc) + (size_t)ptile * 128 * stride;
      const uint32_t ta = tmem + ((uint32_t)(ew * 32) << 16) + (uint32_t)(grp * 128);
#pragma unroll 1
      for (int c0 = 0; c0 < 128; c0 += 32) {
        uint32_t v[32];
        TMEM_LD32(ta + c0, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + 32 == 128) {  // the accumulator is read out: its next tile's MMAs may start
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&s.acc_empty[grp]);
        }
        const int left = in ? a.n_items - ptile * 128 - c0 : 0;
        drain_f32(buf, lane, v, a.inv, dst + (size_t)c0 * stride, stride, left);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256));
}

}  // namespace zeb

using namespace zeb;

static bool x2_dims_ok(const zeb_so3_dims_t* d) {
  return d && d->L >= X2_MIN_L && x2_kblocks(d->L, 0) <= X2_MAX_KB && d->n >= 2 * d->L - 1 && (d->n & (d->n - 1)) == 0 &&
         d->nb == d->n / 2 + 1 && d->fold >= 1 && d->nc == d->n / d->fold && (d->nc & (d->nc - 1)) == 0 && d->nc >= 2 &&
         d->mu_max == (d->L - 1) / d->fold && d->n_pairs == d->L * (d->L + 1) / 2;
}

static int x2_mtiles(const zeb_so3_dims_t* d) { return (2 * d->nb * d->nc + 127) / 128; }

extern "C" size_t zeb_x2_master_bytes(const zeb_so3_dims_t* d) {
  if (!x2_dims_ok(d)) return 0;
  return (size_t)x2_blocks_before(d->L, d->L) * x2_mtiles(d) * 2 * X2_BLOCK;
}

extern "C" size_t zeb_x2_patterns_bytes(const zeb_so3_dims_t* d, int n_items) {
  if (!x2_dims_ok(d) || n_items <= 0) return 0;
  return (size_t)x2_blocks_before(d->L, d->L) * ((n_items + 127) / 128) * 2 * X2_BLOCK;
}

extern "C" int zeb_x2_pack_master(const zeb_so3_dims_t* d, const double* Y, float scale, void* A, void* stream) {
  ZEB_REQUIRE(Y && A, ZEB_EARG, "x2_pack_master: null argument");
  ZEB_REQUIRE(x2_dims_ok(d), ZEB_EARG, "x2_pack_master: unsupported dims (L=%d)", d ? d->L : -1);
  ZEB_REQUIRE(scale > 0.f && scale < 1e30f, ZEB_EARG, "x2_pack_master: scale %g", (double)scale);
  const int mtiles = x2_mtiles(d);
  for (int mp = 0; mp < d->L; ++mp) {
    const long long chunks = (long long)mtiles * x2_kblocks(d->L, mp) * 128 * 8;
    k_x2_pack_master<<<(unsigned)((chunks + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        (const double2*)Y, d->L, d->nb * d->nc, mtiles, mp, (double)scale,
        (uint8_t*)A + (size_t)x2_blocks_before(d->L, mp) * mtiles * 2 * X2_BLOCK);
  }
  return zeb_launch_check("x2_pack_master");
}

extern "C" int zeb_spectrum_x2(const float* alm, int n_items, const zeb_so3_dims_t* d, const void* A, float scale,
                               void* B, float* U, int* status, void* stream) {
  ZEB_REQUIRE(alm && A && B && U && status, ZEB_EARG, "spectrum_x2: null argument");
  ZEB_REQUIRE(x2_dims_ok(d), ZEB_EARG, "spectrum_x2: unsupported dims (L=%d)", d ? d->L : -1);
  ZEB_REQUIRE(scale > 0.f && scale < 1e30f, ZEB_EARG, "spectrum_x2: scale %g", (double)scale);
  if (n_items <= 0) return ZEB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  X2Args a{};
  a.L = d->L; a.nb = d->nb; a.nc = d->nc; a.mtiles = x2_mtiles(d); a.ptiles = (n_items + 127) / 128;
  a.n_items = n_items; a.A = (const uint8_t*)A; a.B = (const uint8_t*)B; a.U = U; a.status = status;
  a.stall = test_stall_ns();
  a.limit = a.stall > 0 ? a.stall : kWaitNs;
  a.kbmax = x2_kblocks(d->L, 0);
  a.stages = x2_stages(a.kbmax);
  a.inv = 1.f / (scale * X2_PATTERN_SCALE);
  const dim3 gp((unsigned)a.kbmax * a.ptiles, d->L);
  k_x2_pack_patterns<<<gp, 256, 0, st>>>((const float2*)alm, n_items, d->n_pairs, d->L, a.ptiles, a.kbmax, (uint8_t*)B);
  int rc = zeb_launch_check("x2_pack_patterns");
  if (rc) return rc;
  ZEB_REQUIRE(((uintptr_t)U & 15) == 0, ZEB_EARG, "spectrum_x2: U must be 16-byte aligned");
  const size_t smem = x2_smem(a.kbmax);
  cudaFuncSetAttribute(k_spectrum_x2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // Row tiles split into groups when the pattern tiles are few: the split of least waves × (row tiles of
  // a CTA + 4), a CTA's start (tensor memory, the patterns' operand, the first table blocks) costing
  // about four row tiles' time.
  const long long base = (long long)a.ptiles * d->L;
  long long least = -1;
  for (int per = a.mtiles; per >= 1; --per) {
    const long long groups = (a.mtiles + per - 1) / per, waves = (base * groups + sms - 1) / sms;
    const long long cost = waves * (per + 4);
    if (least < 0 || cost < least) {
      least = cost;
      a.per = per;
    }
    if (waves > 16) break;
  }
  const int groups = (a.mtiles + a.per - 1) / a.per;
  k_spectrum_x2<<<dim3(a.ptiles, d->L, groups), X2_THREADS, smem, st>>>(a);
  return zeb_launch_check("spectrum_x2");
}
