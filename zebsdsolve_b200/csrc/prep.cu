// Pattern preprocessing: one thread block per pattern does the whole chain (unpack, static
// background, dynamic background, mask and normalization) with the image held in shared memory
// when it fits, so a pattern is read from HBM once and written once.
//
// The arithmetic follows shaders/prep.wgsl: the direct Gaussian (taps to ceil(3σ), renormalized
// over the taps inside the image) below σ = 12 pixels, the box-sum construction above it
// (box sums of s = ⌊σ/6⌋ pixels, a coarse Gaussian over them with a margin of cpad = 3 cells,
// and a spread of deviation s back over the pixels).
#include "abi_util.cuh"

namespace zeb {

struct PrepArgs {
  const void* raw;
  int pixel, n, h, w;
  int sh, sw;      // the stored pattern's size (h, w when nothing is reduced)
  double factor;   // reduction factor (1: none)
  int kwhole;      // the factor as a whole number, 0 when it is not one
  const float* static_bg;
  int dynamic;  // 0 none, 1 subtract, 2 divide, 3 the blur itself
  float sigma;
  float mask[3];
  int normalize;
  float* out;
  float* scratch;  // per pattern: scratch_per floats
  long long scratch_per;
  int use_smem;
  // direct blur
  int radius;
  float k0;
  // wide blur
  int bin, cpad, wradius;
  float kx, kz;
};

// the image against its blurred self: 1 subtract, 2 divide (the dynamic background), 3 the
// blurred image itself (a band pass's Gaussians)
__device__ __forceinline__ float with_background(int dynamic, float v, float bg) {
  return dynamic == 1 ? v - bg : (dynamic == 2 ? v / fmaxf(bg, 1e-6f) : bg);
}

__device__ __forceinline__ float2 wide_cell(int jr, int n, int s) {
  int lo = jr * s;
  int hi = lo + s;
  if (jr >= 0 && lo < n) hi = min(hi, n);
  return make_float2(0.5f * (float)(lo + hi - 1), (float)(hi - lo));
}

// a thread's pixels i = threadIdx.x, + blockDim.x, … by row and column, without a division a pixel
struct PixelWalk {
  int i, r, c, dr, dc, w;
  __device__ __forceinline__ explicit PixelWalk(int width) : i(threadIdx.x), w(width) {
    r = i / w;
    c = i - r * w;
    dr = blockDim.x / w;
    dc = blockDim.x - dr * w;
  }
  __device__ __forceinline__ void next() {
    i += blockDim.x;
    r += dr;
    c += dc;
    if (c >= w) {
      c -= w;
      ++r;
    }
  }
};

// zero mean and unit norm under the mask (prep.wgsl:405-443), or the plain copy out (img: the image in
// shared memory, or out itself)
__device__ void prep_finish(const PrepArgs& a, float* img, float* out, float* red) {
  const int hw = a.h * a.w;
  if (!a.normalize) {
    if (img != out)
      for (int i = threadIdx.x; i < hw; i += blockDim.x) out[i] = img[i];
    return;
  }
  float v2[2] = {0.f, 0.f};
  for (PixelWalk p(a.w); p.i < hw; p.next()) {
    float dr = (float)p.r - a.mask[0], dc = (float)p.c - a.mask[1];
    if (zeb_in_circle(dr, dc, a.mask[2])) {
      v2[0] += img[p.i];
      v2[1] += 1.f;
    }
  }
  block_sums<2>(v2, red);
  const float mean = v2[0] / fmaxf(v2[1], 1.f);
  float ss[1] = {0.f};
  for (PixelWalk p(a.w); p.i < hw; p.next()) {
    float dr = (float)p.r - a.mask[0], dc = (float)p.c - a.mask[1];
    float v = 0.f;
    if (zeb_in_circle(dr, dc, a.mask[2])) v = img[p.i] - mean;
    img[p.i] = v;
    ss[0] += v * v;
  }
  block_sums<1>(ss, red);
  const float inv = rsqrtf(fmaxf(ss[0], 1e-30f));
  for (int i = threadIdx.x; i < hw; i += blockDim.x) out[i] = img[i] * inv;
}

__device__ __forceinline__ float stored_px(const PrepArgs& a, size_t i) {
  if (a.pixel == 0) return (float)((const uint8_t*)a.raw)[i];
  if (a.pixel == 1) return (float)((const uint16_t*)a.raw)[i];
  return ((const float*)a.raw)[i];
}

// Output pixel (r, c) of stored pattern b reduced by a.factor (reduce.zig:44-131): for a whole
// factor k the k × k block's mean (integer pixels summed exactly, f32 ones row by row); otherwise
// the source area the output pixel covers, each source row's part summed in FP64 then shared
// between the one or two output rows it lies in, in the order of the source rows (products and
// sums rounded one at a time, as the host reduction does).
__device__ float reduced_px(const PrepArgs& a, int b, int r, int c) {
  const size_t base = (size_t)b * a.sh * a.sw;
  if (a.kwhole > 0) {
    const int k = a.kwhole;
    const float inv = 1.f / (float)(k * k);
    if (a.pixel != 2) {
      uint32_t acc = 0;
      for (int i = 0; i < k; ++i)
        for (int j = 0; j < k; ++j) acc += (uint32_t)stored_px(a, base + (size_t)(r * k + i) * a.sw + c * k + j);
      return __fmul_rn((float)acc, inv);
    }
    float out = 0.f;
    for (int i = 0; i < k; ++i) {
      float acc = 0.f;
      for (int j = 0; j < k; ++j) acc = __fadd_rn(acc, stored_px(a, base + (size_t)(r * k + i) * a.sw + c * k + j));
      out = __fadd_rn(out, acc);
    }
    return __fmul_rn(out, inv);
  }
  const double f = a.factor;
  const int rows = (int)ceil((double)a.h * f - 1e-9);
  const double x0 = (double)c * f, x1 = x0 + f;
  const int j0 = (int)floor(x0);
  float out = 0.f;
  const int lo = max(0, (int)floor(((double)r - 1.0) * f) - 1), hi = min(rows - 1, (int)ceil(((double)r + 1.0) * f) + 1);
  for (int rs = lo; rs <= hi; ++rs) {
    const double y0 = (double)rs;
    const int top = (int)floor(y0 / f + 1e-12);
    const double edge = (double)(top + 1) * f;
    const float w0 = (float)(fmin(y0 + 1.0, edge) - y0);
    float wt;
    if (top == r) wt = w0;
    else if (top + 1 == r && w0 < 1.f) wt = __fsub_rn(1.f, w0);
    else continue;
    double acc = 0.0;
    for (int j = j0; (double)j < x1 - 1e-12; ++j) {
      const double aa = fmax(x0, (double)j), bb = fmin(x1, (double)(j + 1));
      acc = __dadd_rn(acc, __dmul_rn(bb - aa, (double)stored_px(a, base + (size_t)rs * a.sw + j)));
    }
    out = __fadd_rn(out, __fmul_rn(wt, (float)acc));
  }
  return __fmul_rn(out, (float)(1.0 / (f * f)));
}

// one pixel of pattern b as the chain starts from it: stored (or reduced), static background off
__device__ __forceinline__ float prep_pixel(const PrepArgs& a, int b, int i) {
  float v;
  if (a.factor == 1.0) {
    v = stored_px(a, (size_t)b * a.h * a.w + i);
  } else {
    const int r = i / a.w;
    v = reduced_px(a, b, r, i - r * a.w);
  }
  if (a.static_bg) v -= __ldg(a.static_bg + i);
  return v;
}

// every pixel of pattern b, put(pixel walk, value) in the block's order; the usual case (nothing reduced,
// a static background) without a branch a pixel
template <typename T, typename Put>
__device__ __forceinline__ void unpack_as(const PrepArgs& a, int b, Put put) {
  const T* raw = (const T*)a.raw + (size_t)b * a.h * a.w;
  for (PixelWalk p(a.w); p.i < a.h * a.w; p.next()) put(p, (float)raw[p.i] - __ldg(a.static_bg + p.i));
}
template <typename Put>
__device__ __forceinline__ void unpack(const PrepArgs& a, int b, Put put) {
  if (a.factor == 1.0 && a.static_bg) {
    if (a.pixel == 0) unpack_as<uint8_t>(a, b, put);
    else if (a.pixel == 1) unpack_as<uint16_t>(a, b, put);
    else unpack_as<float>(a, b, put);
  } else {
    for (PixelWalk p(a.w); p.i < a.h * a.w; p.next()) put(p, prep_pixel(a, b, p.i));
  }
}

__global__ void __launch_bounds__(256) k_prep(PrepArgs a) {
  extern __shared__ float sm[];
  __shared__ float taps[64];
  __shared__ float red[2 * 8];
  const int b = blockIdx.x;
  const int h = a.h, w = a.w, hw = h * w;
  float* img = a.use_smem ? sm : a.out + (size_t)b * hw;
  float* tmp = a.use_smem ? sm + hw : a.scratch + (size_t)b * a.scratch_per;

  // unpack
  const size_t base = (size_t)b * hw;
  for (int i = threadIdx.x; i < hw; i += blockDim.x) img[i] = prep_pixel(a, b, i);
  __syncthreads();

  if (a.dynamic != 0 && a.sigma > 0.f) {
    float* bg;  // the blurred image, one value per pixel
    if (a.bin < 2) {
      for (int d = threadIdx.x; d <= min(a.radius, 63); d += blockDim.x) taps[d] = expf(-(float)(d * d) * a.k0);
      __syncthreads();
      const int R = a.radius;
      // along the rows into tmp
      for (int i = threadIdx.x; i < hw; i += blockDim.x) {
        int r = i / w, c = i - r * w;
        float s = 0.f, g = 0.f;
        for (int x = max(c - R, 0); x <= min(c + R, w - 1); ++x) {
          int dd = abs(x - c);
          float t = dd <= R ? taps[min(dd, 63)] : 0.f;
          s += t * img[r * w + x];
          g += t;
        }
        tmp[i] = s / g;
      }
      __syncthreads();
      // along the columns: the background, combined with the image in place
      for (int i = threadIdx.x; i < hw; i += blockDim.x) {
        int r = i / w, c = i - r * w;
        float s = 0.f, g = 0.f;
        for (int y = max(r - R, 0); y <= min(r + R, h - 1); ++y) {
          int dd = abs(y - r);
          float t = dd <= R ? taps[min(dd, 63)] : 0.f;
          s += t * tmp[y * w + c];
          g += t;
        }
        float bgv = s / g;
        img[i] = with_background(a.dynamic, img[i], bgv);
      }
      __syncthreads();
      bg = nullptr;
    } else {
      const int s = a.bin, cp = a.cpad;
      const int hs = (h + s - 1) / s, ws = (w + s - 1) / s, wp = ws + 2 * cp, hp = hs + 2 * cp;
      float2* box = (float2*)(a.scratch + (size_t)b * a.scratch_per + (a.use_smem ? 0 : (hw + 1) & ~1));
      float2* rows = box + hs * ws;
      float2* cols = rows + hs * wp;
      float2* spread = cols + hp * wp;
      for (int t = threadIdx.x; t < hs * ws; t += blockDim.x) {
        int i = t / ws, j = t - i * ws;
        int r1 = min((i + 1) * s, h), c1 = min((j + 1) * s, w);
        float acc = 0.f;
        for (int r = i * s; r < r1; ++r)
          for (int c = j * s; c < c1; ++c) acc += img[r * w + c];
        box[t] = make_float2(acc, (float)((r1 - i * s) * (c1 - j * s)));
      }
      __syncthreads();
      const float reach = (float)a.wradius;
      for (int t = threadIdx.x; t < hs * wp; t += blockDim.x) {
        int line = t / wp, tc = t - line * wp;
        float c = wide_cell(tc - cp, w, s).x;
        int j0 = max((int)floorf((c - reach) / (float)s), 0);
        int j1 = min((int)floorf((c + reach) / (float)s), ws - 1);
        float2 acc = make_float2(0.f, 0.f);
        for (int j = j0; j <= j1; ++j) {
          float d = wide_cell(j, w, s).x - c;
          float e = expf(-d * d * a.kx);
          float2 v = box[line * ws + j];
          acc.x += e * v.x; acc.y += e * v.y;
        }
        rows[t] = acc;
      }
      __syncthreads();
      for (int t = threadIdx.x; t < hp * wp; t += blockDim.x) {
        int tr = t / wp, col = t - tr * wp;
        float c = wide_cell(tr - cp, h, s).x;
        int i0 = max((int)floorf((c - reach) / (float)s), 0);
        int i1 = min((int)floorf((c + reach) / (float)s), hs - 1);
        float2 acc = make_float2(0.f, 0.f);
        for (int i = i0; i <= i1; ++i) {
          float d = wide_cell(i, h, s).x - c;
          float e = expf(-d * d * a.kx);
          float2 v = rows[i * wp + col];
          acc.x += e * v.x; acc.y += e * v.y;
        }
        cols[t] = acc;
      }
      __syncthreads();
      for (int t = threadIdx.x; t < hp * w; t += blockDim.x) {
        int tr = t / w, x = t - tr * w;
        int own = x / s;
        float2 acc = make_float2(0.f, 0.f);
        for (int q = 0; q <= 2 * cp; ++q) {
          float2 cw = wide_cell(own + q - cp, w, s);
          float d = (float)x - cw.x;
          float e = cw.y * expf(-d * d * a.kz);
          float2 v = cols[tr * wp + own + q];
          acc.x += e * v.x; acc.y += e * v.y;
        }
        spread[t] = acc;
      }
      __syncthreads();
      for (int i = threadIdx.x; i < hw; i += blockDim.x) {
        int y = i / w, x = i - y * w;
        int own = y / s;
        float2 acc = make_float2(0.f, 0.f);
        for (int q = 0; q <= 2 * cp; ++q) {
          float2 cw = wide_cell(own + q - cp, h, s);
          float d = (float)y - cw.x;
          float e = cw.y * expf(-d * d * a.kz);
          float2 v = spread[(own + q) * w + x];
          acc.x += e * v.x; acc.y += e * v.y;
        }
        float bgv = acc.x / acc.y;
        img[i] = with_background(a.dynamic, img[i], bgv);
      }
      __syncthreads();
      bg = nullptr;
    }
    (void)bg;
  }

  prep_finish(a, img, a.out + base, red);
}


// The direct blur in shared memory: the image inside its zero-padded rows P[h][pw] (R zeros on
// the left, at least R + 14 on the right, pw odd so that rows at stride pw fall in different
// banks) and the zero-padded row-blurred image Q[R + h + R + 16][w].  A thread takes eight
// consecutive outputs along the blur's direction and walks the taps eight at a time: eight taps
// (two 16-byte loads) and the 23 inputs they reach go into registers, then 128 FMAs, so a shared
// load serves several FMAs (the taps beyond 2R are zeros, adding exact zeros).  Each output sums
// its taps in increasing order with fmaf, the order of k_prep, so the results are the same bits;
// the taps inside the image are summed once per column and per row for the edge renormalization.
// Bound by instruction issue: steps wholly in the padding are skipped, and no loop over the pixels
// divides (16 384 u16 patterns of 60 × 60: 1187 → 949 µs).
constexpr int PD_OUT = 16;  // outputs a thread takes along the blur
constexpr int PD_TB = 8;    // taps a step

__host__ __device__ inline int pd_pw(int w, int R) { return ((w + 2 * R + 2 * PD_OUT) | 1); }
__host__ __device__ inline int pd_qrows(int h, int R) { return h + 2 * R + 2 * PD_OUT; }
__host__ __device__ inline size_t pd_smem(int h, int w, int R) {
  return 4 * ((size_t)h * pd_pw(w, R) + (size_t)pd_qrows(h, R) * w);
}

__global__ void __launch_bounds__(256) k_prep_direct(PrepArgs a) {
  extern __shared__ float sm[];
  __shared__ __align__(16) float taps[128 + PD_TB];
  __shared__ float gsum[2][512];  // Σ taps inside the image, per column and per row
  __shared__ float red[2 * 8];
  const int b = blockIdx.x;
  const int h = a.h, w = a.w, hw = h * w, R = a.radius;
  const int pw = pd_pw(w, R), qr = pd_qrows(h, R);
  const int ntap = 2 * R + 1, nblk = (ntap + PD_TB - 1) / PD_TB;
  float* P = sm;           // [h][pw], the image at columns R … R + w − 1
  float* Q = P + h * pw;   // [qr][w], the row-blurred image at rows R … R + h − 1
  const size_t base = (size_t)b * hw;
  for (int d = threadIdx.x; d < nblk * PD_TB; d += blockDim.x) {
    const int dd = abs(d - R);
    taps[d] = d < ntap ? expf(-(float)(dd * dd) * a.k0) : 0.f;
  }
  for (int i = threadIdx.x; i < h * pw; i += blockDim.x) P[i] = 0.f;
  for (int i = threadIdx.x; i < R * w; i += blockDim.x) Q[i] = 0.f;
  for (int i = threadIdx.x; i < (qr - R - h) * w; i += blockDim.x) Q[(R + h) * w + i] = 0.f;
  __syncthreads();
  unpack(a, b, [&](const PixelWalk& p, float v) { P[p.r * pw + R + p.c] = v; });
  for (int k = threadIdx.x; k < w + h; k += blockDim.x) {
    const int n = k < w ? w : h, c = k < w ? k : k - w;
    float g = 0.f;
    for (int x = max(c - R, 0); x <= min(c + R, n - 1); ++x) g += taps[x - c + R];
    gsum[k < w ? 0 : 1][c] = g;
  }
  __syncthreads();
  // along the rows: Q[R + r][c] = Σ_d taps[d] P[r][c + d] / gsum_col[c]; a thread takes row r,
  // columns c0 … c0 + 7 (threads of a warp: consecutive rows)
  const int cg = (w + PD_OUT - 1) / PD_OUT;
  for (int t = threadIdx.x; t < cg * h; t += blockDim.x) {
    const int r = t % h, c0 = (t / h) * PD_OUT;
    const float* src = P + r * pw + c0;
    float acc[PD_OUT];
#pragma unroll
    for (int k = 0; k < PD_OUT; ++k) acc[k] = 0.f;
    // only the steps that reach the image (the others add exact zeros)
    const int first = c0 + PD_OUT + PD_TB - 2 < R ? (R - c0 - PD_OUT - PD_TB + 2 + PD_TB - 1) & ~(PD_TB - 1) : 0;
    for (int d0 = first; d0 < nblk * PD_TB && c0 + d0 < R + w; d0 += PD_TB) {
      float x[PD_OUT + PD_TB - 1];
      const float4 ta = *reinterpret_cast<const float4*>(taps + d0);
      const float4 tb = *reinterpret_cast<const float4*>(taps + d0 + 4);
      const float tv[PD_TB] = {ta.x, ta.y, ta.z, ta.w, tb.x, tb.y, tb.z, tb.w};
#pragma unroll
      for (int k = 0; k < PD_OUT + PD_TB - 1; ++k) x[k] = src[d0 + k];
#pragma unroll
      for (int dd = 0; dd < PD_TB; ++dd)
#pragma unroll
        for (int k = 0; k < PD_OUT; ++k) acc[k] = fmaf(tv[dd], x[k + dd], acc[k]);
    }
#pragma unroll
    for (int k = 0; k < PD_OUT; ++k)
      if (c0 + k < w) Q[(R + r) * w + c0 + k] = acc[k] / gsum[0][c0 + k];
  }
  __syncthreads();
  // along the columns: the background, combined with the image in place (P's interior); a thread
  // takes column c, rows r0 … r0 + 7 (threads of a warp: consecutive columns)
  const int rg = (h + PD_OUT - 1) / PD_OUT;
  for (int t = threadIdx.x; t < rg * w; t += blockDim.x) {
    const int c = t % w, r0 = (t / w) * PD_OUT;
    const float* src = Q + r0 * w + c;
    float acc[PD_OUT];
#pragma unroll
    for (int k = 0; k < PD_OUT; ++k) acc[k] = 0.f;
    const int first = r0 + PD_OUT + PD_TB - 2 < R ? (R - r0 - PD_OUT - PD_TB + 2 + PD_TB - 1) & ~(PD_TB - 1) : 0;
    for (int d0 = first; d0 < nblk * PD_TB && r0 + d0 < R + h; d0 += PD_TB) {
      float x[PD_OUT + PD_TB - 1];
      const float4 ta = *reinterpret_cast<const float4*>(taps + d0);
      const float4 tb = *reinterpret_cast<const float4*>(taps + d0 + 4);
      const float tv[PD_TB] = {ta.x, ta.y, ta.z, ta.w, tb.x, tb.y, tb.z, tb.w};
#pragma unroll
      for (int k = 0; k < PD_OUT + PD_TB - 1; ++k) x[k] = src[(d0 + k) * w];
#pragma unroll
      for (int dd = 0; dd < PD_TB; ++dd)
#pragma unroll
        for (int k = 0; k < PD_OUT; ++k) acc[k] = fmaf(tv[dd], x[k + dd], acc[k]);
    }
#pragma unroll
    for (int k = 0; k < PD_OUT; ++k) {
      if (r0 + k < h) {
        float* px = P + (r0 + k) * pw + R + c;
        const float bgv = acc[k] / gsum[1][r0 + k];
        *px = with_background(a.dynamic, *px, bgv);
      }
    }
  }
  __syncthreads();
  // the combined image, contiguous, where Q was
  for (PixelWalk p(w); p.i < hw; p.next()) Q[p.i] = P[p.r * pw + R + p.c];
  __syncthreads();
  prep_finish(a, Q, a.out + base, red);
}

// The wide blur with what does not depend on the pattern made once a call (k_wide_tables): the coarse
// Gaussian's weights, the spread's weights and the weights' own sum at every pixel. k_prep forms all of
// them again for each pattern, two exponentials a tap and pixel, and passes its partial sums through
// global memory; here a block keeps the partial sums (and the image, where two blocks fit an SM) in
// shared memory, and the two coarse passes, most of the products, run in register tiles. Every sum runs
// in k_prep's order over the same weights: the results are the same bits. Bound by instruction issue.
// u16 patterns with their background off and normalized: 3072 of 96 × 96 1378 → 509 µs, 4096 of 120 × 120
// 2350 → 1173, 2048 of 160 × 160 1468 → 980, 5 of 160 × 80 158 → 116.
struct WideTables {
  float *den;       // [h][w]: the weights' sum
  float *wx, *wy;   // [ws4][wp], [hs][hp8]: the coarse Gaussian, box j to coarse cell t; 0 out of reach
  float *sx, *sy;   // [kWideQ][w], [kWideQ][h]: a coarse cell's spread to a pixel
};
constexpr int kWideCpad = 3, kWideQ = 2 * kWideCpad + 1;
constexpr int kWideRowTile = 6, kWideColTile = 8;  // box lines, coarse cells down the columns, a thread

struct WideShape {
  int hs, ws, hp, wp, ws4, hp8;
  __host__ __device__ WideShape(int h, int w, int s) {
    hs = (h + s - 1) / s;
    ws = (w + s - 1) / s;
    hp = hs + 2 * kWideCpad;
    wp = ws + 2 * kWideCpad;
    ws4 = (ws + 3) & ~3;
    hp8 = (hp + 7) & ~7;
  }
  __host__ __device__ int lines() const { return (hs + kWideRowTile - 1) / kWideRowTile * kWideRowTile; }
  // the tables in floats; den first, wy on a 16-byte boundary
  __host__ __device__ long long table_floats(int h, int w) const {
    return (((long long)h * w + (long long)ws4 * wp + 3) & ~3LL) + (long long)hs * hp8 + kWideQ * (long long)(h + w);
  }
  __host__ __device__ WideTables tables(float* t, int h, int w) const {
    WideTables o;
    o.den = t;
    o.wx = t + (long long)h * w;
    o.wy = t + (((long long)h * w + (long long)ws4 * wp + 3) & ~3LL);
    o.sx = o.wy + (long long)hs * hp8;
    o.sy = o.sx + kWideQ * (long long)w;
    return o;
  }
  // shared memory of k_prep_wide without the image, in floats: box sums and their rows, or the spread; then
  // the coarse image
  __host__ __device__ int first(int w) const {
    const int coarse = lines() * (ws4 + wp);
    return ((hp * w > coarse ? hp * w : coarse) + 3) & ~3;
  }
  __host__ __device__ int part(int w) const { return first(w) + hp8 * wp; }
};

// weight of box j for coarse cell t of an axis of n pixels in `cells` boxes (0 out of reach)
__device__ __forceinline__ float wide_coarse(const PrepArgs& a, int t, int j, int n, int cells) {
  const int s = a.bin;
  const float reach = (float)a.wradius;
  const float c = wide_cell(t - kWideCpad, n, s).x;
  const int j0 = max((int)floorf((c - reach) / (float)s), 0);
  const int j1 = min((int)floorf((c + reach) / (float)s), cells - 1);
  if (j < j0 || j > j1) return 0.f;
  const float d = wide_cell(j, n, s).x - c;
  return expf(-d * d * a.kx);
}
// weight of coarse cell x / s + q − cpad for pixel x of an axis of n pixels
__device__ __forceinline__ float wide_spread(const PrepArgs& a, int x, int q, int n) {
  const float2 cw = wide_cell(x / a.bin + q - kWideCpad, n, a.bin);
  const float d = (float)x - cw.x;
  return cw.y * expf(-d * d * a.kz);
}

// A block makes the weights' sum of one pixel row; the first block writes the other tables too. The box
// lines of a pattern hold s rows each but the last, so two lines' row sums stand for all.
__global__ void __launch_bounds__(256) k_wide_tables(PrepArgs a, float* out) {
  extern __shared__ float sm[];
  const int h = a.h, w = a.w, s = a.bin, y = blockIdx.x, own = y / s;
  const WideShape d(h, w, s);
  const WideTables T = d.tables(out, h, w);
  float* ex = sm;                       // [ws][wp]
  float* ey = ex + d.ws * d.wp;         // [kWideQ][hs]: the weights of the row's coarse cells
  float* line = ey + kWideQ * d.hs;     // [2][wp]: the row sums of a whole line and of the last
  float* cols = line + 2 * d.wp;        // [kWideQ][wp]
  for (int t = threadIdx.x; t < d.ws * d.wp; t += blockDim.x) ex[t] = wide_coarse(a, t % d.wp, t / d.wp, w, d.ws);
  for (int t = threadIdx.x; t < kWideQ * d.hs; t += blockDim.x) ey[t] = wide_coarse(a, own + t / d.hs, t % d.hs, h, d.hs);
  if (y == 0) {
    for (int t = threadIdx.x; t < d.ws4 * d.wp; t += blockDim.x)
      T.wx[t] = t < d.ws * d.wp ? wide_coarse(a, t % d.wp, t / d.wp, w, d.ws) : 0.f;
    for (int t = threadIdx.x; t < d.hs * d.hp8; t += blockDim.x) {
      const int tr = t % d.hp8;
      T.wy[t] = tr < d.hp ? wide_coarse(a, tr, t / d.hp8, h, d.hs) : 0.f;
    }
    for (int t = threadIdx.x; t < kWideQ * w; t += blockDim.x) T.sx[t] = wide_spread(a, t % w, t / w, w);
    for (int t = threadIdx.x; t < kWideQ * h; t += blockDim.x) T.sy[t] = wide_spread(a, t % h, t / h, h);
  }
  __syncthreads();
  for (int t = threadIdx.x; t < 2 * d.wp; t += blockDim.x) {
    const int last = t / d.wp, tc = t - last * d.wp;
    const int rows = last ? h - (d.hs - 1) * s : s;
    float acc = 0.f;
    for (int j = 0; j < d.ws; ++j) {
      const float e = ex[j * d.wp + tc];
      if (e != 0.f) acc = fmaf(e, (float)(rows * (min((j + 1) * s, w) - j * s)), acc);
    }
    line[t] = acc;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < kWideQ * d.wp; t += blockDim.x) {
    const int q = t / d.wp, col = t - q * d.wp;
    float acc = 0.f;
    for (int i = 0; i < d.hs; ++i) {
      const float e = ey[q * d.hs + i];
      if (e != 0.f) acc = fmaf(e, line[(i == d.hs - 1 ? d.wp : 0) + col], acc);
    }
    cols[t] = acc;
  }
  __syncthreads();
  for (int x = threadIdx.x; x < w; x += blockDim.x) {
    float e[kWideQ], acc = 0.f;
#pragma unroll
    for (int k = 0; k < kWideQ; ++k) e[k] = wide_spread(a, x, k, w);
#pragma unroll
    for (int q = 0; q < kWideQ; ++q) {
      float sp = 0.f;
#pragma unroll
      for (int k = 0; k < kWideQ; ++k) sp = fmaf(e[k], cols[q * d.wp + x / s + k], sp);
      acc = fmaf(wide_spread(a, y, q, h), sp, acc);
    }
    T.den[(size_t)y * w + x] = acc;
  }
}

__global__ void __launch_bounds__(256) k_prep_wide(PrepArgs a, float* tables, int img_smem) {
  extern __shared__ __align__(16) float sm[];
  __shared__ float red[2 * 8];
  const int h = a.h, w = a.w, hw = h * w, s = a.bin;
  const WideShape d(h, w, s);
  const WideTables T = d.tables(tables, h, w);
  const size_t base = (size_t)blockIdx.x * hw;
  float* spread = sm;                     // [hp][w]; before it:
  float* box = sm;                        // [lines][ws4]
  float* rows = sm + d.lines() * d.ws4;   // [lines][wp]
  float* cols = sm + d.first(w);          // [hp8][wp]
  float* img = img_smem ? sm + d.part(w) : a.out + base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  unpack(a, blockIdx.x, [&](const PixelWalk& p, float v) { img[p.i] = v; });
  __syncthreads();
  for (int i = warp; i < d.lines(); i += nw) {
    const int r1 = min((i + 1) * s, h);
    for (int j = lane; j < d.ws4; j += 32) {
      const int c1 = min((j + 1) * s, w);
      float acc = 0.f;
      for (int r = i * s; r < r1; ++r)
        for (int c = j * s; c < c1; ++c) acc += img[r * w + c];
      box[i * d.ws4 + j] = acc;
    }
  }
  __syncthreads();
  // the coarse Gaussian along the rows: a thread takes six lines of one coarse column
  const int tx = (d.wp + 31) / 32;
  for (int t = warp; t < d.lines() / kWideRowTile * tx; t += nw) {
    const int i0 = t / tx * kWideRowTile, tc = (t % tx) * 32 + lane;
    float acc[kWideRowTile];
#pragma unroll
    for (int k = 0; k < kWideRowTile; ++k) acc[k] = 0.f;
    const float* wx = T.wx + min(tc, d.wp - 1);
    for (int j = 0; j < d.ws4; j += 4) {
      float e[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) e[q] = __ldg(wx + (j + q) * d.wp);
#pragma unroll
      for (int k = 0; k < kWideRowTile; ++k) {
        const float4 v = *(const float4*)(box + (i0 + k) * d.ws4 + j);
        if (e[0] != 0.f) acc[k] = fmaf(e[0], v.x, acc[k]);
        if (e[1] != 0.f) acc[k] = fmaf(e[1], v.y, acc[k]);
        if (e[2] != 0.f) acc[k] = fmaf(e[2], v.z, acc[k]);
        if (e[3] != 0.f) acc[k] = fmaf(e[3], v.w, acc[k]);
      }
    }
    if (tc < d.wp)
#pragma unroll
      for (int k = 0; k < kWideRowTile; ++k) rows[(i0 + k) * d.wp + tc] = acc[k];
  }
  __syncthreads();
  // and along the columns: eight coarse cells of one column
  for (int t = warp; t < d.hp8 / kWideColTile * tx; t += nw) {
    const int tr0 = t / tx * kWideColTile, col = (t % tx) * 32 + lane;
    float acc[kWideColTile];
#pragma unroll
    for (int k = 0; k < kWideColTile; ++k) acc[k] = 0.f;
    const float* src = rows + min(col, d.wp - 1);
#pragma unroll 2
    for (int i = 0; i < d.hs; ++i) {
      const float4 ea = __ldg((const float4*)(T.wy + i * d.hp8 + tr0)), eb = __ldg((const float4*)(T.wy + i * d.hp8 + tr0 + 4));
      const float v = src[i * d.wp];
      if (ea.x != 0.f) acc[0] = fmaf(ea.x, v, acc[0]);
      if (ea.y != 0.f) acc[1] = fmaf(ea.y, v, acc[1]);
      if (ea.z != 0.f) acc[2] = fmaf(ea.z, v, acc[2]);
      if (ea.w != 0.f) acc[3] = fmaf(ea.w, v, acc[3]);
      if (eb.x != 0.f) acc[4] = fmaf(eb.x, v, acc[4]);
      if (eb.y != 0.f) acc[5] = fmaf(eb.y, v, acc[5]);
      if (eb.z != 0.f) acc[6] = fmaf(eb.z, v, acc[6]);
      if (eb.w != 0.f) acc[7] = fmaf(eb.w, v, acc[7]);
    }
    if (col < d.wp)
#pragma unroll
      for (int k = 0; k < kWideColTile; ++k) cols[(tr0 + k) * d.wp + col] = acc[k];
  }
  __syncthreads();
  // the coarse cells spread to the pixels, along the rows and then down the columns
  for (int x = lane; x < w; x += 32) {
    float e[kWideQ];
#pragma unroll
    for (int q = 0; q < kWideQ; ++q) e[q] = __ldg(T.sx + q * w + x);
    const float* src = cols + x / s;
    for (int tr = warp; tr < d.hp; tr += nw) {
      float acc = 0.f;
#pragma unroll
      for (int q = 0; q < kWideQ; ++q) acc = fmaf(e[q], src[tr * d.wp + q], acc);
      spread[tr * w + x] = acc;
    }
  }
  __syncthreads();
  for (int y = warp; y < h; y += nw) {
    float e[kWideQ];
#pragma unroll
    for (int q = 0; q < kWideQ; ++q) e[q] = __ldg(T.sy + q * h + y);
    const float* src = spread + y / s * w;
    for (int x = lane; x < w; x += 32) {
      float acc = 0.f;
#pragma unroll
      for (int q = 0; q < kWideQ; ++q) acc = fmaf(e[q], src[q * w + x], acc);
      const float bgv = acc / __ldg(T.den + y * w + x);
      img[y * w + x] = with_background(a.dynamic, img[y * w + x], bgv);
    }
  }
  __syncthreads();
  prep_finish(a, img, a.out + base, red);
}

struct WideDims {
  int bin, hs, ws, hp, wp;
};

static WideDims wide_dims(int h, int w, float sigma) {
  WideDims d{};
  d.bin = (int)floorf(sigma / 6.f);
  if (d.bin < 2) return d;
  d.hs = (h + d.bin - 1) / d.bin;
  d.ws = (w + d.bin - 1) / d.bin;
  d.hp = d.hs + 6;
  d.wp = d.ws + 6;
  return d;
}

static long long scratch_floats(int h, int w, float sigma, int dynamic, bool smem) {
  long long per = 0;
  if (!smem) per += ((long long)h * w + 1) & ~1LL;  // the row-blurred image, to an even count
  if (dynamic && sigma > 0.f) {
    WideDims d = wide_dims(h, w, sigma);
    if (d.bin >= 2) per += 2LL * (d.hs * d.ws + d.hs * d.wp + d.hp * d.wp + (long long)d.hp * w);
  }
  return per;
}

static bool prep_smem(int h, int w) { return 2LL * h * w * 4 <= 160 * 1024; }

}  // namespace zeb

using namespace zeb;

extern "C" size_t zeb_prep_scratch_bytes(int n, int h, int w, float sigma) {
  if (n <= 0 || h <= 0 || w <= 0) return 0;
  long long per = scratch_floats(h, w, sigma, 1, prep_smem(h, w));
  if (!prep_smem(h, w) && per == 0) per = (long long)h * w;
  return (size_t)per * 4 * (size_t)n;
}

static int prep_launch(const void* raw, int pixel, int n, int src_h, int src_w, double factor, const float* static_bg,
                       int dynamic, float sigma, const float mask[3], int normalize, float* out, void* scratch,
                       void* stream) {
  ZEB_REQUIRE(raw && out && mask, ZEB_EARG, "prep: null pointer");
  ZEB_REQUIRE(factor >= 1.0 && factor <= 64.0, ZEB_EARG, "prep: reduction factor %g", factor);
  const int h = (int)floor((double)src_h / factor + 1e-9), w = (int)floor((double)src_w / factor + 1e-9);
  ZEB_REQUIRE(pixel >= 0 && pixel <= 2 && n >= 0 && h >= 4 && w >= 4 && dynamic >= 0 && dynamic <= 3, ZEB_EARG,
              "prep: bad arguments pixel=%d n=%d h=%d w=%d dynamic=%d", pixel, n, h, w, dynamic);
  if (n == 0) return ZEB_OK;
  PrepArgs a{};
  a.raw = raw; a.pixel = pixel; a.n = n; a.h = h; a.w = w; a.static_bg = static_bg;
  a.sh = src_h; a.sw = src_w; a.factor = factor;
  a.kwhole = fabs(factor - round(factor)) < 1e-9 && factor > 1.0 ? (int)round(factor) : 0;
  if (a.kwhole == 1) { a.kwhole = 0; a.factor = 1.0; }
  a.dynamic = (sigma > 0.f) ? dynamic : 0; a.sigma = sigma;
  a.mask[0] = mask[0]; a.mask[1] = mask[1]; a.mask[2] = mask[2];
  a.normalize = normalize; a.out = out;
  a.use_smem = prep_smem(h, w) ? 1 : 0;
  a.scratch_per = scratch_floats(h, w, sigma, a.dynamic, a.use_smem);
  a.scratch = (float*)scratch;
  ZEB_REQUIRE(a.scratch_per == 0 || scratch, ZEB_EARG, "prep: scratch needed (%lld floats per pattern)",
              a.scratch_per);
  if (a.dynamic) {
    WideDims d = wide_dims(h, w, sigma);
    a.bin = d.bin;
    if (d.bin < 2) {
      a.radius = (int)fmaxf(1.f, ceilf(3.f * sigma));
      ZEB_REQUIRE(a.radius <= 63, ZEB_ESIZE, "prep: blur radius %d", a.radius);
      a.k0 = (float)(1.0 / (2.0 * (double)sigma * sigma));
    } else {
      double sf = d.bin;
      double cs = sqrt((double)sigma * sigma - sf * sf - (sf * sf - 1.0) / 12.0);
      a.cpad = 3;
      a.wradius = (int)ceil(4.0 * cs);
      a.kx = (float)(1.0 / (2.0 * cs * cs));
      a.kz = (float)(1.0 / (2.0 * sf * sf));
    }
  }
  if (a.dynamic && a.bin < 2 && a.use_smem && h <= 512 && w <= 512 && 2 * a.radius + 1 <= 128) {
    const size_t dsm = pd_smem(h, w, a.radius);
    if (dsm <= 200 * 1024) {
      cudaFuncSetAttribute(k_prep_direct, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dsm);
      k_prep_direct<<<n, 256, dsm, (cudaStream_t)stream>>>(a);
      return zeb_launch_check("prep (direct blur)");
    }
  }
  if (a.dynamic && a.bin >= 2) {
    const WideShape d(h, w, a.bin);
    const size_t part = (size_t)d.part(w) * 4, whole = part + (size_t)h * w * 4;
    // the image in shared memory while two blocks fit an SM, else where the result goes (L2 holds it)
    const bool in = whole <= 113 * 1024;
    const size_t wsm = in ? whole : part, tsm = (size_t)(d.ws * d.wp + kWideQ * (d.hs + d.wp) + 2 * d.wp) * 4;
    // the tables take the place of the partial sums in the caller's scratch, whose size stays what it was:
    // one pattern of a large detector may not have the room
    if (d.table_floats(h, w) <= a.scratch_per * n && wsm <= 200 * 1024 && tsm <= 200 * 1024 && ((uintptr_t)scratch & 15) == 0) {
      // (the most either may ask for, whatever this call does: 48 KB beside a static array is already over)
      cudaFuncSetAttribute(k_wide_tables, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
      k_wide_tables<<<h, 256, tsm, (cudaStream_t)stream>>>(a, a.scratch);
      int rc = zeb_launch_check("prep (wide blur tables)");
      if (rc) return rc;
      cudaFuncSetAttribute(k_prep_wide, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
      k_prep_wide<<<n, 256, wsm, (cudaStream_t)stream>>>(a, a.scratch, in ? 1 : 0);
      return zeb_launch_check("prep (wide blur)");
    }
  }
  size_t smem = a.use_smem ? 2 * (size_t)h * w * 4 : 0;
  if (smem > 40 * 1024) cudaFuncSetAttribute(k_prep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_prep<<<n, 256, smem, (cudaStream_t)stream>>>(a);
  return zeb_launch_check("prep");
}

extern "C" int zeb_prep_ex(const void* raw, int pixel, int n, int h, int w, const float* static_bg, int dynamic,
                           float sigma, const float mask[3], int normalize, float* out, void* scratch,
                           void* stream) {
  return prep_launch(raw, pixel, n, h, w, 1.0, static_bg, dynamic, sigma, mask, normalize, out, scratch, stream);
}

extern "C" int zeb_prep_reduced(const void* raw, int pixel, int n, int src_h, int src_w, double factor,
                                const float* static_bg, int dynamic, float sigma, const float mask[3], int normalize,
                                float* out, void* scratch, void* stream) {
  return prep_launch(raw, pixel, n, src_h, src_w, factor, static_bg, dynamic, sigma, mask, normalize, out, scratch,
                     stream);
}

extern "C" int zeb_prep(const void* raw, int pixel, int n, int h, int w, const float* static_bg, int dynamic,
                        float sigma, const float mask[3], int normalize, float* out, void* stream) {
  ZEB_REQUIRE(zeb_prep_scratch_bytes(n, h, w, dynamic ? sigma : 0.f) == 0, ZEB_EARG,
              "prep: this size needs scratch (zeb_prep_ex)");
  return zeb_prep_ex(raw, pixel, n, h, w, static_bg, dynamic, sigma, mask, normalize, out, nullptr, stream);
}
