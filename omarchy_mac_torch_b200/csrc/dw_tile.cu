// Depthwise convolution of dense channels-last tensors by tiles: forward, stride-1 input gradient (mirrored taps) and weight
// gradient, ks 3, 5 and 7, stride 1 and 2, any channel count.
//
// A block owns a slab of 32 channels, a tile of up to 64 output columns of one to several images, and walks DOWN their
// rows. Each input row of the tile is copied once to a ring in shared memory by cp.async (zeros outside the image), DEPTH - 1
// rows ahead, and read from there by every output column it reaches: HBM and L2 see each pixel once per tile, not once
// per four columns, and no thread computes addresses for its own halo. A thread owns two channels (one 64-bit lane pair of
// fma.rn.f32x2) and four output columns; the ceil(ks / stride) output rows that an input row overlaps wait in registers, and
// the walk is unrolled over that period, so that their slots are compile-time indices. 16 consecutive lanes are the 16
// channel pairs of one pixel: 128 contiguous bytes, no bank conflicts, whole sectors in global memory.
// The copies are 16 bytes when c % 4 == 0 and the tensors are 16-byte aligned (weight gradient only: see the dispatch in dw.cu), else
// 4 bytes (32 lanes = one pixel's slab).
// What bounds them: issue, at two blocks per SM. Forward 5x5 on 128 x 97 x 56 x 56 (274 us) issues in 57 % of the cycles with 3.4 warps per
// scheduler; the largest stall is a sum's own previous multiply-add, then the row barrier; DRAM is at 12 %.
#include <algorithm>
#include <mutex>

#include "dw.cuh"

namespace omt {

typedef unsigned long long u64;
constexpr int SLAB = 32, TX = 4, DEPTH = 5, TILE_THREADS = 256;

__device__ __forceinline__ u64 lds2(uint32_t a) {
  u64 v;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void fma2(u64& d, u64 a, u64 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ float2 unpack2(u64 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ bool finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }
__host__ __device__ constexpr int fdiv(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }
__host__ __device__ constexpr int pmod(int a, int b) { return ((a % b) + b) % b; }

// one row of `cols` pixels x 32 channels into shared memory; `row` points at channel ch0 of the pixel in column x0 and is only
// followed for columns in [0, width) and channels below c (the rest becomes zeros)
template <int VEC>
__device__ __forceinline__ void copy_row(uint32_t dst, const float* row, const float* safe, int t, int nt, int cols, int x0, int width, int c, int ch0) {
  constexpr int PP = SLAB / VEC;  // copies per pixel
  for (int e = t; e < cols * PP; e += nt) {
    const int k = e / PP, v = (e % PP) * VEC;
    const bool in = (unsigned)(x0 + k) < (unsigned)width && ch0 + v < c;
    const float* src = in ? row + ((int64_t)k * c + v) : safe;
    const uint32_t d = dst + (uint32_t)(k * SLAB + v) * 4u;
    const int n = in ? VEC * 4 : 0;
    if constexpr (VEC == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
  }
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void wait_oldest() { asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 2) : "memory"); }

struct TilePlan {
  int G, Z;            // column groups of four and images per block: threads (16 G, Z)
  int xtiles;          // column tiles per row
  int seg_rows, segs;  // output rows per strip, strips per image
  int imgs;            // image groups
};

// Zeros stand for the pixels outside the image, and zero times infinity is not zero. Only pixels inside the image have a part in a
// result, so the kernels below fall back to the two functions here, which skip the others, where a non-finite value would meet one of
// those zeros: a block whose filters are not all finite, and a tap sum that is not finite. (That covers every such product, and a
// finite run never gets here.)
template <int KS, int S>
__device__ __forceinline__ void direct_outputs(const DwArgs& a, const TilePlan& p, const float* ws) {
  const int slabs = (a.c + SLAB - 1) / SLAB, cols = p.G * TX;
  int b = blockIdx.x;
  const int ch0 = (b % slabs) * SLAB; b /= slabs;
  const int tile0 = b % p.xtiles * cols; b /= p.xtiles;
  const int oy0 = b % p.segs * p.seg_rows, img = b / p.segs * p.Z + threadIdx.y, nrows = min(p.seg_rows, a.oh - oy0);
  if (img >= a.n) return;
  const float* x = a.x.p + (int64_t)img * a.ih * a.iw * a.c;
  float* y = a.y.p + (int64_t)img * a.oh * a.ow * a.c;
  for (int e = threadIdx.x; e < nrows * cols * SLAB; e += blockDim.x) {
    const int cc = e % SLAB, k = e / SLAB, ox = tile0 + k % cols, oy = oy0 + k / cols, ch = ch0 + cc;
    if (ch >= a.c || ox >= a.ow) continue;
    float s = 0.f;
    for (int ky = 0; ky < KS; ky++)
      for (int kx = 0; kx < KS; kx++) {
        const int sy = oy * S - a.pad + ky, sx = ox * S - a.pad + kx;
        if ((unsigned)sy < (unsigned)a.ih && (unsigned)sx < (unsigned)a.iw) s = fmaf(__ldg(x + ((int64_t)sy * a.iw + sx) * a.c + ch), ws[(ky * KS + kx) * SLAB + cc], s);
      }
    if (a.flags & OMT_EPI_BIAS) s += __ldg(a.bias + ch);
    if (a.flags & OMT_EPI_RELU) s = fmaxf(s, 0.f);
    y[((int64_t)oy * a.ow + ox) * a.c + ch] = s;
  }
}
// the sum of tap (ky, kx) of channel ch over the strips of weight-gradient block sl; ends at the first NaN, which stays one
template <int S>
__device__ __forceinline__ float direct_tap_sum(const DwArgs& a, const TilePlan& p, int sl, int SL, int ch, int ky, int kx) {
  float s = 0.f;
  for (int it = sl; it < p.imgs * p.segs * p.xtiles; it += SL) {
    const int tile0 = it % p.xtiles * p.G * TX, q = it / p.xtiles, oy0 = q % p.segs * p.seg_rows, img0 = q / p.segs * p.Z;
    for (int img = img0; img < min(img0 + p.Z, a.n); img++)
      for (int oy = oy0; oy < min(oy0 + p.seg_rows, a.oh); oy++) {
        const int sy = oy * S - a.pad + ky;
        if ((unsigned)sy >= (unsigned)a.ih) continue;
        const float* g = a.y.p + ((int64_t)img * a.oh + oy) * a.ow * a.c + ch;
        const float* x = a.x.p + ((int64_t)img * a.ih + sy) * a.iw * a.c + ch;
        for (int ox = tile0; ox < min(tile0 + p.G * TX, a.ow); ox++) {
          const int sx = ox * S - a.pad + kx;
          if ((unsigned)sx < (unsigned)a.iw) s = fmaf(__ldg(g + (int64_t)ox * a.c), __ldg(x + (int64_t)sx * a.c), s);
        }
        if (s != s) return s;
      }
  }
  return s;
}

// Forward (FLIP = false) and stride-1 input gradient (FLIP = true: taps mirrored, pad = ks-1-pad, the caller swaps the tensors).
template <int KS, int S, bool FLIP>
__global__ void __launch_bounds__(TILE_THREADS, KS == 3 ? 3 : 2) dw_tile_kernel(const __grid_constant__ DwArgs a, const __grid_constant__ TilePlan p) {
  pdl_wait();
  constexpr int SPAN = (TX - 1) * S + KS, R = (KS + S - 1) / S, U = R * S, KK = KS * KS;
  constexpr int WROWS = KS == 3 ? 3 : (KS == 5 ? 4 : 0);  // filter rows of the thread's two channels in registers; the fifth row of 5x5 would spill
  extern __shared__ __align__(16) float sm[];
  const int nt = 16 * p.G, t = threadIdx.x, z = threadIdx.y, cp = t & 15, gr = t >> 4;
  const int slabs = (a.c + SLAB - 1) / SLAB;
  int b = blockIdx.x;
  const int ch0 = (b % slabs) * SLAB; b /= slabs;
  const int xt = b % p.xtiles; b /= p.xtiles;
  const int seg = b % p.segs, img = (b / p.segs) * p.Z + z;
  const int ch = ch0 + 2 * cp, tile0 = xt * p.G * TX, ox0 = tile0 + gr * TX;
  const int oy0 = seg * p.seg_rows, nrows = min(p.seg_rows, a.oh - oy0), n_in = (nrows - 1) * S + KS;
  const int sy0 = oy0 * S - a.pad, x0 = tile0 * S - a.pad, cols = (p.G * TX - 1) * S + KS;
  // the slab's filters, transposed to [tap][channel]
  float* ws = sm;
  for (int e = z * nt + t; e < KK * SLAB; e += nt * p.Z) {
    const int cc = e / KK, tap = e - cc * KK;
    ws[(FLIP ? KK - 1 - tap : tap) * SLAB + cc] = ch0 + cc < a.c ? __ldg(a.w + (int64_t)(ch0 + cc) * KK + tap) : 0.f;
  }
  const uint32_t wbase = (uint32_t)__cvta_generic_to_shared(ws) + cp * 8;
  const uint32_t slot_bytes = (uint32_t)p.Z * cols * SLAB * 4;
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(sm + KK * SLAB) + (uint32_t)z * cols * SLAB * 4;
  const int64_t rs = (int64_t)a.iw * a.c;
  const bool img_ok = img < a.n;
  const float* xbase = a.x.p + (((int64_t)img * a.ih + sy0) * a.iw + x0) * a.c + ch0;
  auto valid = [&](int r) { return img_ok && r < n_in && (unsigned)(sy0 + r) < (unsigned)a.ih; };
  uint32_t wr = 0, rd = 0;  // byte offsets of the slots written and read next
  auto request = [&](int r) {
    if (valid(r)) copy_row<1>(ring + wr, xbase + r * rs, a.x.p, t, nt, cols, x0, a.iw, a.c, ch0);
    commit();
    wr += slot_bytes;
    if (wr == DEPTH * slot_bytes) wr = 0;
  };
  for (int d = 0; d < DEPTH - 1; d++) request(d);
  u64 acc[R][TX];
#pragma unroll
  for (int q = 0; q < R; q++)
#pragma unroll
    for (int j = 0; j < TX; j++) acc[q][j] = 0;
  float b0 = 0.f, b1 = 0.f;
  if (a.flags & OMT_EPI_BIAS) {
    if (ch < a.c) b0 = __ldg(a.bias + ch);
    if (ch + 1 < a.c) b1 = __ldg(a.bias + ch + 1);
  }
  const bool relu = a.flags & OMT_EPI_RELU;
  __syncthreads();
  u64 wreg[WROWS ? WROWS * KS : 1];
#pragma unroll
  for (int k = 0; k < WROWS * KS; k++) wreg[k] = lds2(wbase + k * SLAB * 4);
  float* yrow = a.y.p + (((int64_t)img * a.oh + oy0) * a.ow + ox0) * a.c + ch;
  const int64_t ys = (int64_t)a.ow * a.c;
  const uint32_t lane = ring + (uint32_t)(gr * TX * S * SLAB) * 4 + cp * 8;
  for (int base = 0; base < n_in; base += U) {
    const int qb = base / S;
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int r = base + u;
      if (r >= n_in) break;
      wait_oldest();
      __syncthreads();  // row r is there for everyone, and everyone has read row r - 1: its slot is free
      request(r + DEPTH - 1);
      if (valid(r)) {
        u64 in[SPAN];
#pragma unroll
        for (int k = 0; k < SPAN; k++) in[k] = lds2(lane + rd + k * SLAB * 4);
#pragma unroll
        for (int ky = 0; ky < KS; ky++) {
          if (pmod(u - ky, S) != 0) continue;  // (known at compile time once u and ky are unrolled)
          const int dq = fdiv(u - ky, S), slot = pmod(dq, R), q = qb + dq;  // input row r is filter row ky of output row q
          if (q < 0 || q >= nrows) continue;
#pragma unroll
          for (int kx = 0; kx < KS; kx++) {
            const u64 wv = ky < WROWS ? wreg[ky * KS + kx] : lds2(wbase + (ky * KS + kx) * SLAB * 4);
#pragma unroll
            for (int j = 0; j < TX; j++) fma2(acc[slot][j], in[j * S + kx], wv);
          }
        }
      }
      rd += slot_bytes;
      if (rd == DEPTH * slot_bytes) rd = 0;
      if (pmod(u - (KS - 1), S) == 0) {  // this was the last input row of an output row
        const int dq = fdiv(u - (KS - 1), S), slot = pmod(dq, R), q = qb + dq;
        if (q >= 0 && q < nrows) {
          float* yp = yrow + q * ys;
#pragma unroll
          for (int j = 0; j < TX; j++) {
            if (img_ok && ox0 + j < a.ow) {
              float2 o = unpack2(acc[slot][j]);
              o.x += b0; o.y += b1;
              if (relu) { o.x = fmaxf(o.x, 0.f); o.y = fmaxf(o.y, 0.f); }
              if (ch < a.c) yp[(int64_t)j * a.c] = o.x;
              if (ch + 1 < a.c) yp[(int64_t)j * a.c + 1] = o.y;
            }
            acc[slot][j] = 0;
          }
        }
      }
    }
  }
  bool good = true;  // (looked at last: a branch in front of the walk costs it registers)
  for (int e = threadIdx.y * blockDim.x + threadIdx.x; e < KK * SLAB; e += blockDim.x * blockDim.y) good = good && finite(sm[e]);
  if (!__syncthreads_and(good)) direct_outputs<KS, S>(a, p, sm);
}

// Weight gradient: the same walk with a second ring for the rows of gy. A thread keeps the ks * ks tap sums of its two channels
// in registers over all strips of its block (blockIdx.y, SL blocks per slab); the block's column groups and images are summed
// through shared memory in a fixed order, the blocks by dw_wgrad_fin_kernel: the same result on every run.
template <int KS, int S, int VEC>
__global__ void __launch_bounds__(TILE_THREADS, KS == 7 ? 1 : 2) dw_wgrad_tile_kernel(DwArgs a, TilePlan p, int SL, float* __restrict__ part) {
  pdl_wait();
  constexpr int SPAN = (TX - 1) * S + KS, R = (KS + S - 1) / S, U = R * S, KK = KS * KS;
  extern __shared__ __align__(16) float sm[];
  const int nt = 16 * p.G, t = threadIdx.x, z = threadIdx.y, cp = t & 15, gr = t >> 4;
  const int ch0 = blockIdx.x * SLAB, sl = blockIdx.y;
  const int cols = (p.G * TX - 1) * S + KS, gcols = p.G * TX;
  const uint32_t slot_bytes = (uint32_t)p.Z * (cols + gcols) * SLAB * 4;
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(sm) + (uint32_t)z * (cols + gcols) * SLAB * 4;
  const uint32_t lane = ring + (uint32_t)(gr * TX * S * SLAB) * 4 + cp * 8;
  const uint32_t glane = ring + (uint32_t)(cols + gr * TX) * SLAB * 4 + cp * 8;
  const int64_t rs = (int64_t)a.iw * a.c, gs = (int64_t)a.ow * a.c;
  u64 acc[KK];
#pragma unroll
  for (int k = 0; k < KK; k++) acc[k] = 0;
  const int items = p.imgs * p.segs * p.xtiles;
  for (int it = sl; it < items; it += SL) {
    int b = it;
    const int xt = b % p.xtiles; b /= p.xtiles;
    const int seg = b % p.segs, img = (b / p.segs) * p.Z + z;
    const int tile0 = xt * p.G * TX, oy0 = seg * p.seg_rows, nrows = min(p.seg_rows, a.oh - oy0), n_in = (nrows - 1) * S + KS;
    const int sy0 = oy0 * S - a.pad, x0 = tile0 * S - a.pad;
    const bool img_ok = img < a.n;
    const float* xbase = a.x.p + (((int64_t)img * a.ih + sy0) * a.iw + x0) * a.c + ch0;
    const float* gbase = a.y.p + (((int64_t)img * a.oh + oy0) * a.ow + tile0) * a.c + ch0;
    auto valid = [&](int r) { return img_ok && r < n_in && (unsigned)(sy0 + r) < (unsigned)a.ih; };
    uint32_t wr = 0, rd = 0;
    auto request = [&](int r) {
      if (valid(r)) copy_row<VEC>(ring + wr, xbase + r * rs, a.x.p, t, nt, cols, x0, a.iw, a.c, ch0);
      if (img_ok && r % S == 0 && r / S < nrows)  // the first input row of an output row brings its gy row along
        copy_row<VEC>(ring + wr + (uint32_t)cols * SLAB * 4, gbase + (r / S) * gs, a.y.p, t, nt, gcols, tile0, a.ow, a.c, ch0);
      commit();
      wr += slot_bytes;
      if (wr == DEPTH * slot_bytes) wr = 0;
    };
    __syncthreads();  // everyone has left the strip before
    for (int d = 0; d < DEPTH - 1; d++) request(d);
    u64 g[R][TX];
#pragma unroll
    for (int q = 0; q < R; q++)
#pragma unroll
      for (int j = 0; j < TX; j++) g[q][j] = 0;
    for (int base = 0; base < n_in; base += U) {
      const int qb = base / S;
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int r = base + u;
        if (r >= n_in) break;
        wait_oldest();
        __syncthreads();
        request(r + DEPTH - 1);
        if (u % S == 0 && img_ok) {
          const int q = qb + u / S;
          if (q < nrows) {
#pragma unroll
            for (int j = 0; j < TX; j++) g[(u / S) % R][j] = lds2(glane + rd + j * SLAB * 4);
          }
        }
        if (valid(r)) {
          u64 in[SPAN];
#pragma unroll
          for (int k = 0; k < SPAN; k++) in[k] = lds2(lane + rd + k * SLAB * 4);
#pragma unroll
          for (int ky = 0; ky < KS; ky++) {
            if (pmod(u - ky, S) != 0) continue;
            const int dq = fdiv(u - ky, S), slot = pmod(dq, R), q = qb + dq;
            if (q < 0 || q >= nrows) continue;
#pragma unroll
            for (int kx = 0; kx < KS; kx++)
#pragma unroll
              for (int j = 0; j < TX; j++) fma2(acc[ky * KS + kx], g[slot][j], in[j * S + kx]);
          }
        }
        rd += slot_bytes;
        if (rd == DEPTH * slot_bytes) rd = 0;
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  u64* red = reinterpret_cast<u64*>(sm);  // [KS][Z G][16]
  const int lanes = p.Z * p.G, me = z * p.G + gr, tid = z * nt + t;
  bool good = true;
#pragma unroll
  for (int ky = 0; ky < KS; ky++) {
    __syncthreads();
#pragma unroll
    for (int kx = 0; kx < KS; kx++) red[(kx * lanes + me) * 16 + cp] = acc[ky * KS + kx];
    __syncthreads();
    for (int e = tid; e < KS * 16; e += nt * p.Z) {
      const int kx = e >> 4, c2 = e & 15, ch = ch0 + 2 * c2;
      float s0 = 0.f, s1 = 0.f;
      for (int k = 0; k < lanes; k++) {
        const float2 v = unpack2(red[(kx * lanes + k) * 16 + c2]);
        s0 += v.x; s1 += v.y;
      }
      good = good && finite(s0) && finite(s1);
      if (ch < a.c) part[((int64_t)ch * SL + sl) * KK + ky * KS + kx] = s0;
      if (ch + 1 < a.c) part[((int64_t)(ch + 1) * SL + sl) * KK + ky * KS + kx] = s1;
    }
  }
  if (__syncthreads_and(good)) return;
  for (int e = tid; e < SLAB * KK; e += nt * p.Z) {
    const int ch = ch0 + e % SLAB, tap = e / SLAB;
    float* o = part + ((int64_t)ch * SL + sl) * KK + tap;
    if (ch < a.c && !finite(*o)) *o = direct_tap_sum<S>(a, p, sl, SL, ch, tap / KS, tap % KS);
  }
}

// Tiles of a layer: up to 16 column groups and as many images as fit 256 threads; then smaller image groups and strips down to
// min_rows until the launch has `want` blocks (a strip re-reads ks - stride input rows of its upper neighbour)
static TilePlan plan_tiles(const DwArgs& a, int64_t want, int min_rows) {
  TilePlan p{};
  const int gx = (int)cdiv(a.ow, TX);
  p.xtiles = (int)cdiv(gx, TILE_THREADS / 16);
  p.G = (int)cdiv(gx, p.xtiles);
  p.xtiles = (int)cdiv(gx, p.G);
  const int64_t per = cdiv(a.c, SLAB) * p.xtiles;
  p.Z = std::max(1, std::min(a.n, TILE_THREADS / (16 * p.G)));
  while (p.Z > 1 && p.Z * p.G * 16 > 64 && per * cdiv(a.n, p.Z) < want) p.Z = (p.Z + 1) / 2;
  p.imgs = (int)cdiv(a.n, p.Z);
  const int most = std::max(1, a.oh / std::min(a.oh, min_rows));
  p.seg_rows = (int)cdiv(a.oh, std::min<int64_t>(std::max<int64_t>(1, cdiv(want, per * p.imgs)), most));
  p.segs = (int)cdiv(a.oh, p.seg_rows);
  return p;
}
static size_t tile_smem(const DwArgs& a, const TilePlan& p, bool wgrad) {
  const size_t cols = (size_t)(p.G * TX - 1) * a.stride + a.ks, gcols = (size_t)p.G * TX;
  if (!wgrad) return ((size_t)a.ks * a.ks + DEPTH * p.Z * cols) * SLAB * 4;
  return std::max(DEPTH * p.Z * (cols + gcols) * SLAB * 4, (size_t)a.ks * p.Z * p.G * 16 * 8);
}
constexpr size_t TILE_SMEM_MAX = 200 * 1024;  // (the largest tile, one group of four columns of 16 images at 7x7 stride 2, takes 174 KB)

bool dw_tile_ok(const DwArgs& a) {
  if (!((a.ks == 3 || a.ks == 5 || a.ks == 7) && (a.stride == 1 || a.stride == 2))) return false;
  // block and item counts in 32 bits
  return (int64_t)a.n * a.oh * cdiv(a.ow, TX) * cdiv(a.c, SLAB) < (1ll << 30) && a.c < (1 << 20);
}

template <auto Kernel>
static void allow_smem() {
  static std::once_flag once;
  std::call_once(once, [] {
    if (cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TILE_SMEM_MAX) != cudaSuccess) cudaGetLastError();  // (the launch reports it)
  });
}
template <int KS, int S, bool FLIP>
static void run_conv(const DwArgs& a, const TilePlan& p, cudaStream_t s) {
  allow_smem<dw_tile_kernel<KS, S, FLIP>>();
  launch(dw_tile_kernel<KS, S, FLIP>, (unsigned)(cdiv(a.c, SLAB) * p.xtiles * p.segs * p.imgs), dim3(16 * p.G, p.Z), tile_smem(a, p, false), s, a, p);
}
template <int KS>
static void run_conv_ks(const DwArgs& a, const TilePlan& p, bool flip, cudaStream_t s) {
  if (a.stride == 2) run_conv<KS, 2, false>(a, p, s);
  else if (flip) run_conv<KS, 1, true>(a, p, s);
  else run_conv<KS, 1, false>(a, p, s);
}
int dw_tile_conv(const DwArgs& a, bool flip, cudaStream_t s) {
  const TilePlan p = plan_tiles(a, (int64_t)8 * sm_count(), (a.ks + a.stride) / a.stride);  // 8 x 501 x 60 x 60 3x3 stride 2: 55 us with strips twice as tall, 47 so
  if (a.ks == 3) run_conv_ks<3>(a, p, flip, s);
  else if (a.ks == 5) run_conv_ks<5>(a, p, flip, s);
  else run_conv_ks<7>(a, p, flip, s);
  return check_launch(flip ? "dw_dgrad_tile" : "dw_fwd_tile");
}

template <int KS, int S, int VEC>
static void run_wgrad(const DwArgs& a, const TilePlan& p, int SL, float* part, cudaStream_t s) {
  allow_smem<dw_wgrad_tile_kernel<KS, S, VEC>>();
  launch(dw_wgrad_tile_kernel<KS, S, VEC>, dim3((unsigned)cdiv(a.c, SLAB), (unsigned)SL), dim3(16 * p.G, p.Z), tile_smem(a, p, true), s, a, p, SL, part);
}
template <int KS, int VEC>
static void run_wgrad_ks(const DwArgs& a, const TilePlan& p, int SL, float* part, cudaStream_t s) {
  if (a.stride == 2) run_wgrad<KS, 2, VEC>(a, p, SL, part, s);
  else run_wgrad<KS, 1, VEC>(a, p, SL, part, s);
}
int dw_tile_wgrad(const DwArgs& a, bool vec, float scale, float* dw, omt_stream_t stream) {
  const int64_t slabs = cdiv(a.c, SLAB);
  const int per_sm = a.ks == 7 ? 1 : 2;
  const int64_t resident = std::max<int64_t>(1, (int64_t)per_sm * sm_count() / slabs);  // blocks per slab that run at once
  const TilePlan p = plan_tiles(a, 4 * resident * slabs, a.ks + 1);
  const int64_t small = std::max<int64_t>(1, std::min<int64_t>(4, TILE_THREADS / (16 * p.G * p.Z)));  // blocks of few threads: more per SM (27 x 301 x 23 x 21 7x7 stride 2 110 -> 63 us, 64 x 96 x 56 x 56 77 -> 52)
  // Every thread adds its share of the output pixels one after the other in float32. 7x7 takes up to four times the blocks, one after the other on an SM,
  // to keep that share to about 192: 128 x 96 x 56 x 56 4.3e-7 of the float64 result without, 2.5e-7 with, 3.5e-7 in the kernel that this one replaces, at
  // 198 -> 208 us. (3x3 and 5x5 have shorter shares, two blocks being resident, and are within a tenth of the error of the kernels they replace, or below it.)
  const int64_t items = (int64_t)p.imgs * p.segs * p.xtiles, once = std::min(resident * small, items);
  const int64_t rounds = a.ks == 7 ? std::min<int64_t>(4, std::max<int64_t>(1, std::min(cdiv((int64_t)a.n * a.oh * a.ow, once * p.G * p.Z * 192), items / once))) : 1;
  const int SL = (int)(once * rounds);
  const int kk = a.ks * a.ks;
  Scratch sc;
  int r = sc.get(nullptr, 0, (size_t)a.c * SL * kk * sizeof(float), stream);
  if (r) return r;
  float* part = (float*)sc.p;
  cudaStream_t s = st(stream);
  if (a.ks == 3) vec ? run_wgrad_ks<3, 4>(a, p, SL, part, s) : run_wgrad_ks<3, 1>(a, p, SL, part, s);
  else if (a.ks == 5) vec ? run_wgrad_ks<5, 4>(a, p, SL, part, s) : run_wgrad_ks<5, 1>(a, p, SL, part, s);
  else vec ? run_wgrad_ks<7, 4>(a, p, SL, part, s) : run_wgrad_ks<7, 1>(a, p, SL, part, s);
  r = check_launch("dw_wgrad_tile");
  if (r) return r;
  return dw_wgrad_finish(part, (int64_t)a.c * kk, kk, SL, scale, dw, s);
}

}  // namespace omt
