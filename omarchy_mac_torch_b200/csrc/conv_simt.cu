// fp32 implicit-GEMM convolution on the CUDA cores: forward, input gradient (all stride phases in one launch) and
// weight gradient (split-K + deterministic slab sum). This is the exact-fp32 path: it serves every geometry the op
// layer accepts (ks <= 11, stride 1..4, pad <= ks, any activation strides) and cross-checks the tensor-core path.
//
// Behaviour follows the reference's generated kernels (omarchy_mac_torch/gemm.py: kinds 0, 1, 5, 2) and their host
// side (csrc/conv.cpp:70-114); the structure does not: one templated kernel, im2col index decomposition hoisted out
// of the K loop (rows/columns are decomposed once per thread, the K index once per thread per step), register
// prefetch with double-buffered shared tiles, 128-bit shared loads and stores.
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace omt {

struct ConvArgs {
  ActView a;  // GEMM A-side activation: x (fwd), gy (dgrad), gy (wgrad)
  ActView b;  // second activation: y (fwd, output), dx (dgrad, output), x (wgrad, B operand)
  const float* w;
  const float* bias;
  float* out;  // wgrad: partial slabs [slices][M][N] (or dw when slices == 1)
  int n, ci, co, ih, iw, oh, ow, ks, stride, pad;
  int M, N, K, kslice, slices;
  uint32_t flags;
  float scale;
};

constexpr int BK = 8;

// ---- forward: m=(img,oy,ox) k=(ci,ky,kx) n=co ---------------------------------------------------------------------
struct Fwd {
  static constexpr bool A_MFAST = true, B_NFAST = false, SEQ = false;
  const ConvArgs& g;
  int M, N, kbeg, kend;
  __device__ Fwd(const ConvArgs& g_, int) : g(g_), M(g_.M), N(g_.N), kbeg(0), kend(g_.K) {}
  struct Row { int64_t base; int iy0, ix0; };  // iy0 = INT_MIN/2 marks an out-of-range row
  struct KIdx { int64_t off; int ky, kx; bool ok; };
  struct Col { const float* p; };
  __device__ Row row(int m) const {
    if (m >= M) return {0, -(1 << 28), 0};
    int ohw = g.oh * g.ow, img = m / ohw, r = m - img * ohw, oy = r / g.ow, ox = r - oy * g.ow;
    int iy0 = oy * g.stride - g.pad, ix0 = ox * g.stride - g.pad;
    return {img * g.a.sn + iy0 * g.a.sh + ix0 * g.a.sw, iy0, ix0};
  }
  __device__ KIdx kidx(int k) const {
    if (k >= kend) return {0, 0, 0, false};
    int kk = g.ks * g.ks, c = k / kk, r = k - c * kk, ky = r / g.ks, kx = r - ky * g.ks;
    return {c * g.a.sc + ky * g.a.sh + kx * g.a.sw, ky, kx, true};
  }
  __device__ float loadA(const Row& r, const KIdx& k) const {
    int y = r.iy0 + k.ky, x = r.ix0 + k.kx;
    if (!k.ok || y < 0 || y >= g.ih || x < 0 || x >= g.iw) return 0.f;
    return __ldg(g.a.p + r.base + k.off);
  }
  __device__ Col col(int nn) const { return {nn < N ? g.w + (int64_t)nn * g.K : nullptr}; }
  __device__ float loadB(const Col& c, const KIdx& k, int kabs) const { return (c.p && k.ok) ? __ldg(c.p + kabs) : 0.f; }
  // 4 consecutive rows (m..m+3) x 4 consecutive columns (nn..nn+3)
  __device__ void store(int m, int nn, const float (&v)[4][4]) const {
    int ohw = g.oh * g.ow;
    if (g.b.sc == 1 && nn + 3 < N) {  // channels-last output: the 4 columns of a row are contiguous
      float bv[4];
#pragma unroll
      for (int j = 0; j < 4; j++) bv[j] = (g.flags & OMT_EPI_BIAS) ? __ldg(g.bias + nn + j) : 0.f;
      bool done = true;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        int mm = m + i;
        if (mm >= M) break;
        int im2 = mm / ohw, r2 = mm - im2 * ohw, oy = r2 / g.ow, ox = r2 - oy * g.ow;
        float* p = g.b.p + g.b.off(im2, nn, oy, ox);
        if (reinterpret_cast<uintptr_t>(p) & 15) { done = false; break; }
        float4 o = make_float4(v[i][0] + bv[0], v[i][1] + bv[1], v[i][2] + bv[2], v[i][3] + bv[3]);
        if (g.flags & OMT_EPI_RELU) o = make_float4(fmaxf(o.x, 0.f), fmaxf(o.y, 0.f), fmaxf(o.z, 0.f), fmaxf(o.w, 0.f));
        *reinterpret_cast<float4*>(p) = o;
      }
      if (done) return;
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      int c = nn + j;
      if (c >= N) break;
      float bv = (g.flags & OMT_EPI_BIAS) ? __ldg(g.bias + c) : 0.f;
      float o[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        o[i] = v[i][j] + bv;
        if (g.flags & OMT_EPI_RELU) o[i] = fmaxf(o[i], 0.f);
      }
      int img = m / ohw, r = m - img * ohw;
      if (g.b.sw == 1 && g.b.sh == g.ow && m + 3 < M && r + 3 < ohw) {
        float* p = g.b.p + img * g.b.sn + c * g.b.sc + r;
        if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
          *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
          continue;
        }
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        int mm = m + i;
        if (mm >= M) break;
        int im2 = mm / ohw, r2 = mm - im2 * ohw, oy = r2 / g.ow, ox = r2 - oy * g.ow;
        g.b.p[g.b.off(im2, c, oy, ox)] = o[i];
      }
    }
  }
};

// ---- input gradient, one stride phase per blockIdx.z: m=(img,i,j) k=(co,ty,tx) n=ci -----------------------------------
// Phase (py,px) covers input pixels y=py+s*i, x=px+s*j. Only taps ky=ky0+s*ty, kx=kx0+s*tx reach them, from output
// pixel (i+qy-ty, j+qx-tx). Same index algebra as the reference host loop (csrc/conv.cpp:78-95).
struct Dgrad {
  static constexpr bool A_MFAST = true, B_NFAST = true, SEQ = false;
  const ConvArgs& g;
  int M, N, kbeg, kend;
  int py, px, ky0, kx0, qy, qx, hi, wi, jy, jx;
  __device__ Dgrad(const ConvArgs& g_, int z) : g(g_) {
    int s = g.stride;
    py = z / s; px = z - py * s;
    hi = (g.ih - py + s - 1) / s; wi = (g.iw - px + s - 1) / s;
    if (hi < 0) hi = 0;
    if (wi < 0) wi = 0;
    ky0 = (py + g.pad) % s; kx0 = (px + g.pad) % s;
    jy = ky0 < g.ks ? (g.ks - ky0 + s - 1) / s : 0;
    jx = kx0 < g.ks ? (g.ks - kx0 + s - 1) / s : 0;
    qy = (py + g.pad - ky0) / s; qx = (px + g.pad - kx0) / s;
    M = g.n * hi * wi; N = g.ci; kbeg = 0; kend = g.co * jy * jx;
  }
  struct Row { int64_t base; int oy0, ox0; };
  struct KIdx { int64_t off; int ty, tx, wofs; bool ok; };
  struct Col { int64_t wofs; bool ok; };
  __device__ Row row(int m) const {
    if (m >= M) return {0, -(1 << 28), 0};
    int hw = hi * wi, img = m / hw, r = m - img * hw, i = r / wi, j = r - i * wi;
    int oy0 = i + qy, ox0 = j + qx;
    return {img * g.a.sn + oy0 * g.a.sh + ox0 * g.a.sw, oy0, ox0};
  }
  __device__ KIdx kidx(int k) const {
    if (k >= kend) return {0, 0, 0, 0, false};
    int jj = jy * jx, co = k / jj, r = k - co * jj, ty = r / jx, tx = r - ty * jx;
    int ky = ky0 + g.stride * ty, kx = kx0 + g.stride * tx;
    return {co * g.a.sc - ty * g.a.sh - tx * g.a.sw, ty, tx, (co * g.ci * g.ks + ky) * g.ks + kx, true};
  }
  __device__ float loadA(const Row& r, const KIdx& k) const {
    int oy = r.oy0 - k.ty, ox = r.ox0 - k.tx;
    if (!k.ok || oy < 0 || oy >= g.oh || ox < 0 || ox >= g.ow) return 0.f;
    return __ldg(g.a.p + r.base + k.off);
  }
  __device__ Col col(int nn) const { return {(int64_t)nn * g.ks * g.ks, nn < N}; }
  __device__ float loadB(const Col& c, const KIdx& k, int) const {
    return (c.ok && k.ok) ? __ldg(g.w + k.wofs + c.wofs) : 0.f;
  }
  __device__ void store(int m, int nn, const float (&v)[4][4]) const {
    int hw = hi * wi;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      int c = nn + j;
      if (c >= N) break;
      int img = m / hw, r = m - img * hw, i0 = r / wi, j0 = r - i0 * wi;
      if (g.stride == 1 && g.b.sw == 1 && m + 3 < M && j0 + 3 < wi) {
        float* p = g.b.p + g.b.off(img, c, i0, j0);
        if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
          *reinterpret_cast<float4*>(p) = make_float4(v[0][j], v[1][j], v[2][j], v[3][j]);
          continue;
        }
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        int mm = m + i;
        if (mm >= M) break;
        int im2 = mm / hw, r2 = mm - im2 * hw, ii = r2 / wi, jj2 = r2 - ii * wi;
        g.b.p[g.b.off(im2, c, py + g.stride * ii, px + g.stride * jj2)] = v[i][j];
      }
    }
  }
};

// ---- weight gradient, one K slice per blockIdx.z: m=co k=(img,oy,ox) n=(ci,ky,kx) -------------------------------------
struct Wgrad {
  static constexpr bool A_MFAST = false, B_NFAST = false, SEQ = false;
  const ConvArgs& g;
  int M, N, kbeg, kend, z;
  __device__ Wgrad(const ConvArgs& g_, int z_) : g(g_), M(g_.M), N(g_.N), z(z_) {
    kbeg = z_ * g.kslice;
    kend = min(g.K, kbeg + g.kslice);
  }
  struct Row { int64_t off; bool ok; };
  struct KIdx { int64_t aoff, boff; int iy0, ix0; bool ok; };
  struct Col { int64_t off; int ky, kx; bool ok; };
  __device__ Row row(int m) const { return {m * g.a.sc, m < M}; }
  __device__ KIdx kidx(int k) const {
    if (k >= kend) return {0, 0, 0, 0, false};
    int ohw = g.oh * g.ow, img = k / ohw, r = k - img * ohw, oy = r / g.ow, ox = r - oy * g.ow;
    int iy0 = oy * g.stride - g.pad, ix0 = ox * g.stride - g.pad;
    return {img * g.a.sn + oy * g.a.sh + ox * g.a.sw, img * g.b.sn + iy0 * g.b.sh + ix0 * g.b.sw, iy0, ix0, true};
  }
  __device__ float loadA(const Row& r, const KIdx& k) const { return (r.ok && k.ok) ? __ldg(g.a.p + r.off + k.aoff) : 0.f; }
  __device__ Col col(int nn) const {
    if (nn >= N) return {0, 0, 0, false};
    int kk = g.ks * g.ks, c = nn / kk, r = nn - c * kk, ky = r / g.ks, kx = r - ky * g.ks;
    return {c * g.b.sc + ky * g.b.sh + kx * g.b.sw, ky, kx, true};
  }
  __device__ float loadB(const Col& c, const KIdx& k, int) const {
    int y = k.iy0 + c.ky, x = k.ix0 + c.kx;
    if (!c.ok || !k.ok || y < 0 || y >= g.ih || x < 0 || x >= g.iw) return 0.f;
    return __ldg(g.b.p + k.boff + c.off);
  }
  __device__ void store(int m, int nn, const float (&v)[4][4]) const {
    float* base = g.out + (int64_t)z * M * N;
    float sc = g.slices == 1 ? g.scale : 1.f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (m + i >= M) break;
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (nn + j < N) base[(int64_t)(m + i) * N + nn + j] = v[i][j] * sc;
    }
  }
};

// ---- channels-last operands ---------------------------------------------------------------------------------------------
// The loaders above walk the reduction as (channel, ky, kx): neighbouring lanes then read a channel count apart in a channels-last
// tensor, one sector per float. These walk it as (block of 8 channels, ky, kx, channel), 8 lanes to a pixel's channels, so that a
// sector is used whole; the taps of one channel block follow each other, so that their weights (ks * ks consecutive floats per
// channel) and the shifted rows of the activation are still in L1. A thread's position advances tap by tap: no division per step.
struct FwdCl : Fwd {
  static constexpr bool A_MFAST = false, B_NFAST = false, SEQ = true;
  __device__ FwdCl(const ConvArgs& g_, int z) : Fwd(g_, z) { kend = (g_.ci + 7) / 8 * 8 * g_.ks * g_.ks; }
  struct KIdx { int64_t off; int ky, kx, c, wofs; };
  __device__ KIdx kidx(int k) const {  // k: any multiple of 8 plus the lane's channel
    const int kk = g.ks * g.ks, step = k >> 3, blk = step / kk, tap = step - blk * kk, ky = tap / g.ks, kx = tap - ky * g.ks, c = blk * 8 + (k & 7);
    return {c * g.a.sc + ky * g.a.sh + kx * g.a.sw, ky, kx, c, c * kk + tap};
  }
  __device__ void advance(KIdx& k) const {
    k.kx++; k.wofs++; k.off += g.a.sw;
    if (k.kx == g.ks) {
      k.kx = 0; k.ky++; k.off += g.a.sh - g.ks * g.a.sw;
      if (k.ky == g.ks) { k.ky = 0; k.c += 8; k.off += 8 * g.a.sc - g.ks * g.a.sh; k.wofs += 7 * g.ks * g.ks; }
    }
  }
  __device__ float loadA(const Row& r, const KIdx& k) const {
    const int y = r.iy0 + k.ky, x = r.ix0 + k.kx;
    return k.c < g.ci && (unsigned)y < (unsigned)g.ih && (unsigned)x < (unsigned)g.iw ? __ldg(g.a.p + r.base + k.off) : 0.f;
  }
  __device__ float loadB(const Col& c, const KIdx& k, int) const { return c.p && k.c < g.ci ? __ldg(c.p + k.wofs) : 0.f; }
  __device__ void store(int m, int nn, const float (&v)[4][4]) const {
    const int ohw = g.oh * g.ow;
    float bv[4];
#pragma unroll
    for (int j = 0; j < 4; j++) bv[j] = (g.flags & OMT_EPI_BIAS) && nn + j < N ? __ldg(g.bias + nn + j) : 0.f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (m + i >= M) break;
      const int img = (m + i) / ohw, r = m + i - img * ohw, oy = r / g.ow, ox = r - oy * g.ow;
      float* p = g.b.p + g.b.off(img, nn, oy, ox);
      float o[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        o[j] = v[i][j] + bv[j];
        if (g.flags & OMT_EPI_RELU) o[j] = fmaxf(o[j], 0.f);
      }
      if (nn + 3 < N && (reinterpret_cast<uintptr_t>(p) & 15) == 0) *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
      else {
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (nn + j < N) p[j] = o[j];
      }
    }
  }
};

struct DgradCl : Dgrad {
  static constexpr bool A_MFAST = false, B_NFAST = true, SEQ = true;
  __device__ DgradCl(const ConvArgs& g_, int z) : Dgrad(g_, z) { kend = (g_.co + 7) / 8 * 8 * jy * jx; }
  struct KIdx { int64_t off; int ty, tx, c, wofs; };
  __device__ int wofs_of(int c, int ty, int tx) const { return (c * g.ci * g.ks + ky0 + g.stride * ty) * g.ks + kx0 + g.stride * tx; }
  __device__ KIdx kidx(int k) const {
    const int jj = max(1, jy * jx), step = k >> 3, blk = step / jj, tap = step - blk * jj, ty = tap / max(1, jx), tx = tap - ty * jx, c = blk * 8 + (k & 7);
    return {c * g.a.sc - ty * g.a.sh - tx * g.a.sw, ty, tx, c, wofs_of(c, ty, tx)};
  }
  __device__ void advance(KIdx& k) const {
    k.tx++; k.off -= g.a.sw;
    if (k.tx == jx) {
      k.tx = 0; k.ty++; k.off += jx * g.a.sw - g.a.sh;
      if (k.ty == jy) { k.ty = 0; k.c += 8; k.off += 8 * g.a.sc + jy * g.a.sh; }
    }
    k.wofs = wofs_of(k.c, k.ty, k.tx);
  }
  __device__ float loadA(const Row& r, const KIdx& k) const {
    const int oy = r.oy0 - k.ty, ox = r.ox0 - k.tx;
    return k.c < g.co && (unsigned)oy < (unsigned)g.oh && (unsigned)ox < (unsigned)g.ow ? __ldg(g.a.p + r.base + k.off) : 0.f;
  }
  __device__ float loadB(const Col& c, const KIdx& k, int) const { return c.ok && k.c < g.co ? __ldg(g.w + k.wofs + c.wofs) : 0.f; }
  __device__ void store(int m, int nn, const float (&v)[4][4]) const {  // (neighbouring threads hold neighbouring columns: see the kernel)
    const int hw = hi * wi;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (m + i >= M) break;
      const int img = (m + i) / hw, r = m + i - img * hw, ii = r / wi, jj = r - ii * wi;
      float* p = g.b.p + g.b.off(img, nn, py + g.stride * ii, px + g.stride * jj);
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (nn + j < N) p[j] = v[i][j];
    }
  }
};

// columns as (tap, channel): neighbouring lanes read neighbouring channels of x; the stores put them back into [ci][ky][kx]
struct WgradCl : Wgrad {
  static constexpr bool A_MFAST = true, B_NFAST = true, SEQ = false;
  using Wgrad::Wgrad;
  __device__ Col col(int nn) const {
    if (nn >= N) return {0, 0, 0, false};
    const int tap = nn / g.ci, c = nn - tap * g.ci, ky = tap / g.ks, kx = tap - ky * g.ks;
    return {c * g.b.sc + ky * g.b.sh + kx * g.b.sw, ky, kx, true};
  }
  __device__ void store(int m, int nn, const float (&v)[4][4]) const {
    float* base = g.out + (int64_t)z * M * N;
    const float sc = g.slices == 1 ? g.scale : 1.f;
    const int kk = g.ks * g.ks;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      if (nn + j >= N) break;
      const int tap = (nn + j) / g.ci, c = nn + j - tap * g.ci;
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (m + i < M) base[(int64_t)(m + i) * N + c * kk + tap] = v[i][j] * sc;
    }
  }
};

// C tile BM x BN, KG groups of (BM / TM) * (BN / TN) threads. Each thread of a group owns TM x TN outputs as (TM/4) x (TN/4) groups of
// 4x4, groups BM/2 or BN/2 apart, threads m-fastest so stores along m coalesce for NCHW outputs. The KG groups work on the
// same tile and take every KG-th step of the reduction, each with its own shared tiles; their sums meet in shared memory, in group
// order, at the end. That is for launches with fewer tiles than the SMs need warps (KG = 2) and for weight gradients of a few
// outputs over very many pixels (16 x 32 outputs, eight groups), which a 128 x 64 tile computes almost entirely as padding: 252 us
// for 16 x 27 outputs over 401 408 pixels, 7 % of a MobileNetV3 step. With the channels-last loaders the three passes of a
// 90 -> 50 channel 3x3 stride-2 layer (13 x 57 x 43) go from 217 to 151 us, that step from 3783 to 3592.
// The minimum number of blocks: none as a rule, for a minimum of one lets the compiler spend registers freely (155 against 126 for the 128 x 128 weight
// gradient, so one block per SM and not two: 32 x 130 x 56 x 56 -> 129 3x3 1945 us -> 2087). One where two groups share a tile, as those launches have no second
// block for an SM (8 x 50 x 7 x 7 -> 250 3x3 input gradient 129 us -> 113). Two with the channels-last loaders at 128 x 128, whose 100 bytes of spills cost less
// than the second block gives (32 x 130 x 56 x 56 -> 129 3x3 input gradient 1990 us -> 1650).
template <class L, int BM, int BN, int TM, int TN, int KG = 1>
__global__ void __launch_bounds__((BM / TM) * (BN / TN) * KG, L::SEQ && BM * BN == 128 * 128 ? 2 : (KG == 2 ? 1 : 0)) conv_gemm_simt(ConvArgs g) {
  pdl_wait();
  constexpr int TY = BM / TM, GM = TM / 4, GN = TN / 4, TG = (BM / TM) * (BN / TN);
  constexpr bool A_MF = L::A_MFAST && TG == 256, B_NF = L::B_NFAST && TG == 256;  // small groups: lanes along k, one position per thread
  constexpr int RS = TG / 8;  // rows (columns) that one pass of a group's threads covers
  constexpr int RA = BM / RS, RB = (BN + RS - 1) / RS;
  static_assert(BM % RS == 0 && (TG == 256 || BN % RS == 0), "whole passes");
  constexpr int TILE_F = 2 * BK * (BM + 4) + 2 * BK * (BN + 4);
  constexpr int SMEM_F = KG > 1 && BM * BN > KG * TILE_F ? BM * BN : KG * TILE_F;
  __shared__ __align__(16) float sm[SMEM_F];
  const int kg = KG > 1 ? threadIdx.x / TG : 0, tid = KG > 1 ? threadIdx.x % TG : threadIdx.x;
  float (*As)[BK][BM + 4] = reinterpret_cast<float (*)[BK][BM + 4]>(sm + kg * TILE_F);
  float (*Bs)[BK][BN + 4] = reinterpret_cast<float (*)[BK][BN + 4]>(sm + kg * TILE_F + 2 * BK * (BM + 4));
  L ld(g, blockIdx.z);
  const int M = ld.M, N = ld.N;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;  // M tiles on x: its limit is 2^31-1, y's is 65535
  if (m0 >= M) return;
  const int a_k = A_MF ? (tid >> 5) : (tid & 7), a_r = A_MF ? (tid & 31) : (tid >> 3);
  const int b_k = B_NF ? (tid >> 5) : (tid & 7), b_r = B_NF ? (tid & 31) : (tid >> 3);
  typename L::Row ra[RA];
  typename L::Col cb[RB];
#pragma unroll
  for (int i = 0; i < RA; i++) ra[i] = ld.row(m0 + a_r + RS * i);
#pragma unroll
  for (int i = 0; i < RB; i++) cb[i] = ld.col((b_r + RS * i < BN) ? n0 + b_r + RS * i : N);
  float acc[GM][GN][4][4];
#pragma unroll
  for (int a = 0; a < GM; a++)
#pragma unroll
    for (int b = 0; b < GN; b++)
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[a][b][i][j] = 0.f;
  float pa[RA], pb[RB];
  typename L::KIdx ka = ld.kidx(ld.kbeg + kg * BK + a_k), kb = ld.kidx(ld.kbeg + kg * BK + b_k);  // (SEQ loaders: the position to fetch next)
  auto fetch = [&](int k0) {
    if constexpr (!L::SEQ) {
      ka = ld.kidx(k0 + a_k);
      if constexpr (A_MF != B_NF) kb = ld.kidx(k0 + b_k);
    }
#pragma unroll
    for (int i = 0; i < RA; i++) pa[i] = ld.loadA(ra[i], ka);
    if constexpr (A_MF == B_NF) {
#pragma unroll
      for (int i = 0; i < RB; i++) pb[i] = ld.loadB(cb[i], ka, k0 + b_k);
    } else {
#pragma unroll
      for (int i = 0; i < RB; i++) pb[i] = ld.loadB(cb[i], kb, k0 + b_k);
    }
    if constexpr (L::SEQ) {
#pragma unroll
      for (int q = 0; q < KG; q++) {
        ld.advance(ka);
        if constexpr (A_MF != B_NF) ld.advance(kb);
      }
    }
  };
  auto commit = [&](int buf) {
#pragma unroll
    for (int i = 0; i < RA; i++) As[buf][a_k][a_r + RS * i] = pa[i];
#pragma unroll
    for (int i = 0; i < RB; i++)
      if (b_r + RS * i < BN) Bs[buf][b_k][b_r + RS * i] = pb[i];
  };
  const int tm = tid % TY, tn = tid / TY;
  int buf = 0;
  if (ld.kbeg < ld.kend) {  // (loads at and beyond kend give zeros: the last round of the groups may be partly empty)
    fetch(ld.kbeg + kg * BK);
    commit(0);
  }
  __syncthreads();
  for (int k0 = ld.kbeg; k0 < ld.kend; k0 += BK * KG) {
    const bool more = k0 + BK * KG < ld.kend;
    if (more) fetch(k0 + BK * KG + kg * BK);
#pragma unroll
    for (int kk = 0; kk < BK; kk++) {
      float4 av[GM], bv[GN];
#pragma unroll
      for (int a = 0; a < GM; a++) av[a] = *reinterpret_cast<const float4*>(&As[buf][kk][tm * 4 + a * (BM / 2)]);
#pragma unroll
      for (int b = 0; b < GN; b++) bv[b] = *reinterpret_cast<const float4*>(&Bs[buf][kk][tn * 4 + b * (BN / 2)]);
#pragma unroll
      for (int a = 0; a < GM; a++) {
        const float ar[4] = {av[a].x, av[a].y, av[a].z, av[a].w};
#pragma unroll
        for (int b = 0; b < GN; b++) {
          const float br[4] = {bv[b].x, bv[b].y, bv[b].z, bv[b].w};
#pragma unroll
          for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[a][b][i][j] = fmaf(ar[i], br[j], acc[a][b][i][j]);
        }
      }
    }
    if (more) commit(buf ^ 1);
    __syncthreads();
    buf ^= 1;
  }
  if constexpr (KG > 1) {
    static_assert(GM == 1 && GN == 1, "one 4x4 group per thread");
    float4* red = reinterpret_cast<float4*>(sm);  // [4][TG] float4: one group's tile at a time
    for (int q = 1; q < KG; q++) {
      if (kg == q) {
#pragma unroll
        for (int i = 0; i < 4; i++) red[i * TG + tid] = make_float4(acc[0][0][i][0], acc[0][0][i][1], acc[0][0][i][2], acc[0][0][i][3]);
      }
      __syncthreads();
      if (kg == 0) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float4 v = red[i * TG + tid];
          acc[0][0][i][0] += v.x; acc[0][0][i][1] += v.y; acc[0][0][i][2] += v.z; acc[0][0][i][3] += v.w;
        }
      }
      __syncthreads();
    }
    if (kg != 0) return;
  }
#pragma unroll
  for (int a = 0; a < GM; a++)
#pragma unroll
    for (int b = 0; b < GN; b++) {
      int m = m0 + tm * 4 + a * (BM / 2), nn = n0 + tn * 4 + b * (BN / 2);
      if (m < M && nn < N) ld.store(m, nn, acc[a][b]);
    }
}

// dw[i] = scale * sum_z part[z][i]   (reference csrc/kernels/gemm_reduce.wgsl:7-13, vectorised)
__global__ void __launch_bounds__(256) slab_sum_kernel(const float* __restrict__ part, float* __restrict__ out, int64_t total,
                                                       int slices, float scale) {
  pdl_wait();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  float s = 0.f;
  for (int z = 0; z < slices; z++) s += __ldg(part + (int64_t)z * total + i);
  out[i] = s * scale;
}

template <class L, int BM, int BN, int TM, int TN, int KG = 1>
static void launch_tile(const ConvArgs& a, int64_t Mmax, int64_t N, int gz, cudaStream_t s) {
  const dim3 grid((unsigned)cdiv(Mmax, BM), (unsigned)cdiv(N, BN), gz);
  launch(conv_gemm_simt<L, BM, BN, TM, TN, KG>, grid, (BM / TM) * (BN / TN) * KG, 0, s, a);
}
template <class L>
static int launch_gemm(const ConvArgs& a, int64_t Mmax, int64_t N, int gz, cudaStream_t s, const char* name) {
  constexpr bool WGRAD = std::is_base_of_v<Wgrad, L>;
  // tile choice: narrow-N tiles for tiny channel counts, smaller tiles when the grid would not fill the SMs
  int sms = sm_count();
  auto blocks = [&](int bm, int bn) { return cdiv(Mmax, bm) * cdiv(N, bn) * gz; };
  // M tiles on grid.x (limit 2^31-1), N tiles on grid.y (limit 65535: N is a channel count, or ci*ks*ks for the weight gradient)
  OMT_REQUIRE(cdiv(N, N <= 16 ? 16 : 64) <= 65535 && gz <= 65535, "%s: %lld GEMM columns exceed the launch grid", name, (long long)N);
  if constexpr (WGRAD) {
    bool done = true;
    if (Mmax <= 16 && N <= 32) launch_tile<L, 16, 32, 4, 4, 8>(a, Mmax, N, gz, s);  // a few outputs (first layers): small tiles, the reduction
    else if (Mmax <= 32 && N <= 32) launch_tile<L, 32, 32, 4, 4, 4>(a, Mmax, N, gz, s);  // shared by the block's groups
    else if (Mmax <= 64 && N > 64 && blocks(128, 128) >= sms) launch_tile<L, 64, 128, 4, 8>(a, Mmax, N, gz, s);
    else done = false;
    if (done) return check_launch(name);
  }
  if (N <= 16) {
    launch_tile<L, 256, 16, 4, 4>(a, Mmax, N, gz, s);
  } else if (N <= 64 || blocks(128, 128) < sms) {
    if (blocks(128, 64) < sms) {
      if (blocks(64, 64) <= sms) launch_tile<L, 64, 64, 4, 4, 2>(a, Mmax, N, gz, s);  // one block per SM at most: twice the warps
      else launch_tile<L, 64, 64, 4, 4>(a, Mmax, N, gz, s);
    } else {
      launch_tile<L, 128, 64, 8, 4>(a, Mmax, N, gz, s);
    }
  } else {
    launch_tile<L, 128, 128, 8, 8>(a, Mmax, N, gz, s);
  }
  return check_launch(name);
}

static ConvArgs base_args(const OmtConvGeo* g) {
  ConvArgs a{};
  a.n = g->n; a.ci = g->ci; a.co = g->co; a.ih = g->ih; a.iw = g->iw; a.oh = g->oh; a.ow = g->ow;
  a.ks = g->ks; a.stride = g->stride; a.pad = g->pad;
  a.slices = 1; a.scale = 1.f;
  return a;
}

// Whether the loaders that walk the reduction in steps of eight channels pay, for a reduction over c channels: the last step is partly padding, and so
// are the products of all its taps. One tap costs little against whole sectors; with 3x3 the padding may be 3/5 of the channels (32 x 56 x 56
// forward, 9 -> 64 channels: 57 -> 74 us, 10 -> 90: 165 -> 125), with more taps a third (5x5 17 -> 33: 225 -> 252, 25 -> 50: even).
static bool steps_of_eight_pay(int c, int ks) {
  const int padded = (c + 7) / 8 * 8;
  return c >= 8 && (ks == 1 || (ks <= 3 ? 5 * padded <= 8 * c : 3 * padded <= 4 * c));
}

int simt_conv_fwd(const OmtConvGeo* g, const OmtAct* x, const float* w, const float* bias, const OmtAct* y,
                  uint32_t flags, cudaStream_t s) {
  ConvArgs a = base_args(g);
  a.a = view(x); a.b = view(y); a.w = w; a.bias = bias; a.flags = flags;
  a.M = g->n * g->oh * g->ow; a.N = g->co; a.K = g->ci * g->ks * g->ks;
  if (x->sc == 1 && y->sc == 1 && steps_of_eight_pay(g->ci, g->ks)) return launch_gemm<FwdCl>(a, a.M, a.N, 1, s, "conv_fwd_simt");
  return launch_gemm<Fwd>(a, a.M, a.N, 1, s, "conv_fwd_simt");
}

// ---------------------------------------------------------------------------------------------------------------------
// Input gradient for <= 4 input channels (a network's first layer): the GEMM would have N = ci <= 4 columns, so instead
// one thread owns one input pixel and all its channels. A block works on one stride phase (py, px) of one image: every
// thread then needs the same filter taps (ky = ky0 + s*ty, kx = kx0 + s*tx; the phase algebra of csrc/conv.cpp:78-95),
// whose weights sit in shared memory as float4 per (tap, co) and are read as warp-wide broadcasts, while consecutive
// lanes read consecutive output pixels of gy.
// ---------------------------------------------------------------------------------------------------------------------
struct DgSmallArgs {
  ActView gy, dx;
  const float* w;
  int n, ci, co, ih, iw, oh, ow, ks, stride, pad;
};

__global__ void __launch_bounds__(128) dgrad_small_ci_kernel(DgSmallArgs a) {
  pdl_wait();
  extern __shared__ float4 wsm[];  // [jy * jx][co]
  const int s = a.stride;
  const int py = blockIdx.y / s, px = blockIdx.y - py * s, img = blockIdx.z;
  const int hi = (a.ih - py + s - 1) / s, wi = (a.iw - px + s - 1) / s;  // pixels of this phase
  const int ky0 = (py + a.pad) % s, kx0 = (px + a.pad) % s;
  const int jy = ky0 < a.ks ? (a.ks - ky0 + s - 1) / s : 0, jx = kx0 < a.ks ? (a.ks - kx0 + s - 1) / s : 0;
  const int taps = jy * jx;
  for (int i = threadIdx.x; i < taps * a.co; i += blockDim.x) {
    const int t = i / a.co, o = i - t * a.co;
    const int ky = ky0 + s * (t / jx), kx = kx0 + s * (t % jx);
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c = 0; c < a.ci; c++) v[c] = __ldg(a.w + (((int64_t)o * a.ci + c) * a.ks + ky) * a.ks + kx);
    wsm[i] = make_float4(v[0], v[1], v[2], v[3]);
  }
  __syncthreads();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= hi * wi) return;
  const int yi = p / wi, xi = p - yi * wi;
  const int y = py + s * yi, x = px + s * xi;
  // output pixel reached through tap (ty, tx): oy = (y + pad - ky) / s = qy - ty with qy = (y + pad - ky0) / s
  const int qy = (y + a.pad - ky0) / s, qx = (x + a.pad - kx0) / s;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  const bool vec = a.gy.sc == 1 && (a.co & 3) == 0 && ((reinterpret_cast<uintptr_t>(a.gy.p) & 15) == 0) && (a.gy.sw & 3) == 0 &&
                   (a.gy.sh & 3) == 0 && (a.gy.sn & 3) == 0;
  for (int ty = 0; ty < jy; ty++) {
    const int oy = qy - ty;
    if (oy < 0 || oy >= a.oh) continue;
    for (int tx = 0; tx < jx; tx++) {
      const int ox = qx - tx;
      if (ox < 0 || ox >= a.ow) continue;
      const float4* wt = wsm + (ty * jx + tx) * a.co;
      const float* gp = a.gy.p + a.gy.off(img, 0, oy, ox);
      if (vec) {
        for (int o = 0; o < a.co; o += 4) {
          const float4 g4 = __ldg(reinterpret_cast<const float4*>(gp + o));
          const float gv[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const float4 wv = wt[o + k];
            acc[0] = fmaf(gv[k], wv.x, acc[0]); acc[1] = fmaf(gv[k], wv.y, acc[1]);
            acc[2] = fmaf(gv[k], wv.z, acc[2]); acc[3] = fmaf(gv[k], wv.w, acc[3]);
          }
        }
      } else {
#pragma unroll 4
        for (int o = 0; o < a.co; o++) {
          const float gv = __ldg(gp + (int64_t)o * a.gy.sc);
          const float4 wv = wt[o];
          acc[0] = fmaf(gv, wv.x, acc[0]); acc[1] = fmaf(gv, wv.y, acc[1]);
          acc[2] = fmaf(gv, wv.z, acc[2]); acc[3] = fmaf(gv, wv.w, acc[3]);
        }
      }
    }
  }
  float* out = a.dx.p + a.dx.off(img, 0, y, x);
  for (int c = 0; c < a.ci; c++) out[(int64_t)c * a.dx.sc] = acc[c];
}

bool dgrad_small_ci_ok(const OmtConvGeo* g) {
  if (g->ci > 4 || g->groups != 1 || g->n > 65535 || g->stride * g->stride > 65535) return false;
  const int jmax = (int)cdiv(g->ks, g->stride);
  return (size_t)jmax * jmax * g->co * sizeof(float4) <= 200 * 1024;
}
int dgrad_small_ci(const OmtConvGeo* g, const OmtAct* gy, const float* w, const OmtAct* dx, cudaStream_t s) {
  DgSmallArgs a{view(gy), view(dx), w, g->n, g->ci, g->co, g->ih, g->iw, g->oh, g->ow, g->ks, g->stride, g->pad};
  const int jmax = (int)cdiv(g->ks, g->stride);
  const size_t smem = (size_t)jmax * jmax * g->co * sizeof(float4);
  static size_t attr = 0;
  if (smem > 48 * 1024 && smem > attr) {
    OMT_CUDA(cudaFuncSetAttribute(dgrad_small_ci_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr = smem;
  }
  const int64_t per_phase = cdiv(g->ih, g->stride) * cdiv(g->iw, g->stride);
  dim3 grid((unsigned)cdiv(per_phase, 128), (unsigned)(g->stride * g->stride), (unsigned)g->n);
  launch(dgrad_small_ci_kernel, grid, 128, smem, s, a);
  return check_launch("conv_dgrad_small_ci");
}

int simt_conv_dgrad(const OmtConvGeo* g, const OmtAct* gy, const float* w, const OmtAct* dx, cudaStream_t s) {
  if (dgrad_small_ci_ok(g)) return dgrad_small_ci(g, gy, w, dx, s);
  ConvArgs a = base_args(g);
  a.a = view(gy); a.b = view(dx); a.w = w;
  int st_ = g->stride;
  int64_t hi = cdiv(g->ih, st_), wi = cdiv(g->iw, st_);  // phase (0,0) is the largest
  a.N = g->ci;
  if (gy->sc == 1 && dx->sc == 1 && steps_of_eight_pay(g->co, g->ks)) return launch_gemm<DgradCl>(a, (int64_t)g->n * hi * wi, a.N, st_ * st_, s, "conv_dgrad_simt");
  return launch_gemm<Dgrad>(a, (int64_t)g->n * hi * wi, a.N, st_ * st_, s, "conv_dgrad_simt");
}

// Split-K slicing: enough slices to fill the machine about twice over, each at least 64 deep (the reference's
// bound, csrc/conv.cpp:106-109, with the M1's "512 workgroups" target replaced by 2 x SM count).
void wgrad_slices(const OmtConvGeo* g, int* slices, int* kslice) {
  int64_t M = g->co, N = (int64_t)g->ci * g->ks * g->ks, K = (int64_t)g->n * g->oh * g->ow;
  int bm = 128, bn = N <= 16 ? 16 : (N <= 64 ? 64 : 128);
  if (N <= 16) bm = 256;
  int64_t tiles = cdiv(M, bm) * cdiv(N, bn);
  int64_t want = std::max<int64_t>(1, (2 * sm_count()) / tiles);
  int64_t sl = std::max<int64_t>(1, std::min<int64_t>(want, K / 64));
  int64_t ks = cdiv(cdiv(K, sl), BK) * BK;
  *kslice = (int)ks;
  *slices = (int)cdiv(K, ks);
}

int simt_conv_wgrad(const OmtConvGeo* g, const OmtAct* x, const OmtAct* gy, float* dw, float scale, float* part,
                    cudaStream_t s) {
  ConvArgs a = base_args(g);
  a.a = view(gy); a.b = view(x); a.scale = scale;
  a.M = g->co; a.N = g->ci * g->ks * g->ks; a.K = g->n * g->oh * g->ow;
  wgrad_slices(g, &a.slices, &a.kslice);
  a.out = a.slices == 1 ? dw : part;
  // (columns as (tap, channel): 3 to 7 % slower below, even around 66, 1 to 3 % faster at 90 where there are pixels enough, 5 % from 130 on)
  int r = x->sc == 1 && gy->sc == 1 && g->ci >= 64 ? launch_gemm<WgradCl>(a, a.M, a.N, a.slices, s, "conv_wgrad_simt")
                                                   : launch_gemm<Wgrad>(a, a.M, a.N, a.slices, s, "conv_wgrad_simt");
  if (r != OMT_OK || a.slices == 1) return r;
  int64_t total = (int64_t)a.M * a.N;
  launch(slab_sum_kernel, (unsigned)cdiv(total, 256), 256, 0, s, part, dw, total, a.slices, scale);
  return check_launch("conv_wgrad_slab_sum");
}

size_t simt_wgrad_workspace(const OmtConvGeo* g) {
  int slices, kslice;
  wgrad_slices(g, &slices, &kslice);
  if (slices == 1) return 0;
  return (size_t)slices * g->co * g->ci * g->ks * g->ks * sizeof(float);
}

// ---------------------------------------------------------------------------------------------------------------------
// weight gradient without any allocation
// ---------------------------------------------------------------------------------------------------------------------
// Scratch for the split-K slabs of omt_conv_wgrad_noalloc. It lives in the library image: every GPU that loads the
// library holds these 16 MiB until the process exits. All calls on a device share it.
constexpr size_t NOALLOC_SCRATCH_FLOATS = (size_t)4 << 20;
static __device__ __align__(256) float g_noalloc_scratch[NOALLOC_SCRATCH_FLOATS];

constexpr int NOALLOC_MAX_DEVICES = 64;
static float* g_noalloc_ptr[NOALLOC_MAX_DEVICES];  // device address of g_noalloc_scratch, per device ordinal

}  // namespace omt

using namespace omt;

extern "C" size_t omt_conv_wgrad_noalloc_capacity(void) { return NOALLOC_SCRATCH_FLOATS * sizeof(float); }

extern "C" int omt_conv_wgrad_noalloc(const OmtConvGeo* g, const OmtAct* x, const OmtAct* gy, float* dw, float scale,
                                      omt_stream_t stream) {
  int r = check_dense(g, "omt_conv_wgrad_noalloc");  // the same checks as omt_conv_wgrad (extents below 2^31 included)
  if (r) return r;
  OMT_REQUIRE(x && gy && x->p && gy->p && dw, "omt_conv_wgrad_noalloc: null pointer");
  const size_t need = simt_wgrad_workspace(g);
  if (need > NOALLOC_SCRATCH_FLOATS * sizeof(float)) {
    set_error("omt_conv_wgrad_noalloc: this geometry needs %zu bytes of split-K scratch, the built-in scratch holds %zu", need,
              NOALLOC_SCRATCH_FLOATS * sizeof(float));
    return OMT_ETOOBIG;
  }
  int dev = -1;
  OMT_CUDA(cudaGetDevice(&dev));
  OMT_REQUIRE(dev >= 0 && dev < NOALLOC_MAX_DEVICES, "omt_conv_wgrad_noalloc: device ordinal %d out of range", dev);
  if (!g_noalloc_ptr[dev]) {
    // The array's name is only a host-side handle; the kernels need its address on the current device. Looked up once per
    // device (this first call should therefore come before any stream capture).
    float* p = nullptr;
    OMT_CUDA(cudaGetSymbolAddress((void**)&p, g_noalloc_scratch));
    g_noalloc_ptr[dev] = p;
  }
  return simt_conv_wgrad(g, x, gy, dw, scale, g_noalloc_ptr[dev], st(stream));
}

namespace omt {

// ---- bias gradient: db[c] = sum gy[:, c, :, :] ---------------------------------------------------------------------
// One block per (channel, slice) with 128-bit loads when the plane is contiguous, then a second tiny kernel; the
// reference used one workgroup per channel (csrc/kernels/csum_nchw.wgsl), i.e. 64 blocks for 64 channels.
__global__ void __launch_bounds__(256) csum_part_kernel(ActView gy, int n, int c, int h, int w, int S, float* part) {
  pdl_wait();
  __shared__ float red[32];
  int ch = blockIdx.x, sl = blockIdx.y;
  int hw = h * w;
  float s = 0.f;
  bool plane = gy.sw == 1 && gy.sh == w;
  for (int img = sl; img < n; img += S) {
    if (plane) {
      const float* p = gy.p + img * gy.sn + ch * gy.sc;
      if (((reinterpret_cast<uintptr_t>(p) & 15) == 0) && (hw & 3) == 0) {
        const float4* p4 = reinterpret_cast<const float4*>(p);
        for (int e = threadIdx.x; e < hw / 4; e += blockDim.x) {
          float4 v = __ldg(p4 + e);
          s += (v.x + v.y) + (v.z + v.w);
        }
      } else {
        for (int e = threadIdx.x; e < hw; e += blockDim.x) s += __ldg(p + e);
      }
    } else {
      for (int e = threadIdx.x; e < hw; e += blockDim.x) s += __ldg(gy.p + gy.off(img, ch, e / w, e % w));
    }
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) part[ch * S + sl] = s;
}
__global__ void csum_fin_kernel(const float* part, int c, int S, float scale, float* out) {
  pdl_wait();
  int ch = blockIdx.x * blockDim.x + threadIdx.x;
  if (ch >= c) return;
  float s = 0.f;
  for (int k = 0; k < S; k++) s += part[ch * S + k];
  out[ch] = s * scale;
}
// Channels-last: a block is CL channel groups of VEC x 256 / CL pixel lanes over `per` pixels; the lanes meet in a tree in shared
// memory. HBM-bound: every lane keeps four independent loads in flight, and a block has at least 32 KB to read. One thread per
// channel walking pixels (what this replaces) left most of the block idle below 256 channels and had one load in flight: with its
// second launch 74 us for 16 x 64 x 55 x 55 (12 MB), and a PlainCNN step with three such layers went from 568 to 438 us. With one slice the sums are final, else csum_nhwc_fin_kernel adds the slices.
template <int VEC>
__global__ void __launch_bounds__(256) csum_nhwc_kernel(const float* __restrict__ gy, int64_t pixels, int c, int CL, int64_t per, float scale, float div,
                                                        float* __restrict__ out) {  // out[image][slice][c], images of `pixels` pixels each
  pdl_wait();
  gy += (int64_t)blockIdx.z * pixels * c;
  out += (int64_t)blockIdx.z * gridDim.y * c;
  __shared__ float red[256][VEC];
  const int PL = 256 / CL, cl = threadIdx.x % CL, pl = threadIdx.x / CL;
  const int ch = ((int)blockIdx.x * CL + cl) * VEC;
  const bool live = pl < PL && ch < c;
  float s[4][VEC];
#pragma unroll
  for (int k = 0; k < 4; k++)
#pragma unroll
    for (int e = 0; e < VEC; e++) s[k][e] = 0.f;
  if (live) {
    const int64_t end = min(pixels, ((int64_t)blockIdx.y + 1) * per);
    int64_t p = (int64_t)blockIdx.y * per + pl;
    auto add = [&](float (&t)[VEC], int64_t q) {
      if constexpr (VEC == 4) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(gy + q * c + ch));
        t[0] += v.x; t[1] += v.y; t[2] += v.z; t[3] += v.w;
      } else {
        t[0] += __ldg(gy + q * c + ch);
      }
    };
    for (; p + 3 * PL < end; p += 4 * PL) {
#pragma unroll
      for (int k = 0; k < 4; k++) add(s[k], p + k * PL);
    }
    for (; p < end; p += PL) add(s[0], p);
  }
#pragma unroll
  for (int e = 0; e < VEC; e++) red[threadIdx.x][e] = (s[0][e] + s[1][e]) + (s[2][e] + s[3][e]);
  __syncthreads();
  for (int n = PL; n > 1;) {
    const int h = (n + 1) / 2;
    if (pl < n - h) {
#pragma unroll
      for (int e = 0; e < VEC; e++) red[threadIdx.x][e] += red[threadIdx.x + h * CL][e];
    }
    __syncthreads();
    n = h;
  }
  if (pl == 0 && live) {
#pragma unroll
    for (int e = 0; e < VEC; e++) out[(int64_t)blockIdx.y * c + ch + e] = red[threadIdx.x][e] * scale / div;
  }
}
// 32 channels x 16 slice lanes per block
__global__ void __launch_bounds__(512) csum_nhwc_fin_kernel(const float* __restrict__ part, int c, int S, float scale, float div, float* __restrict__ out) {
  pdl_wait();
  part += (int64_t)blockIdx.y * S * c;
  out += (int64_t)blockIdx.y * c;
  __shared__ float red[16][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5, ch = blockIdx.x * 32 + x;
  float s = 0.f;
  if (ch < c) {
#pragma unroll 4
    for (int k = y; k < S; k += 16) s += __ldg(part + (int64_t)k * c + ch);
  }
  red[y][x] = s;
  __syncthreads();
  if (y == 0 && ch < c) {
    for (int k = 1; k < 16; k++) s += red[k][x];
    out[ch] = s * scale / div;
  }
}
struct CsumPlan {
  bool vec;          // four channels per lane
  int CL;            // channel groups per block
  int64_t gx, S, per;  // blocks over the channels, slices of an image, pixels per slice
};
static CsumPlan plan_csum(const float* x, int64_t images, int64_t pixels, int c) {
  CsumPlan p;
  p.vec = c % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const int groups = p.vec ? c / 4 : c;
  p.CL = groups <= 64 ? groups : 32;
  p.gx = cdiv(groups, p.CL);
  // slices of 32 KB and more, at most about four blocks per SM
  const int64_t want = std::min<int64_t>(pixels * c * 4 / p.gx / (32 << 10), 4 * sm_count() / (p.gx * images));
  p.per = cdiv(pixels, std::max<int64_t>(1, want));
  p.S = cdiv(pixels, p.per);
  return p;
}
// out[image][ch] = scale / div * sum over the image's pixels, for images of channels-last pixels
static int csum_nhwc(const float* x, int64_t images, int64_t pixels, int c, float scale, float div, float* out, omt_stream_t stream) {
  cudaStream_t s = st(stream);
  const CsumPlan p = plan_csum(x, images, pixels, c);
  Scratch sc;
  if (p.S > 1) {
    int r = sc.get(nullptr, 0, (size_t)images * c * p.S * sizeof(float), stream);
    if (r) return r;
  }
  float* part = p.S > 1 ? (float*)sc.p : out;
  const float sc1 = p.S > 1 ? 1.f : scale, dv1 = p.S > 1 ? 1.f : div;
  const dim3 grid((unsigned)p.gx, (unsigned)p.S, (unsigned)images);
  if (p.vec) launch(csum_nhwc_kernel<4>, grid, 256, 0, s, x, pixels, c, p.CL, p.per, sc1, dv1, part);
  else launch(csum_nhwc_kernel<1>, grid, 256, 0, s, x, pixels, c, p.CL, p.per, sc1, dv1, part);
  int r = check_launch("channel_sum_nhwc");
  if (r || p.S == 1) return r;
  launch(csum_nhwc_fin_kernel, dim3((unsigned)cdiv(c, 32), (unsigned)images), 512, 0, s, part, c, (int)p.S, scale, div, out);
  return check_launch("channel_sum_nhwc_fin");
}

}  // namespace omt

using namespace omt;

extern "C" int omt_conv_bias_grad(const OmtAct* gy, int32_t n, int32_t c, int32_t h, int32_t w, float* db, float scale,
                                  omt_stream_t stream) {
  OMT_REQUIRE(gy && gy->p && db && n > 0 && c > 0 && h > 0 && w > 0, "omt_conv_bias_grad: bad arguments");
  cudaStream_t s = st(stream);
  if (is_nhwc(gy, c, h, w) && c > 1) return csum_nhwc(gy->p, 1, (int64_t)n * h * w, c, scale, 1.f, db, stream);
  const int S = (int)std::min<int64_t>(n, std::max<int64_t>(1, (4 * sm_count()) / c));
  Scratch sc;
  int r = sc.get(nullptr, 0, (size_t)c * S * sizeof(float), stream);
  if (r) return r;
  float* part = (float*)sc.p;
  launch(csum_part_kernel, dim3(c, S), 256, 0, s, view(gy), n, c, h, w, S, part);
  r = check_launch("bias_grad_part");
  if (r) return r;
  launch(csum_fin_kernel, (unsigned)cdiv(c, 128), 128, 0, s, part, c, S, scale, db);
  return check_launch("bias_grad_fin");
}

extern "C" int omt_channel_sum(const float* x, int32_t images, int64_t pixels, int32_t c, int32_t mean, float* out, omt_stream_t stream) {
  OMT_REQUIRE(x && out && images > 0 && images <= 65535 && pixels > 0 && c > 0, "omt_channel_sum: bad arguments");
  return csum_nhwc(x, images, pixels, c, 1.f, mean ? (float)pixels : 1.f, out, stream);
}

// Against ATen's reduction and the adaptive pooling kernel, warm and with L2 flushed, over 1 to 60 000 images of 4 to 10^6 pixels: faster (by 12 to 70 %) as
// long as one wave of blocks covers the call and a lane has little to add up one after the other. More blocks than that have too little
// to read each (60 000 x 16 x 3 x 3 8.5 -> 183 us, 256 x 2048 x 7 x 7 17.8 -> 27, a 16 x 10^6 matrix 10.6 -> 24.6), and slices of single-float loads
// keep too few bytes in flight from HBM (50 000 x 257 33 -> 48 with L2 flushed).
extern "C" int omt_channel_sum_pays(const float* x, int32_t images, int64_t pixels, int32_t c) {
  if (!x || images <= 0 || images > 65535 || pixels <= 0 || c <= 0) return 0;
  const CsumPlan p = plan_csum(x, images, pixels, c);
  return p.gx * p.S * images <= 4 * sm_count() && p.per <= 32 * (256 / p.CL) && (p.vec || p.S == 1);
}
