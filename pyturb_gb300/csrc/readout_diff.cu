// Differentiable multi-layer readout: a forward gather and its two adjoints.
//
// Layer screens phi (B, L, S, S) are sampled at the pupil grid of each
// direction and frame and summed with per-layer weights:
//   out[b,t,d,i,j] = sum_l w_l * bilerp(phi[b,l], u_r(i), u_c(j)),
//   u_r(i) = pos0[t,d,l,0] + mag[d,l] * i,   u_c(j) = pos0[t,d,l,1] + mag[d,l] * j,
// with periodic wrap on the S x S screen. This is the cone zoom of
// Atmosphere._build_lgs_zoom / _lgs_zoom (src/pyturb/atmosphere.py:581-616,
// 1048-1090: pupil scaled about the screen centre by mag = 1 - h/H) with the
// frozen-flow + direction displacement of _integrate_lgs (atmosphere.py:
// 1012-1022) applied as a sub-pixel bilinear shift instead of a phase ramp.
//
// Positions are 32.32 fixed point (k_lr_fix), reduced modulo S, so all three
// kernels form bit-identical taps. The adjoints are deterministic: the
// parameter gradients are block reductions written per (band, image), and the
// screen gradient is a gather in which each warp owns one screen tile and walks
// every (frame, direction) in a fixed order, using the separability of the
// axis-aligned bilinear map (columns, then rows).

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "common.cuh"

namespace pt {
uint64_t* launch_counter();
static inline void count_launch_r(int k = 1) {
  __atomic_add_fetch(launch_counter(), (uint64_t)k, __ATOMIC_RELAXED);
}

constexpr int kLrMaxLayers = 32;
constexpr int kLrMaxMag = 256;   // D * L entries of the magnification table
constexpr int kLrBand = 64;      // pupil rows per CTA (forward, parameter gradients)
constexpr int kLrTogether = 10;  // layers of a forward launch
constexpr long long kLrOne = 1ll << 32;

struct LrMag {
  double m[kLrMaxMag];
};

// fix[(t*D + d)*L + l] = {p0r, p0c, m}: positions of pupil pixel (0, 0)
// reduced into [0, S) and the per-pixel step, in units of 2^-32 px.
__global__ void k_lr_fix(int T, int D, int L, int S, const double* __restrict__ pos0, LrMag mag,
                         long long* __restrict__ fix) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= T * D * L) return;
  const int l = k % L, d = (k / L) % D;
  const long long span = (long long)S * kLrOne;
  long long out[2];
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    const double p = pos0[2 * k + a];
    const double x = p - floor(p / S) * (double)S;
    long long v = llrint(ldexp(x, 32));
    if (v < 0) v += span;
    if (v >= span) v -= span;
    out[a] = v;
  }
  fix[3 * k + 0] = out[0];
  fix[3 * k + 1] = out[1];
  fix[3 * k + 2] = llrint(ldexp(mag.m[d * L + l], 32));
}

// One axis tap: u = p0 + i*m (p0 in [0, S), m*(n-1) < S - 2, so u < 2S).
struct Tap {
  int a0, a1;
  float f;
};
__device__ __forceinline__ Tap lr_tap(long long p0, long long m, int i, int S) {
  const long long u = p0 + (long long)i * m;
  int i0 = (int)(u >> 32);
  if (i0 >= S) i0 -= S;
  Tap t;
  t.a0 = i0;
  t.a1 = (i0 + 1 == S) ? 0 : i0 + 1;
  t.f = (float)(uint32_t)(u & 0xffffffffll) * 2.3283064365386963e-10f;
  return t;
}

struct RowTab {
  int o0, o1;  // row offsets (row * S)
  float f;
};

// The sampling kernels address a float at a byte offset below 2^32 from a base
// that is the same for the whole CTA: one 32-bit add a load.
__device__ __forceinline__ float ld_at(const float* base, uint32_t byte_off) {
  return __ldg((const float*)((const char*)base + byte_off));
}

// Row tables of NL layers l0, l0 + 1, ... (clamped to L - 1) for a band of
// pupil rows: byte offsets of the upper and lower sample row from a realisation's
// first screen of the launch, and the fraction between them. Layers are adjacent, so
// a thread reads a row's entries with 16-byte loads.
template <int NL>
struct BandTab {
  static constexpr int NP = (NL + 3) & ~3;
  __align__(16) uint32_t up[kLrBand][NP], lo[kLrBand][NP];
  __align__(16) float f[kLrBand][NP];
};
template <int NL>
__device__ __forceinline__ void band_table(BandTab<NL>& tab, const long long* __restrict__ fx, int l0,
                                           int L, int S, int band0) {
  for (int k = threadIdx.x; k < BandTab<NL>::NP * kLrBand; k += blockDim.x) {
    const int q = k % BandTab<NL>::NP, r = k / BandTab<NL>::NP;
    const int l = min(l0 + min(q, NL - 1), L - 1);
    const Tap t = lr_tap(fx[3 * l], fx[3 * l + 2], band0 + r, S);
    tab.up[r][q] = 4u * ((uint32_t)l * S + t.a0) * S;
    tab.lo[r][q] = 4u * ((uint32_t)l * S + t.a1) * S;
    tab.f[r][q] = t.f;
  }
}
template <int NL, class V>
__device__ __forceinline__ void table_row(const V (&row)[BandTab<NL>::NP], V (&out)[NL]) {
#pragma unroll
  for (int q = 0; q < NL; q += 4) {
    const uint4 v = *(const uint4*)&row[q];
    const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (q + i < NL) memcpy(&out[q + i], &x[i], 4);
  }
}

// Whether layers l0 .. l0 + NL - 1 of an image all step one screen pixel per
// pupil pixel (a natural guide star).
template <int NL>
__device__ __forceinline__ bool all_unit(const long long* __restrict__ fx, int l0, int L) {
  bool unit = true;
  for (int q = 0; q < NL; ++q) unit = unit && fx[3 * min(l0 + q, L - 1) + 2] == kLrOne;
  return unit;
}

// Forward: CTA = (band of kLrBand pupil rows, t*D + d, b); threads walk
// columns, then the rows of the band, the NL layers of a pixel together. A launch
// takes at most kLrTogether of the L layers and as many as 32-bit byte offsets reach;
// screens, w and fix start at its first layer. A further launch (ADD) adds its layers
// to the output, which keeps the order of the sum: 16 layers in 8 + 8 took 76 us for
// 2 x 2 frames of 4 directions, 768^2 screens, 512^2 pupils, and 452 us in one form
// for up to 32 layers. (k_lr_forward_any takes the screens that pass 32 bits by
// themselves.)
//
// Bound by instruction issue and the L1 data path (scattered 4-byte taps; issue
// active 75%, L1 68%). Where every layer of the image has unit magnification
// the samples step one screen row per pupil row, so the lower row of one pixel
// is the upper row of the next: its horizontal interpolation stays in a
// register, a sample costs two loads instead of four, and the next row's taps
// are in flight while a row is summed. A layer count known at compile time and
// 32-bit offsets take the address and predicate instructions from 45 a sample
// to 16. 4 x 8 frames of 9 directions, 9 layers, 768^2 screens, 512^2 pupils:
// 1093 us with four loads and 64-bit offsets, 411 us so.
template <int NL, bool ADD>
__global__ void __launch_bounds__(256, NL <= 6 ? 3 : 2)
k_lr_forward(int L, int S, int T, int D, int n, const float* __restrict__ screens,
             const float* __restrict__ w, const long long* __restrict__ fix,
             float* __restrict__ out) {
  __shared__ BandTab<NL> tab;
  const int band0 = blockIdx.x * kLrBand;
  const int td = blockIdx.y, b = blockIdx.z;
  const int rows = min(kLrBand, n - band0);
  const long long* fx = fix + (size_t)td * L * 3;
  const bool unit = all_unit<NL>(fx, 0, NL);
  band_table<NL>(tab, fx, 0, NL, S, band0);
  __syncthreads();
  const float* scr = screens + (size_t)b * L * S * S;
  float* o = out + ((size_t)b * T * D + td) * n * n + (size_t)band0 * n;
  float wl[NL];
#pragma unroll
  for (int l = 0; l < NL; ++l) wl[l] = __ldg(w + l);
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    uint32_t c0[NL], c1[NL];
    float cf[NL];
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      const Tap c = lr_tap(fx[3 * l + 1], fx[3 * l + 2], j, S);
      c0[l] = 4u * c.a0;
      c1[l] = 4u * c.a1;
      cf[l] = c.f;
    }
    uint32_t ro[NL];
    float fr[NL];
    if (unit) {
      float top[NL], v0[NL], v1[NL];
      table_row<NL>(tab.up[0], ro);
      table_row<NL>(tab.f[0], fr);
#pragma unroll
      for (int l = 0; l < NL; ++l) {
        const float t0 = ld_at(scr, ro[l] + c0[l]);
        top[l] = fmaf(cf[l], ld_at(scr, ro[l] + c1[l]) - t0, t0);
      }
      table_row<NL>(tab.lo[0], ro);
#pragma unroll
      for (int l = 0; l < NL; ++l) {
        v0[l] = ld_at(scr, ro[l] + c0[l]);
        v1[l] = ld_at(scr, ro[l] + c1[l]);
      }
#pragma unroll 2
      for (int r = 0; r < rows; ++r) {
        float n0[NL], n1[NL];
        table_row<NL>(tab.lo[min(r + 1, rows - 1)], ro);
#pragma unroll
        for (int l = 0; l < NL; ++l) {
          n0[l] = ld_at(scr, ro[l] + c0[l]);
          n1[l] = ld_at(scr, ro[l] + c1[l]);
        }
        float acc = ADD ? o[(size_t)r * n + j] : 0.f;
#pragma unroll
        for (int l = 0; l < NL; ++l) {
          const float bot = fmaf(cf[l], v1[l] - v0[l], v0[l]);
          acc = fmaf(wl[l], fmaf(fr[l], bot - top[l], top[l]), acc);
          top[l] = bot;
          v0[l] = n0[l];
          v1[l] = n1[l];
        }
        o[(size_t)r * n + j] = acc;
      }
      continue;
    }
    for (int r = 0; r < rows; ++r) {
      uint32_t rl[NL];
      table_row<NL>(tab.up[r], ro);
      table_row<NL>(tab.lo[r], rl);
      table_row<NL>(tab.f[r], fr);
      float acc = ADD ? o[(size_t)r * n + j] : 0.f;
#pragma unroll
      for (int l = 0; l < NL; ++l) {
        const float v00 = ld_at(scr, ro[l] + c0[l]), v01 = ld_at(scr, ro[l] + c1[l]);
        const float v10 = ld_at(scr, rl[l] + c0[l]), v11 = ld_at(scr, rl[l] + c1[l]);
        const float top = fmaf(cf[l], v01 - v00, v00);
        const float bot = fmaf(cf[l], v11 - v10, v10);
        acc = fmaf(wl[l], fmaf(fr[l], bot - top, top), acc);
      }
      o[(size_t)r * n + j] = acc;
    }
  }
}

// nl <= LM layers of screens whose byte offsets pass 32 bits.
template <int LM>
__global__ void __launch_bounds__(256)
k_lr_forward_any(int L, int nl, int add, int S, int T, int D, int n, const float* __restrict__ screens,
                 const float* __restrict__ w, const long long* __restrict__ fix,
                 float* __restrict__ out) {
  __shared__ RowTab rt[LM][kLrBand];
  const int band0 = blockIdx.x * kLrBand;
  const int td = blockIdx.y, b = blockIdx.z;
  const int rows = min(kLrBand, n - band0);
  const long long* fx = fix + (size_t)td * L * 3;
  for (int k = threadIdx.x; k < nl * kLrBand; k += blockDim.x) {
    const int l = k / kLrBand, r = k % kLrBand;
    const Tap t = lr_tap(fx[3 * l], fx[3 * l + 2], band0 + r, S);
    rt[l][r] = RowTab{t.a0, t.a1, t.f};
  }
  __syncthreads();
  const float* scr = screens + (size_t)b * L * S * S;
  float* o = out + ((size_t)b * T * D + td) * n * n + (size_t)band0 * n;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    Tap c[LM];
#pragma unroll
    for (int l = 0; l < LM; ++l)
      if (l < nl) c[l] = lr_tap(fx[3 * l + 1], fx[3 * l + 2], j, S);
    for (int r = 0; r < rows; ++r) {
      float acc = add ? o[(size_t)r * n + j] : 0.f;
#pragma unroll
      for (int l = 0; l < LM; ++l) {
        if (l < nl) {
          const float* sl = scr + (size_t)l * S * S;
          const RowTab q = rt[l][r];
          const float* s0 = sl + (size_t)q.o0 * S;
          const float* s1 = sl + (size_t)q.o1 * S;
          const float v00 = __ldg(s0 + c[l].a0), v01 = __ldg(s0 + c[l].a1);
          const float v10 = __ldg(s1 + c[l].a0), v11 = __ldg(s1 + c[l].a1);
          const float top = fmaf(c[l].f, v01 - v00, v00);
          const float bot = fmaf(c[l].f, v11 - v10, v10);
          acc = fmaf(__ldg(w + l), fmaf(q.f, bot - top, top), acc);
        }
      }
      o[(size_t)r * n + j] = acc;
    }
  }
}

// Parameter gradients: per (band, image) and layer, the sums over the band's
// pixels of g * val, g * w * d val / d u_r and g * w * d val / d u_c (the
// derivative of the bilinear cell the sample lies in). Layers go in groups of
// NL so that taps and accumulators stay in registers; the band of g is re-read
// from L2 once per group (NL = 5 takes the 9-layer profile in two; the last
// group repeats its last layer in its unused places and does not write them). A
// launch takes `count` of the L layers, screens, w, fix and partial starting at its
// first: all of them, but for stacks that pass 32-bit byte offsets.
// Bounds and row reuse as in the forward: at unit magnification the
// interpolated value and the column difference of a sample's lower row serve
// the next pixel. The forward's workload: 1393 us before, 737 us so (issue
// active 63%, the rest load latency at two CTAs an SM).
constexpr int kLrGroupMax = 5;
template <int NL>
__global__ void __launch_bounds__(256, 2)
k_lr_grad_params(int L, int count, int S, int T, int D, int n, const float* __restrict__ screens,
                 const float* __restrict__ w, const long long* __restrict__ fix,
                 const float* __restrict__ g, float* __restrict__ partial) {
  __shared__ BandTab<NL> tab;
  __shared__ float red[8][3 * NL];
  const int band0 = blockIdx.x * kLrBand;
  const int td = blockIdx.y, b = blockIdx.z;
  const int rows = min(kLrBand, n - band0);
  const long long* fx = fix + (size_t)td * L * 3;
  const float* scr = screens + (size_t)b * L * S * S;
  const float* gi = g + ((size_t)b * T * D + td) * n * n + (size_t)band0 * n;
  const int nb = gridDim.x;
  float* pp = partial + (((size_t)b * T * D + td) * nb + blockIdx.x) * L * 3;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int l0 = 0; l0 < count; l0 += NL) {
    const bool unit = all_unit<NL>(fx, l0, count);
    band_table<NL>(tab, fx, l0, count, S, band0);
    __syncthreads();
    float sv[NL], sr[NL], sc[NL];
#pragma unroll
    for (int q = 0; q < NL; ++q) sv[q] = sr[q] = sc[q] = 0.f;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
      uint32_t c0[NL], c1[NL], ro[NL];
      float cf[NL], fr[NL];
#pragma unroll
      for (int q = 0; q < NL; ++q) {
        const int l = min(l0 + q, count - 1);
        const Tap c = lr_tap(fx[3 * l + 1], fx[3 * l + 2], j, S);
        c0[q] = 4u * c.a0;
        c1[q] = 4u * c.a1;
        cf[q] = c.f;
      }
      if (unit) {
        float top[NL], dtop[NL], v0[NL], v1[NL];
        table_row<NL>(tab.up[0], ro);
        table_row<NL>(tab.f[0], fr);
#pragma unroll
        for (int q = 0; q < NL; ++q) {
          const float t0 = ld_at(scr, ro[q] + c0[q]);
          dtop[q] = ld_at(scr, ro[q] + c1[q]) - t0;
          top[q] = fmaf(cf[q], dtop[q], t0);
        }
        table_row<NL>(tab.lo[0], ro);
#pragma unroll
        for (int q = 0; q < NL; ++q) {
          v0[q] = ld_at(scr, ro[q] + c0[q]);
          v1[q] = ld_at(scr, ro[q] + c1[q]);
        }
        float gv = gi[j];
#pragma unroll 2
        for (int r = 0; r < rows; ++r) {
          const int rn = min(r + 1, rows - 1);
          float n0[NL], n1[NL];
          const float gn = gi[(size_t)rn * n + j];
          table_row<NL>(tab.lo[rn], ro);
#pragma unroll
          for (int q = 0; q < NL; ++q) {
            n0[q] = ld_at(scr, ro[q] + c0[q]);
            n1[q] = ld_at(scr, ro[q] + c1[q]);
          }
#pragma unroll
          for (int q = 0; q < NL; ++q) {
            const float dbot = v1[q] - v0[q];
            const float bot = fmaf(cf[q], dbot, v0[q]);
            const float rise = bot - top[q];
            sv[q] = fmaf(gv, fmaf(fr[q], rise, top[q]), sv[q]);
            sr[q] = fmaf(gv, rise, sr[q]);
            sc[q] = fmaf(gv, fmaf(fr[q], dbot - dtop[q], dtop[q]), sc[q]);
            top[q] = bot;
            dtop[q] = dbot;
            v0[q] = n0[q];
            v1[q] = n1[q];
          }
          gv = gn;
        }
        continue;
      }
      for (int r = 0; r < rows; ++r) {
        uint32_t rl[NL];
        table_row<NL>(tab.up[r], ro);
        table_row<NL>(tab.lo[r], rl);
        table_row<NL>(tab.f[r], fr);
        const float gv = gi[(size_t)r * n + j];
#pragma unroll
        for (int q = 0; q < NL; ++q) {
          const float v00 = ld_at(scr, ro[q] + c0[q]), v01 = ld_at(scr, ro[q] + c1[q]);
          const float v10 = ld_at(scr, rl[q] + c0[q]), v11 = ld_at(scr, rl[q] + c1[q]);
          const float dtop = v01 - v00, dbot = v11 - v10;
          const float top = fmaf(cf[q], dtop, v00);
          const float bot = fmaf(cf[q], dbot, v10);
          sv[q] = fmaf(gv, fmaf(fr[q], bot - top, top), sv[q]);
          sr[q] = fmaf(gv, bot - top, sr[q]);
          sc[q] = fmaf(gv, fmaf(fr[q], dbot - dtop, dtop), sc[q]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < NL; ++q) {
      float a = sv[q], r = sr[q], c = sc[q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        r += __shfl_xor_sync(0xffffffffu, r, o);
        c += __shfl_xor_sync(0xffffffffu, c, o);
      }
      if (lane == 0) {
        red[warp][3 * q] = a;
        red[warp][3 * q + 1] = r;
        red[warp][3 * q + 2] = c;
      }
    }
    __syncthreads();
    if (threadIdx.x < 3 * NL) {
      const int k = threadIdx.x, l = l0 + k / 3;
      if (l < count) {
        float s = 0.f;
        for (int q = 0; q < 8; ++q) s += red[q][k];
        pp[3 * l + k % 3] = (k % 3 == 0) ? s : s * w[l];
      }
    }
    __syncthreads();
  }
}

// The same sums, one layer at a time, for screens whose byte offsets pass 32 bits.
__global__ void __launch_bounds__(256)
k_lr_grad_params_any(int L, int S, int T, int D, int n, const float* __restrict__ screens,
                     const float* __restrict__ w, const long long* __restrict__ fix,
                     const float* __restrict__ g, float* __restrict__ partial) {
  __shared__ float red[8][3];
  const int band0 = blockIdx.x * kLrBand;
  const int td = blockIdx.y, b = blockIdx.z;
  const int rows = min(kLrBand, n - band0);
  const float* gi = g + ((size_t)b * T * D + td) * n * n + (size_t)band0 * n;
  float* pp = partial + (((size_t)b * T * D + td) * gridDim.x + blockIdx.x) * L * 3;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int l = 0; l < L; ++l) {
    const long long* fx = fix + ((size_t)td * L + l) * 3;
    const float* sl = screens + ((size_t)b * L + l) * S * S;
    float s[3] = {0.f, 0.f, 0.f};
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
      const Tap c = lr_tap(fx[1], fx[2], j, S);
      for (int r = 0; r < rows; ++r) {
        const Tap t = lr_tap(fx[0], fx[2], band0 + r, S);
        const float gv = gi[(size_t)r * n + j];
        const float* s0 = sl + (size_t)t.a0 * S;
        const float* s1 = sl + (size_t)t.a1 * S;
        const float v00 = __ldg(s0 + c.a0), v10 = __ldg(s1 + c.a0);
        const float dtop = __ldg(s0 + c.a1) - v00, dbot = __ldg(s1 + c.a1) - v10;
        const float top = fmaf(c.f, dtop, v00);
        const float bot = fmaf(c.f, dbot, v10);
        s[0] = fmaf(gv, fmaf(t.f, bot - top, top), s[0]);
        s[1] = fmaf(gv, bot - top, s[1]);
        s[2] = fmaf(gv, fmaf(t.f, dbot - dtop, dtop), s[2]);
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
      if (lane == 0) red[warp][k] = s[k];
    }
    __syncthreads();
    if (threadIdx.x < 3) {
      float v = 0.f;
      for (int q = 0; q < 8; ++q) v += red[q][threadIdx.x];
      pp[3 * l + threadIdx.x] = threadIdx.x == 0 ? v : v * w[l];
    }
    __syncthreads();
  }
}

// First pupil index x with p0 + x*m > a (m > 0): a float estimate (|x| < 2^17,
// so off by less than one) corrected with exact 64-bit products, so the result
// equals the integer floor form. FP32 keeps it off the slow FP64 pipe.
__device__ __forceinline__ long long first_above(long long a, long long p0, long long m,
                                                 float inv_m) {
  long long x = (long long)floorf((float)(a - p0) * inv_m) + 1;
  if (p0 + (x - 1) * m > a) --x;
  if (p0 + x * m <= a) ++x;
  return x;
}

// Screen gradient, the transpose of the bilinear gather as a gather: a warp
// owns a block of screen pixels of one (layer, b), walks the (t, d) in a fixed
// order and adds what the pupil samples near each pixel give,
//   grad[r][c] = sum_td sum_y (row weight) sum_x (column weight) g[y][x],
// in registers; each pixel is written once (times w_l, or added). A lane holds
// columns lane and lane + 32, so a warp's loads are contiguous stretches of a
// pupil row; no shared memory and no barriers. Two kernels share the (t, d):
// k_lr_grad_unit takes those where the layer has unit magnification (a natural
// guide star), k_lr_grad_cone the others.
//
// Every layer maps the same pupil pixels onto other screen pixels, so each
// reads the gradient stack again, from L2 (reading an image once would mean
// scattering it with atomics); the bound is instruction issue. 4 x 8 frames of
// 8 stars and a laser star, 9 layers, 768^2 screens, 512^2 pupils: 2704 us
// with tiles staged in shared memory and general weights for every star,
// 515 + 339 us so. Rows a warp, measured on that workload: 16 rows 515 us,
// 32 rows 547 us (spills) at unit magnification; 8 rows 376 us, 16 rows 388 us and
// 32 rows 562 us on the cone with each tap at its own address (one address a
// column took the 8-row form to 339 us).
constexpr int kGsCols = 64;       // screen columns a warp owns (two a lane)
constexpr int kGsWarps = 4;       // warps a CTA, one below the other
constexpr int kUnitRows = 16;     // screen rows a warp owns
constexpr int kConeRows = 8;

// Block (rows x kGsCols) of this warp, or false below the screen.
struct GsTile {
  int R0, C0, lane;
};
template <int ROWS>
__device__ __forceinline__ bool gs_tile(int S, int tiles_c, GsTile& t) {
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  t.lane = threadIdx.x & 31;
  t.R0 = ((int)(blockIdx.x / tiles_c) * kGsWarps + warp) * ROWS;
  t.C0 = (int)(blockIdx.x % tiles_c) * kGsCols;
  return t.R0 < S;
}
template <int ROWS>
__device__ __forceinline__ void gs_store(const float (&acc)[2][ROWS], const GsTile& t, int S,
                                         float wl, int accumulate, float* __restrict__ gl) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = t.C0 + t.lane + 32 * h;
    if (c >= S) continue;
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      if (t.R0 + j >= S) break;
      float* o = gl + (size_t)(t.R0 + j) * S + c;
      *o = accumulate ? *o + wl * acc[h][j] : wl * acc[h][j];
    }
  }
}

// Unit magnification: the weights are the same for every pixel and the samples
// of a screen row are one pupil row, so a pixel costs two loads and four
// multiply-adds, the row above kept in registers. A lane whose column meets
// the pupil's first or last column keeps both its addresses inside and moves
// the weight; rows outside are skipped (n >= 2).
__global__ void __launch_bounds__(32 * kGsWarps, 6)
k_lr_grad_unit(int L, int S, int T, int D, int n, int tiles_c, const float* __restrict__ w,
               const long long* __restrict__ fix, const float* __restrict__ g, int accumulate,
               float* __restrict__ grad) {
  GsTile t;
  if (!gs_tile<kUnitRows>(S, tiles_c, t)) return;
  const int l = blockIdx.y, b = blockIdx.z;
  float acc[2][kUnitRows];
#pragma unroll
  for (int j = 0; j < kUnitRows; ++j) acc[0][j] = acc[1][j] = 0.f;
  for (int td = 0; td < T * D; ++td) {
    const long long* fx = fix + ((size_t)td * L + l) * 3;
    if (fx[2] != kLrOne) continue;
    const float* gi = g + ((size_t)b * T * D + td) * n * n;
    const long long p0r = fx[0], p0c = fx[1];
    const int ir = (int)(p0r >> 32), ic = (int)(p0c >> 32);
    const float fr = (float)(uint32_t)(p0r & 0xffffffffll) * 2.3283064365386963e-10f;
    const float fc = (float)(uint32_t)(p0c & 0xffffffffll) * 2.3283064365386963e-10f;
    const float gr = 1.f - fr;
    // the two wrap images of the block along each axis; a pupil smaller than
    // the screen by two rows meets a block in at most these
    for (int k = 0; k < 4; ++k) {
      const int y0 = t.R0 - ir + (k >> 1) * S;  // pupil row whose upper tap is screen row R0
      const int x0 = t.C0 - ic + (k & 1) * S;
      if (y0 + kUnitRows <= 0 || y0 > n || x0 + kGsCols <= 0 || x0 > n) continue;
      const float* p[2];
      float wa[2], wb[2];  // weights of p[.][0] and p[.][-1]
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int x = x0 + t.lane + 32 * h;
        wa[h] = x == n ? fc : 1.f - fc;
        wb[h] = x == 0 ? 1.f - fc : fc;
        if (x <= 0 || x > n) wa[h] = 0.f;
        if (x < 0 || x >= n) wb[h] = 0.f;
        p[h] = gi + ((long long)(y0 - 1) * n + min(max(x, 1), n - 1));
      }
      if (y0 >= 1 && y0 + kUnitRows <= n) {
        float h0 = fmaf(wa[0], __ldg(p[0]), wb[0] * __ldg(p[0] - 1));
        float h1 = fmaf(wa[1], __ldg(p[1]), wb[1] * __ldg(p[1] - 1));
#pragma unroll
        for (int j = 0; j < kUnitRows; ++j) {
          p[0] += n;
          p[1] += n;
          const float v0 = fmaf(wa[0], __ldg(p[0]), wb[0] * __ldg(p[0] - 1));
          const float v1 = fmaf(wa[1], __ldg(p[1]), wb[1] * __ldg(p[1] - 1));
          acc[0][j] = fmaf(gr, v0, fmaf(fr, h0, acc[0][j]));
          acc[1][j] = fmaf(gr, v1, fmaf(fr, h1, acc[1][j]));
          h0 = v0;
          h1 = v1;
        }
      } else {
        float h0 = 0.f, h1 = 0.f;
#pragma unroll
        for (int j = -1; j < kUnitRows; ++j) {
          float v0 = 0.f, v1 = 0.f;
          if ((unsigned)(y0 + j) < (unsigned)n) {
            v0 = fmaf(wa[0], __ldg(p[0]), wb[0] * __ldg(p[0] - 1));
            v1 = fmaf(wa[1], __ldg(p[1]), wb[1] * __ldg(p[1] - 1));
          }
          p[0] += n;
          p[1] += n;
          if (j >= 0) {
            acc[0][j < 0 ? 0 : j] = fmaf(gr, v0, fmaf(fr, h0, acc[0][j < 0 ? 0 : j]));
            acc[1][j < 0 ? 0 : j] = fmaf(gr, v1, fmaf(fr, h1, acc[1][j < 0 ? 0 : j]));
          }
          h0 = v0;
          h1 = v1;
        }
      }
    }
  }
  gs_store<kUnitRows>(acc, t, S, w[l], accumulate, grad + ((size_t)b * L + l) * S * S);
}

// Any magnification: the pupil rows that end in screen row r are walked in
// turn (their count depends only on the row, so the warp does not diverge);
// KM = ceil(2 / mag) bounds the samples whose footprint covers one pixel along
// an axis; a pupil of fewer has SMALL. Entries of unit magnification are left to
// k_lr_grad_unit with `skip_unit`.
template <int KM, bool SMALL>
__global__ void __launch_bounds__(32 * kGsWarps, KM <= 4 ? 7 : 4)
k_lr_grad_cone(int L, int S, int T, int D, int n, int tiles_c, int skip_unit,
               const float* __restrict__ w, const long long* __restrict__ fix,
               const float* __restrict__ g, int accumulate, float* __restrict__ grad) {
  GsTile t;
  if (!gs_tile<kConeRows>(S, tiles_c, t)) return;
  const int l = blockIdx.y, b = blockIdx.z;
  const long long span = (long long)S * kLrOne;
  float acc[2][kConeRows];
#pragma unroll
  for (int j = 0; j < kConeRows; ++j) acc[0][j] = acc[1][j] = 0.f;
  bool any = false;
  for (int td = 0; td < T * D; ++td) {
    const long long* fx = fix + ((size_t)td * L + l) * 3;
    const long long p0r = fx[0], p0c = fx[1], m = fx[2];
    if (skip_unit && m == kLrOne) continue;
    any = true;
    const float* gi = g + ((size_t)b * T * D + td) * n * n;
    const float inv_m = 1.0f / (float)m;
    const long long ur1 = p0r + (long long)(n - 1) * m, uc1 = p0c + (long long)(n - 1) * m;
    for (int img = 0; img < 4; ++img) {
      const int kr = img >> 1, kc = img & 1;
      // samples reaching rows [R0, R0 + kConeRows): u_r in the open window + kr S
      const long long wr0 = (long long)(t.R0 - 1) * kLrOne + kr * span;
      const long long wr1 = (long long)(t.R0 + kConeRows) * kLrOne + kr * span;
      const long long wc0 = (long long)(t.C0 - 1) * kLrOne + kc * span;
      const long long wc1 = (long long)(t.C0 + kGsCols) * kLrOne + kc * span;
      if (!(wr0 < ur1 && wr1 > p0r && wc0 < uc1 && wc1 > p0c)) continue;
      int y = (int)max(0ll, first_above(wr0, p0r, m, inv_m));
      // each column's KM consecutive samples, moved inside the pupil row; the
      // weight of a sample that does not reach the column is zero
      float cw[2][KM];
      const float* p[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const long long pf = (long long)(t.C0 + t.lane + 32 * h) * kLrOne + kc * span;
        const long long xa = first_above(pf - kLrOne, p0c, m, inv_m);
        const int xb = (int)max(0ll, min(xa, (long long)(n - KM)));
#pragma unroll
        for (int k = 0; k < KM; ++k) {
          const long long dl = p0c + (long long)(xb + k) * m - pf;
          const long long ad = dl < 0 ? -dl : dl;
          cw[h][k] = ad < kLrOne && (!SMALL || k < n) ? 1.f - (float)ad * 2.3283064365386963e-10f : 0.f;
        }
        p[h] = gi + ((size_t)y * n + xb);
      }
      long long u = p0r + (long long)y * m - kr * span;  // row position of sample row y
      float a0[2] = {0.f, 0.f}, a1[2] = {0.f, 0.f};      // what rows r and r + 1 get
#pragma unroll
      for (int j = -1; j < kConeRows; ++j) {
        while (y < n && (int)(u >> 32) == t.R0 + j) {
          const float f = (float)(uint32_t)(u & 0xffffffffll) * 2.3283064365386963e-10f;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float v = 0.f;
#pragma unroll
            for (int k = 0; k < KM; ++k) v = fmaf(cw[h][k], __ldg(p[h] + (SMALL ? min(k, n - 1) : k)), v);
            a0[h] = fmaf(1.f - f, v, a0[h]);
            a1[h] = fmaf(f, v, a1[h]);
            p[h] += n;
          }
          ++y;
          u += m;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (j >= 0) acc[h][j < 0 ? 0 : j] += a0[h];
          a0[h] = a1[h];
          a1[h] = 0.f;
        }
      }
    }
  }
  if (accumulate && !any) return;  // nothing to add
  gs_store<kConeRows>(acc, t, S, w[l], accumulate, grad + ((size_t)b * L + l) * S * S);
}

// ----------------------------------------------------------------- host side
static int lr_check(const char* who, int B, int L, int S, int T, int D, int n, const double* mag) {
  if (B < 1 || L < 1 || S < 2 || T < 1 || D < 1 || n < 1)
    return fail(PT_ERR_ARG, std::string(who) + ": bad sizes");
  if (L > kLrMaxLayers) return fail(PT_ERR_UNSUPPORTED, std::string(who) + ": at most 32 layers");
  if (D * L > kLrMaxMag)
    return fail(PT_ERR_UNSUPPORTED, std::string(who) + ": at most 256 direction-layer pairs");
  if (S > (1 << 20) || n > (1 << 16))
    return fail(PT_ERR_UNSUPPORTED, std::string(who) + ": screen or pupil too large");
  if (!mag) return fail(PT_ERR_ARG, std::string(who) + ": NULL magnification table");
  for (int k = 0; k < D * L; ++k) {
    const double m = mag[k];
    if (!(m >= 0.25 && m <= 4.0))
      return fail(PT_ERR_ARG, std::string(who) + ": magnification must lie in [0.25, 4]");
    if (!(m * (n - 1) + 2.0 < S))
      return fail(PT_ERR_ARG, std::string(who) + ": the pupil footprint must be smaller than the screen");
  }
  return PT_OK;
}

// L screens lie within 32-bit byte offsets of the first one's base.
static bool small_offsets(int L, int S) { return 4.0 * L * S * S < 4294967296.0; }

}  // namespace pt

using namespace pt;

extern "C" int pt_lr_fix(int T, int D, int L, int S, int n, const double* pos0, const double* mag,
                         int64_t* fix, void* stream) {
  if (int rc = lr_check("pt_lr_fix", 1, L, S, T, D, n, mag)) return rc;
  if (!pos0 || !fix) return fail(PT_ERR_ARG, "pt_lr_fix: NULL pointer");
  LrMag M{};
  for (int k = 0; k < D * L; ++k) M.m[k] = mag[k];
  cudaStream_t s = (cudaStream_t)stream;
  const int cnt = T * D * L;
  k_lr_fix<<<(cnt + 255) / 256, 256, 0, s>>>(T, D, L, S, pos0, M, (long long*)fix);
  count_launch_r();
  return check_launch("pt_lr_fix");
}

extern "C" int pt_lr_forward(int B, int L, int S, int T, int D, int n, const double* mag,
                             const float* screens, const float* weights, const int64_t* fix,
                             float* out, void* stream) {
  if (int rc = lr_check("pt_lr_forward", B, L, S, T, D, n, mag)) return rc;
  if (!screens || !weights || !fix || !out) return fail(PT_ERR_ARG, "pt_lr_forward: NULL pointer");
  if ((long long)T * D > 65535 || B > 65535)
    return fail(PT_ERR_UNSUPPORTED, "pt_lr_forward: T*D and B must be <= 65535");
  cudaStream_t s = (cudaStream_t)stream;
  dim3 grid((n + kLrBand - 1) / kLrBand, T * D, B);
  const long long* fx = (const long long*)fix;
  ProfScope ps("k_lr_forward", s);
  // equal groups of the layers that one launch takes together
  const bool wide = !small_offsets(1, S);
  int most = wide ? 8 : kLrTogether;
  while (!wide && !small_offsets(most, S)) --most;
  for (int l0 = 0, left = (L + most - 1) / most; left > 0; --left) {
    const int nl = (L - l0 + left - 1) / left;
    const float *scr = screens + (size_t)l0 * S * S, *w = weights + l0;
    auto go = [&](auto first, auto add) {
      (l0 ? add : first)<<<grid, 256, 0, s>>>(L, S, T, D, n, scr, w, fx + 3 * l0, out);
    };
    switch (wide ? 0 : nl) {
      case 0: {
        auto kern = nl <= 4 ? k_lr_forward_any<4> : k_lr_forward_any<8>;
        kern<<<grid, 256, 0, s>>>(L, nl, l0 > 0, S, T, D, n, scr, w, fx + 3 * l0, out);
        break;
      }
#define PT_CASE(k) case k: go(k_lr_forward<k, false>, k_lr_forward<k, true>); break;
      PT_CASE(1) PT_CASE(2) PT_CASE(3) PT_CASE(4) PT_CASE(5)
      PT_CASE(6) PT_CASE(7) PT_CASE(8) PT_CASE(9) PT_CASE(10)
#undef PT_CASE
    }
    count_launch_r();
    l0 += nl;
  }
  return check_launch("pt_lr_forward");
}

extern "C" int pt_lr_grad_params(int B, int L, int S, int T, int D, int n, const double* mag,
                                 const float* screens, const float* weights, const int64_t* fix,
                                 const float* grad_out, float* partial, void* stream) {
  if (int rc = lr_check("pt_lr_grad_params", B, L, S, T, D, n, mag)) return rc;
  if (!screens || !weights || !fix || !grad_out || !partial)
    return fail(PT_ERR_ARG, "pt_lr_grad_params: NULL pointer");
  if ((long long)T * D > 65535 || B > 65535)
    return fail(PT_ERR_UNSUPPORTED, "pt_lr_grad_params: T*D and B must be <= 65535");
  cudaStream_t s = (cudaStream_t)stream;
  dim3 grid((n + kLrBand - 1) / kLrBand, T * D, B);
  const long long* fx = (const long long*)fix;
  ProfScope ps("k_lr_grad_params", s);
  if (!small_offsets(1, S)) {
    k_lr_grad_params_any<<<grid, 256, 0, s>>>(L, S, T, D, n, screens, weights, fx, grad_out, partial);
    count_launch_r();
    return check_launch("pt_lr_grad_params");
  }
  // as many layers a launch as lie within 32-bit byte offsets, in equal groups of at
  // most kLrGroupMax
  int most = L;
  while (!small_offsets(most, S)) --most;
  for (int l0 = 0; l0 < L; l0 += most) {
    const int count = std::min(most, L - l0);
    auto go = [&](auto kern) {
      kern<<<grid, 256, 0, s>>>(L, count, S, T, D, n, screens + (size_t)l0 * S * S, weights + l0,
                                fx + 3 * l0, grad_out, partial + 3 * l0);
    };
    const int passes = (count + kLrGroupMax - 1) / kLrGroupMax, nl = (count + passes - 1) / passes;
    if (nl == 1) go(k_lr_grad_params<1>);
    else if (nl == 2) go(k_lr_grad_params<2>);
    else if (nl == 3) go(k_lr_grad_params<3>);
    else if (nl == 4) go(k_lr_grad_params<4>);
    else go(k_lr_grad_params<5>);
    count_launch_r();
  }
  return check_launch("pt_lr_grad_params");
}

extern "C" size_t pt_lr_partial_count(int B, int L, int T, int D, int n) {
  if (B < 1 || L < 1 || T < 1 || D < 1 || n < 1) return 0;
  return (size_t)B * T * D * ((n + kLrBand - 1) / kLrBand) * L * 3;
}

extern "C" int pt_lr_grad_screens(int B, int L, int S, int T, int D, int n, const double* mag,
                                  const float* weights, const int64_t* fix, const float* grad_out,
                                  int accumulate, float* grad_screens, void* stream) {
  if (int rc = lr_check("pt_lr_grad_screens", B, L, S, T, D, n, mag)) return rc;
  if (!weights || !fix || !grad_out || !grad_screens)
    return fail(PT_ERR_ARG, "pt_lr_grad_screens: NULL pointer");
  // which kernels have work: unit magnifications (exactly 1 in fixed point, and two
  // pixels of the pupil side by side), and the taps per screen pixel and axis of the
  // others, at most ceil(2 / mag)
  double mmin = 4.0;
  int unit = 0, cone = 0;
  for (int k = 0; k < D * L; ++k) {
    if (n > 1 && std::llrint(std::ldexp(mag[k], 32)) == kLrOne) {
      unit = 1;
    } else {
      cone = 1;
      mmin = std::min(mmin, mag[k]);
    }
  }
  const int km = (int)std::ceil(2.0 / mmin);
  if (km > 8) return fail(PT_ERR_UNSUPPORTED, "pt_lr_grad_screens: magnification too small");
  if (B > 65535) return fail(PT_ERR_UNSUPPORTED, "pt_lr_grad_screens: B must be <= 65535");
  cudaStream_t s = (cudaStream_t)stream;
  const int tiles_c = (S + kGsCols - 1) / kGsCols;
  auto tiles = [&](int rows) {
    return dim3(tiles_c * ((S + rows * kGsWarps - 1) / (rows * kGsWarps)), L, B);
  };
  const long long* fx = (const long long*)fix;
  ProfScope ps("k_lr_grad_screens", s);
  if (unit) {
    k_lr_grad_unit<<<tiles(kUnitRows), 32 * kGsWarps, 0, s>>>(
        L, S, T, D, n, tiles_c, weights, fx, grad_out, accumulate, grad_screens);
    accumulate = 1;
  }
  if (cone) {
    auto go = [&](auto kern) {
      kern<<<tiles(kConeRows), 32 * kGsWarps, 0, s>>>(L, S, T, D, n, tiles_c, unit, weights, fx,
                                                      grad_out, accumulate, grad_screens);
    };
#define PT_CASE(K) go(n < K ? k_lr_grad_cone<K, true> : k_lr_grad_cone<K, false>)
    if (km <= 2) PT_CASE(2);
    else if (km <= 3) PT_CASE(3);
    else if (km <= 4) PT_CASE(4);
    else PT_CASE(8);
#undef PT_CASE
    count_launch_r(unit);
  }
  count_launch_r();
  return check_launch("pt_lr_grad_screens");
}
