// Register-resident Bluestein transforms (fft_bluestein of fft.cuh on the
// register FFT of fft_reg.cuh), included by spectral.cu inside namespace pt after
// the power-of-two fast path: lengths n with a prime factor above 61 whose padded
// length M, the power of two >= 2n - 1, is 256 .. 4096. A team of M / 8 threads
// holds the padded vector eight elements a thread; n <= M / 2, so the upper four
// start at zero (the first butterflies drop them) and only the lower four of the
// result are kept. Both length-M transforms, the product with the chirp's
// spectrum between them and the chirp products around them stay in registers; a
// row CTA walks several rows so that its twiddle staging serves all of them. Eight
// transforms of 586^2 (M = 2048), screens of 8 levels: rows 223 us and columns
// 256 us on the shared-memory stages, 66 us and 103 us so (instruction issue).
#pragma once

template <int M>
struct BluCfg {
  static constexpr int T = M / 8;
  static constexpr int NV = T >= 256 ? 1 : 256 / T;         // teams of a row CTA
  static constexpr int THREADS = NV * T;
  static constexpr int RPT = 4;                             // rows a team walks
  static constexpr int C = M >= 4096 ? 2 : (M == 2048 ? 4 : (M == 1024 ? 8 : 16));
  static constexpr int COL_THREADS = C * T;
  static constexpr bool SWAP = (Pow2Plan<M>::stages - 1) % 2 == 1;  // odd exchange count
};
static bool blu_fast(const FftDesc& d) { return d.M >= 256 && d.M <= 4096; }

// The length-n transform of the team's vector: x[i], i < 4, element j + T i of the
// input (zero at n and beyond) and of the output; a and b as in reg_fft_db, free
// again in the same order after the call.
template <int M, class Lay, class Sync>
__device__ __forceinline__ void reg_bluestein(float2 (&x)[8], int j, const FftDesc& d,
                                              const float2* stw, const Lay& a, const Lay& b,
                                              const Sync& sync) {
  constexpr int T = M / 8;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int e = j + T * i;
    x[i] = e < d.n ? cmul(x[i], __ldg(d.chirp + e)) : make_float2(0.f, 0.f);
    x[i + 4] = make_float2(0.f, 0.f);
  }
  reg_fft_db<M>(x, j, stw, a, b, sync);
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = cconj(cmul(x[i], __ldg(d.bhat + j + T * i)));
  // the first exchange of this transform must not meet the last of the one above
  if constexpr (BluCfg<M>::SWAP) reg_fft_db<M>(x, j, stw, b, a, sync);
  else reg_fft_db<M>(x, j, stw, a, b, sync);
  const float inv = 1.0f / (float)M;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int e = j + T * i;
    if (e < d.n) x[i] = cscale(cmul(__ldg(d.chirp + e), cconj(x[i])), inv);
  }
}

// Rows: plain complex input (in may be work itself: a team reads its row before
// it writes it) or generate's coloured noise, as k_rows.
template <int M>
__global__ void __launch_bounds__(BluCfg<M>::THREADS)
k_rows_blu(FftDesc d, const float2* in, int gen, GenRowArgs ga, float2* work) {
  using Cfg = BluCfg<M>;
  constexpr int T = Cfg::T, NV = Cfg::NV;
  extern __shared__ float2 sm[];
  float2* stw = sm;
  const int n = d.n, v = threadIdx.x / T, j = threadIdx.x % T;
  const RowLayout s{sm + M + v * fft_padded(M)}, s2{sm + M + (NV + v) * fft_padded(M)};
  asm volatile("griddepcontrol.launch_dependents;");
  load_stage_tw<M>(stw, d.twM);
  const int img = blockIdx.y;
  if (gen) gen_coef_pair(ga, img);
  __syncthreads();
  const TeamSync team{1 + v, T};
  for (int q = 0; q < Cfg::RPT; ++q) {
    const int kx = (blockIdx.x * Cfg::RPT + q) * NV + v;
    if (kx >= n) return;  // the whole team
    float2 x[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int ky = j + T * i;
      x[i] = make_float2(0.f, 0.f);
      if (ky >= n) continue;
      if (gen) {
        float2 z;
        if (ga.noise) {
          const size_t e = ((size_t)(ga.img0 + img) * n + kx) * n + ky, plane = (size_t)ga.n_fft * n * n;
          z = make_float2(ga.noise[e], ga.noise[plane + e]);
        } else {
          z = screen_normal(ga.seed, (uint64_t)(ga.img0 + img) * n + kx, ky, n, ga.call);
        }
        const float amp = __ldg(ga.amplitude + (size_t)kx * n + ky);
        x[i] = make_float2(z.x * amp, z.y * amp);
      } else {
        x[i] = in[((size_t)img * n + kx) * n + ky];
      }
    }
    reg_bluestein<M>(x, j, d, stw, s, s2, team);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int ky = j + T * i;
      if (ky < n) work[((size_t)img * n + kx) * n + ky] = x[i];
    }
  }
}

// Columns, plain complex output. (work is the row pass's result, written while
// this kernel's first CTAs may already run: not a pointer to promise constant.)
template <int M>
__global__ void __launch_bounds__(BluCfg<M>::COL_THREADS)
k_plain_cols_blu(FftDesc d, const float2* work, float2* __restrict__ out) {
  using Cfg = BluCfg<M>;
  constexpr int T = Cfg::T, C = Cfg::C;
  extern __shared__ float2 sm[];
  float2* stw = sm;
  const int n = d.n, c = threadIdx.x % C, j = threadIdx.x / C;
  const ColLayout<C> s{sm + M + c}, s2{sm + M + M * C + c};
  load_stage_tw<M>(stw, d.twM);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int y = blockIdx.x * C + c, img = blockIdx.y;
  float2 x[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = j + T * i;
    x[i] = r < n && y < n ? __ldcs(work + ((size_t)img * n + r) * n + y) : make_float2(0.f, 0.f);
  }
  __syncthreads();
  reg_bluestein<M>(x, j, d, stw, s, s2, CtaSync{});
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = j + T * i;
    if (r < n && y < n) out[((size_t)img * n + r) * n + y] = x[i];
  }
}

// Columns with the paired real epilogue of k_pair_cols_reg.
template <int M>
__global__ void __launch_bounds__(BluCfg<M>::COL_THREADS)
k_pair_cols_blu(FftDesc d, const float2* work, int pair0, PairStore st) {
  using Cfg = BluCfg<M>;
  constexpr int T = Cfg::T, C = Cfg::C;
  extern __shared__ float2 sm[];
  float2* stw = sm;
  float2* buf = sm + M;
  const int n = d.n, P = st.P;
  float2* mtab = buf + 2 * M * C;  // (2, 3P, C), then (P, C) float4
  const int c = threadIdx.x % C, j = threadIdx.x / C;
  const ColLayout<C> s{buf + c}, s2{buf + M * C + c};
  load_stage_tw<M>(stw, d.twM);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int y = blockIdx.x * C + c, pl = blockIdx.y, pair = pair0 + pl;
  const bool ok = y < n;
  const int img_re = pair * st.re_mul + st.re_add, img_im = pair * st.im_mul + st.im_add;
  const bool do_re = img_re < st.count, do_im = img_im < st.count;
  const int row_re = pl * st.crow_mul + st.crow_re, row_im = pl * st.crow_mul + st.crow_im;
  // m[o][p*3+i][c] = sum_j coef[o][p][i][j] basis[p][j][y]
  for (int i = threadIdx.x; i < 2 * 3 * P * C; i += Cfg::COL_THREADS) {
    const int cc = i % C, pi = (i / C) % (3 * P), o = i / (C * 3 * P);
    const int yy = blockIdx.x * C + cc;
    float2 m = make_float2(0.f, 0.f);
    if ((o == 0 ? do_re : do_im) && yy < n) {
      const float2* cf = st.coef + ((size_t)(o == 0 ? row_re : row_im) * P * 3 + pi) * 3;
#pragma unroll
      for (int q = 0; q < 3; ++q) m = cfma(cf[q], st.basis[((size_t)(pi / 3) * 3 + q) * n + yy], m);
    }
    mtab[i] = m;
  }
  float2 x[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = j + T * i;
    x[i] = ok && r < n ? __ldcs(work + ((size_t)pl * n + r) * n + y) : make_float2(0.f, 0.f);
  }
  __syncthreads();
  // symmetric bases: (U_re, W_re, U_im, W_im) of a level and column, and the
  // constant K of the column in registers
  float4* utab = (float4*)(mtab + 2 * 3 * P * C);
  float k0 = 0.f, k1 = 0.f;
  if (st.sym) {
    for (int p = 0; p < P; ++p) {
      k0 += mtab[(3 * p + 1) * C + c].x;
      k1 += mtab[(3 * P + 3 * p + 1) * C + c].x;
    }
    for (int i = threadIdx.x; i < P * C; i += Cfg::COL_THREADS) {
      const int p = i / C, cc = i % C;
      const float2 m00 = mtab[(3 * p) * C + cc], m02 = mtab[(3 * p + 2) * C + cc];
      const float2 m10 = mtab[(3 * P + 3 * p) * C + cc], m12 = mtab[(3 * P + 3 * p + 2) * C + cc];
      utab[i] = make_float4(m00.x + m02.x, m02.y - m00.y, m10.x + m12.x, m12.y - m10.y);
    }
  }
  if (P > 0 && do_re) k0 -= st.mean[row_re];
  if (P > 0 && do_im) k1 -= st.mean[row_im];
  reg_bluestein<M>(x, j, d, stw, s, s2, CtaSync{});  // its barriers order utab
  if (!ok) return;
  const int yo = y - st.crop;
  if (yo < 0 || yo >= st.n_out) return;
  // the low-order screens on their own, then added: one rounding at full scale
  float2 low[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) low[i] = make_float2(k0, k1);
  if (st.sym) {
    for (int p = 0; p < P; ++p) {
      const float4 u = utab[p * C + c];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 b = __ldg(st.basis + (size_t)(3 * p) * n + min(j + T * i, n - 1));
        low[i].x = fmaf(b.x, u.x, fmaf(b.y, u.y, low[i].x));
        low[i].y = fmaf(b.x, u.z, fmaf(b.y, u.w, low[i].y));
      }
    }
  } else {
    for (int pi = 0; pi < 3 * P; ++pi) {
      const float2 m0 = mtab[pi * C + c], m1 = mtab[(3 * P + pi) * C + c];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 b = __ldg(st.basis + (size_t)pi * n + min(j + T * i, n - 1));
        low[i].x = fmaf(b.x, m0.x, fmaf(-b.y, m0.y, low[i].x));
        low[i].y = fmaf(b.x, m1.x, fmaf(-b.y, m1.y, low[i].y));
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = cadd(x[i], low[i]);
  const size_t plane = (size_t)st.n_out * st.n_out;
  const float sre = img_scale_of(st, img_re), sim = img_scale_of(st, img_im);
  float* ore = st.out + (size_t)(do_re ? img_re : 0) * plane + yo;
  float* oim = st.out + (size_t)(do_im ? img_im : 0) * plane + yo;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = j + T * i, xo = r - st.crop;
    if (r >= n || xo < 0 || xo >= st.n_out) continue;
    const size_t o = (size_t)xo * st.n_out;
    if (st.accumulate) {
      if (do_re) ore[o] += sre * x[i].x;
      if (do_im) oim[o] += sim * x[i].y;
    } else {
      if (do_re) __stcs(ore + o, sre * x[i].x);
      if (do_im) __stcs(oim + o, sim * x[i].y);
    }
  }
}
