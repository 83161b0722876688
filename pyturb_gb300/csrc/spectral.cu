// Spectral synthesis on the GB300: PhaseScreen.generate, the frozen-flow
// frame readout of the spectral engine, per-layer LGS screens, the LGS cone
// zoom and spectral boiling.
//
// A 2-D inverse transform is two shared-memory passes:
//   pass 1 (rows, axis 1): a producer writes one complex row into shared
//     memory (coloured noise, or the phasor-weighted layer sum), the row is
//     transformed and written to the workspace;
//   pass 2 (columns, axis 0): tiles of C columns are transformed and the
//     epilogue writes the real/imaginary parts as two real screens with the
//     subharmonic low-frequency sum added, cropped and scaled.
// Two real outputs share one complex transform: generate() uses the
// reference's own Re/Im pairing, frames are paired through their
// Hermitian parts, H = (X(k) + conj X(-k)) / 2, so Re ifft2(X1) + i Re
// ifft2(X2) = ifft2(H1 + i H2).
#include <cuda.h>  // CUtensorMap (types only; the encoder comes from the runtime's entry point)
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "fft.cuh"
#include "fft_reg.cuh"

namespace pt {
uint64_t* launch_counter();
}

struct pt_grid {
  int ns;
  double dx;
  int P;
  pt::FftDesc desc;
  float2* tw;       // (ns) exp(+2 pi i k / ns)
  float2* basis;    // (P, 3, ns) exp(2 pi i f_p (x - ns/2) dx)
  double* sh_freq;  // (P, 3)
  double* beta;     // (P, 3, 2) grid mean of each basis row
  int sym;          // every level's frequencies are {-a, 0, +a}
  int cols_variant; // power-of-two column pass: 0 register-fed, 1 TMA-fed
  float2* blu;      // Bluestein tables of desc (chirp, bhat, twM), or NULL
};

namespace pt {

constexpr int kMaxLevels = 16;
constexpr int kThreads = 256;
constexpr int kColThreads = 512;  // shared-memory column passes
// Largest P * ns (float2) of first basis rows the column kernels stage in
// shared memory for the subharmonic epilogue.
constexpr int kColBasisMax = 4096;

static inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Number of complex ns x ns images one internal pass batches.
static inline int image_chunk(int ns) {
  size_t per = (size_t)ns * ns * sizeof(float2);
  size_t c = (size_t)(64u << 20) / per;
  return (int)std::max<size_t>(1, std::min<size_t>(32, c));
}
// Transforms per chunk of generate / ifft2: up to 256 as long as the row-pass
// intermediate of a chunk stays within 64 MB (L2-resident between the passes),
// so small screens run as a few large launches.
static inline int gen_chunk(int ns) {
  size_t per = (size_t)ns * ns * sizeof(float2);
  size_t c = (size_t)(64u << 20) / per;
  return (int)std::max<size_t>(1, std::min<size_t>(256, c));
}
// Rows / columns a CTA of the shared-memory passes transforms, from the buffer
// length (fft_buf_len: M for a Bluestein grid): about 4096 elements of columns, and
// of rows 3072 (more CTAs to fill the last wave; 4096 in brackets: 8 screens of
// 700^2 81 (83) us, 4 of 1000^2 91 (95) us, three images of 728^2 2 us more) or, of
// vectors below 320 elements, 2048 (3072 in brackets: 100 screens of 200^2 71 (73)
// us, 20 of 250^2 42 (44) us, but 64 of 280^2 89 (85) us). 2048 also below 350 CTAs
// of 3072 (9% faster below 100 such CTAs, 3% at 200 to 300, even at 350, 2 to 5% slower
// from 400 on, over 20 lengths from 330 to 1500; four screens of 640^2 43 us, 47 us
// with 3072), and for
// plans with a direct-sum stage, which want many warps (40 images of 331^2 so 2064 us,
// with 3072 2585 us). A frame pass takes the 4096 where that makes its rows two to
// three CTAs an SM in one wave (five directions on 728^2: 95 us without, 90 us so; 64
// frames of 9 layers on 200^2 64 us and 60 us; below two, 20 frames on 300^2, 55 us
// without and 60 us so).
static inline int rows_per_cta(const FftDesc& d, int nimg, bool frames = false) {
  const int nb = fft_buf_len(d);
  const auto rows = [&](int elements) { return std::max(1, std::min(16, elements / nb)); };
  const auto ctas = [&](int r) { return (long long)((d.n + r - 1) / r) * nimg; };
  const int some = rows(nb < 320 || fft_direct(d) ? 2048 : 3072);
  if (frames && ctas(some) > 3 * 152 && ctas(rows(4096)) <= 3 * 152 && ctas(rows(4096)) > 2 * 152)
    return rows(4096);
  return ctas(some) < 350 ? rows(2048) : some;
}
static inline int cols_per_cta(int nb) { return std::max(1, std::min(16, 4096 / nb)); }
// The shape of a column pass over `nimg` images: where such CTAs would not fill
// the SMs three times over, more columns and threads a CTA (three 728^2 images:
// 41.4 us at 4096 elements and 256 threads, 34.2 us at 6144 and 512; vectors of
// fewer than 320 elements measured slower so, 278^2: 55.5 us against 59.0 us).
struct ColShape {
  int C, threads;
};
static inline ColShape col_shape(int ns, int nb, int nimg) {
  const int C = cols_per_cta(nb);
  if (nb < 320 || (long long)((ns + C - 1) / C) * nimg >= 3 * 152) return {C, kThreads};
  return {std::max(1, std::min(16, 6144 / nb)), kColThreads};
}

static inline void count_launch(int k = 1) {
  __atomic_add_fetch(launch_counter(), (uint64_t)k, __ATOMIC_RELAXED);
}

// fftfreq index: k for k < (n+1)/2, else k - n
__device__ __forceinline__ int signed_freq(int k, int n) { return k < (n + 1) / 2 ? k : k - n; }

// ---------------------------------------------------------------- workspace
struct SpecWork {
  float2* img;     // (chunk, ns, ns)
  float2* coef;    // (2 chunk, P, 9)
  float* mean;     // (2 chunk)
  float2* px;      // (2 chunk, J, ns)
  float2* py;      // (2 chunk, J, ns)
  float2* hn;      // (2 chunk, 2 ns) Hermitian parts on the Nyquist cross
  size_t bytes;
};

static SpecWork carve(const pt_grid* g, int L, void* base) {
  const int ns = g->ns, ch = image_chunk(ns), gch = gen_chunk(ns), P = std::max(1, g->P);
  const int F = 2 * ch;
  const int J = std::max(1, L);
  size_t off = 0;
  SpecWork w{};
  char* b = (char*)base;
  auto take = [&](size_t bytes) {
    char* p = b ? b + off : nullptr;
    off += align256(bytes);
    return p;
  };
  w.img = (float2*)take((size_t)std::max(ch, gch) * ns * ns * sizeof(float2));
  w.coef = (float2*)take((size_t)2 * std::max(ch, gch) * P * 9 * sizeof(float2));
  w.mean = (float*)take((size_t)2 * std::max(ch, gch) * sizeof(float));
  w.px = (float2*)take((size_t)F * J * ns * sizeof(float2));
  w.py = (float2*)take((size_t)F * J * ns * sizeof(float2));
  w.hn = (float2*)take((size_t)F * 2 * ns * sizeof(float2));
  w.bytes = off;
  return w;
}

// ================================================================ pass 1 producers
// Generate: X[kx, ky] = (n0 + i n1) * amplitude[kx, ky]
struct GenRowArgs {
  const float* amplitude;
  const float* noise;  // (2, n_fft, ns, ns) or null
  int n_fft;
  int img0;            // first FFT index of this chunk
  uint64_t seed, call;
  // subharmonic coefficients of the chunk's screens (P = 0: none), made by
  // warps 0 and 1 of each pair's first row CTA
  const float* sh_amp;    // (P, 9)
  const float* sh_noise;  // (P, 2, count, 3, 3) or null
  const double* beta;     // (P, 3, 2) grid means of the basis rows
  float2* coef;           // (2 ch, P, 9)
  float* mean;            // (2 ch)
  int count, ch, P;
};

// coef[slot][p][ij] = (n0 + i n1) * sh_amp[p][ij] of screen gc and
// mean[slot] = Re sum_p,ij coef beta_i beta_j: one warp, a lane per (level,
// 3x3 cell), the mean reduced by shuffles.
__device__ __forceinline__ void gen_coef_warp(const GenRowArgs& a, int gc, int slot, int lane) {
  double mr = 0.0;
  for (int q = lane; q < a.P * 9; q += 32) {
    const int p = q / 9, ij = q - 9 * p;
    float2 z;
    if (a.sh_noise) {
      // layout (P, 2, count, 3, 3)
      const size_t base = (size_t)p * 2 * a.count * 9;
      z = make_float2(a.sh_noise[base + (size_t)gc * 9 + ij],
                      a.sh_noise[base + (size_t)a.count * 9 + (size_t)gc * 9 + ij]);
    } else {
      z = philox_cnormal(a.seed, ((uint64_t)gc * kMaxLevels + p) * 9 + ij, a.call, kDomainSub);
    }
    const float amp = a.sh_amp[q];
    const float2 cf = make_float2(z.x * amp, z.y * amp);
    a.coef[(size_t)slot * a.P * 9 + q] = cf;
    const int i = ij / 3, j = ij % 3;
    const double bir = a.beta[(p * 3 + i) * 2], bii = a.beta[(p * 3 + i) * 2 + 1];
    const double bjr = a.beta[(p * 3 + j) * 2], bji = a.beta[(p * 3 + j) * 2 + 1];
    const double br = bir * bjr - bii * bji, bi = bir * bji + bii * bjr;
    mr += (double)cf.x * br - (double)cf.y * bi;
  }
  for (int o = 16; o > 0; o >>= 1) mr += __shfl_xor_sync(0xffffffffu, mr, o);
  if (lane == 0) a.mean[slot] = (float)mr;
}

// In the first row CTA (blockIdx.x == 0) of transform pair `img` of the
// chunk, warp 0 makes the coefficients of its real-part screen b0 + img
// (slot img) and warp 1 those of its imaginary-part screen n_fft + b0 + img
// (slot ch + img), when they exist. No barrier is involved.
__device__ __forceinline__ void gen_coef_pair(const GenRowArgs& a, int img) {
  if (a.P <= 0 || blockIdx.x != 0 || threadIdx.x >= 64) return;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gc = (w == 0 ? 0 : a.n_fft) + a.img0 + img;
  if (gc >= a.count) return;  // warp-uniform
  gen_coef_warp(a, gc, w == 0 ? img : a.ch + img, lane);
}

// Plain complex rows (pt_ifft2; frames, in place) and generate rows share this
// kernel: `gen` selects the producer. rpc rows per CTA, one transform per row; a
// CTA has read its rows before it writes them, so `in` may be `work`.
template <bool PRIME>
__global__ void __launch_bounds__(kThreads)
k_rows(FftDesc d, const float2* __restrict__ tw, int rpc, const float2* in,
       int gen, GenRowArgs ga, float2* work) {
  extern __shared__ float2 sm[];
  const int ns = d.n;
  const int row0 = blockIdx.x * rpc;
  const int img = blockIdx.y;  // image within this chunk
  if (gen) gen_coef_pair(ga, img);
  const int vs = fft_buf_len(d) + 1;
  float2* bufA = sm;
  float2* bufB = sm + rpc * vs;
  float2* stw = sm + 2 * rpc * vs;
  for (int i = threadIdx.x; i < ns; i += blockDim.x) stw[i] = tw[i];
  for (int i = threadIdx.x; i < rpc * ns; i += blockDim.x) {
    const int r = i / ns, ky = i % ns;
    const int kx = row0 + r;
    float2 v = make_float2(0.f, 0.f);
    if (kx < ns) {
      if (gen) {
        const size_t e = ((size_t)(ga.img0 + img) * ns + kx) * ns + ky;
        float2 z;
        if (ga.noise) {
          const size_t plane = (size_t)ga.n_fft * ns * ns;
          z = make_float2(ga.noise[e], ga.noise[plane + e]);
        } else {
          z = screen_normal(ga.seed, (uint64_t)(ga.img0 + img) * ns + kx, ky, ns, ga.call);
        }
        const float amp = ga.amplitude[(size_t)kx * ns + ky];
        v = make_float2(z.x * amp, z.y * amp);
      } else {
        v = in[((size_t)img * ns + kx) * ns + ky];
      }
    }
    bufA[r * vs + ky] = v;
  }
  __syncthreads();
  float2* res = fft_smem<PRIME>(bufA, bufB, d, stw, rpc, vs, 1, false);
  for (int i = threadIdx.x; i < rpc * ns; i += blockDim.x) {
    const int r = i / ns, ky = i % ns;
    const int kx = row0 + r;
    if (kx < ns) work[((size_t)img * ns + kx) * ns + ky] = res[r * vs + ky];
  }
}

// Frames: CTA = (row pair {kx, ns-kx}, frame pair). Each frame's row is the
// phasor-weighted layer sum X_f[kx, ky] = sum_j S_l[kx,ky] Px[f,j,kx] Py[f,j,ky]
// (l = j, or l = the frame's own layer in per-layer mode); the pair is then
// folded through its Hermitian parts into one complex row per kx.
struct FrameRowArgs {
  const float2* spectra;  // (L, ns, ns)
  const float2* px;       // (F, J, ns) for this chunk
  const float2* py;       // (F, J, ns)
  int J, F;               // J = terms per frame (L, or 1 per-layer); F frames in chunk
  int frame0;             // global index of the chunk's first frame (per-layer: its layer)
  int per_layer;
};

// (PRIME as in k_rows: 64 frames of 9 layers on 64^2, no levels: 28.5 us
// with, 22.6 us without.)
template <bool PRIME>
__global__ void __launch_bounds__(kThreads)
k_frame_rows(FftDesc d, const float2* __restrict__ tw, FrameRowArgs a, float2* __restrict__ work) {
  extern __shared__ float2 sm[];
  const int ns = d.n;
  const int rp = blockIdx.x;  // 0 .. ns/2
  const int pair = blockIdx.y;
  const int kxa = rp, kxb = (ns - rp) % ns;
  const int nrows = (kxa == kxb) ? 1 : 2;
  const int vs = fft_buf_len(d) + 1;
  // X rows: [frame 0 row a, frame 0 row b, frame 1 row a, frame 1 row b]
  float2* X = sm;                // 4 * vs
  float2* bufA = sm + 4 * vs;    // 2 * vs
  float2* bufB = bufA + 2 * vs;  // 2 * vs
  float2* stw = bufB + 2 * vs;   // ns
  for (int i = threadIdx.x; i < ns; i += blockDim.x) stw[i] = tw[i];
  const int f0 = 2 * pair, f1 = 2 * pair + 1;
  const bool has1 = f1 < a.F;
  for (int i = threadIdx.x; i < nrows * ns; i += blockDim.x) {
    const int r = i / ns, ky = i % ns;
    const int kx = r == 0 ? kxa : kxb;
    float2 acc0 = make_float2(0.f, 0.f), acc1 = make_float2(0.f, 0.f);
    for (int j = 0; j < a.J; ++j) {
      const int l0 = a.per_layer ? (a.frame0 + f0) : j;
      const float2 s0 = a.spectra[((size_t)l0 * ns + kx) * ns + ky];
      const size_t t0 = ((size_t)f0 * a.J + j) * ns;
      acc0 = cfma(s0, cmul(a.px[t0 + kx], a.py[t0 + ky]), acc0);
      if (has1) {
        const float2 s1 =
            a.per_layer ? a.spectra[((size_t)(a.frame0 + f1) * ns + kx) * ns + ky] : s0;
        const size_t t1 = ((size_t)f1 * a.J + j) * ns;
        acc1 = cfma(s1, cmul(a.px[t1 + kx], a.py[t1 + ky]), acc1);
      }
    }
    X[(0 * 2 + r) * vs + ky] = acc0;
    X[(1 * 2 + r) * vs + ky] = acc1;
  }
  __syncthreads();
  // Y[kx] = H0[kx] + i H1[kx], H_f[kx,ky] = (X_f[kx,ky] + conj X_f[-kx,-ky]) / 2
  for (int i = threadIdx.x; i < nrows * ns; i += blockDim.x) {
    const int r = i / ns, ky = i % ns;
    const int ro = (nrows == 1) ? 0 : 1 - r;  // row holding -kx
    const int kyn = (ns - ky) % ns;
    const float2 a0 = X[(0 * 2 + r) * vs + ky], b0 = X[(0 * 2 + ro) * vs + kyn];
    const float2 a1 = X[(1 * 2 + r) * vs + ky], b1 = X[(1 * 2 + ro) * vs + kyn];
    const float2 h0 = make_float2(0.5f * (a0.x + b0.x), 0.5f * (a0.y - b0.y));
    const float2 h1 = make_float2(0.5f * (a1.x + b1.x), 0.5f * (a1.y - b1.y));
    bufA[r * vs + ky] = make_float2(h0.x - h1.y, h0.y + h1.x);
  }
  __syncthreads();
  float2* res = fft_smem<PRIME>(bufA, bufB, d, stw, nrows, vs, 1, false);
  for (int i = threadIdx.x; i < nrows * ns; i += blockDim.x) {
    const int r = i / ns, ky = i % ns;
    const int kx = r == 0 ? kxa : kxb;
    work[((size_t)pair * ns + kx) * ns + ky] = res[r * vs + ky];
  }
}

// Uniformly spaced frames (shift of frame f, layer l = s0_l + f delta_l):
// only the Hermitian part Sh_l = (S_l(k) + conj S_l(-k)) / 2 of each layer
// contributes to a real frame, and its phasor is a geometric sequence in f,
//   H_f(k) = sum_l Sh_l(k) Q_l(k) R_l(k)^f,
// so each thread keeps A_l = Sh_l Q_l R_l^f and R_l in registers and advances
// a frame with one complex multiply-add per layer — no phasor tables. Anchors
// (exact 64-bit fixed-point phases, u0 + f du mod 1) are re-taken every
// kAnchor frames at most, bounding the float32 drift of the recurrence. Frame
// pairs are packed as Y = H_f0 + i H_f1.
constexpr int kMaxUniformLayers = 16;
constexpr int kAnchor = 64;

struct UniformParams {
  uint64_t ux0[kMaxUniformLayers], uy0[kMaxUniformLayers];  // frac(s0 df) of frame 0
  uint64_t dux[kMaxUniformLayers], duy[kMaxUniformLayers];  // frac(delta df) per frame
};

__device__ __forceinline__ float2 phasor2(int kxs, int kys, uint64_t ux, uint64_t uy) {
  return phasor_from_fixed((uint64_t)(int64_t)kxs * ux + (uint64_t)(int64_t)kys * uy);
}

// The phasor of the Nyquist index ns/2 is exp(-i pi ns u) on both k and -k
// (fftfreq gives -ns/2 for it), so Q(-k) = conj Q(k) fails on the Nyquist
// row and column and the shortcut through Sh does not hold there: the prep launch
// forms H_f(k) = (X_f(k) + conj X_f(-k)) / 2 exactly on that cross (element e:
// e < ns is (ns/2, e), else (e - ns, ns/2)) for every frame of the chunk.

// ================================================================ pass 2
// Column transform of a tile of C columns plus the paired real epilogue:
// Re -> output image (pair*re_mul + re_add), Im -> (pair*im_mul + im_add),
// each plus its subharmonic sum (coefficient row pl*crow_mul + crow_add_*)
// minus that sum's grid mean, cropped and scaled.
struct PairStore {
  float* out;
  int n_out, crop;
  float scale;
  int accumulate;
  int count;  // valid output images (global)
  int re_mul, re_add, im_mul, im_add;
  int crow_mul, crow_re, crow_im;
  const float2* coef;   // (rows, P, 9)
  const float* mean;    // (rows)
  const float2* basis;  // (P, 3, ns)
  int P;
  int sym;  // symmetric subharmonic frequencies (see k_pair_cols_reg)
  const float* img_scale;  // per output image factor on top of `scale` (NULL: none)
};

// (An odd count's last pair has one image: the table ends before the other.)
__device__ __forceinline__ float img_scale_of(const PairStore& st, int img) {
  return st.img_scale && img < st.count ? st.scale * __ldg(st.img_scale + img) : st.scale;
}

template <int THREADS, bool PRIME>
__global__ void __launch_bounds__(THREADS)
k_pair_cols(FftDesc d, const float2* __restrict__ tw, const float2* __restrict__ work, int C,
            int pair0, PairStore st) {
  extern __shared__ float2 sm[];
  const int ns = d.n;
  const int y0 = blockIdx.x * C;
  const int pl = blockIdx.y;  // pair within chunk
  const int pair = pair0 + pl;
  const int nb = fft_buf_len(d);
  float2* bufA = sm;
  float2* bufB = sm + nb * C;
  float2* stw = bufB + nb * C;
  // column tables from an even float2 offset: utab below is read as float4
  float2* mtab = stw + ((ns + 1) & ~1);  // (2, 3P, C)
  for (int i = threadIdx.x; i < ns; i += blockDim.x) stw[i] = tw[i];
  for (int i = threadIdx.x; i < ns * C; i += blockDim.x) {
    const int x = i / C, c = i % C;
    const int y = y0 + c;
    bufA[i] = y < ns ? __ldcs(work + ((size_t)pl * ns + x) * ns + y) : make_float2(0.f, 0.f);
  }
  const int img_re = pair * st.re_mul + st.re_add;
  const int img_im = pair * st.im_mul + st.im_add;
  const bool do_re = img_re < st.count, do_im = img_im < st.count;
  const int row_re = pl * st.crow_mul + st.crow_re, row_im = pl * st.crow_mul + st.crow_im;
  const int P = st.P;
  // m[o][p*3+i][c] = sum_j coef[o][p][i][j] basis[p][j][y]
  for (int i = threadIdx.x; i < 2 * 3 * P * C; i += blockDim.x) {
    const int c = i % C;
    const int pi = (i / C) % (3 * P);
    const int o = i / (C * 3 * P);
    const bool ok = o == 0 ? do_re : do_im;
    const int row = o == 0 ? row_re : row_im;
    const int y = y0 + c;
    float2 m = make_float2(0.f, 0.f);
    if (ok && y < ns) {
      const int p = pi / 3, ii = pi % 3;
      const float2* cf = st.coef + ((size_t)row * P + p) * 9 + ii * 3;
#pragma unroll
      for (int j = 0; j < 3; ++j) m = cfma(cf[j], st.basis[((size_t)p * 3 + j) * ns + y], m);
    }
    mtab[i] = m;
  }
  __syncthreads();
  // symmetric bases (b1 = 1, b2 = conj b0): per column K = sum_p m[p][1].x
  // minus the mean, per (level, column) (U_re, W_re, U_im, W_im), and the
  // first basis row of each level staged when it fits, as in the register
  // column pass; the transform's barriers order these writes before the reads
  float4* utab = (float4*)(mtab + 2 * 3 * P * C);   // P * C
  float2* ktab = mtab + 8 * (P > 0 ? P : 1) * C;     // C: (K_re, K_im)
  float2* sbasis = ktab + C;                         // P * ns
  const bool sb = st.sym && P * ns <= kColBasisMax;
  if (st.sym) {
    for (int i = threadIdx.x; i < P * C; i += blockDim.x) {
      const int p = i / C, c = i % C;
      const float2 m00 = mtab[(0 * 3 * P + 3 * p) * C + c], m02 = mtab[(0 * 3 * P + 3 * p + 2) * C + c];
      const float2 m10 = mtab[(1 * 3 * P + 3 * p) * C + c], m12 = mtab[(1 * 3 * P + 3 * p + 2) * C + c];
      utab[i] = make_float4(m00.x + m02.x, m02.y - m00.y, m10.x + m12.x, m12.y - m10.y);
    }
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
      float k0 = 0.f, k1 = 0.f;
      for (int p = 0; p < P; ++p) {
        k0 += mtab[(0 * 3 * P + 3 * p + 1) * C + c].x;
        k1 += mtab[(1 * 3 * P + 3 * p + 1) * C + c].x;
      }
      if (P > 0 && do_re) k0 -= st.mean[row_re];
      if (P > 0 && do_im) k1 -= st.mean[row_im];
      ktab[c] = make_float2(k0, k1);
    }
    if (sb)
      for (int i = threadIdx.x; i < P * ns; i += blockDim.x)
        sbasis[i] = __ldg(st.basis + (size_t)(3 * (i / ns)) * ns + (i % ns));
  }
  float2* res = fft_smem<PRIME>(bufA, bufB, d, stw, C, 1, C, true);
  const float mre = (P > 0 && do_re) ? st.mean[row_re] : 0.f;
  const float mim = (P > 0 && do_im) ? st.mean[row_im] : 0.f;
  const float sre = img_scale_of(st, img_re), sim = img_scale_of(st, img_im);
  const size_t plane = (size_t)st.n_out * st.n_out;
  for (int i = threadIdx.x; i < ns * C; i += blockDim.x) {
    const int x = i / C, c = i % C;
    const int y = y0 + c;
    if (y >= ns) continue;
    const int xo = x - st.crop, yo = y - st.crop;
    if (xo < 0 || yo < 0 || xo >= st.n_out || yo >= st.n_out) continue;
    const float2 v = res[i];
    float lre, lim;
    if (st.sym) {
      const float2 k = ktab[c];
      lre = k.x;
      lim = k.y;
      for (int p = 0; p < P; ++p) {
        const float2 b = sb ? sbasis[p * ns + x] : __ldg(st.basis + (size_t)(3 * p) * ns + x);
        const float4 u = utab[p * C + c];
        lre = fmaf(b.x, u.x, fmaf(b.y, u.y, lre));
        lim = fmaf(b.x, u.z, fmaf(b.y, u.w, lim));
      }
    } else {
      lre = -mre;
      lim = -mim;
      for (int pi = 0; pi < 3 * P; ++pi) {
        const float2 b = st.basis[(size_t)pi * ns + x];
        const float2 m0 = mtab[(0 * 3 * P + pi) * C + c];
        const float2 m1 = mtab[(1 * 3 * P + pi) * C + c];
        lre = fmaf(b.x, m0.x, fmaf(-b.y, m0.y, lre));
        lim = fmaf(b.x, m1.x, fmaf(-b.y, m1.y, lim));
      }
    }
    const size_t o = (size_t)xo * st.n_out + yo;
    if (st.accumulate) {
      if (do_re) st.out[(size_t)img_re * plane + o] += sre * (v.x + lre);
      if (do_im) st.out[(size_t)img_im * plane + o] += sim * (v.y + lim);
    } else {
      if (do_re) __stcs(st.out + (size_t)img_re * plane + o, sre * (v.x + lre));
      if (do_im) __stcs(st.out + (size_t)img_im * plane + o, sim * (v.y + lim));
    }
  }
}

using RowsKernel = void (*)(FftDesc, const float2*, int, const float2*, int, GenRowArgs, float2*);
static RowsKernel rows_kernel(const FftDesc& d) { return fft_primes(d) ? k_rows<true> : k_rows<false>; }
using PairColsKernel = void (*)(FftDesc, const float2*, const float2*, int, int, PairStore);
template <int THREADS>
static PairColsKernel pair_cols_kernel(const FftDesc& d) {
  return fft_primes(d) ? k_pair_cols<THREADS, true> : k_pair_cols<THREADS, false>;
}

// plain complex column pass (pt_ifft2)
__global__ void __launch_bounds__(kThreads)
k_plain_cols(FftDesc d, const float2* __restrict__ tw, const float2* __restrict__ work, int C,
             float2* __restrict__ out) {
  extern __shared__ float2 sm[];
  const int ns = d.n;
  const int y0 = blockIdx.x * C;
  const int img = blockIdx.y;
  const int nb = fft_buf_len(d);
  float2* bufA = sm;
  float2* bufB = sm + nb * C;
  float2* stw = bufB + nb * C;
  for (int i = threadIdx.x; i < ns; i += blockDim.x) stw[i] = tw[i];
  for (int i = threadIdx.x; i < ns * C; i += blockDim.x) {
    const int x = i / C, c = i % C;
    const int y = y0 + c;
    bufA[i] = y < ns ? work[((size_t)img * ns + x) * ns + y] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  float2* res = fft_smem(bufA, bufB, d, stw, C, 1, C, true);
  for (int i = threadIdx.x; i < ns * C; i += blockDim.x) {
    const int x = i / C, c = i % C;
    const int y = y0 + c;
    if (y < ns) out[((size_t)img * ns + x) * ns + y] = res[i];
  }
}

// frames: per frame f of a chunk, shifted-and-summed subharmonic
// coefficients (FP64 phases), their grid mean, and the main-grid phasor tables.
// Displacements travel to the device inside the launch parameters (no
// pageable copy, hence no stream synchronisation on the frame path).
constexpr int kShiftDoubles = 1792;
struct ShiftParams {
  double v[kShiftDoubles];  // (nf, J, 2) for frames [fbeg, fbeg + nf) of the chunk
};

struct FramePrepArgs {
  const float2* sh_coef;  // (P, L, 3, 3)
  const double* sh_freq;  // (P, 3)
  const double* beta;     // (P, 3, 2)
  float2* coef;           // (F, P, 9)
  float* mean;            // (F)
  float2* px;             // (F, J, ns)
  float2* py;
  int F, L, J, P, ns, per_layer, frame0;
  double df;
};

// Subharmonic coefficients of chunk frame f and their grid mean, by one CTA: a
// thread per (level, 3x3 cell). The per-layer phases f_p . s are FP64 products
// reduced mod 1 (so the error does not grow with the travel), the phasors and
// the layer sum are float32 (the reference's own complex64 path), and the CTA
// reduces the grid mean of the low-order screen. shift(j, sx, sy) gives the
// displacement of term j. Every thread of the CTA calls it.
template <class Shift>
__device__ __forceinline__ void frame_coef(const FramePrepArgs& a, int f, const Shift& shift) {
  __shared__ double part[32];
  const int t = threadIdx.x;
  double term = 0.0;
  for (int q = t; q < a.P * 9; q += blockDim.x) {
    const int p = q / 9, ij = q % 9, i = ij / 3, k = ij % 3;
    const double fi = a.sh_freq[p * 3 + i], fk = a.sh_freq[p * 3 + k];
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll 3
    for (int j = 0; j < a.J; ++j) {
      const int l = a.per_layer ? a.frame0 + f : j;
      double sx, sy;
      shift(j, sx, sy);
      double ph = fi * sx + fk * sy;
      ph -= floor(ph);
      float sn, cs;
      sincospif(2.0f * (float)ph, &sn, &cs);
      const float2 c = a.sh_coef[(((size_t)p * a.L + l) * 3 + i) * 3 + k];
      acc = cfma(c, make_float2(cs, sn), acc);
    }
    a.coef[((size_t)f * a.P + p) * 9 + ij] = acc;
    const double bir = a.beta[(p * 3 + i) * 2], bii = a.beta[(p * 3 + i) * 2 + 1];
    const double bkr = a.beta[(p * 3 + k) * 2], bki = a.beta[(p * 3 + k) * 2 + 1];
    const double br = bir * bkr - bii * bki, bi = bir * bki + bii * bkr;
    term += (double)acc.x * br - (double)acc.y * bi;
  }
  for (int o = 16; o > 0; o >>= 1) term += __shfl_down_sync(0xffffffffu, term, o);
  if ((t & 31) == 0) part[t >> 5] = term;
  __syncthreads();
  if (t == 0) {
    double m = 0.0;
    for (int w = 0; w < (int)(blockDim.x + 31) / 32; ++w) m += part[w];
    a.mean[f] = (float)m;
  }
}

__global__ void k_frame_coef(FramePrepArgs a, ShiftParams sp, int fbeg, int nf) {
  const int fl = blockIdx.x;
  if (fl >= nf) return;
  frame_coef(a, fbeg + fl, [&](int j, double& sx, double& sy) {
    sx = sp.v[(fl * a.J + j) * 2];
    sy = sp.v[(fl * a.J + j) * 2 + 1];
  });
}

// px[f][j][k] = exp(2 pi i f_k sx[f][j]), f_k = k' df, phase wrapped exactly
// in 64-bit fixed point.
__global__ void k_frame_phasors(FramePrepArgs a, ShiftParams sp, int fbeg) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int fjl = blockIdx.y;  // (frame - fbeg) * J + j
  if (k >= a.ns) return;
  const double sx = sp.v[fjl * 2];
  const double sy = sp.v[fjl * 2 + 1];
  const size_t fj = (size_t)fbeg * a.J + fjl;
  const uint64_t ux = phase_fixed(sx * a.df), uy = phase_fixed(sy * a.df);
  const uint64_t kk = (uint64_t)(int64_t)signed_freq(k, a.ns);
  a.px[fj * a.ns + k] = phasor_from_fixed(kk * ux);
  a.py[fj * a.ns + k] = phasor_from_fixed(kk * uy);
}

// ================================================================ layers / boiling
struct SeedTable {
  uint64_t s[64];
};

__global__ void k_fill_spectra(int ns, const float* __restrict__ amplitude,
                               const float* __restrict__ noise, SeedTable seeds,
                               float2* __restrict__ spectra) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t plane = (size_t)ns * ns;
  const int l = blockIdx.y;
  if (e >= plane) return;
  float2 z;
  if (noise) {
    const float* nl = noise + (size_t)l * 2 * plane;
    z = make_float2(nl[e], nl[plane + e]);
  } else {
    z = philox_cnormal(seeds.s[l], e, 0, kDomainLayer);
  }
  const float amp = amplitude[(size_t)l * plane + e];
  spectra[(size_t)l * plane + e] = make_float2(z.x * amp, z.y * amp);
}

__global__ void k_fill_sh(int L, int P, const float* __restrict__ sh_amp,
                          const float* __restrict__ sh_noise, SeedTable seeds,
                          float2* __restrict__ sh_coef) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P * L * 9) return;
  const int ij = i % 9, l = (i / 9) % L, p = i / (9 * L);
  float2 z;
  if (sh_noise) {
    // (L, P, 2, 3, 3)
    const float* b = sh_noise + ((size_t)l * P + p) * 18;
    z = make_float2(b[ij], b[9 + ij]);
  } else {
    z = philox_cnormal(seeds.s[l], (uint64_t)p * 9 + ij, 0, kDomainLayerSub);
  }
  const float amp = sh_amp[i];
  sh_coef[i] = make_float2(z.x * amp, z.y * amp);
}

// One AR(1) step of both tables: the grid modes, then the subharmonic ones (the
// last elements, a few hundred) in the same launch.
struct BoilPart {
  size_t n;
  float2* s;
  const float* amplitude;
  const float* tau;
  const float* noise;  // (2, n) or NULL
  uint64_t idx_base;
};
__device__ __forceinline__ void boil(const BoilPart& p, size_t e, float dt, uint64_t seed, uint64_t call) {
  if (e >= p.n) return;
  const float a = expf(-dt / p.tau[e]);
  const float b = sqrtf(fmaxf(1.0f - a * a, 0.0f));
  const float2 z = p.noise ? make_float2(p.noise[e], p.noise[p.n + e])
                           : philox_cnormal(seed, p.idx_base + e, call, kDomainBoil);
  const float amp = p.amplitude[e];
  const float2 v = p.s[e];
  p.s[e] = make_float2(fmaf(a, v.x, b * (z.x * amp)), fmaf(a, v.y, b * (z.y * amp)));
}
// The last CTAs take the subharmonic modes: a part chosen by the thread is read
// through an address, not from the parameter bank (9 layers of
// 1024^2: 75.8 us so, 67.7 us by CTA).
__global__ void __launch_bounds__(256)
k_boil(const __grid_constant__ BoilPart main, const __grid_constant__ BoilPart sh, unsigned main_ctas,
       float dt, uint64_t seed, uint64_t call) {
  if (blockIdx.x < main_ctas) boil(main, (size_t)blockIdx.x * 256 + threadIdx.x, dt, seed, call);
  else boil(sh, (size_t)(blockIdx.x - main_ctas) * 256 + threadIdx.x, dt, seed, call);
}

// ================================================================ LGS zoom
__global__ void k_lgs_zoom(int L, int ns, int n, int T, const int32_t* __restrict__ idx,
                           const float* __restrict__ w, const float* __restrict__ screens,
                           float scale, float* __restrict__ out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y;
  if (j >= n) return;
  float acc = 0.f;
  for (int l = 0; l < L; ++l) {
    const float* s = screens + (size_t)l * ns * ns;
    const int32_t* il = idx + (size_t)l * T * n;
    const float* wl = w + (size_t)l * T * n;
    float v = 0.f;
    for (int a = 0; a < T; ++a) {
      const float* row = s + (size_t)il[a * n + i] * ns;
      float rs = 0.f;
      for (int b = 0; b < T; ++b) rs = fmaf(wl[b * n + j], row[il[b * n + j]], rs);
      v = fmaf(wl[a * n + i], rs, v);
    }
    acc += v;
  }
  out[(size_t)i * n + j] = scale * acc;
}

// The same zoom by tiles of kZoomRows x kZoomCols output pixels: the taps are
// separable, so each source row that a tile meets is interpolated along its
// columns once, into shared memory, and the rows are combined from there: T
// loads a pixel and layer (plus T rows in kZoomRows) instead of T^2. The cost of
// a tile is load latency, layer after layer, so kZoomGroups groups of threads
// take every kZoomGroups-th layer (their sums are added in order at the end),
// the row taps of all layers are staged first, and a layer's source values are
// in flight while the one before is combined. A layer whose tile spans more
// source rows than the buffer (a magnification above one) takes the direct sum.
// 9 layers, 512^2, T = 4: 41 us by the direct sum a pixel, 43 us by tiles with
// one group and no prefetch, 13.4 us so.
constexpr int kZoomRows = 16, kZoomCols = 64, kZoomThreads = 128, kZoomGroups = 3;
template <int T>
static size_t zoom_smem(int L) {
  return (size_t)L * T * kZoomRows * 8 + (size_t)L * 8 +
         (size_t)kZoomGroups * 2 * (kZoomRows + T) * kZoomCols * sizeof(float);
}
template <int T>
__global__ void __launch_bounds__(kZoomThreads * kZoomGroups)
k_lgs_zoom_tile(int L, int ns, int n, const int32_t* __restrict__ idx, const float* __restrict__ w,
                const float* __restrict__ screens, float scale, float* __restrict__ out) {
  constexpr int SPAN = kZoomRows + T, G = kZoomThreads / kZoomCols, PX = kZoomRows / G;
  constexpr int NR = (SPAN + G - 1) / G;  // source rows a thread interpolates
  extern __shared__ float zs[];
  float* hbuf = zs;                                                  // (groups, 2, SPAN, cols)
  float* rw = hbuf + kZoomGroups * 2 * SPAN * kZoomCols;             // (L, T, rows)
  int* ri = (int*)(rw + (size_t)L * T * kZoomRows);                  // (L, T, rows)
  int* span = ri + (size_t)L * T * kZoomRows;                        // (L, 2) first and last row
  const int grp = threadIdx.x / kZoomThreads, t = threadIdx.x % kZoomThreads;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = t % kZoomCols, g = t / kZoomCols;
  const int j = blockIdx.x * kZoomCols + c, i0 = blockIdx.y * kZoomRows;
  const int jc = min(j, n - 1), rows = min(kZoomRows, n - i0);
  for (int l = warp; l < L; l += kZoomGroups * kZoomThreads / 32) {
    int lo = ns, hi = -1;
    for (int q = lane; q < T * kZoomRows; q += 32) {
      const size_t e = ((size_t)l * T + q / kZoomRows) * n + min(i0 + q % kZoomRows, n - 1);
      const int v = idx[e];
      ri[l * T * kZoomRows + q] = v;
      rw[l * T * kZoomRows + q] = w[e];
      lo = min(lo, v);
      hi = max(hi, v);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0) {
      span[2 * l] = lo;
      span[2 * l + 1] = hi;
    }
  }
  float acc[PX];
#pragma unroll
  for (int q = 0; q < PX; ++q) acc[q] = 0.f;
  int ci[T];
  float cw[T], nw[T];
  float v[NR][T];
  auto columns = [&](int l) {  // column taps of layer l
#pragma unroll
    for (int a = 0; a < T; ++a) {
      ci[a] = idx[((size_t)l * T + a) * n + jc];
      nw[a] = w[((size_t)l * T + a) * n + jc];
    }
  };
  auto fetch = [&](int l) {  // this thread's source values of layer l
    const int lo = span[2 * l], last = min(span[2 * l + 1] - lo, SPAN - 1);
    const float* s = screens + (size_t)l * ns * ns + (size_t)lo * ns;
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      const float* row = s + (size_t)min(g + q * G, last) * ns;
#pragma unroll
      for (int a = 0; a < T; ++a) v[q][a] = __ldg(row + ci[a]);
    }
  };
  if (grp < L) columns(grp);
  __syncthreads();
  if (grp < L) fetch(grp);
  int b = 0;
  for (int l = grp; l < L; l += kZoomGroups) {
    float* h = hbuf + (size_t)(grp * 2 + b) * SPAN * kZoomCols;
    const int lo = span[2 * l];
    const bool fits = span[2 * l + 1] - lo < SPAN;
    const int* rl = ri + l * T * kZoomRows;
    const float* wl = rw + l * T * kZoomRows;
    if (!fits) {
#pragma unroll
      for (int q = 0; q < PX; ++q) {
        float sum = 0.f;
        for (int a = 0; a < T; ++a) {
          const float* row = screens + (size_t)l * ns * ns + (size_t)rl[a * kZoomRows + g + q * G] * ns;
          float rs = 0.f;
#pragma unroll
          for (int k = 0; k < T; ++k) rs = fmaf(nw[k], __ldg(row + ci[k]), rs);
          sum = fmaf(wl[a * kZoomRows + g + q * G], rs, sum);
        }
        acc[q] += sum;
      }
    }
#pragma unroll
    for (int a = 0; a < T; ++a) cw[a] = nw[a];
    if (l + kZoomGroups < L) columns(l + kZoomGroups);
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      float rs = 0.f;
#pragma unroll
      for (int a = 0; a < T; ++a) rs = fmaf(cw[a], v[q][a], rs);
      if (g + q * G < SPAN) h[(g + q * G) * kZoomCols + c] = rs;
    }
    if (l + kZoomGroups < L) fetch(l + kZoomGroups);
    // the other buffer was last read before the barrier of the layer before
    asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(kZoomThreads) : "memory");
    if (fits) {
#pragma unroll
      for (int q = 0; q < PX; ++q) {
        float sum = 0.f;
#pragma unroll
        for (int a = 0; a < T; ++a)
          sum = fmaf(wl[a * kZoomRows + g + q * G],
                     h[(rl[a * kZoomRows + g + q * G] - lo) * kZoomCols + c], sum);
        acc[q] += sum;
      }
    }
    b ^= 1;
  }
  // the groups' sums, in group order (hbuf is free once every group is here)
  __syncthreads();
#pragma unroll
  for (int q = 0; q < PX; ++q) hbuf[(grp * kZoomRows + g + q * G) * kZoomCols + c] = acc[q];
  __syncthreads();
  for (int e = threadIdx.x; e < kZoomRows * kZoomCols; e += kZoomThreads * kZoomGroups) {
    const int r = e / kZoomCols, jj = blockIdx.x * kZoomCols + e % kZoomCols;
    float s = hbuf[e];
#pragma unroll
    for (int q = 1; q < kZoomGroups; ++q) s += hbuf[q * kZoomRows * kZoomCols + e];
    if (r < rows && jj < n) out[(size_t)(i0 + r) * n + jj] = scale * s;
  }
}

#include "frames_fast.cuh"  // power-of-two fast path kernels
#include "cols_tma.cuh"     // TMA-fed column pass
#include "gt_fast.cuh"       // register transforms of length 3 * 2^k (Good-Thomas)
#include "blu_fast.cuh"      // register Bluestein transforms

// Layer sums of equally spaced frames on grids without a fused row kernel:
// Y[pair][kx][ky] = H_f0 + i H_f1 for every element off the Nyquist cross (the prep
// launch writes that), to be transformed in place by the row pass of the grid's
// form. A thread owns a column ky of the row pair {kx, -kx} and advances the
// recurrence of k_frame_rows_uniform_reg over `run` frames, its anchor and its ratio
// each one rounded phasor of the exact combined phase (as products of two rounded
// table entries they left the last of 16 frames of white noise on 1000^2 at 1.07e-6,
// 0.72e-6 so).
// Half the sums of a kernel that owns one row, and the transforms get the grid's
// own row pass instead of four rows at a time in shared memory. 64 frames of 9
// layers on 500^2: 230 us for sums and rows in that kernel, 36 us here and 112 us in
// the row pass, bound by issue and the stores. Windows of 256 such frames: 500^2
// 1436 -> 1183 us, 586^2 8703 -> 2357 us, 384^2 925 -> 384 us, 278^2 2015 -> 535 us,
// 100^2 97 -> 82 us, 128^2 84 -> 54 us, 64^2 62 -> 39 us.
constexpr int kSumThreads = 128;
template <int LM>
__global__ void __launch_bounds__(kSumThreads, LM <= 4 ? 8 : LM <= 9 ? 5 : 4)
k_uniform_sum(int n, const float2* __restrict__ spectra, int L, int F, int run,
              const __grid_constant__ UniformParams up, float2* __restrict__ img) {
  constexpr int LP = (LM + 1) / 2;  // packed layer pairs
  const int ky = blockIdx.x * kSumThreads + threadIdx.x, kx = blockIdx.y;
  const int f0 = blockIdx.z * run, nfr = min(run, F - f0);
  if (ky >= n || 2 * ky == n) return;
  const int nkx = kx ? n - kx : 0, nky = ky ? n - ky : 0;
  const int kxs = signed_freq(kx, n), kys = signed_freq(ky, n);
  f2x Ax[LP], Ay[LP], Rx[LP], Ry[LP], NRy[LP];
#pragma unroll
  for (int q = 0; q < LP; ++q) {
    float ax[2], ay[2], rx[2], ry[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int l = 2 * q + h;
      ax[h] = ay[h] = ry[h] = 0.f;
      rx[h] = 1.f;
      if (l < LM && l < L) {
        const float2 sa = spectra[((size_t)l * n + kx) * n + ky];
        const float2 sb = spectra[((size_t)l * n + nkx) * n + nky];
        const float2 sh = make_float2(0.5f * (sa.x + sb.x), 0.5f * (sa.y - sb.y));
        const uint64_t dx = up.dux[l], dy = up.duy[l];
        const float2 a = cmul(sh, phasor2(kxs, kys, up.ux0[l] + (uint64_t)f0 * dx, up.uy0[l] + (uint64_t)f0 * dy));
        const float2 r = phasor2(kxs, kys, dx, dy);
        ax[h] = a.x;
        ay[h] = a.y;
        rx[h] = r.x;
        ry[h] = r.y;
      }
    }
    Ax[q] = pk2(ax[0], ax[1]);
    Ay[q] = pk2(ay[0], ay[1]);
    Rx[q] = pk2(rx[0], rx[1]);
    Ry[q] = pk2(ry[0], ry[1]);
    NRy[q] = pk2(-ry[0], -ry[1]);
  }
  const size_t plane = (size_t)n * n;
  float2* ra = img + (size_t)(f0 / 2) * plane + (size_t)kx * n + ky;
  float2* rb = img + (size_t)(f0 / 2) * plane + (size_t)nkx * n + nky;
  for (int f = 0; f < nfr; f += 2) {
    float2 h[2];
#pragma unroll
    for (int fr = 0; fr < 2; ++fr) {
      f2x hxa = 0ull, hya = 0ull, hxb = 0ull, hyb = 0ull;
      if (fr == 0 || f + 1 < nfr) {
#pragma unroll
        for (int q = 0; q < LP; ++q) {
          if (q & 1) {
            hxb = add2(hxb, Ax[q]);
            hyb = add2(hyb, Ay[q]);
          } else {
            hxa = add2(hxa, Ax[q]);
            hya = add2(hya, Ay[q]);
          }
          const f2x nx = fma2(Ax[q], Rx[q], mul2(Ay[q], NRy[q]));
          Ay[q] = fma2(Ax[q], Ry[q], mul2(Ay[q], Rx[q]));
          Ax[q] = nx;
        }
      }
      float a0, a1, b0, b1;
      upk2(add2(hxa, hxb), a0, a1);
      upk2(add2(hya, hyb), b0, b1);
      h[fr] = make_float2(a0 + a1, b0 + b1);
    }
    *ra = make_float2(h[0].x - h[1].y, h[0].y + h[1].x);
    // Y(-k) = conj H0(k) + i conj H1(k)
    if (kx) *rb = make_float2(h[0].x + h[1].y, h[1].x - h[0].y);
    ra += plane;
    rb += plane;
  }
}

// Layer sums of frames at arbitrary shifts on grids that are not a power of two:
// Y[pair][kx][ky] = H_f0 + i H_f1 for every row, to be transformed in place by
// the row pass of the grid's form. A thread owns one column ky and RB row pairs
// {kx, -kx} of NF frames, so a phasor of the column serves RB rows and a value of
// the spectra NF frames; the phasors are made here, from the exact fixed-point
// phases. As in k_frame_rows_reg a layer costs one product an element and frame,
// both products only on the Nyquist row and column of an even grid, and the CTAs
// of the last block row make the subharmonic coefficients. Five frames of 9
// layers on 728^2 took 81.6 us for coefficients, phasor tables and rows in one
// shared-memory kernel, 44.3 us in this one and the row pass. A CTA walks all
// layers, so where few CTAs of RB = 4 make the launch its latency counts: RB = 1
// there (three frames of 16 layers on 200^2, whole call: 55 us with four row pairs
// a thread, 47 us with one).
template <int NF, int RB, int CAP>
__global__ void __launch_bounds__(kSumThreads)
k_frame_sum(int n, const float2* __restrict__ spectra, const __grid_constant__ FramePrepArgs a,
            const __grid_constant__ FrameShifts<CAP> sh, int fbeg, int nf, float2* __restrict__ work) {
  extern __shared__ float2 pxs[];  // (NF, J, RB) row phasors
  const int f0 = NF * blockIdx.z;  // within this launch
  const int live = min(NF, nf - f0);
  const int J = a.J, rows = n / 2 + 1;
  const FrameShift* fs = sh.v + f0 * J;
  if ((int)blockIdx.y * RB >= rows) {  // subharmonic coefficients, a frame a CTA
    if ((int)blockIdx.x < live) {
      const FrameShift* q = fs + blockIdx.x * J;
      frame_coef(a, fbeg + f0 + blockIdx.x, [&](int j, double& x, double& y) { x = q[j].sx; y = q[j].sy; });
    }
    return;
  }
  const int kx0 = blockIdx.y * RB;
  for (int i = threadIdx.x; i < live * J * RB; i += kSumThreads) {
    const int r = i % RB, fj = i / RB;
    pxs[i] = phasor_from_fixed((uint64_t)(int64_t)signed_freq(min(kx0 + r, rows - 1), n) * fs[fj].ux);
  }
  __syncthreads();
  const int ky = blockIdx.x * kSumThreads + threadIdx.x;
  if (ky >= n) return;
  const int nky = ky == 0 ? 0 : n - ky;
  const bool even = (n & 1) == 0, nyq_col = even && ky == n / 2;
  const uint64_t kys = (uint64_t)(int64_t)signed_freq(ky, n);
  const size_t plane = (size_t)n * n;
  float2 h[NF][RB];
#pragma unroll
  for (int f = 0; f < NF; ++f)
#pragma unroll
    for (int r = 0; r < RB; ++r) h[f][r] = make_float2(0.f, 0.f);
  auto load = [&](int l, float2 (&s)[RB], float2 (&t)[RB]) {
    const float2* sl = spectra + (size_t)l * plane;
#pragma unroll
    for (int r = 0; r < RB; ++r) {
      const int kx = min(kx0 + r, rows - 1), nkx = kx == 0 ? 0 : n - kx;
      s[r] = __ldg(sl + (size_t)kx * n + ky);
      t[r] = __ldg(sl + (size_t)nkx * n + nky);
    }
  };
  auto add = [&](int f, int j, const float2 (&s)[RB], const float2 (&t)[RB]) {
    const float2 py = phasor_from_fixed(kys * fs[f * J + j].uy);
    const float2* px = pxs + (size_t)(f * J + j) * RB;
#pragma unroll
    for (int r = 0; r < RB; ++r) {
      const bool nyq_row = even && kx0 + r == n / 2;
      if (nyq_row || nyq_col) {
        const float2 qc = cmul(nyq_row ? cconj(px[r]) : px[r], nyq_col ? cconj(py) : py);
        const float2 x = cfma(s[r], cmul(px[r], py), cmul(cconj(t[r]), qc));
        h[f][r] = cadd(h[f][r], cscale(x, 0.5f));
      } else {
        const float2 m = make_float2(0.5f * (s[r].x + t[r].x), 0.5f * (s[r].y - t[r].y));
        h[f][r] = cfma(m, cmul(px[r], py), h[f][r]);
      }
    }
  };
  // with one row pair a thread, several layers' loads in flight
#pragma unroll (RB == 1 ? 4 : 1)
  for (int j = 0; j < J; ++j) {
    float2 s[RB], t[RB];
    if (!a.per_layer) load(j, s, t);
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      if (f >= live) break;
      if (a.per_layer) load(a.frame0 + fbeg + f0 + f, s, t);
      add(f, j, s, t);
    }
  }
#pragma unroll
  for (int f = 0; f < NF; f += 2) {
    if (f >= live) break;
    float2* img = work + (size_t)((fbeg + f0 + f) / 2) * plane;
#pragma unroll
    for (int r = 0; r < RB; ++r) {
      const int kx = kx0 + r;
      if (kx >= rows) break;
      const float2 p = h[f][r], q = h[f + 1][r];
      img[(size_t)kx * n + ky] = make_float2(p.x - q.y, p.y + q.x);
      if (kx != 0 && 2 * kx != n)  // Y(-k) = conj H0(k) + i conj H1(k)
        img[(size_t)(n - kx) * n + nky] = make_float2(p.x + q.y, q.x - p.y);
    }
  }
}

// ================================================================ host helpers
// shared memory of the generic passes: nb = fft_buf_len of the grid's
// transform (exchange buffers), ns twiddles
static size_t rows_smem(int ns, int nb, int rpc) {
  return (size_t)(2 * rpc * (nb + 1) + ns) * sizeof(float2);
}
static size_t frame_rows_smem(int ns, int nb) {
  return (size_t)(8 * (nb + 1) + ns) * sizeof(float2);
}
static size_t cols_smem(int ns, int nb, int C, int P) {
  // exchange buffers, twiddles, (m, U/W, K) column tables, staged basis rows
  return (size_t)(2 * nb * C + ((ns + 1) & ~1) + 8 * std::max(P, 1) * C + C +
                  (P * ns <= kColBasisMax ? P * ns : 0)) *
         sizeof(float2);
}

// The grid's transform for the frame passes: the Bluestein form only when
// its buffers fit (the frame row kernel holds eight rows); otherwise the
// direct-sum stages.
static FftDesc frame_desc(const pt_grid* g) {
  FftDesc d = g->desc;
  const int ns = g->ns;
  if (d.M > 0) {
    const size_t cap = 220 * 1024;
    if (frame_rows_smem(ns, d.M) > cap || cols_smem(ns, d.M, cols_per_cta(d.M), g->P) > cap)
      d.M = 0;
  }
  return d;
}

template <class K>
static int set_smem(K kernel, size_t bytes, const char* name) {
  if (bytes > 227 * 1024)
    return fail(PT_ERR_UNSUPPORTED, std::string(name) + ": grid too large for shared memory");
  return allow_smem((const void*)kernel, bytes, true, name);
}

// M of a length 3 M that the Good-Thomas register path takes (M = 64 .. 512), or 0.
static int gt_m(int ns) {
  if (ns % 3 != 0) return 0;
  const int m = ns / 3;
  return (m >= 64 && m <= 512 && (m & (m - 1)) == 0) ? m : 0;
}

static int check_grid(const pt_grid* g, const char* who) {
  if (!g) return fail(PT_ERR_ARG, std::string(who) + ": grid is NULL");
  return PT_OK;
}

// 64-bit binary fraction of frac(x), host side (matches phase_fixed on the device).
static uint64_t host_fixed(double x) {
  double f = x - std::floor(x);
  double v = std::ldexp(f, 64);
  if (!(v < 18446744073709551615.0)) return ~0ull;
  return (uint64_t)v;
}

// Frames [f0, f0 + nf) of a layer-sum request are equally spaced in shift
// (s_f = s_0 + f delta for every layer, to 1e-9 m + 1e-12 relative), on a grid
// the register-recurrence kernel handles (ns <= 1024, L <= 16).
static bool uniform_ok(const double* sx, const double* sy, int per_layer, int L, int f0, int nf,
                       int ns) {
  if (per_layer || nf < 2 || L > kMaxUniformLayers || ns > 1024) return false;
  for (int l = 0; l < L; ++l) {
    const double* v[2] = {sx, sy};
    for (const double* a : v) {
      const double s0 = a[(size_t)f0 * L + l];
      const double d = (a[(size_t)(f0 + nf - 1) * L + l] - s0) / (nf - 1);
      for (int f = 1; f < nf; ++f) {
        const double sf = a[(size_t)(f0 + f) * L + l];
        if (std::fabs(sf - (s0 + f * d)) > 1e-9 + 1e-12 * std::fabs(sf)) return false;
      }
    }
  }
  return true;
}

// ---- uniform frames on the 256/512/1024 register path: one prep launch + rows
template <int LM>
static int uniform_reg_rows_t(const pt_grid* g, const float2* spectra, int L, int nf,
                              const UniformTables& ut, const float2* hn, float2* img,
                              cudaStream_t s) {
  const int ns = g->ns;
  const dim3 pgrid(ns / 2 + 1, (nf + kAnchor - 1) / kAnchor);  // row pairs {kx, ns - kx}
  auto go = [&](auto kern, int threads, int nv) -> int {
    const size_t smem = (size_t)(ns + 2 * nv * fft_padded(ns)) * sizeof(float2);
    if (int rc = set_smem(kern, smem, "k_frame_rows_uniform_reg")) return rc;
    ProfScope ps("k_frame_rows_uniform", s);
    kern<<<pgrid, threads, smem, s>>>(g->tw, spectra, L, nf, ut, hn, img);
    return PT_OK;
  };
  if (ns == 256) return go(k_frame_rows_uniform_reg<LM, 256>, 256, 8);
  if (ns == 512) return go(k_frame_rows_uniform_reg<LM, 512>, 512, 8);
  return go(k_frame_rows_uniform_reg<LM, 1024>, 512, 4);
}

// Nyquist cross and subharmonic coefficients of frames [f0, f0 + nf); with `ut` the
// cross goes to w.hn, and tables with an anchor every kAnchor frames are made for the
// fused row kernel, else it goes straight to the images
static int launch_uniform_prep(const pt_grid* g, const float2* spectra, const float2* sh_coef,
                               int L, const double* sx, const double* sy, int f0, int nf,
                               const SpecWork& w, UniformTables* ut, UniformParams* up, cudaStream_t s) {
  const int ns = g->ns;
  const double df = 1.0 / (ns * g->dx);
  UniformPrep a{};
  for (int l = 0; l < L; ++l) {
    const double x0 = sx[(size_t)f0 * L + l], y0 = sy[(size_t)f0 * L + l];
    const double dx = (sx[(size_t)(f0 + nf - 1) * L + l] - x0) / (nf - 1);
    const double dy = (sy[(size_t)(f0 + nf - 1) * L + l] - y0) / (nf - 1);
    a.up.ux0[l] = host_fixed(x0 * df);
    a.up.uy0[l] = host_fixed(y0 * df);
    a.up.dux[l] = host_fixed(dx * df);
    a.up.duy[l] = host_fixed(dy * df);
    a.s0x[l] = x0;
    a.s0y[l] = y0;
    a.dsx[l] = dx;
    a.dsy[l] = dy;
  }
  const int nb = (nf + kAnchor - 1) / kAnchor;
  float2* ptab = w.px;
  a.px0 = ptab;
  a.py0 = ptab + (size_t)nb * L * ns;
  a.rx = ptab + (size_t)2 * nb * L * ns;
  a.ry = ptab + (size_t)(2 * nb + 1) * L * ns;
  a.spectra = spectra;
  a.sh_coef = sh_coef;
  a.sh_freq = g->sh_freq;
  a.beta = g->beta;
  a.hn = w.hn;
  a.coef = w.coef;
  a.mean = w.mean;
  a.N = ns;
  a.L = L;
  a.P = g->P;
  a.F = nf;
  a.nb = nb;
  a.img = ut ? nullptr : w.img;
  a.blocks_tab = ut ? ((nb + 1) * L * ns + 255) / 256 : 0;
  a.blocks_nyq = ns & 1 ? 0 : (2 * ns * ((nf + kNyqGroup - 1) / kNyqGroup) + 255) / 256;
  {
    ProfScope ps("k_uniform_prep", s);
    k_uniform_prep<<<a.blocks_tab + a.blocks_nyq + nf, 256, 0, s>>>(a);
  }
  count_launch();
  if (ut) *ut = UniformTables{a.px0, a.py0, a.rx, a.ry};
  if (up) *up = a.up;
  return PT_OK;
}

static int launch_uniform_reg_chunk(const pt_grid* g, const float2* spectra, const float2* sh_coef,
                                    int L, const double* sx, const double* sy, int f0, int nf,
                                    const SpecWork& w, cudaStream_t s) {
  UniformTables ut;
  if (int rc = launch_uniform_prep(g, spectra, sh_coef, L, sx, sy, f0, nf, w, &ut, nullptr, s)) return rc;
  if (L <= 1) return uniform_reg_rows_t<1>(g, spectra, L, nf, ut, w.hn, w.img, s);
  if (L <= 2) return uniform_reg_rows_t<2>(g, spectra, L, nf, ut, w.hn, w.img, s);
  if (L <= 3) return uniform_reg_rows_t<3>(g, spectra, L, nf, ut, w.hn, w.img, s);
  if (L <= 4) return uniform_reg_rows_t<4>(g, spectra, L, nf, ut, w.hn, w.img, s);
  if (L <= 6) return uniform_reg_rows_t<6>(g, spectra, L, nf, ut, w.hn, w.img, s);
  if (L <= 9) return uniform_reg_rows_t<9>(g, spectra, L, nf, ut, w.hn, w.img, s);
  if (L <= 12) return uniform_reg_rows_t<12>(g, spectra, L, nf, ut, w.hn, w.img, s);
  return uniform_reg_rows_t<16>(g, spectra, L, nf, ut, w.hn, w.img, s);
}

// ---- uniform frames on other grids: layer sums, to be transformed by the row pass
template <int LM>
static int uniform_sum_t(const pt_grid* g, const float2* spectra, int L, int nf, int run,
                         const UniformParams& up, float2* img, cudaStream_t s) {
  const int n = g->ns;
  ProfScope ps("k_uniform_sum", s);
  k_uniform_sum<LM><<<dim3((n + kSumThreads - 1) / kSumThreads, (n + 1) / 2, (nf + run - 1) / run),
                      kSumThreads, 0, s>>>(n, spectra, L, nf, run, up, img);
  count_launch();
  return PT_OK;
}
static int launch_uniform_sum(const pt_grid* g, const float2* spectra, const float2* sh_coef, int L,
                              const double* sx, const double* sy, int f0, int nf, const SpecWork& w,
                              cudaStream_t s) {
  // frames in runs, each from its own anchor: as few as give every SM ten CTAs,
  // but of eight frames at least (the spectra are read once a run)
  const int n = g->ns, ctas = (n + kSumThreads - 1) / kSumThreads * ((n + 1) / 2);
  const int runs = std::min(8, (1520 + ctas - 1) / ctas);
  const int run = std::max(8, ((nf + runs - 1) / runs + 1) & ~1);
  UniformParams up;
  if (int rc = launch_uniform_prep(g, spectra, sh_coef, L, sx, sy, f0, nf, w, nullptr, &up, s)) return rc;
  if (L <= 2) return uniform_sum_t<2>(g, spectra, L, nf, run, up, w.img, s);
  if (L <= 4) return uniform_sum_t<4>(g, spectra, L, nf, run, up, w.img, s);
  if (L <= 6) return uniform_sum_t<6>(g, spectra, L, nf, run, up, w.img, s);
  if (L <= 9) return uniform_sum_t<9>(g, spectra, L, nf, run, up, w.img, s);
  if (L <= 12) return uniform_sum_t<12>(g, spectra, L, nf, run, up, w.img, s);
  return uniform_sum_t<16>(g, spectra, L, nf, run, up, w.img, s);
}

// shifts of global frames [f0, f0 + nf), term by term
static void fill_shifts(FrameShift* v, const FramePrepArgs& pa, const double* sx, const double* sy,
                        int f0, int nf) {
  for (int f = 0; f < nf; ++f)
    for (int j = 0; j < pa.J; ++j) {
      const size_t src = pa.per_layer ? (size_t)f0 + f : ((size_t)f0 + f) * pa.J + j;
      v[f * pa.J + j] = FrameShift{sx[src], sy[src], host_fixed(sx[src] * pa.df), host_fixed(sy[src] * pa.df)};
    }
}

// ---- frames at arbitrary shifts on power-of-two grids
static bool frames_reg(int ns, int J) {
  return ns >= 128 && ns <= 2048 && (ns & (ns - 1)) == 0 && 2 * J <= kShiftTermsMany;
}

template <int N, int CAP>
static int frame_rows_reg_t(const pt_grid* g, const float2* spectra, const FramePrepArgs& pa,
                            const double* sx, const double* sy, int f0, float2* img,
                            cudaStream_t s) {
  using Cfg = FrameRowsCfg<N>;
  const size_t smem = (size_t)(N + 4 * fft_padded(N) + 2 * pa.J) * sizeof(float2);
  auto kern = k_frame_rows_reg<N, CAP>;
  if (int rc = set_smem(kern, smem, "k_frame_rows_reg")) return rc;
  const int fsub = CAP / pa.J & ~1;  // frames a launch takes, whole pairs
  for (int fb = 0; fb < pa.F; fb += fsub) {
    const int nf = std::min(fsub, pa.F - fb);
    FrameShifts<CAP> sh;
    fill_shifts(sh.v, pa, sx, sy, f0 + fb, nf);
    ProfScope ps("k_frame_rows", s);
    kern<<<dim3(N / 2 + 1 + (pa.P > 0), (nf + 1) / 2), Cfg::THREADS, smem, s>>>(g->tw, spectra, pa,
                                                                               sh, fb, nf, img);
    if (fb) count_launch();  // the caller counts one
  }
  return PT_OK;
}

static int launch_frame_rows_reg(const pt_grid* g, const float2* spectra, const FramePrepArgs& pa,
                                 const double* sx, const double* sy, int f0, float2* img,
                                 cudaStream_t s) {
  // a few shifts travel in 2 KB of launch parameters, many in 16 KB
  const bool few = pa.F * pa.J <= kShiftTermsFew && 2 * pa.J <= kShiftTermsFew;
  switch (g->ns) {
#define PT_CASE(n)                                                                             \
  case n:                                                                                      \
    return few ? frame_rows_reg_t<n, kShiftTermsFew>(g, spectra, pa, sx, sy, f0, img, s)       \
               : frame_rows_reg_t<n, kShiftTermsMany>(g, spectra, pa, sx, sy, f0, img, s);
    PT_CASE(128) PT_CASE(256) PT_CASE(512) PT_CASE(1024) PT_CASE(2048)
#undef PT_CASE
  }
  return fail(PT_ERR_UNSUPPORTED, "frame_rows_reg: not an instantiated size");
}

// ---- frames at arbitrary shifts on other grids
// Sums and a row pass against phasor tables and one kernel for sums and rows, by
// whole calls of F frames, J layers each (us, tables / sums):
//  - without subharmonic levels the tables' way has no launch more, and wins below
//    about 1.2e6 pixels: 9 layers, 100^2 F = 5 25 / 33, 288^2 F = 3 40 / 41 and
//    F = 10 54 / 49, 400^2 F = 5 46 / 51 and F = 10 68 / 58; with the register row pass
//    of 3 x 2^k below 0.7e6, and on 384^2 never;
//  - with levels the tables take a launch for the coefficients: below 256^2 they win
//    from four frames and four layers on (150^2, 9 layers, F = 5 41 / 47; F = 3 41 / 41);
//  - many layers that take several launches of shifts go to the tables up to 320^2
//    (60 layers, F = 20: 288^2 293 / 395, 400^2 593 / 471).
// Bluestein grids have the register transforms in the row pass only: always sums.
static bool frames_sum(const pt_grid* g, int J, int F) {
  const int ns = g->ns;
  if ((ns & (ns - 1)) == 0 || 4 * J > kShiftTermsMany) return false;
  if (blu_fast(g->desc)) return true;
  const double px = (double)F * ns * ns;
  const bool gt = gt_m(ns) != 0;
  if (J > 40 && ns < 320 && F * J > kShiftTermsMany && !fft_direct(g->desc)) return false;
  if (g->P == 0) return ns > 512 || px >= (!gt ? 1.2e6 : ns < 256 ? 0.7e6 : 0.0);
  return !(ns < 256 && F >= 4 && J >= 4 && (px < (gt ? 0.5e6 : 1.2e6) || J > 16));
}
// Equally spaced frames pay for their tables and anchors from this many on (the
// general way below). Whole calls, us, general / equally spaced: 500^2, 16 layers,
// F = 2 51 / 62; 586^2, 9 layers, F = 5 78 / 72; 150^2, 16 layers, F = 10 47 / 47 and
// F = 20 62 / 47; without levels 240^2, 3 layers, F = 10 35 / 40 and 9 layers, F = 20
// 51 / 47; 64^2, 9 layers, F = 16 17 / 23, with levels 25 / 23; 128^2, 9 layers,
// F = 16 16 / 27 and F = 64 37 / 27.
static int uniform_from(const pt_grid* g) {
  const int ns = g->ns;
  if (blu_fast(g->desc)) return 4;
  if (ns <= 128 && (ns & (ns - 1)) == 0) return ns == 128 ? 32 : g->P > 0 ? 12 : 24;
  const double f = std::ceil((g->P > 0 ? 0.3e6 : 0.62e6) / ((double)ns * ns));
  return (int)std::max(4.0, std::min(24.0, f));
}

template <int NF, int CAP, int RB>
static int frame_sum_t(const pt_grid* g, const float2* spectra, const FramePrepArgs& pa,
                       const double* sx, const double* sy, int f0, float2* img, cudaStream_t s) {
  const int n = g->ns;
  auto kern = k_frame_sum<NF, RB, CAP>;
  const size_t smem = (size_t)NF * pa.J * RB * sizeof(float2);
  const int fsub = CAP / pa.J / NF * NF;  // frames a launch takes
  for (int fb = 0; fb < pa.F; fb += fsub) {
    const int nf = std::min(fsub, pa.F - fb);
    FrameShifts<CAP> sh;
    fill_shifts(sh.v, pa, sx, sy, f0 + fb, nf);
    ProfScope ps("k_frame_sum", s);
    const int cols = (n + kSumThreads - 1) / kSumThreads, rows = (n / 2 + RB) / RB;
    kern<<<dim3(std::max(cols, pa.P > 0 ? NF : 0), rows + (pa.P > 0), (nf + NF - 1) / NF), kSumThreads, smem,
           s>>>(n, spectra, pa, sh, fb, nf, img);
    count_launch();
  }
  return PT_OK;
}
static int launch_frame_sum(const pt_grid* g, const float2* spectra, const FramePrepArgs& pa,
                            const double* sx, const double* sy, int f0, float2* img, cudaStream_t s) {
  // four frames to a pass over the spectra, but no more than there are; one row pair
  // a thread where four would leave less than two CTAs an SM over all launches (15
  // grids, up to 60 layers: one is 12% faster below 100 CTAs of four, 5% to 300, as
  // fast at 330, 4% slower to 1000 and 10% beyond; 64 frames of 60 layers on 331^2, in
  // eight launches of 252 CTAs of four: 822 us with four, 1043 us with one)
  const int n = g->ns, nf = pa.F <= 2 ? 2 : 4;
  const bool few = (pa.F + 3) / 4 * 4 * pa.J <= kShiftTermsFew;
  const bool thin = (long long)((n + kSumThreads - 1) / kSumThreads) * ((n / 2 + 4) / 4) *
                        ((pa.F + nf - 1) / nf) < 2 * 152;
  auto go = [&](auto kern) { return kern(g, spectra, pa, sx, sy, f0, img, s); };
  constexpr int A = kShiftTermsFew, B = kShiftTermsMany;
  if (nf == 2)
    return thin ? go(few ? frame_sum_t<2, A, 1> : frame_sum_t<2, B, 1>)
                : go(few ? frame_sum_t<2, A, 4> : frame_sum_t<2, B, 4>);
  return thin ? go(few ? frame_sum_t<4, A, 1> : frame_sum_t<4, B, 1>)
              : go(few ? frame_sum_t<4, A, 4> : frame_sum_t<4, B, 4>);
}

// ---- power-of-two dispatch (runtime ns -> template N)
static bool pow2_fast(int ns) { return ns >= 8 && ns <= 4096 && (ns & (ns - 1)) == 0; }

#define PT_POW2_CASES(X) X(8) X(16) X(32) X(64) X(128) X(256) X(512) X(1024) X(2048) X(4096)

template <int N>
static int rows_reg_t(const pt_grid* g, const float2* in, int gen, const GenRowArgs& ga, int nimg,
                      float2* work, cudaStream_t s) {
  using Cfg = RegCfg<N>;
  const size_t smem = (size_t)(N + 2 * Cfg::NV * fft_padded(N)) * sizeof(float2);
  if (int rc = set_smem(k_rows_reg<N>, smem, "k_rows_reg")) return rc;
  ProfScope ps("k_rows", s);
  k_rows_reg<N><<<dim3((N + Cfg::NV - 1) / Cfg::NV, nimg), Cfg::THREADS, smem, s>>>(g->tw, in, gen,
                                                                                   ga, work);
  return PT_OK;
}

static int rows_reg(const pt_grid* g, const float2* in, int gen, const GenRowArgs& ga, int nimg,
                    float2* work, cudaStream_t s) {
  switch (g->ns) {
#define PT_CASE(n) \
  case n: return rows_reg_t<n>(g, in, gen, ga, nimg, work, s);
    PT_POW2_CASES(PT_CASE)
#undef PT_CASE
  }
  return fail(PT_ERR_UNSUPPORTED, "rows_reg: not a power of two");
}

template <int N>
static int plain_cols_reg_t(const pt_grid* g, const float2* work, int nimg, float2* out,
                            cudaStream_t s) {
  using Cfg = RegCfg<N>;
  const size_t smem = (size_t)(N + 2 * Cfg::C * N) * sizeof(float2);
  if (int rc = set_smem(k_plain_cols_reg<N>, smem, "k_plain_cols_reg")) return rc;
  ProfScope ps("k_plain_cols", s);
  k_plain_cols_reg<N><<<dim3((N + Cfg::C - 1) / Cfg::C, nimg), Cfg::THREADS, smem, s>>>(g->tw, work,
                                                                                        out);
  return PT_OK;
}

static int plain_cols_reg(const pt_grid* g, const float2* work, int nimg, float2* out,
                          cudaStream_t s) {
  switch (g->ns) {
#define PT_CASE(n) \
  case n: return plain_cols_reg_t<n>(g, work, nimg, out, s);
    PT_POW2_CASES(PT_CASE)
#undef PT_CASE
  }
  return fail(PT_ERR_UNSUPPORTED, "plain_cols_reg: not a power of two");
}

template <int N>
static int pair_cols_reg_t(const pt_grid* g, const float2* work, int npair, int pair0,
                           const PairStore& st, cudaStream_t s) {
  using Cfg = PairColCfg<N>;
  const int P = g->P;
  const size_t smem = (size_t)(N + 2 * Cfg::C * N + (2 * 3 + 2) * std::max(P, 1) * Cfg::C +
                               (P * N <= kColBasisMax ? P * N : 0)) *
                      sizeof(float2);
  if (int rc = set_smem(k_pair_cols_reg<N>, smem, "k_pair_cols_reg")) return rc;
  ProfScope ps("k_pair_cols", s);
  // a programmatic dependent of the row pass before it on the stream: its
  // CTAs stage their twiddles while the row pass's last wave runs, then wait
  // (griddepcontrol.wait) for the row pass to complete
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((N + Cfg::C - 1) / Cfg::C, npair);
  cfg.blockDim = dim3(Cfg::THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return check_cuda(cudaLaunchKernelEx(&cfg, k_pair_cols_reg<N>, g->tw, work, pair0, st),
                    "k_pair_cols_reg");
}

// ---- TMA-fed column pass (N = 256, 512, 1024)
typedef CUresult (*TensorMapEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                      const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                      const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                      CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static TensorMapEncodeFn tensor_map_encoder() {
  static std::once_flag once;
  static TensorMapEncodeFn fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<TensorMapEncodeFn>(p);
  });
  return fn;
}

template <int N>
static int pair_cols_tma_t(const pt_grid* g, const float2* work, int npair, int pair0,
                           const PairStore& st, cudaStream_t s) {
  using Cfg = TmaCfg<N>;
  TensorMapEncodeFn enc = tensor_map_encoder();
  if (!enc) return fail(PT_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled unavailable");
  // 2-D view of the (npair, N, N) complex workspace: x = column (inner), y = pair * N + row
  CUtensorMap map;
  const cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)npair * N};
  const cuuint64_t strides[1] = {(cuuint64_t)N * sizeof(float2)};
  const cuuint32_t box[2] = {(cuuint32_t)Cfg::C, (cuuint32_t)Cfg::BOXR};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, (void*)work, dims, strides, box,
                         estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(PT_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  const int P1 = std::max(g->P, 1);
  const size_t smem =
      (size_t)(3 * N * Cfg::C + N + 2 * 3 * P1 * Cfg::C) * sizeof(float2) + 2 * sizeof(uint64_t);
  if (int rc = set_smem(k_pair_cols_tma<N>, smem, "k_pair_cols_tma")) return rc;
  const int xb = N / Cfg::C;
  const int groups = std::max(1, std::min(npair, (2 * 152 + xb - 1) / xb));
  ProfScope ps("k_pair_cols", s);
  k_pair_cols_tma<N><<<dim3(xb, groups), RegCfg<N>::THREADS, smem, s>>>(map, g->tw, npair, pair0,
                                                                        st);
  return PT_OK;
}

// The TMA-fed column pass is selected with PYTURB_GB300_COLS=tma (N = 256, 512,
// 1024). Measured on the GB300 it trails the one-CTA-per-tile register pass,
// whose 2048 short CTAs keep more loads in flight, so the latter is the default.
// default column-pass variant of new grids (PYTURB_GB300_COLS=tma selects TMA)
static int default_cols_variant() {
  static const int v = [] {
    const char* e = std::getenv("PYTURB_GB300_COLS");
    return (e && std::string(e) == "tma") ? 1 : 0;
  }();
  return v;
}

// ---- Good-Thomas register path

template <int M>
static int rows_gt_t(const pt_grid* g, const float2* in, int gen, const GenRowArgs& ga, int nimg,
                     float2* work, cudaStream_t s) {
  using G = GtCfg<3, M>;
  const size_t smem = (size_t)(M + G::ROW_NV * 2 * 3 * G::PAD) * sizeof(float2);
  if (int rc = set_smem(k_rows_gt<3, M>, smem, "k_rows_gt")) return rc;
  ProfScope ps("k_rows", s);
  k_rows_gt<3, M><<<dim3((G::N + G::ROW_NV - 1) / G::ROW_NV, nimg), G::ROW_THREADS, smem, s>>>(
      g->tw, in, gen, ga, work);
  return PT_OK;
}

template <int M>
static int pair_cols_gt_t(const pt_grid* g, const float2* work, int npair, int pair0,
                          const PairStore& st, cudaStream_t s) {
  using G = GtCfg<3, M>;
  const int P = g->P;
  const size_t smem = (size_t)(M + 2 * 3 * M * G::C + 8 * std::max(P, 1) * G::C +
                               (P * G::N <= kColBasisMax ? P * G::N : 0)) *
                      sizeof(float2);
  if (int rc = set_smem(k_pair_cols_gt<3, M>, smem, "k_pair_cols_gt")) return rc;
  ProfScope ps("k_pair_cols", s);
  k_pair_cols_gt<3, M><<<dim3((G::N + G::C - 1) / G::C, npair), G::COL_THREADS, smem, s>>>(
      g->tw, work, pair0, st);
  return PT_OK;
}

static int rows_gt(const pt_grid* g, const float2* in, int gen, const GenRowArgs& ga, int nimg,
                   float2* work, cudaStream_t s) {
  switch (gt_m(g->ns)) {
    case 64: return rows_gt_t<64>(g, in, gen, ga, nimg, work, s);
    case 128: return rows_gt_t<128>(g, in, gen, ga, nimg, work, s);
    case 256: return rows_gt_t<256>(g, in, gen, ga, nimg, work, s);
    case 512: return rows_gt_t<512>(g, in, gen, ga, nimg, work, s);
  }
  return fail(PT_ERR_UNSUPPORTED, "rows_gt: not 3 x 2^k");
}

static int pair_cols_gt(const pt_grid* g, const float2* work, int npair, int pair0,
                        const PairStore& st, cudaStream_t s) {
  switch (gt_m(g->ns)) {
    case 64: return pair_cols_gt_t<64>(g, work, npair, pair0, st, s);
    case 128: return pair_cols_gt_t<128>(g, work, npair, pair0, st, s);
    case 256: return pair_cols_gt_t<256>(g, work, npair, pair0, st, s);
    case 512: return pair_cols_gt_t<512>(g, work, npair, pair0, st, s);
  }
  return fail(PT_ERR_UNSUPPORTED, "pair_cols_gt: not 3 x 2^k");
}

// A launch that is a programmatic dependent of the one before it on the stream:
// its CTAs stage their twiddles while that one's last wave runs, then wait for it
// (griddepcontrol.wait).
template <class... KArgs, class... Args>
static int launch_dependent(const char* name, void (*kern)(KArgs...), dim3 grid, int threads,
                            size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return check_cuda(cudaLaunchKernelEx(&cfg, kern, args...), name);
}

// ---- register Bluestein path
template <int M>
static int rows_blu_t(const FftDesc& d, const float2* in, int gen, const GenRowArgs& ga, int nimg,
                      float2* work, cudaStream_t s) {
  using Cfg = BluCfg<M>;
  const size_t smem = (size_t)(M + 2 * Cfg::NV * fft_padded(M)) * sizeof(float2);
  if (int rc = set_smem(k_rows_blu<M>, smem, "k_rows_blu")) return rc;
  ProfScope ps("k_rows", s);
  const int per = Cfg::NV * Cfg::RPT;
  k_rows_blu<M><<<dim3((d.n + per - 1) / per, nimg), Cfg::THREADS, smem, s>>>(d, in, gen, ga, work);
  return PT_OK;
}
template <int M>
static int cols_blu_t(const pt_grid* g, const FftDesc& d, const float2* work, int nimg, int pair0,
                      const PairStore* st, float2* out, cudaStream_t s) {
  using Cfg = BluCfg<M>;
  const dim3 grid((d.n + Cfg::C - 1) / Cfg::C, nimg);
  const size_t smem = (size_t)(M + 2 * M * Cfg::C + (st ? 8 * g->P * Cfg::C : 0)) * sizeof(float2);
  ProfScope ps(st ? "k_pair_cols" : "k_plain_cols", s);
  if (st) {
    if (int rc = set_smem(k_pair_cols_blu<M>, smem, "k_pair_cols_blu")) return rc;
    return launch_dependent("k_pair_cols_blu", k_pair_cols_blu<M>, grid, Cfg::COL_THREADS, smem, s, d,
                            work, pair0, *st);
  }
  if (int rc = set_smem(k_plain_cols_blu<M>, smem, "k_plain_cols_blu")) return rc;
  return launch_dependent("k_plain_cols_blu", k_plain_cols_blu<M>, grid, Cfg::COL_THREADS, smem, s, d,
                          work, out);
}
static int rows_blu(const FftDesc& d, const float2* in, int gen, const GenRowArgs& ga, int nimg,
                    float2* work, cudaStream_t s) {
  switch (d.M) {
    case 256: return rows_blu_t<256>(d, in, gen, ga, nimg, work, s);
    case 512: return rows_blu_t<512>(d, in, gen, ga, nimg, work, s);
    case 1024: return rows_blu_t<1024>(d, in, gen, ga, nimg, work, s);
    case 2048: return rows_blu_t<2048>(d, in, gen, ga, nimg, work, s);
    case 4096: return rows_blu_t<4096>(d, in, gen, ga, nimg, work, s);
  }
  return fail(PT_ERR_UNSUPPORTED, "rows_blu: padded length not instantiated");
}
// `st`: the paired epilogue; else plain columns to out
static int cols_blu(const pt_grid* g, const FftDesc& d, const float2* work, int nimg, int pair0,
                    const PairStore* st, float2* out, cudaStream_t s) {
  switch (d.M) {
    case 256: return cols_blu_t<256>(g, d, work, nimg, pair0, st, out, s);
    case 512: return cols_blu_t<512>(g, d, work, nimg, pair0, st, out, s);
    case 1024: return cols_blu_t<1024>(g, d, work, nimg, pair0, st, out, s);
    case 2048: return cols_blu_t<2048>(g, d, work, nimg, pair0, st, out, s);
    case 4096: return cols_blu_t<4096>(g, d, work, nimg, pair0, st, out, s);
  }
  return fail(PT_ERR_UNSUPPORTED, "cols_blu: padded length not instantiated");
}

template <int N>
static int pair_cols_pipe_t(const pt_grid* g, const float2* work, int npair, int pair0,
                            const PairStore& st, cudaStream_t s) {
  using Cfg = PipeCfg<N>;
  const size_t smem = pipe_smem<N>(g->P);
  if (int rc = set_smem(k_pair_cols_pipe<N>, smem, "k_pair_cols_pipe")) return rc;
  ProfScope ps("k_pair_cols", s);
  const int grid = std::min(N / Cfg::C * npair, 152 * Cfg::PER_SM);
  return launch_dependent("k_pair_cols_pipe", k_pair_cols_pipe<N>, dim3(grid), Cfg::THREADS, smem, s,
                          (const float2*)g->tw, work, npair, pair0, st);
}
// symmetric bases whose staged rows fit beside the tiles of two CTAs an SM (one at
// 1024), and images that 16-byte pieces can be fetched from
static bool pair_cols_pipe(const pt_grid* g, const float2* work, const PairStore& st) {
  return st.sym && g->P * g->ns <= kColBasisMax && ((uintptr_t)work & 15) == 0 &&
         (g->ns == 256 || g->ns == 512 || g->ns == 1024);
}

static int pair_cols_reg(const pt_grid* g, const float2* work, int npair, int pair0,
                         const PairStore& st, cudaStream_t s) {
  if (g->cols_variant == 0 && pair_cols_pipe(g, work, st)) {
    if (g->ns == 256) return pair_cols_pipe_t<256>(g, work, npair, pair0, st, s);
    if (g->ns == 512) return pair_cols_pipe_t<512>(g, work, npair, pair0, st, s);
    return pair_cols_pipe_t<1024>(g, work, npair, pair0, st, s);
  }
  if (g->cols_variant == 1) {
    if (g->ns == 256) return pair_cols_tma_t<256>(g, work, npair, pair0, st, s);
    if (g->ns == 512) return pair_cols_tma_t<512>(g, work, npair, pair0, st, s);
    if (g->ns == 1024) return pair_cols_tma_t<1024>(g, work, npair, pair0, st, s);
  }
  switch (g->ns) {
#define PT_CASE(n) \
  case n: return pair_cols_reg_t<n>(g, work, npair, pair0, st, s);
    PT_POW2_CASES(PT_CASE)
#undef PT_CASE
  }
  return fail(PT_ERR_UNSUPPORTED, "pair_cols_reg: not a power of two");
}

}  // namespace pt

using namespace pt;

// Device error word set by bounded waits that ran out (0 = none).
namespace pt {
int tc_device_error(int* out, int clear);
int dft_device_error(int* out, int clear);
}

extern "C" int pt_device_error(int* out, int clear) {
  if (!out) return fail(PT_ERR_ARG, "pt_device_error: out is NULL");
  if (int rc = check_cuda(cudaDeviceSynchronize(), "pt_device_error: sync")) return rc;
  if (int rc = check_cuda(cudaMemcpyFromSymbol(out, g_pt_device_error, sizeof(int)),
                          "pt_device_error: read"))
    return rc;
  if (clear) {
    const int zero = 0;
    if (int rc = check_cuda(cudaMemcpyToSymbol(g_pt_device_error, &zero, sizeof(int)),
                            "pt_device_error: clear"))
      return rc;
  }
  int tcw = 0, dftw = 0;  // the tensor-core kernels' own error words (separate modules)
  if (int rc = tc_device_error(&tcw, clear)) return rc;
  if (int rc = dft_device_error(&dftw, clear)) return rc;
  *out |= tcw | dftw;
  return PT_OK;
}

extern "C" int pt_selftest_wait_timeout(long long limit, int* timed_out) {
  if (!timed_out || limit < 1 || limit > (1ll << 24))
    return fail(PT_ERR_ARG, "pt_selftest_wait_timeout: bad arguments");
  int* d = nullptr;
  if (int rc = check_cuda(cudaMalloc(&d, sizeof(int)), "pt_selftest_wait_timeout: cudaMalloc"))
    return rc;
  k_selftest_wait_timeout<<<1, 32>>>(limit, d);
  int rc = check_launch("pt_selftest_wait_timeout");
  if (!rc) rc = check_cuda(cudaMemcpy(timed_out, d, sizeof(int), cudaMemcpyDeviceToHost),
                           "pt_selftest_wait_timeout: read");
  cudaFree(d);
  return rc;
}

using namespace pt;

// ================================================================ C-ABI
// Lengths whose largest prime factor exceeds kBluesteinPrime take the
// Bluestein form (fft_bluestein) when its padded length M fits the passes'
// shared memory: the direct-sum stage costs O(p) per element for a prime p.
constexpr int kBluesteinPrime = 61;
constexpr int kBluesteinMaxM = 8192;

static int largest_prime_factor(int n) {
  int best = 1;
  for (int p = 2; (long long)p * p <= n; ++p)
    while (n % p == 0) {
      best = p;
      n /= p;
    }
  return n > 1 ? std::max(best, n) : best;
}

// In-place radix-2 transform of a power-of-two length, exp(+2 pi i j k / n), FP64.
static void host_fft_pow2(std::vector<double>& re, std::vector<double>& im) {
  const size_t n = re.size();
  for (size_t i = 1, j = 0; i < n; ++i) {
    size_t bit = n >> 1;
    for (; j & bit; bit >>= 1) j ^= bit;
    j ^= bit;
    if (i < j) {
      std::swap(re[i], re[j]);
      std::swap(im[i], im[j]);
    }
  }
  for (size_t len = 2; len <= n; len <<= 1) {
    const double a = 2.0 * M_PI / (double)len;
    for (size_t i = 0; i < n; i += len)
      for (size_t k = 0; k < len / 2; ++k) {
        const double c = std::cos(a * (double)k), sn = std::sin(a * (double)k);
        const size_t u = i + k, v = i + k + len / 2;
        const double tr = re[v] * c - im[v] * sn, ti = re[v] * sn + im[v] * c;
        re[v] = re[u] - tr;
        im[v] = im[u] - ti;
        re[u] += tr;
        im[u] += ti;
      }
  }
}

static int bluestein_plan(pt_grid* g) {
  const int n = g->ns;
  if (largest_prime_factor(n) <= kBluesteinPrime) return PT_OK;
  int M = 1;
  while (M < 2 * n - 1) M <<= 1;
  if (M > kBluesteinMaxM) return PT_OK;  // keeps the direct-sum stage
  const FftDesc dm = make_fft_desc(M);
  std::vector<float2> tab((size_t)n + 2 * M);
  std::vector<double> br(M, 0.0), bi(M, 0.0);
  for (int e = 0; e < n; ++e) {
    const long long q = (long long)e * e % (2LL * n);  // exact phase index
    const double a = M_PI * (double)q / (double)n;
    const double c = std::cos(a), sn = std::sin(a);
    tab[e] = make_float2((float)c, (float)sn);
    br[e] = c;
    bi[e] = -sn;
    if (e > 0) {
      br[M - e] = c;
      bi[M - e] = -sn;
    }
  }
  host_fft_pow2(br, bi);
  for (int k = 0; k < M; ++k) {
    tab[(size_t)n + k] = make_float2((float)br[k], (float)bi[k]);
    const double a = 2.0 * M_PI * (double)k / (double)M;
    tab[(size_t)n + M + k] = make_float2((float)std::cos(a), (float)std::sin(a));
  }
  int rc = check_cuda(cudaMalloc(&g->blu, tab.size() * sizeof(float2)), "pt_grid_create: cudaMalloc");
  if (!rc)
    rc = check_cuda(cudaMemcpy(g->blu, tab.data(), tab.size() * sizeof(float2), cudaMemcpyHostToDevice),
                    "pt_grid_create: cudaMemcpy");
  if (rc) return rc;
  g->desc.M = M;
  g->desc.mstages = dm.nstages;
  for (int i = 0; i < dm.nstages; ++i) g->desc.mradix[i] = dm.radix[i];
  g->desc.chirp = g->blu;
  g->desc.bhat = g->blu + n;
  g->desc.twM = g->blu + n + M;
  return PT_OK;
}

extern "C" int pt_grid_create(pt_grid** out, int ns, double dx, int P, const double* sh_freq) {
  if (!out) return fail(PT_ERR_ARG, "pt_grid_create: out is NULL");
  *out = nullptr;
  if (ns < 2 || ns > 8192) return fail(PT_ERR_ARG, "pt_grid_create: ns must be in [2, 8192]");
  if (!(dx > 0) || !std::isfinite(dx))
    return fail(PT_ERR_ARG, "pt_grid_create: pixel_scale must be positive and finite");
  if (P < 0 || P > kMaxLevels) return fail(PT_ERR_ARG, "pt_grid_create: n_levels must be in [0, 16]");
  if (P > 0 && !sh_freq) return fail(PT_ERR_ARG, "pt_grid_create: sh_freq is NULL");
  pt_grid* g = new pt_grid{};
  g->ns = ns;
  g->dx = dx;
  g->P = P;
  g->cols_variant = default_cols_variant();
  g->desc = make_fft_desc(ns);
  if (g->desc.nstages >= kMaxStages) {
    delete g;
    return fail(PT_ERR_UNSUPPORTED, "pt_grid_create: too many FFT stages");
  }
  std::vector<float2> tw(ns);
  for (int k = 0; k < ns; ++k) {
    const double a = 2.0 * M_PI * (double)k / ns;
    tw[k] = make_float2((float)std::cos(a), (float)std::sin(a));
  }
  const int Pm = std::max(P, 1);
  std::vector<float2> basis((size_t)Pm * 3 * ns, make_float2(0.f, 0.f));
  std::vector<double> beta((size_t)Pm * 3 * 2, 0.0);
  for (int p = 0; p < P; ++p)
    for (int i = 0; i < 3; ++i) {
      const double f = sh_freq[p * 3 + i];
      double br = 0, bi = 0;
      for (int x = 0; x < ns; ++x) {
        const double arg = 2.0 * M_PI * f * (((double)x - ns / 2.0) * dx);
        const double c = std::cos(arg), s = std::sin(arg);
        basis[((size_t)p * 3 + i) * ns + x] = make_float2((float)c, (float)s);
        br += c;
        bi += s;
      }
      beta[(p * 3 + i) * 2] = br / ns;
      beta[(p * 3 + i) * 2 + 1] = bi / ns;
    }
  std::vector<double> freq((size_t)Pm * 3, 0.0);
  for (int i = 0; i < P * 3; ++i) freq[i] = sh_freq[i];
  g->sym = 1;
  for (int p = 0; p < P; ++p)
    if (!(sh_freq[p * 3 + 1] == 0.0 && sh_freq[p * 3] == -sh_freq[p * 3 + 2])) g->sym = 0;
  int rc = check_cuda(cudaMalloc(&g->tw, ns * sizeof(float2)), "pt_grid_create: cudaMalloc");
  if (!rc) rc = check_cuda(cudaMalloc(&g->basis, basis.size() * sizeof(float2)), "pt_grid_create: cudaMalloc");
  if (!rc) rc = check_cuda(cudaMalloc(&g->sh_freq, freq.size() * sizeof(double)), "pt_grid_create: cudaMalloc");
  if (!rc) rc = check_cuda(cudaMalloc(&g->beta, beta.size() * sizeof(double)), "pt_grid_create: cudaMalloc");
  if (!rc) rc = check_cuda(cudaMemcpy(g->tw, tw.data(), ns * sizeof(float2), cudaMemcpyHostToDevice), "pt_grid_create: cudaMemcpy");
  if (!rc) rc = check_cuda(cudaMemcpy(g->basis, basis.data(), basis.size() * sizeof(float2), cudaMemcpyHostToDevice), "pt_grid_create: cudaMemcpy");
  if (!rc) rc = check_cuda(cudaMemcpy(g->sh_freq, freq.data(), freq.size() * sizeof(double), cudaMemcpyHostToDevice), "pt_grid_create: cudaMemcpy");
  if (!rc) rc = check_cuda(cudaMemcpy(g->beta, beta.data(), beta.size() * sizeof(double), cudaMemcpyHostToDevice), "pt_grid_create: cudaMemcpy");
  if (!rc) rc = bluestein_plan(g);
  if (rc) {
    pt_grid_destroy(g);
    return rc;
  }
  *out = g;
  return PT_OK;
}

extern "C" int pt_grid_radices(const pt_grid* g, int* n_stages, int* radices) {
  if (int rc = check_grid(g, "pt_grid_radices")) return rc;
  if (!n_stages || !radices) return fail(PT_ERR_ARG, "pt_grid_radices: NULL pointer");
  *n_stages = g->desc.nstages;
  for (int i = 0; i < g->desc.nstages; ++i) radices[i] = g->desc.radix[i];
  return PT_OK;
}

extern "C" int pt_grid_set_radices(pt_grid* g, int n_stages, const int* radices) {
  if (int rc = check_grid(g, "pt_grid_set_radices")) return rc;
  if (!radices || n_stages < 1 || n_stages >= kMaxStages)
    return fail(PT_ERR_ARG, "pt_grid_set_radices: n_stages must be in [1, 23]");
  long long prod = 1;
  for (int i = 0; i < n_stages; ++i) {
    if (radices[i] < 2) return fail(PT_ERR_ARG, "pt_grid_set_radices: every radix must be >= 2");
    prod *= radices[i];
    if (prod > g->ns) break;
  }
  if (prod != g->ns) return fail(PT_ERR_ARG, "pt_grid_set_radices: radices must multiply to ns");
  g->desc.nstages = n_stages;
  for (int i = 0; i < n_stages; ++i) g->desc.radix[i] = radices[i];
  return PT_OK;
}

extern "C" int pt_grid_set_cols_variant(pt_grid* g, int variant) {
  if (int rc = check_grid(g, "pt_grid_set_cols_variant")) return rc;
  if (variant != 0 && variant != 1)
    return fail(PT_ERR_ARG, "pt_grid_set_cols_variant: variant must be 0 (register) or 1 (TMA)");
  g->cols_variant = variant;
  return PT_OK;
}

extern "C" int pt_grid_destroy(pt_grid* g) {
  if (!g) return PT_OK;
  cudaFree(g->tw);
  cudaFree(g->basis);
  cudaFree(g->sh_freq);
  cudaFree(g->beta);
  cudaFree(g->blu);
  delete g;
  return PT_OK;
}

extern "C" size_t pt_grid_workspace_bytes(const pt_grid* g, int L) {
  if (!g) return 0;
  return carve(g, std::max(1, L), nullptr).bytes;
}

extern "C" int pt_ifft2(const pt_grid* g, const float* in, float* out, int batch, void* work,
                        size_t work_bytes, void* stream) {
  if (int rc = check_grid(g, "pt_ifft2")) return rc;
  if (!in || !out || batch < 0) return fail(PT_ERR_ARG, "pt_ifft2: bad arguments");
  SpecWork w = carve(g, 1, work);
  if (!work || work_bytes < w.bytes) return fail(PT_ERR_ARG, "pt_ifft2: workspace too small");
  cudaStream_t s = (cudaStream_t)stream;
  const int ns = g->ns, blen = fft_buf_len(g->desc), ch = gen_chunk(ns),
            rpc = rows_per_cta(g->desc, std::min(ch, batch)), C = cols_per_cta(blen);
  const size_t rs = rows_smem(ns, blen, rpc), cs = cols_smem(ns, blen, C, 0);
  const bool blu = blu_fast(g->desc);
  if (!pow2_fast(ns) && !blu) {
    if (int rc = set_smem(rows_kernel(g->desc), rs, "k_rows")) return rc;
    if (int rc = set_smem(k_plain_cols, cs, "k_plain_cols")) return rc;
  }
  GenRowArgs none{};
  for (int b0 = 0; b0 < batch; b0 += ch) {
    const int nb = std::min(ch, batch - b0);
    const float2* src = (const float2*)in + (size_t)b0 * ns * ns;
    float2* dst = (float2*)out + (size_t)b0 * ns * ns;
    if (pow2_fast(ns)) {
      if (int rc = rows_reg(g, src, 0, none, nb, w.img, s)) return rc;
      if (int rc = plain_cols_reg(g, w.img, nb, dst, s)) return rc;
    } else if (blu) {
      if (int rc = rows_blu(g->desc, src, 0, none, nb, w.img, s)) return rc;
      if (int rc = cols_blu(g, g->desc, w.img, nb, 0, nullptr, dst, s)) return rc;
    } else {
      {
        ProfScope ps("k_rows", s);
        rows_kernel(g->desc)<<<dim3((ns + rpc - 1) / rpc, nb), kThreads, rs, s>>>(g->desc, g->tw, rpc, src, 0,
                                                                   none, w.img);
      }
      ProfScope ps("k_plain_cols", s);
      k_plain_cols<<<dim3((ns + C - 1) / C, nb), kThreads, cs, s>>>(g->desc, g->tw, w.img, C, dst);
    }
    count_launch(2);
    if (int rc = check_launch("pt_ifft2")) return rc;
  }
  return PT_OK;
}

static int generate_impl(const pt_grid* g, int count, const float* amplitude,
                         const float* sh_amp, const float* noise, const float* sh_noise,
                         uint64_t seed, uint64_t call, int crop, int n_out, float scale,
                         const float* screen_scale, int accumulate, float* out, void* work,
                         size_t work_bytes, void* stream) {
  if (int rc = check_grid(g, "pt_generate")) return rc;
  const int ns = g->ns, P = g->P;
  if (count < 1) return fail(PT_ERR_ARG, "pt_generate: count must be >= 1");
  if (!amplitude || !out) return fail(PT_ERR_ARG, "pt_generate: NULL amplitude or out");
  if (P > 0 && !sh_amp) return fail(PT_ERR_ARG, "pt_generate: sh_amp is NULL");
  if (crop < 0 || n_out < 1 || crop + n_out > ns)
    return fail(PT_ERR_ARG, "pt_generate: crop window outside the grid");
  SpecWork w = carve(g, 1, work);
  if (!work || work_bytes < w.bytes) return fail(PT_ERR_ARG, "pt_generate: workspace too small");
  cudaStream_t s = (cudaStream_t)stream;
  const int n_fft = (count + 1) / 2;
  const int blen = fft_buf_len(g->desc);
  const int ch = gen_chunk(ns), rpc = rows_per_cta(g->desc, std::min(ch, n_fft)), C = cols_per_cta(blen);
  const size_t rs = rows_smem(ns, blen, rpc), cs = cols_smem(ns, blen, C, P);
  const bool blu = blu_fast(g->desc);
  if (!pow2_fast(ns) && !gt_m(ns) && !blu) {
    if (int rc = set_smem(rows_kernel(g->desc), rs, "k_rows")) return rc;
    if (int rc = set_smem(pair_cols_kernel<kThreads>(g->desc), cs, "k_pair_cols")) return rc;
  }
  for (int b0 = 0; b0 < n_fft; b0 += ch) {
    const int nb = std::min(ch, n_fft - b0);
    GenRowArgs ga{amplitude, noise, n_fft, b0, seed, call, sh_amp, sh_noise, g->beta,
                  w.coef, w.mean, count, ch, P};
    if (pow2_fast(ns)) {
      if (int rc = rows_reg(g, nullptr, 1, ga, nb, w.img, s)) return rc;
    } else if (gt_m(ns)) {
      if (int rc = rows_gt(g, nullptr, 1, ga, nb, w.img, s)) return rc;
    } else if (blu) {
      if (int rc = rows_blu(g->desc, nullptr, 1, ga, nb, w.img, s)) return rc;
    } else {
      ProfScope ps("k_rows", s);
      rows_kernel(g->desc)<<<dim3((ns + rpc - 1) / rpc, nb), kThreads, rs, s>>>(g->desc, g->tw, rpc, nullptr, 1,
                                                                 ga, w.img);
    }
    count_launch();
    PairStore st{};
    st.out = out;
    st.n_out = n_out;
    st.crop = crop;
    st.scale = scale;
    st.accumulate = accumulate;
    st.count = count;
    st.re_mul = 1;
    st.re_add = 0;
    st.im_mul = 1;
    st.im_add = n_fft;
    st.crow_mul = 1;
    st.crow_re = 0;   // rows [0, ch): screens b0 + pl
    st.crow_im = ch;  // rows [ch, 2 ch): screens n_fft + b0 + pl
    st.coef = w.coef;
    st.mean = w.mean;
    st.basis = g->basis;
    st.P = P;
    st.sym = g->sym;
    st.img_scale = screen_scale;
    if (pow2_fast(ns)) {
      if (int rc = pair_cols_reg(g, w.img, nb, b0, st, s)) return rc;
    } else if (gt_m(ns)) {
      if (int rc = pair_cols_gt(g, w.img, nb, b0, st, s)) return rc;
    } else if (blu) {
      if (int rc = cols_blu(g, g->desc, w.img, nb, b0, &st, nullptr, s)) return rc;
    } else {
      ProfScope ps("k_pair_cols", s);
      pair_cols_kernel<kThreads>(g->desc)<<<dim3((ns + C - 1) / C, nb), kThreads, cs, s>>>(g->desc, g->tw, w.img, C, b0, st);
    }
    count_launch();
    if (int rc = check_launch("pt_generate")) return rc;
  }
  return PT_OK;
}

extern "C" int pt_generate(const pt_grid* g, int count, const float* amplitude,
                           const float* sh_amp, const float* noise, const float* sh_noise,
                           uint64_t seed, uint64_t call, int crop, int n_out, float scale,
                           int accumulate, float* out, void* work, size_t work_bytes,
                           void* stream) {
  return generate_impl(g, count, amplitude, sh_amp, noise, sh_noise, seed, call, crop, n_out,
                       scale, nullptr, accumulate, out, work, work_bytes, stream);
}

extern "C" int pt_generate_scaled(const pt_grid* g, int count, const float* amplitude,
                                  const float* sh_amp, uint64_t seed, uint64_t call, int crop,
                                  int n_out, float scale, const float* screen_scale, float* out,
                                  void* work, size_t work_bytes, void* stream) {
  if (!screen_scale) return fail(PT_ERR_ARG, "pt_generate_scaled: screen_scale is NULL");
  return generate_impl(g, count, amplitude, sh_amp, nullptr, nullptr, seed, call, crop, n_out,
                       scale, screen_scale, 0, out, work, work_bytes, stream);
}

extern "C" int pt_layers_fill(const pt_grid* g, int L, const float* amplitude,
                              const float* sh_amp, const float* noise, const float* sh_noise,
                              const uint64_t* seeds, float* spectra, float* sh_coef,
                              void* stream) {
  if (int rc = check_grid(g, "pt_layers_fill")) return rc;
  if (L < 1 || L > 64) return fail(PT_ERR_ARG, "pt_layers_fill: n_layers must be in [1, 64]");
  if (!amplitude || !spectra) return fail(PT_ERR_ARG, "pt_layers_fill: NULL amplitude or spectra");
  if (g->P > 0 && (!sh_amp || !sh_coef)) return fail(PT_ERR_ARG, "pt_layers_fill: NULL sh_amp or sh_coef");
  if ((!noise || (g->P > 0 && !sh_noise)) && !seeds)
    return fail(PT_ERR_ARG, "pt_layers_fill: seeds required when noise is not injected");
  SeedTable st{};
  for (int l = 0; l < L; ++l) st.s[l] = seeds ? seeds[l] : 0;
  cudaStream_t s = (cudaStream_t)stream;
  const size_t plane = (size_t)g->ns * g->ns;
  k_fill_spectra<<<dim3((unsigned)((plane + 255) / 256), L), 256, 0, s>>>(
      g->ns, amplitude, noise, st, (float2*)spectra);
  count_launch();
  if (g->P > 0) {
    const int n = g->P * L * 9;
    k_fill_sh<<<(n + 127) / 128, 128, 0, s>>>(L, g->P, sh_amp, sh_noise, st, (float2*)sh_coef);
    count_launch();
  }
  return check_launch("pt_layers_fill");
}

extern "C" int pt_frames(const pt_grid* g, int L, const float* spectra, const float* sh_coef,
                         int F, const double* sx, const double* sy, int per_layer, int crop,
                         int n_out, float scale, float* out, void* work, size_t work_bytes,
                         void* stream) {
  if (int rc = check_grid(g, "pt_frames")) return rc;
  const int ns = g->ns, P = g->P;
  if (L < 1) return fail(PT_ERR_ARG, "pt_frames: n_layers must be >= 1");
  if (F < 1) return fail(PT_ERR_ARG, "pt_frames: n_frames must be >= 1");
  if (!spectra || !out || !sx || !sy) return fail(PT_ERR_ARG, "pt_frames: NULL pointer");
  if (P > 0 && !sh_coef) return fail(PT_ERR_ARG, "pt_frames: sh_coef is NULL");
  if (per_layer && F != L) return fail(PT_ERR_ARG, "pt_frames: per-layer mode needs n_frames == n_layers");
  if (per_layer && (crop != 0 || n_out != ns)) return fail(PT_ERR_ARG, "pt_frames: per-layer screens are uncropped");
  if (crop < 0 || n_out < 1 || crop + n_out > ns)
    return fail(PT_ERR_ARG, "pt_frames: crop window outside the grid");
  SpecWork w = carve(g, L, work);
  if (!work || work_bytes < w.bytes) return fail(PT_ERR_ARG, "pt_frames: workspace too small");
  cudaStream_t s = (cudaStream_t)stream;
  const FftDesc fd = frame_desc(g);
  const int blen = fft_buf_len(fd);
  const int ch = image_chunk(ns);
  const int J = per_layer ? 1 : L;
  if (2 * J > kShiftDoubles) return fail(PT_ERR_UNSUPPORTED, "pt_frames: at most 896 layers");
  const size_t rs = frame_rows_smem(ns, blen);
  const bool blu = blu_fast(g->desc);
  const int fchunk = 2 * ch;
  const int fsub = std::max(1, kShiftDoubles / (2 * J));  // frames per parameter block
  for (int f0 = 0; f0 < F; f0 += fchunk) {
    const int nf = std::min(fchunk, F - f0);
    const int npair = (nf + 1) / 2;
    FramePrepArgs pa{};
    pa.sh_coef = (const float2*)sh_coef;
    pa.sh_freq = g->sh_freq;
    pa.beta = g->beta;
    pa.coef = w.coef;
    pa.mean = w.mean;
    pa.px = w.px;
    pa.py = w.py;
    pa.F = nf;
    pa.L = L;
    pa.J = J;
    pa.P = P;
    pa.ns = ns;
    pa.per_layer = per_layer;
    pa.frame0 = f0;
    pa.df = 1.0 / (ns * g->dx);
    const bool reg_size = ns == 256 || ns == 512 || ns == 1024;
    const bool uni = (reg_size || nf >= uniform_from(g)) && uniform_ok(sx, sy, per_layer, L, f0, nf, ns);
    const bool uni_reg = uni && reg_size;
    if (uni_reg) {
      // one prep launch (tables, Nyquist cross, subharmonics) + the fused rows kernel
      if (int rc = launch_uniform_reg_chunk(g, (const float2*)spectra, (const float2*)sh_coef, L,
                                            sx, sy, f0, nf, w, s))
        return rc;
    }
    const bool reg = !uni && frames_reg(ns, J), sum = !uni && !reg && frames_sum(g, J, nf);
    if (reg) {
      // phasors, layer sums, row transforms and coefficients in one launch
      if (int rc = launch_frame_rows_reg(g, (const float2*)spectra, pa, sx, sy, f0, w.img, s))
        return rc;
    }
    if (sum) {
      // phasors, layer sums and coefficients, then the grid's own row pass in place
      if (int rc = launch_frame_sum(g, (const float2*)spectra, pa, sx, sy, f0, w.img, s)) return rc;
    } else if (uni && !uni_reg) {
      if (int rc = launch_uniform_sum(g, (const float2*)spectra, (const float2*)sh_coef, L, sx, sy, f0,
                                      nf, w, s))
        return rc;
    }
    if (sum || (uni && !uni_reg)) {
      const GenRowArgs none{};
      if (pow2_fast(ns)) {
        if (int rc = rows_reg(g, w.img, 0, none, npair, w.img, s)) return rc;
      } else if (blu) {
        if (int rc = rows_blu(g->desc, w.img, 0, none, npair, w.img, s)) return rc;
      } else if (gt_m(ns)) {
        if (int rc = rows_gt(g, w.img, 0, none, npair, w.img, s)) return rc;
      } else {
        const int rb = fft_buf_len(g->desc), rpc = rows_per_cta(g->desc, npair, true);
        const size_t rsm = rows_smem(ns, rb, rpc);
        if (int rc = set_smem(rows_kernel(g->desc), rsm, "k_rows")) return rc;
        ProfScope ps("k_rows", s);
        rows_kernel(g->desc)<<<dim3((ns + rpc - 1) / rpc, npair), kThreads, rsm, s>>>(g->desc, g->tw, rpc, w.img, 0,
                                                                       none, w.img);
      }
    }
    for (int fb = 0; fb < nf && !uni && !reg && !sum; fb += fsub) {
      const int nb = std::min(fsub, nf - fb);
      ShiftParams sp;
      for (int f = 0; f < nb; ++f)
        for (int j = 0; j < J; ++j) {
          const int gf = f0 + fb + f;
          const size_t src = per_layer ? (size_t)gf : (size_t)gf * L + j;
          sp.v[(f * J + j) * 2] = sx[src];
          sp.v[(f * J + j) * 2 + 1] = sy[src];
        }
      if (P > 0) {
        k_frame_coef<<<nb, 32 * ((P * 9 + 31) / 32), 0, s>>>(pa, sp, fb, nb);
        count_launch();
      }
      ProfScope ps("k_frame_phasors", s);
      k_frame_phasors<<<dim3((ns + 255) / 256, nb * J), 256, 0, s>>>(pa, sp, fb);
      count_launch();
    }
    if (!uni && !reg && !sum) {
      FrameRowArgs fa{(const float2*)spectra, w.px, w.py, J, nf, f0, per_layer};
      auto kern = fft_primes(fd) ? k_frame_rows<true> : k_frame_rows<false>;
      if (int rc = set_smem(kern, rs, "k_frame_rows")) return rc;
      ProfScope ps("k_frame_rows", s);
      kern<<<dim3(ns / 2 + 1, npair), kThreads, rs, s>>>(fd, g->tw, fa, w.img);
    }
    count_launch();
    PairStore st{};
    st.out = out + (size_t)f0 * n_out * n_out;
    st.n_out = n_out;
    st.crop = crop;
    st.scale = scale;
    st.accumulate = 0;
    st.count = nf;
    st.re_mul = 2;
    st.re_add = 0;
    st.im_mul = 2;
    st.im_add = 1;
    st.crow_mul = 2;
    st.crow_re = 0;
    st.crow_im = 1;
    st.coef = w.coef;
    st.mean = w.mean;
    st.basis = g->basis;
    st.P = P;
    st.sym = g->sym;
    if (pow2_fast(ns)) {
      if (int rc = pair_cols_reg(g, w.img, npair, 0, st, s)) return rc;
    } else if (gt_m(ns)) {
      if (int rc = pair_cols_gt(g, w.img, npair, 0, st, s)) return rc;
    } else if (blu) {
      if (int rc = cols_blu(g, g->desc, w.img, npair, 0, &st, nullptr, s)) return rc;
    } else {
      ProfScope ps("k_pair_cols", s);
      const ColShape sh = col_shape(ns, blen, npair);
      const size_t csm = cols_smem(ns, blen, sh.C, P);
      const dim3 grid((ns + sh.C - 1) / sh.C, npair);
      if (sh.threads == kThreads) {
        if (int rc = set_smem(pair_cols_kernel<kThreads>(fd), csm, "k_pair_cols")) return rc;
        pair_cols_kernel<kThreads>(fd)<<<grid, kThreads, csm, s>>>(fd, g->tw, w.img, sh.C, 0, st);
      } else {
        if (int rc = set_smem(pair_cols_kernel<kColThreads>(fd), csm, "k_pair_cols")) return rc;
        pair_cols_kernel<kColThreads>(fd)<<<grid, kColThreads, csm, s>>>(fd, g->tw, w.img, sh.C, 0, st);
      }
    }
    count_launch();
    if (int rc = check_launch("pt_frames")) return rc;
  }
  return PT_OK;
}

extern "C" int pt_lgs_zoom(int L, int ns, int n, int T, const int32_t* idx, const float* w,
                           const float* screens, float scale, float* out, void* stream) {
  if (L < 1 || ns < 1 || n < 1 || T < 1 || T > 6) return fail(PT_ERR_ARG, "pt_lgs_zoom: bad sizes");
  if (!idx || !w || !screens || !out) return fail(PT_ERR_ARG, "pt_lgs_zoom: NULL pointer");
  cudaStream_t s = (cudaStream_t)stream;
  ProfScope ps("k_lgs_zoom", s);
  const dim3 tiles((n + kZoomCols - 1) / kZoomCols, (n + kZoomRows - 1) / kZoomRows);
  auto go = [&](auto kern, size_t smem) -> int {
    if (int rc = set_smem(kern, smem, "k_lgs_zoom_tile")) return rc;
    kern<<<tiles, kZoomThreads * kZoomGroups, smem, s>>>(L, ns, n, idx, w, screens, scale, out);
    return PT_OK;
  };
  // the staged row taps of up to 150 layers fit beside the tiles
  int rc = PT_OK;
  if (T == 2 && L <= 150) rc = go(k_lgs_zoom_tile<2>, zoom_smem<2>(L));
  else if (T == 4 && L <= 150) rc = go(k_lgs_zoom_tile<4>, zoom_smem<4>(L));
  else if (T == 6 && L <= 150) rc = go(k_lgs_zoom_tile<6>, zoom_smem<6>(L));
  else k_lgs_zoom<<<dim3((n + 127) / 128, n), 128, 0, s>>>(L, ns, n, T, idx, w, screens, scale, out);
  if (rc) return rc;
  count_launch();
  return check_launch("pt_lgs_zoom");
}

extern "C" int pt_boil_step(const pt_grid* g, int L, float* spectra, float* sh_coef,
                            const float* amplitude, const float* sh_amp, const float* main_tau,
                            const float* sh_tau, double dt, const float* noise,
                            const float* sh_noise, uint64_t seed, uint64_t call, void* stream) {
  if (int rc = check_grid(g, "pt_boil_step")) return rc;
  if (L < 1 || !spectra || !amplitude || !main_tau) return fail(PT_ERR_ARG, "pt_boil_step: bad arguments");
  if (g->P > 0 && (!sh_coef || !sh_amp || !sh_tau)) return fail(PT_ERR_ARG, "pt_boil_step: NULL subharmonic table");
  if (!(dt > 0)) return fail(PT_ERR_ARG, "pt_boil_step: dt must be positive");
  cudaStream_t s = (cudaStream_t)stream;
  const size_t n_main = (size_t)L * g->ns * g->ns, n_sh = (size_t)g->P * L * 9;
  const BoilPart mp{n_main, (float2*)spectra, amplitude, main_tau, noise, 0};
  const BoilPart sp{n_sh, (float2*)sh_coef, sh_amp, sh_tau, sh_noise, 1ull << 40};
  const unsigned main_ctas = (unsigned)((n_main + 255) / 256), sh_ctas = (unsigned)((n_sh + 255) / 256);
  k_boil<<<main_ctas + sh_ctas, 256, 0, s>>>(mp, sp, main_ctas, (float)dt, seed, call);
  count_launch();
  return check_launch("pt_boil_step");
}

// ================================================================ allocation-free inverse FFT
// pt_ifft2_noalloc serves callers that cannot call cudaMalloc: code running
// inside a host framework that owns all device memory, or a process that must
// not grow its footprint after start-up. Its scratch is not a caller
// workspace but a file-scope device array of fixed size, which every GPU that
// loads this library holds until the process exits. Host code cannot use the
// array's name as a device address, so every call resolves the addresses with
// cudaGetSymbolAddress on the current device (a device reset or a rebuilt
// primary context can move the arrays, so an address kept from an earlier
// call could be stale). While the stream is being captured the address from
// the last uncaptured call on that device is used instead; make one call on
// each device before any stream capture. All calls
// share the arrays and the last call's contents stay in them; the row pass
// overwrites every scratch element it later reads and the twiddle table is
// rewritten by each call, so nothing has to start at zero. Calls from several
// streams or threads follow one another on a device: each waits for an event that
// the one before records behind its launches. Captured calls carry no event: a
// replay must not overlap another use of the arrays.
#include <mutex>

namespace pt {

constexpr size_t kNoAllocScratchBytes = size_t(8) << 20;  // one 1024^2 complex image
constexpr int kNoAllocMaxN = 1024;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
static __device__ __align__(256) float2 g_noalloc_tw[kNoAllocMaxN];

struct NoAllocPtrs {
  void* scratch;
  void* tw;
  cudaEvent_t last;        // behind the last call's launches
  unsigned long long ctx;  // the context it belongs to
  bool captured;
};

constexpr int kNoAllocMaxDevices = 64;
static std::mutex g_noalloc_mu;
static NoAllocPtrs g_noalloc_ptrs[kNoAllocMaxDevices];
static bool g_noalloc_ready[kNoAllocMaxDevices];

static int noalloc_setup(cudaStream_t s, NoAllocPtrs* out) {
  int dev = 0;
  if (int rc = check_cuda(cudaGetDevice(&dev), "pt_ifft2_noalloc: cudaGetDevice")) return rc;
  if (dev < 0 || dev >= kNoAllocMaxDevices)
    return fail(PT_ERR_UNSUPPORTED, "pt_ifft2_noalloc: device index beyond 63");
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (int rc = check_cuda(cudaStreamIsCapturing(s, &cap), "pt_ifft2_noalloc: cudaStreamIsCapturing"))
    return rc;
  if (cap == cudaStreamCaptureStatusNone || !g_noalloc_ready[dev]) {
    NoAllocPtrs p = g_noalloc_ptrs[dev];
    if (int rc = check_cuda(cudaGetSymbolAddress(&p.scratch, g_noalloc_scratch),
                            "pt_ifft2_noalloc: cudaGetSymbolAddress(scratch)"))
      return rc;
    if (int rc = check_cuda(cudaGetSymbolAddress(&p.tw, g_noalloc_tw),
                            "pt_ifft2_noalloc: cudaGetSymbolAddress(twiddles)"))
      return rc;
    const unsigned long long ctx = context_id();
    if (!p.last || p.ctx != ctx) {  // an event of an earlier context is gone with it
      if (int rc = check_cuda(cudaEventCreateWithFlags(&p.last, cudaEventDisableTiming),
                              "pt_ifft2_noalloc: event"))
        return rc;
      p.ctx = ctx;
    } else if (cap == cudaStreamCaptureStatusNone) {
      if (int rc = check_cuda(cudaStreamWaitEvent(s, p.last, 0), "pt_ifft2_noalloc: event")) return rc;
    }
    g_noalloc_ptrs[dev] = p;
    g_noalloc_ready[dev] = true;
  }
  *out = g_noalloc_ptrs[dev];
  out->captured = cap != cudaStreamCaptureStatusNone;
  return PT_OK;
}

// exp(+2 pi i k / n) from the FP64 sincospi of the exact fraction k / n
__global__ void k_noalloc_twiddles(float2* tw, int n) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  double s, c;
  sincospi(2.0 * (double)k / (double)n, &s, &c);
  tw[k] = make_float2((float)c, (float)s);
}

static int noalloc_run(int ns, const float* in, float* out, int batch, const NoAllocPtrs& p,
                       cudaStream_t s) {
  pt_grid g{};  // a stack view over the static arrays: nothing is allocated
  g.ns = ns;
  g.dx = 1.0;
  g.P = 0;
  g.desc = make_fft_desc(ns);
  g.tw = (float2*)p.tw;
  float2* scratch = (float2*)p.scratch;
  const size_t per = (size_t)ns * ns;
  // images per pass: what the scratch holds, and at most 65535 (grid y limit)
  const int chunk = (int)std::min<size_t>(
      65535, std::max<size_t>(1, kNoAllocScratchBytes / (per * sizeof(float2))));
  k_noalloc_twiddles<<<(ns + 127) / 128, 128, 0, s>>>(g.tw, ns);
  count_launch();
  const int rpc = rows_per_cta(g.desc, std::min(chunk, batch)), C = cols_per_cta(ns);  // no Bluestein form here
  const size_t rs = rows_smem(ns, ns, rpc), cs = cols_smem(ns, ns, C, 0);
  if (!pow2_fast(ns)) {
    if (int rc = set_smem(rows_kernel(g.desc), rs, "k_rows")) return rc;
    if (int rc = set_smem(k_plain_cols, cs, "k_plain_cols")) return rc;
  }
  GenRowArgs none{};
  for (int b0 = 0; b0 < batch; b0 += chunk) {
    const int nb = std::min(chunk, batch - b0);
    const float2* src = (const float2*)in + (size_t)b0 * per;
    float2* dst = (float2*)out + (size_t)b0 * per;
    if (pow2_fast(ns)) {
      if (int rc = rows_reg(&g, src, 0, none, nb, scratch, s)) return rc;
      if (int rc = plain_cols_reg(&g, scratch, nb, dst, s)) return rc;
    } else {
      rows_kernel(g.desc)<<<dim3((ns + rpc - 1) / rpc, nb), kThreads, rs, s>>>(g.desc, g.tw, rpc, src, 0, none,
                                                                 scratch);
      k_plain_cols<<<dim3((ns + C - 1) / C, nb), kThreads, cs, s>>>(g.desc, g.tw, scratch, C, dst);
    }
    count_launch(2);
    if (int rc = check_launch("pt_ifft2_noalloc")) return rc;
  }
  return PT_OK;
}

}  // namespace pt

extern "C" int pt_ifft2_noalloc(int ns, const float* in, float* out, int batch, void* stream) {
  if (ns < 2 || ns > kNoAllocMaxN)
    return fail(PT_ERR_ARG, "pt_ifft2_noalloc: ns must be in [2, 1024] (fixed 8 MiB scratch)");
  if (!in || !out || batch < 0) return fail(PT_ERR_ARG, "pt_ifft2_noalloc: bad arguments");
  if (batch == 0) return PT_OK;
  NoAllocPtrs p{};
  cudaStream_t s = (cudaStream_t)stream;
  std::lock_guard<std::mutex> lk(g_noalloc_mu);  // calls launch, and wait, one after another
  if (int rc = noalloc_setup(s, &p)) return rc;
  const int rc = noalloc_run(ns, in, out, batch, p, s);
  if (!p.captured) {
    const int er = check_cuda(cudaEventRecord(p.last, s), "pt_ifft2_noalloc: event");
    if (!rc) return er;
  }
  return rc;
}

// ------------------------------------------------------------------ translate
// Layer spectra and subharmonic coefficients moved by a displacement per
// layer, out = in * exp(2 pi i (f_x sx[l] + f_y sy[l])): the shift theorem of
// FourierFlowScreen.translate / Atmosphere._integrate (src/pyturb/flow.py:
// 96-129, src/pyturb/atmosphere.py:904-916) applied to the stored state, so
// that frames rendered from the result at displacement s equal frames of the
// original at sx[l] + s. Main-grid phases are exact 64-bit fixed point
// (k' frac(s df) mod 1, fftfreq signs); subharmonic phases are FP64 mod 1.
namespace pt {
constexpr int kMaxTranslateLayers = 64;
struct TranslateArgs {
  uint64_t ux[kMaxTranslateLayers], uy[kMaxTranslateLayers];
  double sx[kMaxTranslateLayers], sy[kMaxTranslateLayers];
};

__global__ void k_translate_spectra(int ns, int L, TranslateArgs a, const float2* __restrict__ in,
                                    float2* __restrict__ out) {
  const size_t npix = (size_t)ns * ns;
  const size_t total = npix * L;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const int l = (int)(i / npix);
    const size_t k = i % npix;
    const int kx = (int)(k / ns), ky = (int)(k % ns);
    const int64_t sx = kx <= (ns - 1) / 2 ? kx : kx - ns;
    const int64_t sy = ky <= (ns - 1) / 2 ? ky : ky - ns;
    const uint64_t ph = (uint64_t)sx * a.ux[l] + (uint64_t)sy * a.uy[l];
    out[i] = cmul(in[i], phasor_from_fixed(ph));
  }
}

__global__ void k_translate_sh(int P, int L, TranslateArgs a, const double* __restrict__ sh_freq,
                               const float2* __restrict__ in, float2* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P * L * 9) return;
  const int ij = i % 9, l = (i / 9) % L, p = i / (9 * L);
  const double fi = sh_freq[p * 3 + ij / 3], fk = sh_freq[p * 3 + ij % 3];
  double ph = fi * a.sx[l] + fk * a.sy[l];
  ph -= floor(ph);
  float sn, cs;
  sincospif(2.0f * (float)ph, &sn, &cs);
  out[i] = cmul(in[i], make_float2(cs, sn));
}
}  // namespace pt

// ================================================================ adjoint: subharmonics
// The subharmonic sum of a frame is Re sum_pij C_pij (b_pi(x) b_pj(y) - mean)
// with b_pi(x) = exp(2 pi i f_pi (x - ns/2) dx) (the grid's basis rows). Its
// adjoint needs, per frame f of an upstream gradient g (F, n_out, n_out) on the
// crop window, the projections
//   out[f][((p*3 + i)*3 + j)*2 + {re, im}] = sum_{x,y} g_f(x, y) b_pi(crop + x) b_pj(crop + y)
//   out[f][18 P] = sum_{x,y} g_f(x, y)
// Symmetric frequencies (b_1 = 1, b_2 = conj b_0; g is real): a level needs the
// complex column sums u(y) = sum_x g b_0 and nine real sums over y. One CTA per
// frame, kShCols columns x kShSlices row slices of threads, float sums along a
// slice (short runs in flight together) added over the slices, NL levels a pass
// over g; then kShCols threads a level form the sums over y in FP64, a fixed
// order throughout. FP64 runs at 1/64 of the FP32 rate here, so its products
// are what the symmetry leaves. 32 frames of 256^2, 3 levels: 102 us with 256
// threads walking whole columns, all nine complex products in FP64 and one pass
// a level (k_adj_sh, still the form for other frequencies), 21.7 us so.
constexpr int kShCols = 128, kShSlices = 8;
template <int NL>
__global__ void __launch_bounds__(kShCols * kShSlices)
k_adj_sh_sym(int ns, int P, int p0, int crop, int n_out, const float2* __restrict__ basis,
             const float* __restrict__ g, double* __restrict__ out) {
  __shared__ float part[kShSlices][2 * NL + 1][kShCols];
  __shared__ double red[NL][kShCols / 32][9];
  const int f = blockIdx.x;
  const float* gf = g + (size_t)f * n_out * n_out;
  const int c = threadIdx.x % kShCols, sl = threadIdx.x / kShCols;
  const int rows = (n_out + kShSlices - 1) / kShSlices;
  const int xb = min(n_out, sl * rows), xe = min(n_out, xb + rows);
  const float2* bp = basis + (size_t)p0 * 3 * ns + crop;  // row 0 of each level
  double acc[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) acc[q] = 0.0;
  for (int y0 = 0; y0 < n_out; y0 += kShCols) {
    const int y = y0 + c;
    float2 u[NL];
    float sum = 0.f;
#pragma unroll
    for (int l = 0; l < NL; ++l) u[l] = make_float2(0.f, 0.f);
    if (y < n_out) {
#pragma unroll 8
      for (int x = xb; x < xe; ++x) {
        const float v = __ldg(gf + (size_t)x * n_out + y);
        sum += v;
#pragma unroll
        for (int l = 0; l < NL; ++l) {
          const float2 b = __ldg(bp + (size_t)(3 * l) * ns + x);
          u[l].x = fmaf(b.x, v, u[l].x);
          u[l].y = fmaf(b.y, v, u[l].y);
        }
      }
    }
    part[sl][0][c] = sum;
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      part[sl][1 + 2 * l][c] = u[l].x;
      part[sl][2 + 2 * l][c] = u[l].y;
    }
    __syncthreads();
    if (sl < NL && y < n_out) {  // threads of slice l sum level l
      float t = 0.f, ux = 0.f, uy = 0.f;
#pragma unroll
      for (int q = 0; q < kShSlices; ++q) {
        t += part[q][0][c];
        ux += part[q][1 + 2 * sl][c];
        uy += part[q][2 + 2 * sl][c];
      }
      const float2 b = __ldg(bp + (size_t)(3 * sl) * ns + y);
      const double dx = ux, dy = uy, dt = t, bx = b.x, by = b.y;
      acc[0] += dx * bx;
      acc[1] += dy * by;
      acc[2] += dx * by;
      acc[3] += dy * bx;
      acc[4] += dx;
      acc[5] += dy;
      acc[6] += dt * bx;
      acc[7] += dt * by;
      acc[8] += dt;
    }
    __syncthreads();
  }
  if (sl >= NL) return;
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    double v = acc[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((c & 31) == 0) red[sl][c >> 5][q] = v;
  }
  asm volatile("bar.sync %0, %1;" ::"r"(1 + sl), "n"(kShCols) : "memory");
  if (c != 0) return;
  double v[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    v[q] = 0.0;
#pragma unroll
    for (int w = 0; w < kShCols / 32; ++w) v[q] += red[sl][w][q];
  }
  const double G[18] = {v[0] - v[1], v[2] + v[3], v[4],  v[5],  v[0] + v[1], v[3] - v[2],
                        v[6],        v[7],        v[8],  0.0,   v[6],        -v[7],
                        v[0] + v[1], v[2] - v[3], v[4],  -v[5], v[0] - v[1], -(v[2] + v[3])};
  double* of = out + (size_t)f * (18 * P + 1);
#pragma unroll
  for (int q = 0; q < 18; ++q) of[(size_t)(p0 + sl) * 18 + q] = G[q];
  if (p0 + sl == 0) of[(size_t)18 * P] = v[8];
}

// One CTA per frame; thread t owns columns y = t, t + 256, ...; one pass over
// g per level; float sums along x, double products and a fixed-order reduce.
__global__ void __launch_bounds__(256)
k_adj_sh(int ns, int P, int crop, int n_out, const float2* __restrict__ basis,
         const float* __restrict__ g, double* __restrict__ out) {
  __shared__ double red[8][19];
  const int f = blockIdx.x;
  const float* gf = g + (size_t)f * n_out * n_out;
  const size_t stride = (size_t)18 * P + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int p = 0; p < P; ++p) {
    const float2* b0 = basis + (size_t)p * 3 * ns + crop;
    double acc[19];
#pragma unroll
    for (int q = 0; q < 19; ++q) acc[q] = 0.0;
    for (int y = threadIdx.x; y < n_out; y += blockDim.x) {
      float2 u[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      float sum = 0.f;
      for (int x = 0; x < n_out; ++x) {
        const float v = gf[(size_t)x * n_out + y];
        sum += v;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const float2 b = __ldg(b0 + (size_t)i * ns + x);
          u[i].x = fmaf(b.x, v, u[i].x);
          u[i].y = fmaf(b.y, v, u[i].y);
        }
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const float2 b = __ldg(b0 + (size_t)j * ns + y);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          acc[(i * 3 + j) * 2] += (double)u[i].x * b.x - (double)u[i].y * b.y;
          acc[(i * 3 + j) * 2 + 1] += (double)u[i].x * b.y + (double)u[i].y * b.x;
        }
      }
      acc[18] += sum;
    }
#pragma unroll
    for (int q = 0; q < 19; ++q) {
      double v = acc[q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) red[warp][q] = v;
    }
    __syncthreads();
    if (threadIdx.x < 19) {
      const int q = threadIdx.x;
      double v = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += red[w][q];
      if (q < 18) out[f * stride + (size_t)p * 18 + q] = v;
      else if (p == 0) out[f * stride + (size_t)18 * P] = v;
    }
    __syncthreads();
  }
}

// Level gradients from the projections. With C_fpij = sum_l w_l c_lpij E_flpij,
// E = exp(2 pi i (sx f_pi + sy f_pj)) and Q = scale (G - beta_pi beta_pj sum g),
//   dL/dw_l += sum Re(c E Q), dL/dsx_fl -= 2 pi sum f_pi Im(w c E Q) (sy: f_pj),
//   dL/dc_lpij += conj(w_l sum_f E Q),
// in FP64. k_adj_terms: CTA = (frame, layer), thread = (p, i, j); it writes
// E Q and the frame's shift gradient (with the grid part's, if given).
// k_adj_levels: CTA = layer, sums over the frames in order.
struct AdjLevels {
  int L, F, P, f0;        // F frames of this chunk, the first is frame f0
  double scale;
  const double* freq;     // (P, 3)
  const double* beta;     // (P, 3, 2)
  const float* w;         // (L)
  const float2* c;        // (P, L, 9)
  const double* sx;       // (F, L)
  const double* sy;
  const double* proj;     // (F, 18 P + 1), or NULL: no levels
  const double* part;     // (L, F, 3) of pt_synth_adj_params, or NULL
  double2* eq;            // (F, L, 9 P)
  double* fw;             // (F, L) weight contributions
  double* gw;             // (L)
  double* gsh;            // (all frames, L, 2)
  double2* gc;            // (L, P, 9), or NULL
  int accumulate;
};

__global__ void __launch_bounds__(160)
k_adj_terms(AdjLevels a) {
  __shared__ double red[5][3];
  const int f = blockIdx.x, l = blockIdx.y, t = threadIdx.x;
  double v[3] = {0.0, 0.0, 0.0};
  if (a.proj && t < 9 * a.P) {
    const int p = t / 9, ij = t % 9, i = ij / 3, j = ij % 3;
    const double* pr = a.proj + (size_t)f * (18 * a.P + 1);
    const double fi = a.freq[3 * p + i], fj = a.freq[3 * p + j];
    const double bir = a.beta[(3 * p + i) * 2], bii = a.beta[(3 * p + i) * 2 + 1];
    const double bjr = a.beta[(3 * p + j) * 2], bji = a.beta[(3 * p + j) * 2 + 1];
    const double S = pr[18 * a.P];
    const double qr = a.scale * (pr[2 * t] - (bir * bjr - bii * bji) * S);
    const double qi = a.scale * (pr[2 * t + 1] - (bir * bji + bii * bjr) * S);
    double ph = a.sx[(size_t)f * a.L + l] * fi + a.sy[(size_t)f * a.L + l] * fj;
    ph -= floor(ph);
    double sn, cs;
    sincospi(2.0 * ph, &sn, &cs);
    const double er = cs * qr - sn * qi, ei = cs * qi + sn * qr;
    a.eq[((size_t)f * a.L + l) * 9 * a.P + t] = make_double2(er, ei);
    const float2 c = a.c[((size_t)p * a.L + l) * 9 + ij];
    v[0] = (double)c.x * er - (double)c.y * ei;
    const double im = (double)a.w[l] * ((double)c.x * ei + (double)c.y * er);
    v[1] = fi * im;
    v[2] = fj * im;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if ((t & 31) == 0) red[t >> 5][k] = v[k];
  }
  __syncthreads();
  if (t < 3) {
    double s = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) s += red[q][t];
    const double grid = a.part ? a.part[((size_t)l * a.F + f) * 3 + t] : 0.0;
    if (t == 0) a.fw[(size_t)f * a.L + l] = s + grid;
    else if (a.gsh) a.gsh[((size_t)(a.f0 + f) * a.L + l) * 2 + t - 1] = grid - 2.0 * M_PI * s;
  }
}

__global__ void __launch_bounds__(160)
k_adj_levels(AdjLevels a) {
  const int l = blockIdx.x, t = threadIdx.x;
  const int Q = a.proj && a.gc ? 9 * a.P : 0;
  if (t < Q) {
    double2 s = make_double2(0.0, 0.0);
#pragma unroll 8
    for (int f = 0; f < a.F; ++f) {
      const double2 v = a.eq[((size_t)f * a.L + l) * 9 * a.P + t];
      s.x += v.x;
      s.y += v.y;
    }
    double2* o = a.gc + (size_t)l * Q + t;
    const double w = a.w[l];
    const double2 was = a.accumulate ? *o : make_double2(0.0, 0.0);
    *o = make_double2(was.x + w * s.x, was.y - w * s.y);
  }
  if (t == 159 && a.gw) {
    double s = a.accumulate ? a.gw[l] : 0.0;
#pragma unroll 8
    for (int f = 0; f < a.F; ++f) s += a.fw[(size_t)f * a.L + l];
    a.gw[l] = s;
  }
}

extern "C" size_t pt_synth_adj_levels_workspace_bytes(int L, int F, int P) {
  if (L < 1 || F < 1 || P < 0 || P > kMaxLevels) return 0;
  return ((size_t)18 * P + 1) * L * F * sizeof(double);
}

extern "C" int pt_synth_adj_levels(const pt_grid* g, int L, int F, int f0, float scale, const float* w,
                                   const float* sh_coef, const double* sx, const double* sy,
                                   const double* proj, const double* part, int accumulate,
                                   double* grad_w, double* grad_shifts, double* grad_coef, void* work,
                                   size_t work_bytes, void* stream) {
  if (int rc = check_grid(g, "pt_synth_adj_levels")) return rc;
  if (L < 1 || L > 65535 || F < 1 || f0 < 0) return fail(PT_ERR_ARG, "pt_synth_adj_levels: bad sizes");
  if (!w || (!proj && !part) || (!grad_w != !grad_shifts))
    return fail(PT_ERR_ARG, "pt_synth_adj_levels: NULL pointer");
  if (proj && (g->P < 1 || !sh_coef || !sx || !sy))
    return fail(PT_ERR_ARG, "pt_synth_adj_levels: projections without levels, coefficients or shifts");
  if (grad_coef && !proj) return fail(PT_ERR_ARG, "pt_synth_adj_levels: level gradients need projections");
  const int P = proj ? g->P : 0;
  if (!work || work_bytes < pt_synth_adj_levels_workspace_bytes(L, F, P))
    return fail(PT_ERR_ARG, "pt_synth_adj_levels: workspace too small");
  AdjLevels a{};
  a.L = L;
  a.F = F;
  a.P = P;
  a.f0 = f0;
  a.scale = scale;
  a.freq = g->sh_freq;
  a.beta = g->beta;
  a.w = w;
  a.c = (const float2*)sh_coef;
  a.sx = sx;
  a.sy = sy;
  a.proj = proj;
  a.part = part;
  a.eq = (double2*)work;
  a.fw = (double*)work + (size_t)18 * P * L * F;
  a.gw = grad_w;
  a.gsh = grad_shifts;
  a.gc = (double2*)grad_coef;
  a.accumulate = accumulate;
  cudaStream_t s = (cudaStream_t)stream;
  ProfScope ps("k_adj_levels", s);
  k_adj_terms<<<dim3(F, L), 32 * std::max(1, (9 * P + 31) / 32), 0, s>>>(a);
  k_adj_levels<<<L, 160, 0, s>>>(a);
  count_launch(2);
  return check_launch("pt_synth_adj_levels");
}

extern "C" int pt_synth_adj_sh(const pt_grid* g, int F, int crop, int n_out, const float* grad,
                               double* out, void* stream) {
  if (int rc = check_grid(g, "pt_synth_adj_sh")) return rc;
  if (g->P < 1) return fail(PT_ERR_ARG, "pt_synth_adj_sh: the grid has no subharmonic levels");
  if (F < 1 || n_out < 1 || crop < 0 || crop + n_out > g->ns)
    return fail(PT_ERR_ARG, "pt_synth_adj_sh: crop window outside the grid");
  if (!grad || !out) return fail(PT_ERR_ARG, "pt_synth_adj_sh: NULL pointer");
  cudaStream_t s = (cudaStream_t)stream;
  ProfScope ps("k_adj_sh", s);
  if (!g->sym) {
    k_adj_sh<<<F, 256, 0, s>>>(g->ns, g->P, crop, n_out, g->basis, grad, out);
  } else {
    for (int p = 0; p < g->P;) {  // up to three levels a pass over the gradient
      const int nl = std::min(3, g->P - p), threads = kShCols * kShSlices;
      if (nl == 1) k_adj_sh_sym<1><<<F, threads, 0, s>>>(g->ns, g->P, p, crop, n_out, g->basis, grad, out);
      else if (nl == 2) k_adj_sh_sym<2><<<F, threads, 0, s>>>(g->ns, g->P, p, crop, n_out, g->basis, grad, out);
      else k_adj_sh_sym<3><<<F, threads, 0, s>>>(g->ns, g->P, p, crop, n_out, g->basis, grad, out);
      p += nl;
      if (p < g->P) count_launch();
    }
  }
  count_launch();
  return check_launch("pt_synth_adj_sh");
}

extern "C" int pt_layers_translate(const pt_grid* g, int L, const float* spectra_in,
                                   const float* sh_in, const double* sx, const double* sy,
                                   float* spectra_out, float* sh_out, void* stream) {
  if (int rc = check_grid(g, "pt_layers_translate")) return rc;
  if (L < 1 || L > kMaxTranslateLayers)
    return fail(PT_ERR_ARG, "pt_layers_translate: n_layers must be in [1, 64]");
  if (!spectra_in || !spectra_out || !sx || !sy)
    return fail(PT_ERR_ARG, "pt_layers_translate: NULL pointer");
  if (g->P > 0 && (!sh_in || !sh_out))
    return fail(PT_ERR_ARG, "pt_layers_translate: subharmonic coefficients are NULL");
  TranslateArgs a{};
  const double df = 1.0 / (g->ns * g->dx);
  for (int l = 0; l < L; ++l) {
    if (!std::isfinite(sx[l]) || !std::isfinite(sy[l]))
      return fail(PT_ERR_ARG, "pt_layers_translate: displacement is not finite");
    a.ux[l] = host_fixed(sx[l] * df);
    a.uy[l] = host_fixed(sy[l] * df);
    a.sx[l] = sx[l];
    a.sy[l] = sy[l];
  }
  cudaStream_t s = (cudaStream_t)stream;
  const size_t total = (size_t)g->ns * g->ns * L;
  k_translate_spectra<<<(unsigned)std::min<size_t>((total + 255) / 256, 152 * 16), 256, 0, s>>>(
      g->ns, L, a, (const float2*)spectra_in, (float2*)spectra_out);
  count_launch();
  if (g->P > 0) {
    const int n = g->P * L * 9;
    k_translate_sh<<<(n + 127) / 128, 128, 0, s>>>(g->P, L, a, g->sh_freq,
                                                   (const float2*)sh_in, (float2*)sh_out);
    count_launch();
  }
  return check_launch("pt_layers_translate");
}

// ------------------------------------------------------------------ temporal PSD
// pyturb.analysis.temporal_psd (src/pyturb/analysis.py:183-208): each series
// (samples along the last axis) minus its mean, |DFT|^2 * 2 dt / T, averaged
// over the series. The DFT is the grid's mixed-radix transform of length
// ns = T (|X(f)|^2 of a real series is the same for either sign). CTA b sums
// the power of series b, b + G, ... in shared memory; a second kernel sums
// the G partials in a fixed order.
namespace pt {
__global__ void __launch_bounds__(kThreads)
k_psd_series(FftDesc d, const float2* __restrict__ tw, int count,
             const float* __restrict__ series, float* __restrict__ partial) {
  extern __shared__ float2 sm[];
  __shared__ double red[32];
  const int T = d.n, H = T / 2 + 1, nb = fft_buf_len(d);
  float2* bufA = sm;
  float2* bufB = sm + nb;
  float2* stw = sm + 2 * nb;
  float* acc = (float*)(stw + T);
  for (int i = threadIdx.x; i < T; i += blockDim.x) stw[i] = tw[i];
  for (int f = threadIdx.x; f < H; f += blockDim.x) acc[f] = 0.f;
  for (int s = blockIdx.x; s < count; s += gridDim.x) {
    const float* x = series + (size_t)s * T;
    double m = 0.0;
    for (int i = threadIdx.x; i < T; i += blockDim.x) m += x[i];
    for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    double tot = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
    const float mean = (float)(tot / T);
    for (int i = threadIdx.x; i < T; i += blockDim.x) bufA[i] = make_float2(x[i] - mean, 0.f);
    __syncthreads();
    const float2* res = fft_smem(bufA, bufB, d, stw, 1, nb, 1, false);
    __syncthreads();
    for (int f = threadIdx.x; f < H; f += blockDim.x) {
      const float2 v = res[f];
      acc[f] += v.x * v.x + v.y * v.y;
    }
    __syncthreads();
  }
  for (int f = threadIdx.x; f < H; f += blockDim.x) partial[(size_t)blockIdx.x * H + f] = acc[f];
}

__global__ void k_psd_reduce(int H, int G, double scale, const float* __restrict__ partial,
                             float* __restrict__ psd) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= H) return;
  double s = 0.0;
  for (int b = 0; b < G; ++b) s += partial[(size_t)b * H + f];
  psd[f] = (float)(s * scale);
}

static int psd_blocks(int count) { return std::max(1, std::min(count, 2 * 152)); }
}  // namespace pt

extern "C" size_t pt_temporal_psd_workspace_bytes(const pt_grid* g, int count) {
  if (!g || count < 1) return 0;
  return (size_t)psd_blocks(count) * (g->ns / 2 + 1) * sizeof(float);
}

extern "C" int pt_temporal_psd(const pt_grid* g, int count, const float* series, double dt,
                               float* psd, void* work, size_t work_bytes, void* stream) {
  if (int rc = check_grid(g, "pt_temporal_psd")) return rc;
  if (count < 1 || !(dt > 0)) return fail(PT_ERR_ARG, "pt_temporal_psd: bad count or dt");
  if (!series || !psd) return fail(PT_ERR_ARG, "pt_temporal_psd: NULL pointer");
  if (!work || work_bytes < pt_temporal_psd_workspace_bytes(g, count))
    return fail(PT_ERR_ARG, "pt_temporal_psd: workspace too small");
  const int T = g->ns, H = T / 2 + 1, G = psd_blocks(count);
  const size_t smem = (size_t)(2 * fft_buf_len(g->desc) + T) * sizeof(float2) +
                      (size_t)H * sizeof(float);
  if (smem > 220 * 1024) return fail(PT_ERR_UNSUPPORTED, "pt_temporal_psd: series longer than 8192");
  if (int rc = set_smem(k_psd_series, smem, "k_psd_series")) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  {
    ProfScope ps("k_psd_series", s);
    k_psd_series<<<G, kThreads, smem, s>>>(g->desc, g->tw, count, series, (float*)work);
  }
  k_psd_reduce<<<(H + 127) / 128, 128, 0, s>>>(H, G, 2.0 * dt / T / count, (const float*)work, psd);
  count_launch(2);
  return check_launch("pt_temporal_psd");
}
