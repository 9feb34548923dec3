// Batched 3D real FFTs with fused spectral operators, and 1D spectral
// derivatives, for periodic N^3 grids (N in {16,32,48,64,96,128,192,256}).
//
// These replace AccFFT's accfft_execute_r2c_t / accfft_execute_c2r_t /
// accfft_grad_t / accfft_divergence_t at the reference's call sites
// (src/CLAIRE.cpp:2622, 2662, 2695, 3243, 3261, 3911, 3949, 3984;
// src/Regularization*.cpp) and the diagonal "Hadamard" loops that follow
// them (e.g. src/RegularizationH2.cpp:212-244).
//
// 3D transform = three passes over HBM:
//   rows (x3, r2c via pair packing) -> columns x2 -> x1 pencil.
// The x1 pencil pass of the forward transform, the spectral multiply and the
// x1 pass of the inverse transform are one kernel; then columns x2 (inverse)
// and rows (c2r) with a fused epilogue (store / accumulate / sum of squares).
// Spectral derivatives are separable: d/dx_k of a periodic field only needs
// the 1D transform along axis k, so gradient and divergence are one pass per
// axis over real data.
//
// A butterfly's elements go straight between global memory and registers (a
// compile-time count of independent loads per thread, 4-32 in flight).
#include <atomic>
#include <cstdio>
#include <mutex>
#include <vector>

#include "fft_engine.cuh"
#include "spectral.cuh"
#include "reduce.cuh"

namespace cb {

// ---------------------------------------------------------------------------
// twiddle tables W_N^m = exp(-2 pi i m / N), computed in double on the host
// ---------------------------------------------------------------------------
static std::mutex g_tw_mutex;
static std::vector<std::pair<long long, float2*>> g_tw;  // key: device*1024 + N

static const float2* twiddles(int n) {
  int dev = 0;
  cudaGetDevice(&dev);
  long long key = (long long)dev * 1024 + n;
  std::lock_guard<std::mutex> lock(g_tw_mutex);
  for (auto& e : g_tw)
    if (e.first == key) return e.second;
  std::vector<float2> h(n);
  for (int m = 0; m < n; ++m) {
    double a = kTwoPi * (double)m / (double)n;
    h[m] = make_float2((float)cos(a), (float)(-sin(a)));
  }
  float2* d = nullptr;
  if (cudaMalloc(&d, n * sizeof(float2)) != cudaSuccess) return nullptr;
  cudaMemcpy(d, h.data(), n * sizeof(float2), cudaMemcpyHostToDevice);
  g_tw.push_back({key, d});
  return d;
}

// Lengths with a plan on every axis, and the extra lengths the column and
// pencil passes (axes x1, x2) also take: 150 = 10 x 15 (the x2 length of the
// reference's example brains, 128 x 150 x 128).  Row passes have no plan for it:
// their R0 is a power of two (RowPlan).
bool fft_size_supported(int n) {
  switch (n) {
    case 16: case 32: case 48: case 64: case 96: case 128: case 192: case 256: return true;
    default: return false;
  }
}

bool fft_col_size_supported(int n) { return fft_size_supported(n) || n == 150; }

// Columns per CTA of the column kernels; variant bit 1 selects the alternative
// count the autotuner tries.
template <int N> struct ColLines {
  static constexpr int base = N <= 128 ? 32 : 16;
  static constexpr int alt = N <= 128 ? 16 : (N == 192 ? 32 : 16);
};

// Packed lines (row pairs) per CTA of the row kernels: a power of two P with
// one thread per A butterfly (P * R1), 256 threads at most (128: variant bit 1).
constexpr int row_pairs(int r1, int v) {
  int p = 1;
  while (2 * p * r1 <= ((v & 2) ? 128 : 256)) p *= 2;
  return p;
}

// Row kernels (bound by global traffic: three 256^3 fields 68 us r2c and 70 us
// c2r against a floor of 62; 150 and 165 us when rows were transposed through
// padded shared memory on the way in and out; 128^3: 12.4 and 11.4 against 20
// and 21): a warp's lanes are neighbouring butterflies of a few lines.  The
// shared layout is y[line, k0, j] at line * PL + k0 * PK + j; 64-bit accesses are
// served by half-warps.  A (lanes over j, then lines) has no bank conflicts, as
// PL = R1 (mod 16 float2); B (lanes over k0, odd PK) has none with R0 = 16 and at
// 4 x 4, 4 x 12 and 8 x 8, and two-way ones in the other plans with R0 < 16, where
// the lines of a half-warp meet.  The twiddles tw[j k0] take 1.1 to 2.2
// wavefronts a half-warp on average, 8 at worst (R0 = 16, j a multiple of 8).
// Counted at 128^3 (16 x 8): 25% of r2c's shared wavefronts, 18% of c2r's and 22%
// of the derivative's are conflicts, all of them twiddles.
template <int N, int V> struct RowCfg {
  static constexpr int R0 = RowPlan<N, V>::R0, R1 = RowPlan<N, V>::R1;
  static constexpr int P = row_pairs(R1, V), T = P * R1;
  static constexpr int PK = R1 + 1;
  static constexpr int PL = R0 * PK + ((R1 - R0 * PK) % 16 + 16) % 16;
  static constexpr int NH = N / 2 + 1;
  static constexpr size_t smem = (size_t)(P * PL + N) * sizeof(float2);
  static_assert(T % 32 == 0 && (P * R0) % 32 == 0 && R1 % 2 == 0 && (R0 & (R0 - 1)) == 0, "whole warps of partners");
};

// Column kernels are bound by global traffic (each pass reads and writes its
// spectra once) once their instructions and barriers are few.  Lanes run over
// adjacent columns in both butterflies, so
// every global access is a run of C float2 and every shared access a run of
// 16 consecutive float2 per half-warp (64-bit accesses are served by half-warps):
// no bank conflicts by the layout at pitch C (counted at 128^3: 6% of the
// wavefronts, 11% with the pencil's symbols).  The CTA has one thread per A
// butterfly (C * R1), 256 at most.
template <int N, int V = 0> struct ColCfg {
  static constexpr int C = (V & 2) ? ColLines<N>::alt : ColLines<N>::base;
  static constexpr int R0 = Plan<N, V>::R0, R1 = Plan<N, V>::R1;
  static constexpr int T = C * R1 >= 256 ? 256 : (C * R1 + 31) / 32 * 32;
  static constexpr int B = N * C;  // float2s of one exchange buffer
  static_assert(T % C == 0, "a thread keeps its column");
};

__host__ __device__ inline bool epi_reduces(int epi) {
  return epi == EPI_SUMSQ || epi == EPI_STORE_DOT || epi == EPI_ADD_DOT;
}

// ---------------------------------------------------------------------------
// rows (x3).  Two real rows a, b (2p and 2p + 1) are packed as z = a + i b.
// Elements go straight between global memory and the A butterfly's registers:
// the lanes of a line cover R1 consecutive floats, so with R1 = 8 every 32-byte
// sector of an access is used whole.
// ---------------------------------------------------------------------------
template <class F>
CB_DEVICE void rows_a(const float* __restrict__ ra, bool ok, int p, int j, float2* S) {
  const float* rb = ra + F::R0 * F::R1;
  fft_a<F::R0, F::R1, false>(
      j, [&](int e) { return ok ? make_float2(__ldg(ra + e), __ldg(rb + e)) : make_float2(0.f, 0.f); },
      [&](int k0, float2 v) { S[p * F::PL + k0 * F::PK + j] = v; });
}

// Inverse A butterfly and the epilogue: value e of row a / b is al times the
// real / imaginary part; stored, added to dst or to `oth`, or squared and summed
// (returned), with the product with `oth` summed for the dot epilogues.  Old
// values of a group of elements are loaded before any of them is stored.
template <class F>
CB_DEVICE double rows_out(float* __restrict__ da, const float* __restrict__ oa, bool ok, int p, int j,
                          const float2* S, int epi, float al) {
  constexpr int R0 = F::R0, R1 = F::R1, N = R0 * R1, G = R0 < 8 ? R0 : 8;
  float2 v[R0];
#pragma unroll
  for (int k0 = 0; k0 < R0; ++k0) v[k0] = S[p * F::PL + k0 * F::PK + j];
  Dft<R0, true>::run(v);
  double acc = 0.0;
  if (!ok) return acc;
  if (epi == EPI_STORE) {
#pragma unroll
    for (int r = 0; r < R0; ++r) {
      da[j + R1 * r] = al * v[r].x;
      da[N + j + R1 * r] = al * v[r].y;
    }
    return acc;
  }
  if (epi == EPI_SUMSQ) {
#pragma unroll
    for (int r = 0; r < R0; ++r) {
      const float x = al * v[r].x, y = al * v[r].y;
      acc += (double)x * (double)x + (double)y * (double)y;
    }
    return acc;
  }
  const bool add = epi != EPI_STORE_DOT, dot = epi == EPI_STORE_DOT || epi == EPI_ADD_DOT;
  const float* src = epi == EPI_SUM ? oa : da;
#pragma unroll
  for (int r0 = 0; r0 < R0; r0 += G) {
    float2 old[G], oth[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int e = j + R1 * (r0 + i);
      old[i] = add ? make_float2(src[e], src[N + e]) : make_float2(0.f, 0.f);
      oth[i] = dot ? make_float2(oa[e], oa[N + e]) : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int e = j + R1 * (r0 + i);
      const float x = add ? old[i].x + al * v[r0 + i].x : al * v[r0 + i].x;
      const float y = add ? old[i].y + al * v[r0 + i].y : al * v[r0 + i].y;
      da[e] = x;
      da[N + e] = y;
      if (dot) acc += (double)x * (double)oth[i].x + (double)y * (double)oth[i].y;
    }
  }
  return acc;
}

CB_DEVICE float2 shfl2(float2 v, int lane) {
  return make_float2(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
}

// Lane that holds B butterfly (R0 - k0) mod R0 of this lane's line: the
// butterflies of a line sit in R0 neighbouring lanes of one warp.
template <int R0>
CB_DEVICE int mirror_lane(int k0) {
  return (int)(threadIdx.x & 31 & ~(R0 - 1)) | ((R0 - k0) & (R0 - 1));
}

// r2c: after the complex FFT Z of a row pair, A[k] = (Z[k] + conj Z[N-k]) / 2,
// B[k] = (Z[k] - conj Z[N-k]) / 2i.  Z[N-k] is in the mirror lane's registers,
// element R1 - 1 - k1 (butterfly 0 mirrors itself, element R1 - k1).
template <int N, int V>
__global__ void __launch_bounds__(RowCfg<N, V>::T, 1024 / RowCfg<N, V>::T)
    k_r2c_rows(const float* __restrict__ in, long long ip, long long ifs, float2* __restrict__ out, long long op,
               long long ofs, int nrows, const float2* __restrict__ twg, const int* __restrict__ active) {
  using F = RowCfg<N, V>;
  constexpr int R0 = F::R0, R1 = F::R1, NH = F::NH;
  if (active && !active[blockIdx.z]) return;
  extern __shared__ __align__(16) float2 sm2[];
  float2* tw = sm2 + F::P * F::PL;
  const int row0 = blockIdx.x * 2 * F::P;
  load_twiddles<N, F::T>(tw, twg);
  {
    const int p = threadIdx.x / R1, j = threadIdx.x % R1, row = row0 + 2 * p;
    const float* src = in + blockIdx.z * ip + blockIdx.y * ifs + (long long)row * N;
    rows_a<F>(src, row < nrows, p, j, sm2);
  }
  __syncthreads();
  float2* dst = out + blockIdx.z * op + blockIdx.y * ofs;
  for (int u = threadIdx.x; u < F::P * R0; u += F::T) {
    const int p = u / R0, k0 = u % R0, row = row0 + 2 * p;
    float2 v[R1];
    fft_b<R0, R1, false>(k0, tw, v, [&](int j) { return sm2[p * F::PL + k0 * F::PK + j]; });
    const int lane = mirror_lane<R0>(k0);
    const bool ok = row < nrows;
    float2* da = dst + (long long)row * NH + k0;
#pragma unroll
    for (int k1 = 0; k1 < R1 / 2; ++k1) {
      float2 m = shfl2(v[R1 - 1 - k1], lane);
      if (k0 == 0) m = v[k1 == 0 ? 0 : R1 - k1];
      const float2 z = v[k1];
      if (ok) {
        da[R0 * k1] = make_float2(0.5f * (z.x + m.x), 0.5f * (z.y - m.y));
        da[NH + R0 * k1] = make_float2(0.5f * (z.y + m.y), -0.5f * (z.x - m.x));
      }
    }
    if (ok && k0 == 0) {  // Nyquist
      da[N / 2] = make_float2(v[R1 / 2].x, 0.f);
      da[NH + N / 2] = make_float2(v[R1 / 2].y, 0.f);
    }
  }
}

// c2r with epilogue: Z[k] = A[k] + i B[k], Z[N-k] = conj(A[k]) + i conj(B[k])
// handed to the mirror lane; the imaginary parts of the DC and Nyquist bins
// are ignored (the c2r convention of FFTW / pocketfft).
template <int N, int V>
__global__ void __launch_bounds__(RowCfg<N, V>::T, 1024 / RowCfg<N, V>::T)
    k_c2r_rows(const float2* __restrict__ in, long long ip, long long ifs, float* __restrict__ out, long long op,
               long long ofs, int nrows, const float2* __restrict__ twg, int epi, const float* __restrict__ alpha,
               double* __restrict__ partials, int nparts, const float* __restrict__ other,
               const int* __restrict__ active) {
  using F = RowCfg<N, V>;
  constexpr int R0 = F::R0, R1 = F::R1, NH = F::NH, H = R1 / 2;
  if (active && !active[blockIdx.z]) return;
  extern __shared__ __align__(16) float2 sm2[];
  float2* tw = sm2 + F::P * F::PL;
  const int row0 = blockIdx.x * 2 * F::P;
  load_twiddles<N, F::T>(tw, twg);
  __syncthreads();
  const float2* src = in + blockIdx.z * ip + blockIdx.y * ifs;
  for (int u = threadIdx.x; u < F::P * R0; u += F::T) {
    const int p = u / R0, k0 = u % R0, row = row0 + 2 * p;
    const bool ok = row < nrows;
    const float2* sa = src + (long long)row * NH + k0;
    const float2 zero = make_float2(0.f, 0.f);
    float2 v[R1], hi[H];
#pragma unroll
    for (int k1 = 0; k1 < H; ++k1) {
      v[k1] = ok ? __ldg(sa + R0 * k1) : zero;
      hi[k1] = ok ? __ldg(sa + NH + R0 * k1) : zero;
    }
    float2 nyq = zero;
    if (k0 == 0) {
      if (ok) nyq = make_float2(__ldg(sa + N / 2).x, __ldg(sa + NH + N / 2).x);
      v[0].y = hi[0].y = 0.f;
    }
#pragma unroll
    for (int k1 = 0; k1 < H; ++k1) {
      const float2 a = v[k1], b = hi[k1];
      v[k1] = make_float2(a.x - b.y, a.y + b.x);
      hi[k1] = make_float2(a.x + b.y, b.x - a.y);
    }
    const int lane = mirror_lane<R0>(k0);
#pragma unroll
    for (int k1 = 0; k1 < H; ++k1) {
      const float2 m = shfl2(hi[k1], lane);
      v[R1 - 1 - k1] = k0 ? m : (k1 + 1 < H ? hi[k1 + 1 < H ? k1 + 1 : 0] : nyq);
    }
    fft_b_inverse<R0, R1>(k0, tw, v, [&](int j, float2 x) { sm2[p * F::PL + k0 * F::PK + j] = x; });
  }
  __syncthreads();
  const int p = threadIdx.x / R1, j = threadIdx.x % R1, row = row0 + 2 * p;
  const long long off = blockIdx.z * op + blockIdx.y * ofs + (long long)row * N;
  const double acc = rows_out<F>(out + off, other + off, row < nrows, p, j, sm2, epi, alpha ? alpha[blockIdx.z] : 1.f);
  if (epi_reduces(epi))
    block_reduce_store(acc, partials + (long long)blockIdx.z * nparts, blockIdx.x + gridDim.x * blockIdx.y);
}

// ---------------------------------------------------------------------------
// complex column FFT along a strided axis, in place
// column g starts at (g / cpg) * gs + (g % cpg); elements are es apart
// ---------------------------------------------------------------------------
template <int N, bool INV, int V>
__global__ void __launch_bounds__(ColCfg<N, V>::T, 1024 / ColCfg<N, V>::T)
    k_cols(float2* __restrict__ data, long long pstr, long long fstr,
                                                           int ncols, int cpg, long long gs, int es,
                                                           const float2* __restrict__ twg,
                                                           const int* __restrict__ active) {
  using F = ColCfg<N, V>;
  constexpr int C = F::C, R0 = F::R0, R1 = F::R1;
  if (active && !active[blockIdx.z]) return;
  extern __shared__ __align__(16) float2 sm2[];
  float2* tw = sm2 + F::B;
  const int c = threadIdx.x % C;
  const int g = blockIdx.x * C + c;
  float2* col = g < ncols ? data + blockIdx.z * pstr + blockIdx.y * fstr + (long long)(g / cpg) * gs + (g % cpg)
                          : nullptr;
  load_twiddles<N, F::T>(tw, twg);
  // in place: all reads of the CTA's columns finish before the barrier, all
  // writes follow it
  for (int j = threadIdx.x / C; j < R1; j += F::T / C)
    fft_a<R0, R1, INV>(j, [&](int e) { return col ? col[e * es] : make_float2(0.f, 0.f); },
                       [&](int k0, float2 v) { sm2[(k0 * R1 + j) * C + c] = v; });
  __syncthreads();
  if (!col) return;
  for (int k0 = threadIdx.x / C; k0 < R0; k0 += F::T / C) {
    float2 v[R1];
    fft_b<R0, R1, INV>(k0, tw, v, [&](int j) { return sm2[(k0 * R1 + j) * C + c]; });
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) col[(k0 + R0 * k1) * es] = v[k1];
  }
}

// ---------------------------------------------------------------------------
// spectral symbols (src/Regularization*.cpp, src/CLAIREStokes.cpp:407-540,
// src/CLAIREDivReg.cpp:313-460, src/Preprocessing.cpp:1956-2056)
// ---------------------------------------------------------------------------
// Wavenumber data of one spectral column (x2 index i2, x3 index i3) and a
// spectral element of it along x1 (index i1).
struct ColumnK {
  float k2, k3, l2, l3;   // Nyquist-zeroed and Nyquist-kept wavenumbers
};

CB_DEVICE ColumnK column_k(int i2, int i3, const Dims& d) {
  ColumnK c;
  c.k2 = (float)wavenumber(i2, d.n2);
  c.k3 = (float)wavenumber(i3, d.n3);
  c.l2 = (float)wavenumber_keep_nyquist(i2, d.n2);
  c.l3 = (float)wavenumber_keep_nyquist(i3, d.n3);
  return c;
}

// The diagonal operators without a DiagSymbol: the regularisation functional and
// the Gaussian (one field, component index comp for H3/H3SN).
CB_DEVICE float2 apply_op1(int op, const SpecParams& q, const Dims& d, int i1, const ColumnK& ck, int comp,
                           float2 x, float s) {
  const float k1 = (float)wavenumber(i1, d.n1);
  const float kap = k1 * k1 + ck.k2 * ck.k2 + ck.k3 * ck.k3;
  switch (op) {
    case OP_REG_FUNC: {
      if (q.norm == NORM_L2) {
        const float sig = s * sqrtf(q.beta0);
        return make_float2(x.x * sig, x.y * sig);
      }
      if (q.norm == NORM_H2) {
        const float sig = s * sqrtf(q.beta0) * (-kap + sqrtf(q.beta1));
        return make_float2(x.x * sig, x.y * sig);
      }
      if (q.norm == NORM_H2SN) {
        const float sig = -s * kap;
        return make_float2(x.x * sig, x.y * sig);
      }
      // H3 / H3SN: separate multipliers on real and imaginary parts
      const float kc = comp == 0 ? k1 : (comp == 1 ? ck.k2 : ck.k3);
      const float a = kc * (-kap);
      float mre, mim;
      if (q.norm == NORM_H3) {
        const float sb0 = sqrtf(q.beta0), sb1 = sqrtf(q.beta1);
        mre = s * sb0 * (a + sb1);
        mim = s * sb0 * (-a + sb1);
      } else {
        mre = s * a;
        mim = -s * a;
      }
      return make_float2(x.x * mre, x.y * mim);
    }
    case OP_GAUSS: {
      const float l1 = (float)wavenumber_keep_nyquist(i1, d.n1);
      const float c1 = q.sigma[0] * (float)(kTwoPi / d.n1), c2 = q.sigma[1] * (float)(kTwoPi / d.n2),
                  c3 = q.sigma[2] * (float)(kTwoPi / d.n3);
      const float sik = expf(-0.5f * (l1 * l1 * c1 * c1 + ck.l2 * ck.l2 * c2 * c2 + ck.l3 * ck.l3 * c3 * c3));
      return make_float2(x.x * s * sik, x.y * s * sik);
    }
    default:
      return make_float2(x.x * s, x.y * s);
  }
}

// Coupled 3-field projections b -> F^-1(-c k (k . b^)/kappa): Stokes keeps the
// Nyquist index in kappa, the relaxed model zeroes it and scales by
// c = (beta_v (beta_w (kappa + 1))^-1 + 1)^-1.
CB_DEVICE void apply_op3(int op, const SpecParams& q, const Dims& d, int i1, const ColumnK& ck, float2 (&x)[3],
                         float s) {
  const float k1 = (float)wavenumber(i1, d.n1);
  const float kap = k1 * k1 + ck.k2 * ck.k2 + ck.k3 * ck.k3;
  float kl, c = 1.f;
  if (op == OP_LERAY) {
    const float l1 = (float)wavenumber_keep_nyquist(i1, d.n1);
    kl = l1 * l1 + ck.l2 * ck.l2 + ck.l3 * ck.l3;
  } else {
    kl = kap;
    const float opik = 1.f / (q.beta2 * (kap + 1.f));
    c = 1.f / (q.beta0 * opik + 1.f);
  }
  const float L = (kl == 0.f) ? -1.f : -1.f / kl;
  const float2 kd = make_float2(k1 * x[0].x + ck.k2 * x[1].x + ck.k3 * x[2].x,
                                k1 * x[0].y + ck.k2 * x[1].y + ck.k3 * x[2].y);
  const float g = s * c * L;
  x[0] = make_float2(g * k1 * kd.x, g * k1 * kd.y);
  x[1] = make_float2(g * ck.k2 * kd.x, g * ck.k2 * kd.y);
  x[2] = make_float2(g * ck.k3 * kd.x, g * ck.k3 * kd.y);
}

// The real diagonal operators that run once per Krylov iteration, reduced to
// sig = s coef (t + b1) or s / (coef (t + b1)) with t a power of kappa, so that
// one symbol costs a few instructions per element:
//   gradient   L2 beta0, H1SN hd beta0 kappa, H1 hd beta0 (kappa + beta1),
//              H2SN hd beta0 kappa^2, H2 beta0 (kappa^2 + beta1),
//              H3SN beta0 kappa^3, H3 beta0 (kappa^3 + beta1)
//   inverse    1 / the same without hd, the seminorms' symbol beta0 at kappa = 0;
//              its square root for the square-root inverse
struct DiagSymbol {
  float s, coef, b1;
  int power;
  bool inv, sq, keep0;  // keep0: the inverse seminorms take the symbol beta0 at kappa = 0
  CB_DEVICE DiagSymbol(int op, const SpecParams& q, float scale) {
    s = scale;
    inv = op != OP_REG_GRAD;
    sq = op == OP_REG_SQRTINV;
    const bool h1 = q.norm == NORM_H1 || q.norm == NORM_H1SN, h2 = q.norm == NORM_H2 || q.norm == NORM_H2SN;
    power = q.norm == NORM_L2 ? 0 : (h1 ? 1 : (h2 ? 2 : 3));
    const bool semi = q.norm == NORM_H1SN || q.norm == NORM_H2SN || q.norm == NORM_H3SN;
    b1 = (semi || q.norm == NORM_L2) ? 0.f : q.beta1;
    // the norms whose gradient symbol has the factor hd
    const bool hd = q.norm == NORM_H1SN || q.norm == NORM_H1 || q.norm == NORM_H2SN;
    coef = (!inv && hd) ? q.hd * q.beta0 : q.beta0;
    keep0 = inv && semi;
  }
  CB_DEVICE float operator()(float kap) const {
    const float k2 = kap * kap;
    float t = power == 1 ? kap : (power == 2 ? k2 : (power == 3 ? k2 * kap : 1.f));
    t += b1;
    if (keep0 && kap == 0.f) t = 1.f;
    const float o = coef * t;
    if (!inv) return s * o;
    return s / (sq ? sqrtf(o) : o);
  }
};

// x1 pencil: forward FFT along x1, a diagonal symbol, inverse FFT, of `nf`
// fields one after another in one CTA.  The symbol is the same for every field
// (DIAG: DiagSymbol, computed once per element and kept in shared memory, each
// entry read by the thread that wrote it: its division costs about as much as
// a radix-8 butterfly); otherwise the general apply_op1, one field per CTA
// (grid.y, nf = 1).  Three 256^3 spectra: 98-106 us, 175 with four staged
// passes through shared memory and the symbol per field (traffic floor 62 us);
// 128^3: 16 against 22.
template <int N, int V, bool DIAG>
__global__ void __launch_bounds__(ColCfg<N, V>::T,
                                  (DIAG ? (ColCfg<N, V>::R1 > 12 ? 768 : 1024) : 512) / ColCfg<N, V>::T)
    k_pencil1(float2* __restrict__ spec, long long pstr, long long fstr, int nf, Dims d, int op, float s,
              const SpecParams* __restrict__ params, SpecParams one, const float2* __restrict__ twg,
              const int* __restrict__ active) {
  using F = ColCfg<N, V>;
  constexpr int C = F::C, R0 = F::R0, R1 = F::R1, STEP = F::T / C;
  if (active && !active[blockIdx.z]) return;
  extern __shared__ __align__(16) float2 sm2[];
  float2* tw = sm2 + F::B;
  const int n3h = d.n3 / 2 + 1;
  const int ncols = d.n2 * n3h;
  const int c = threadIdx.x % C, u0 = threadIdx.x / C;
  const int g = blockIdx.x * C + c;
  const bool ok = g < ncols;
  float2* col = spec + blockIdx.z * pstr + blockIdx.y * fstr + (ok ? g : 0);
  float* sig = reinterpret_cast<float*>(tw + N);
  load_twiddles<N, F::T>(tw, twg);
  const SpecParams q = params ? params[blockIdx.z] : one;
  const ColumnK ck = column_k(g / n3h, g % n3h, d);
  if constexpr (DIAG) {
    const DiagSymbol sym(op, q, s);
    const float kap23 = ck.k2 * ck.k2 + ck.k3 * ck.k3;
    for (int k0 = u0; k0 < R0; k0 += STEP)
#pragma unroll 4
      for (int k1 = 0; k1 < R1; ++k1) {
        const float w1 = (float)wavenumber(k0 + R0 * k1, N);
        sig[(k0 * R1 + k1) * C + c] = sym(w1 * w1 + kap23);
      }
  }
#pragma unroll 1
  for (int f = 0; f < nf; ++f, col += fstr) {
    // opaque per field: element offsets and symbols hoisted out of this loop
    // would not fit in registers
    int es = ncols;
    float sf = s;
    asm volatile("" : "+r"(es), "+f"(sf));
    for (int j = u0; j < R1; j += STEP)
      fft_a<R0, R1, false>(j, [&](int e) { return ok ? col[e * es] : make_float2(0.f, 0.f); },
                           [&](int k0, float2 v) { sm2[(k0 * R1 + j) * C + c] = v; });
    __syncthreads();
    // the butterfly's inputs and outputs are the same R1 entries: in place
    for (int k0 = u0; k0 < R0; k0 += STEP) {
      float2 v[R1];
      fft_b<R0, R1, false>(k0, tw, v, [&](int j) { return sm2[(k0 * R1 + j) * C + c]; });
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) {
        if constexpr (DIAG) {
          const float w = sig[(k0 * R1 + k1) * C + c];
          v[k1] = make_float2(v[k1].x * w, v[k1].y * w);
        } else {
          v[k1] = apply_op1(op, q, d, k0 + R0 * k1, ck, blockIdx.y, v[k1], sf);
        }
      }
      fft_b_inverse<R0, R1>(k0, tw, v, [&](int j, float2 x) { sm2[(k0 * R1 + j) * C + c] = x; });
    }
    __syncthreads();
    for (int j = u0; j < R1; j += STEP)
      fft_a_inverse<R0, R1>(j, [&](int k0) { return sm2[(k0 * R1 + j) * C + c]; },
                            [&](int e, float2 v) {
                              if (ok) col[e * es] = v;
                            });
    // the next field's A butterfly j overwrites what this thread's inverse A
    // butterfly j just read: no barrier in between
  }
}

// x1 pencil with the three fields in one CTA (coupled projections): the three
// spectra of an element meet in one thread's registers (128^3: 14 us, 24 when
// they were staged in shared memory between the transforms).
template <int N, int V>
__global__ void __launch_bounds__(ColCfg<N, V>::T, 512 / ColCfg<N, V>::T)
    k_pencil3(float2* __restrict__ spec, long long pstr,
                                                              long long fstr, Dims d, int op, float s,
                                                              const SpecParams* __restrict__ params,
                                                              SpecParams one, const float2* __restrict__ twg,
                                                              const int* __restrict__ active) {
  using F = ColCfg<N, V>;
  constexpr int C = F::C, R0 = F::R0, R1 = F::R1;
  if (active && !active[blockIdx.z]) return;
  extern __shared__ __align__(16) float2 sm2[];
  float2* tw = sm2 + 3 * F::B;
  const int n3h = d.n3 / 2 + 1;
  const int ncols = d.n2 * n3h;
  const int c = threadIdx.x % C, u0 = threadIdx.x / C;
  const int g = blockIdx.x * C + c;
  float2* col = g < ncols ? spec + blockIdx.z * pstr + g : nullptr;
  load_twiddles<N, F::T>(tw, twg);
#pragma unroll 1
  for (int f = 0; f < 3; ++f) {
    const float2* cf = col + f * fstr;
    float2* S = sm2 + f * F::B;
    for (int j = u0; j < R1; j += F::T / C)
      fft_a<R0, R1, false>(j, [&](int e) { return col ? cf[e * ncols] : make_float2(0.f, 0.f); },
                           [&](int k0, float2 v) { S[(k0 * R1 + j) * C + c] = v; });
  }
  __syncthreads();
  const SpecParams q = params ? params[blockIdx.z] : one;
  const ColumnK ck = column_k(g / n3h, g % n3h, d);
  for (int k0 = u0; k0 < R0; k0 += F::T / C) {
    float2 v[3][R1];
#pragma unroll
    for (int f = 0; f < 3; ++f)
      fft_b<R0, R1, false>(k0, tw, v[f], [&](int j) { return sm2[f * F::B + (k0 * R1 + j) * C + c]; });
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) {
      float2 x[3] = {v[0][k1], v[1][k1], v[2][k1]};
      apply_op3(op, q, d, k0 + R0 * k1, ck, x, s);
      v[0][k1] = x[0];
      v[1][k1] = x[1];
      v[2][k1] = x[2];
    }
#pragma unroll
    for (int f = 0; f < 3; ++f)
      fft_b_inverse<R0, R1>(k0, tw, v[f], [&](int j, float2 x) { sm2[f * F::B + (k0 * R1 + j) * C + c] = x; });
  }
  __syncthreads();
  if (!col) return;
#pragma unroll 1
  for (int f = 0; f < 3; ++f) {
    float2* cf = col + f * fstr;
    const float2* S = sm2 + f * F::B;
    for (int j = u0; j < R1; j += F::T / C)
      fft_a_inverse<R0, R1>(j, [&](int k0) { return S[(k0 * R1 + j) * C + c]; },
                            [&](int e, float2 v) { cf[e * ncols] = v; });
  }
}

// ---------------------------------------------------------------------------
// 1D spectral derivative of real fields.  Two real lines a, b are packed as
// a + i b; i*k/N with the Nyquist wavenumber zeroed is Hermitian, so the real
// and imaginary parts of the result are the derivatives of a and b.
// AXIS 2: rows (x3, contiguous).  AXIS 0/1: columns along x1 / x2.
// ---------------------------------------------------------------------------
// i k / N on the outputs k0 + R0 k1 of a B butterfly
template <int N, int R0, int R1>
CB_DEVICE void mul_ik(int k0, float2 (&v)[R1]) {
#pragma unroll
  for (int k1 = 0; k1 < R1; ++k1) {
    const float k = (float)wavenumber(k0 + R0 * k1, N) * (1.f / (float)N);
    v[k1] = make_float2(-k * v[k1].y, k * v[k1].x);
  }
}

template <int N, int V>
__global__ void __launch_bounds__(RowCfg<N, V>::T, 1024 / RowCfg<N, V>::T)
    k_deriv_rows(const float* __restrict__ in, long long ip, long long ifs, float* __restrict__ out, long long op,
                 long long ofs, int nrows, const float2* __restrict__ twg, int epi, double* __restrict__ partials,
                 int nparts, const int* __restrict__ active) {
  using F = RowCfg<N, V>;
  constexpr int R0 = F::R0, R1 = F::R1;
  if (active && !active[blockIdx.z]) return;
  extern __shared__ __align__(16) float2 sm2[];
  float2* tw = sm2 + F::P * F::PL;
  const int row0 = blockIdx.x * 2 * F::P;
  const int p = threadIdx.x / R1, j = threadIdx.x % R1, row = row0 + 2 * p;
  load_twiddles<N, F::T>(tw, twg);
  rows_a<F>(in + blockIdx.z * ip + blockIdx.y * ifs + (long long)row * N, row < nrows, p, j, sm2);
  __syncthreads();
  for (int u = threadIdx.x; u < F::P * R0; u += F::T) {
    const int k0 = u % R0;
    float2* S = sm2 + (u / R0) * F::PL + k0 * F::PK;
    float2 v[R1];
    fft_b<R0, R1, false>(k0, tw, v, [&](int i) { return S[i]; });
    mul_ik<N, R0, R1>(k0, v);
    fft_b_inverse<R0, R1>(k0, tw, v, [&](int i, float2 x) { S[i] = x; });
  }
  __syncthreads();
  const double acc = rows_out<F>(out + blockIdx.z * op + blockIdx.y * ofs + (long long)row * N, nullptr,
                                 row < nrows && (out || epi == EPI_SUMSQ), p, j, sm2, epi, 1.f);
  if (epi == EPI_SUMSQ)
    block_reduce_store(acc, partials + (long long)blockIdx.z * nparts, blockIdx.x + gridDim.x * blockIdx.y);
}

// Column derivative: the thread's packed line holds the real columns 2p (real
// part) and 2p + 1 (imaginary part).  n3 is even, so the two are neighbours in
// memory: one 8-byte access each way when the arrays are 8-byte aligned
// (vin / vout), two 4-byte ones otherwise.  i k / N is applied in registers
// between the forward and the inverse B butterfly.  One 128^3 field: 7.4 us,
// 9.1 with 4-byte accesses and four staged passes.
template <int N, int V>
__global__ void __launch_bounds__(ColCfg<N, V>::T, 1024 / ColCfg<N, V>::T)
    k_deriv_cols(const float* __restrict__ in, long long ip,
                                                                 long long ifs, float* __restrict__ out,
                                                                 long long op, long long ofs, int ncols, int cpg,
                                                                 long long gs, int es,
                                                                 const float2* __restrict__ twg, int epi, bool vin,
                                                                 bool vout, double* __restrict__ partials,
                                                                 int nparts, const int* __restrict__ active) {
  using F = ColCfg<N, V>;
  constexpr int C = F::C, R0 = F::R0, R1 = F::R1;
  if (active && !active[blockIdx.z]) return;
  extern __shared__ __align__(16) float2 sm2[];
  float2* tw = sm2 + F::B;
  const int c = threadIdx.x % C, u0 = threadIdx.x / C;
  const int g = 2 * (blockIdx.x * C + c);
  const bool ok = g < ncols;
  const long long off = ok ? (long long)(g / cpg) * gs + (g % cpg) : 0;
  const float* src = in + blockIdx.z * ip + blockIdx.y * ifs + off;
  float* dst = out ? out + blockIdx.z * op + blockIdx.y * ofs + off : nullptr;
  load_twiddles<N, F::T>(tw, twg);
  auto ld = [&](int e) {
    if (!ok) return make_float2(0.f, 0.f);
    const float* p = src + e * es;
    return vin ? __ldg(reinterpret_cast<const float2*>(p)) : make_float2(__ldg(p), __ldg(p + 1));
  };
  for (int j = u0; j < R1; j += F::T / C)
    fft_a<R0, R1, false>(j, ld, [&](int k0, float2 v) { sm2[(k0 * R1 + j) * C + c] = v; });
  __syncthreads();
  for (int k0 = u0; k0 < R0; k0 += F::T / C) {
    float2 v[R1];
    fft_b<R0, R1, false>(k0, tw, v, [&](int j) { return sm2[(k0 * R1 + j) * C + c]; });
    mul_ik<N, R0, R1>(k0, v);
    fft_b_inverse<R0, R1>(k0, tw, v, [&](int j, float2 x) { sm2[(k0 * R1 + j) * C + c] = x; });
  }
  __syncthreads();
  double acc = 0.0;
  if (ok && (dst || epi == EPI_SUMSQ)) {
    for (int j = u0; j < R1; j += F::T / C)
      fft_a_inverse<R0, R1>(j, [&](int k0) { return sm2[(k0 * R1 + j) * C + c]; },
                            [&](int e, float2 v) {
                              if (epi == EPI_SUMSQ) {  // no output array needed
                                acc += (double)v.x * (double)v.x + (double)v.y * (double)v.y;
                                return;
                              }
                              float* p = dst + e * es;
                              if (vout) {
                                float2* p2 = reinterpret_cast<float2*>(p);
                                if (epi == EPI_ADD) {
                                  const float2 o = *p2;
                                  v = make_float2(o.x + v.x, o.y + v.y);
                                }
                                *p2 = v;
                              } else {
                                p[0] = epi == EPI_ADD ? p[0] + v.x : v.x;
                                p[1] = epi == EPI_ADD ? p[1] + v.y : v.y;
                              }
                            });
  }
  if (epi == EPI_SUMSQ)
    block_reduce_store(acc, partials + (long long)blockIdx.z * nparts, blockIdx.x + gridDim.x * blockIdx.y);
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
// nbuf exchange buffers, the twiddles and (symbol) the pencil's symbol table
template <int N, int V> static size_t col_smem(int nbuf, bool symbol = false) {
  return (size_t)(nbuf * ColCfg<N, V>::B + N) * sizeof(float2) + (symbol ? ColCfg<N, V>::B * sizeof(float) : 0);
}

template <typename K> static int set_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024 && !g_graph_capture) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}

static bool aligned16(const void* p) { return (reinterpret_cast<unsigned long long>(p) & 15) == 0; }

#define CB_DISPATCH_N(n, CALL)                         \
  switch (n) {                                         \
    case 16: { constexpr int NN = 16; CALL; } break;   \
    case 32: { constexpr int NN = 32; CALL; } break;   \
    case 48: { constexpr int NN = 48; CALL; } break;   \
    case 64: { constexpr int NN = 64; CALL; } break;   \
    case 96: { constexpr int NN = 96; CALL; } break;   \
    case 128: { constexpr int NN = 128; CALL; } break; \
    case 192: { constexpr int NN = 192; CALL; } break; \
    case 256: { constexpr int NN = 256; CALL; } break; \
    default: return (int)cudaErrorInvalidValue;        \
  }

// ---------------------------------------------------------------------------
// FFT variants (plan factorization x lines per CTA) chosen per grid size.
// The table is process-wide; the autotuner (fft_autotune) or
// set_fft_variant change it, and every launch reads it, so it must only
// change while no transform of that size is in flight (contexts tune when
// they are created, before any of their work).
// ---------------------------------------------------------------------------
static std::atomic<int> g_fft_var[9];

static int size_slot(int n) {
  switch (n) {
    case 16: return 0;
    case 32: return 1;
    case 48: return 2;
    case 64: return 3;
    case 96: return 4;
    case 128: return 5;
    case 192: return 6;
    case 256: return 7;
    case 150: return 8;
    default: return -1;
  }
}

int fft_variant_candidates(int n, int* out) {
  const int k = size_slot(n);
  if (k < 0) return 0;
  if (n == 16 || n == 256) {  // one factorization: line counts only
    out[0] = 0;
    out[1] = 2;
    return 2;
  }
  if (n == 150) {  // column passes only, one line count: radix orders only
    out[0] = 0;
    out[1] = 1;
    return 2;
  }
  for (int v = 0; v < 4; ++v) out[v] = v;
  return 4;
}

int fft_variant(int n) {
  const int k = size_slot(n);
  return k < 0 ? 0 : g_fft_var[k].load(std::memory_order_relaxed);
}

int set_fft_variant(int n, int v) {
  int cand[4];
  const int nc = fft_variant_candidates(n, cand);
  for (int i = 0; i < nc; ++i)
    if (cand[i] == v) {
      g_fft_var[size_slot(n)].store(v, std::memory_order_relaxed);
      return 0;
    }
  return (int)cudaErrorInvalidValue;
}

#define CB_V(VV_, CALL) \
  case VV_: {           \
    constexpr int VV = VV_; \
    CALL;               \
  } break;
#define CB_VSW4(N_, CALL)                                                                  \
  {                                                                                        \
    constexpr int NN = N_;                                                                 \
    switch (fft_variant(N_)) { CB_V(0, CALL) CB_V(1, CALL) CB_V(2, CALL) CB_V(3, CALL)     \
      default: return (int)cudaErrorInvalidValue; }                                        \
  } break;
#define CB_VSW2(N_, CALL)                                                                  \
  {                                                                                        \
    constexpr int NN = N_;                                                                 \
    switch (fft_variant(N_)) { CB_V(0, CALL) CB_V(2, CALL)                                 \
      default: return (int)cudaErrorInvalidValue; }                                        \
  } break;
#define CB_VSW01(N_, CALL)                                                                 \
  {                                                                                        \
    constexpr int NN = N_;                                                                 \
    switch (fft_variant(N_)) { CB_V(0, CALL) CB_V(1, CALL)                                 \
      default: return (int)cudaErrorInvalidValue; }                                        \
  } break;
// CB_DISPATCH_N with the size's current variant as the constexpr VV.  It is read
// once: kernel, grid and the count of partials of a launch belong together.
#define CB_DISPATCH_NV(n, CALL)      \
  switch (n) {                       \
    case 16: CB_VSW2(16, CALL)       \
    case 32: CB_VSW4(32, CALL)       \
    case 48: CB_VSW4(48, CALL)       \
    case 64: CB_VSW4(64, CALL)       \
    case 96: CB_VSW4(96, CALL)       \
    case 128: CB_VSW4(128, CALL)     \
    case 192: CB_VSW4(192, CALL)     \
    case 256: CB_VSW2(256, CALL)     \
    default: return (int)cudaErrorInvalidValue; \
  }
// the same for column / pencil passes, which also take 150 points
#define CB_DISPATCH_NV_COL(n, CALL)  \
  switch (n) {                       \
    case 16: CB_VSW2(16, CALL)       \
    case 32: CB_VSW4(32, CALL)       \
    case 48: CB_VSW4(48, CALL)       \
    case 64: CB_VSW4(64, CALL)       \
    case 96: CB_VSW4(96, CALL)       \
    case 128: CB_VSW4(128, CALL)     \
    case 150: CB_VSW01(150, CALL)    \
    case 192: CB_VSW4(192, CALL)     \
    case 256: CB_VSW2(256, CALL)     \
    default: return (int)cudaErrorInvalidValue; \
  }

// Partials of a reducing launch: reported through *used; an error where they do
// not fit into nparts.
static int claim_partials(int epi, const dim3& grid, const double* partials, int nparts, int* used) {
  const int count = (int)(grid.x * grid.y);
  if (used) *used = epi_reduces(epi) ? count : 0;
  if (epi_reduces(epi) && (!partials || !used || count > nparts)) return (int)cudaErrorInvalidValue;
  return 0;
}

template <int N, int V>
static int r2c_rows_impl(const float* in, long long ip, long long ifs, float2* out, long long op,
                         long long ofs, int nrows, int nf, int nprob, const int* active,
                         cudaStream_t s) {
  const float2* tw = twiddles(N);
  if (!tw) return (int)cudaErrorMemoryAllocation;
  size_t sm = RowCfg<N, V>::smem;
  int e = set_smem(k_r2c_rows<N, V>, sm);
  if (e) return e;
  dim3 grid((nrows + 2 * RowCfg<N, V>::P - 1) / (2 * RowCfg<N, V>::P), nf, nprob);
  k_r2c_rows<N, V><<<grid, RowCfg<N, V>::T, sm, s>>>(in, ip, ifs, out, op, ofs, nrows, tw, active);
  return (int)cudaGetLastError();
}

template <int N, int V>
static int c2r_rows_impl(const float2* in, long long ip, long long ifs, float* out, long long op,
                         long long ofs, int nrows, int nf, int nprob, int epi, const float* alpha,
                         double* partials, int nparts, int* used, const float* other, const int* active,
                         cudaStream_t s) {
  const float2* tw = twiddles(N);
  if (!tw) return (int)cudaErrorMemoryAllocation;
  size_t sm = RowCfg<N, V>::smem;
  dim3 grid((nrows + 2 * RowCfg<N, V>::P - 1) / (2 * RowCfg<N, V>::P), nf, nprob);
  int e = claim_partials(epi, grid, partials, nparts, used);
  if (!e) e = set_smem(k_c2r_rows<N, V>, sm);
  if (e) return e;
  k_c2r_rows<N, V><<<grid, RowCfg<N, V>::T, sm, s>>>(in, ip, ifs, out, op, ofs, nrows, tw, epi, alpha, partials,
                                            nparts, other, active);
  return (int)cudaGetLastError();
}

template <int N, bool INV, int V>
static int cols_impl(float2* data, long long pstr, long long fstr, int ncols, int cpg, long long gs,
                     long long es, int nf, int nprob, const int* active, cudaStream_t s) {
  const float2* tw = twiddles(N);
  if (!tw) return (int)cudaErrorMemoryAllocation;
  size_t sm = col_smem<N, V>(1);
  int e = set_smem(k_cols<N, INV, V>, sm);
  if (e) return e;
  dim3 grid((ncols + ColCfg<N, V>::C - 1) / ColCfg<N, V>::C, nf, nprob);
  k_cols<N, INV, V><<<grid, ColCfg<N, V>::T, sm, s>>>(data, pstr, fstr, ncols, cpg, gs, (int)es, tw, active);
  return (int)cudaGetLastError();
}

// The fields of a diagonal symbol share a CTA (and the symbol) once that leaves
// two CTAs per SM; fewer columns run one field per CTA.  One problem of three
// fields, one field per CTA against shared: 64^3 4.4 and 6.5 us, 192^3 52.3 and
// 42.7, 256^3 119 and 105; near the line sharing does not pay yet (128 x 150 x 128,
// 305 CTAs shared: 19.6 and 22.4).
static bool pencil_shares_fields(int blocks, int nprob) { return (long long)blocks * nprob >= 2 * 148; }

template <int N, int V>
static int pencil_impl(float2* spec, long long sp, long long fstr, int nprob, const Dims& d, int op,
                       const SpecParams* params, const SpecParams& one, int nin, int nout, const int* active,
                       cudaStream_t s) {
  const float2* tw = twiddles(N);
  if (!tw) return (int)cudaErrorMemoryAllocation;
  const int ncols = d.n2 * (d.n3 / 2 + 1);
  const float scale = 1.f / (float)((double)d.n1 * d.n2 * d.n3);
  const bool coupled = op == OP_LERAY || op == OP_LERAY_RELAXED;
  if (coupled ? (nin != 3 || nout != 3) : nin != nout) return (int)cudaErrorInvalidValue;
  constexpr int T = ColCfg<N, V>::T;
  const bool diag = op == OP_REG_GRAD || op == OP_REG_INV || op == OP_REG_SQRTINV;
  const int blocks = (ncols + ColCfg<N, V>::C - 1) / ColCfg<N, V>::C;
  const bool shared = diag && pencil_shares_fields(blocks, nprob);
  const dim3 grid(blocks, coupled || shared ? 1 : nin, nprob);
  const size_t sm = col_smem<N, V>(coupled ? 3 : 1, diag);
  int e = 0;
  if (coupled) {
    if ((e = set_smem(k_pencil3<N, V>, sm))) return e;
    k_pencil3<N, V><<<grid, T, sm, s>>>(spec, sp, fstr, d, op, scale, params, one, tw, active);
  } else if (diag) {
    if ((e = set_smem(k_pencil1<N, V, true>, sm))) return e;
    k_pencil1<N, V, true><<<grid, T, sm, s>>>(spec, sp, fstr, shared ? nin : 1, d, op, scale, params, one, tw, active);
  } else {
    if ((e = set_smem(k_pencil1<N, V, false>, sm))) return e;
    k_pencil1<N, V, false><<<grid, T, sm, s>>>(spec, sp, fstr, 1, d, op, scale, params, one, tw, active);
  }
  return (int)cudaGetLastError();
}

// Every axis has its own transform (rows: x3, columns: x2, pencils: x1), so
// grids need not be cubic; each axis length must have a plan.
static bool axes_supported(const Dims& d) {
  return fft_col_size_supported(d.n1) && fft_col_size_supported(d.n2) && fft_size_supported(d.n3);
}
static bool cubic_supported(const Dims& d) { return d.n1 == d.n2 && d.n2 == d.n3 && axes_supported(d); }

// Inputs of the row passes have to start on 16 bytes, which callers rely on being
// told (the kernels load single floats and would take any).
int launch_r2c3d(const float* in, long long ip, long long ifs, float2* spec, long long sp, int nf,
                 int nprob, const Dims& d, const int* active, cudaStream_t s) {
  if (!axes_supported(d) || !aligned16(in) || ((ip | ifs) & 3)) return (int)cudaErrorInvalidValue;
  const long long nc = d.nc();
  const int n3h = d.n3 / 2 + 1;
  int e = 0;
  CB_DISPATCH_NV(d.n3, e = (r2c_rows_impl<NN, VV>(in, ip, ifs, spec, sp, nc, d.n1 * d.n2, nf, nprob, active, s)));
  if (e) return e;
  // x2 columns: column g = (i1, k3) starts at i1*n2*n3h + k3, stride n3h
  CB_DISPATCH_NV_COL(d.n2, e = (cols_impl<NN, false, VV>(spec, sp, nc, d.n1 * n3h, n3h, (long long)d.n2 * n3h, n3h,
                                                nf, nprob, active, s)));
  return e;
}

int launch_pencil(float2* spec, long long sp, int nprob, const Dims& d, int op,
                  const SpecParams* dparams, int nin, int nout, const int* active, cudaStream_t s,
                  const SpecParams* one) {
  if (!axes_supported(d) || (!dparams && !one)) return (int)cudaErrorInvalidValue;
  const SpecParams q = one ? *one : SpecParams{};
  int e = 0;
  CB_DISPATCH_NV_COL(d.n1, e = (pencil_impl<NN, VV>(spec, sp, d.nc(), nprob, d, op, dparams, q, nin, nout, active, s)));
  return e;
}

// Packed lines per CTA: the smallest over the size's variants, which sizes
// reduction buffers for any of them.
static int row_lines(int n) {
  auto pairs = [](int k, int v) {
    switch (k) {
      case 16: return row_pairs((v & 1) ? RowPlan<16, 1>::R1 : RowPlan<16, 0>::R1, v);
      case 32: return row_pairs((v & 1) ? RowPlan<32, 1>::R1 : RowPlan<32, 0>::R1, v);
      case 48: return row_pairs((v & 1) ? RowPlan<48, 1>::R1 : RowPlan<48, 0>::R1, v);
      case 64: return row_pairs((v & 1) ? RowPlan<64, 1>::R1 : RowPlan<64, 0>::R1, v);
      case 96: return row_pairs((v & 1) ? RowPlan<96, 1>::R1 : RowPlan<96, 0>::R1, v);
      case 128: return row_pairs((v & 1) ? RowPlan<128, 1>::R1 : RowPlan<128, 0>::R1, v);
      case 192: return row_pairs((v & 1) ? RowPlan<192, 1>::R1 : RowPlan<192, 0>::R1, v);
      case 256: return row_pairs((v & 1) ? RowPlan<256, 1>::R1 : RowPlan<256, 0>::R1, v);
      default: return 0;
    }
  };
  int m = pairs(n, 0);
  for (int v = 1; v < 4; ++v) m = pairs(n, v) < m ? pairs(n, v) : m;
  return m;
}

static int col_lines(int n) {
  int base = 0, alt = 0;
  switch (n) {
    case 16: base = ColLines<16>::base; alt = ColLines<16>::alt; break;
    case 32: base = ColLines<32>::base; alt = ColLines<32>::alt; break;
    case 48: base = ColLines<48>::base; alt = ColLines<48>::alt; break;
    case 64: base = ColLines<64>::base; alt = ColLines<64>::alt; break;
    case 96: base = ColLines<96>::base; alt = ColLines<96>::alt; break;
    case 128: base = ColLines<128>::base; alt = ColLines<128>::alt; break;
    case 192: base = ColLines<192>::base; alt = ColLines<192>::alt; break;
    case 256: base = ColLines<256>::base; alt = ColLines<256>::alt; break;
    case 150: base = ColLines<150>::base; alt = ColLines<150>::alt; break;
    default: return 0;
  }
  return base < alt ? base : alt;
}

int c2r_partials(const Dims& d, int nf) {
  const int P = row_lines(d.n3);
  if (!P) return 0;
  const int nrows = d.n1 * d.n2;
  return ((nrows + 2 * P - 1) / (2 * P)) * nf;
}

int launch_c2r3d(float2* spec, long long sp, float* out, long long op_, long long ofs, int nf,
                 int nprob, const Dims& d, int epi, const float* alpha, double* partials, int nparts,
                 const int* active, cudaStream_t s, const float* other, int* used) {
  if ((epi == EPI_STORE_DOT || epi == EPI_ADD_DOT || epi == EPI_SUM) && !other) return (int)cudaErrorInvalidValue;
  if (!axes_supported(d)) return (int)cudaErrorInvalidValue;
  const long long nc = d.nc();
  const int n3h = d.n3 / 2 + 1;
  int e = 0;
  CB_DISPATCH_NV_COL(d.n2, e = (cols_impl<NN, true, VV>(spec, sp, nc, d.n1 * n3h, n3h, (long long)d.n2 * n3h, n3h,
                                               nf, nprob, active, s)));
  if (e) return e;
  CB_DISPATCH_NV(d.n3, e = (c2r_rows_impl<NN, VV>(spec, sp, nc, out, op_, ofs, d.n1 * d.n2, nf, nprob, epi, alpha,
                                            partials, nparts, used, other, active, s)));
  return e;
}

template <int N, int V>
static int deriv_rows_impl(const float* in, long long ip, long long ifs, float* out, long long op_, long long ofs,
                           int nf, int nprob, const Dims& d, int epi, double* partials, int nparts, int* used,
                           const int* active, cudaStream_t s) {
  const float2* tw = twiddles(N);
  if (!tw) return (int)cudaErrorMemoryAllocation;
  size_t sm = RowCfg<N, V>::smem;
  const int nrows = d.n1 * d.n2;
  dim3 grid((nrows + 2 * RowCfg<N, V>::P - 1) / (2 * RowCfg<N, V>::P), nf, nprob);
  int e = claim_partials(epi, grid, partials, nparts, used);
  if (!e) e = set_smem(k_deriv_rows<N, V>, sm);
  if (e) return e;
  k_deriv_rows<N, V><<<grid, RowCfg<N, V>::T, sm, s>>>(in, ip, ifs, out, op_, ofs, nrows, tw, epi, partials, nparts, active);
  return (int)cudaGetLastError();
}

template <int N, int V>
static int deriv_cols_impl(const float* in, long long ip, long long ifs, float* out, long long op_, long long ofs,
                           int nf, int nprob, const Dims& d, int axis, int epi, double* partials, int nparts,
                           int* used, const int* active, cudaStream_t s) {
  const float2* tw = twiddles(N);
  if (!tw) return (int)cudaErrorMemoryAllocation;
  size_t sm = col_smem<N, V>(1);
  // neighbouring columns as one float2: even strides and 8-byte bases
  auto pairs = [](const float* p, long long a, long long b) {
    return (reinterpret_cast<uintptr_t>(p) & 7) == 0 && ((a | b) & 1) == 0;
  };
  int ncols, cpg;
  long long gs, es;
  if (axis == 1) {  // lines along x2: column (i1, i3)
    ncols = d.n1 * d.n3; cpg = d.n3; gs = (long long)d.n2 * d.n3; es = d.n3;
  } else {          // lines along x1: column (i2, i3)
    ncols = d.n2 * d.n3; cpg = ncols; gs = 0; es = (long long)d.n2 * d.n3;
  }
  constexpr int C = 2 * ColCfg<N, V>::C;
  dim3 grid((ncols + C - 1) / C, nf, nprob);
  int e = claim_partials(epi, grid, partials, nparts, used);
  if (!e) e = set_smem(k_deriv_cols<N, V>, sm);
  if (e) return e;
  k_deriv_cols<N, V><<<grid, ColCfg<N, V>::T, sm, s>>>(in, ip, ifs, out, op_, ofs, ncols, cpg, gs, (int)es, tw, epi,
                                                       pairs(in, ip, ifs), pairs(out, op_, ofs), partials, nparts,
                                                       active);
  return (int)cudaGetLastError();
}

int deriv_partials(const Dims& d, int axis, int nf) {
  const int n = (axis == 0) ? d.n1 : (axis == 1 ? d.n2 : d.n3);
  if (axis == 2) {
    const int P = row_lines(n);
    if (!P) return 0;
    return ((d.n1 * d.n2 + 2 * P - 1) / (2 * P)) * nf;
  }
  const int C = col_lines(n);
  if (!C) return 0;
  const int ncols = (axis == 1) ? d.n1 * d.n3 : d.n2 * d.n3;
  return ((ncols + 2 * C - 1) / (2 * C)) * nf;
}

int launch_deriv(const float* in, long long ip, long long ifs, float* out, long long op_,
                 long long ofs, int nf, int nprob, const Dims& d, int axis, int epi,
                 double* partials, int nparts, const int* active, cudaStream_t s, int* used) {
  if (!axes_supported(d)) return (int)cudaErrorInvalidValue;
  if (axis == 2 && (!aligned16(in) || ((ip | ifs) & 3))) return (int)cudaErrorInvalidValue;
  const int n = (axis == 0) ? d.n1 : (axis == 1 ? d.n2 : d.n3);
  int e = 0;
  if (axis == 2) {
    CB_DISPATCH_NV(n, e = (deriv_rows_impl<NN, VV>(in, ip, ifs, out, op_, ofs, nf, nprob, d, epi, partials, nparts,
                                                   used, active, s)));
  } else {
    CB_DISPATCH_NV_COL(n, e = (deriv_cols_impl<NN, VV>(in, ip, ifs, out, op_, ofs, nf, nprob, d, axis, epi,
                                                       partials, nparts, used, active, s)));
  }
  return e;
}

// 3-field spectral operator (r2c, x1 op, c2r store) on caller-provided
// spectrum workspace and twiddle table: the launches allocate nothing.
template <int N, int V>
static int spectral3_explicit_impl(const float* in, float* out, float2* spec, const SpecParams* params,
                                   const Dims& d, int op, const float2* tw, cudaStream_t s) {
  const long long n = d.n(), nc = d.nc();
  const int n3h = N / 2 + 1;
  const int nrows = d.n1 * d.n2;
  int e = set_smem(k_r2c_rows<N, V>, RowCfg<N, V>::smem);
  if (!e) e = set_smem(k_cols<N, false, V>, col_smem<N, V>(1));
  if (!e) e = set_smem(k_cols<N, true, V>, col_smem<N, V>(1));
  if (!e) e = set_smem(k_pencil1<N, V, true>, col_smem<N, V>(1, true));
  if (!e) e = set_smem(k_c2r_rows<N, V>, RowCfg<N, V>::smem);
  if (e) return e;
  const dim3 rows((nrows + 2 * RowCfg<N, V>::P - 1) / (2 * RowCfg<N, V>::P), 3, 1);
  const int ncx2 = d.n1 * n3h;
  const dim3 cols((ncx2 + ColCfg<N, V>::C - 1) / ColCfg<N, V>::C, 3, 1);
  const int ncx1 = d.n2 * n3h;
  const int blocks = (ncx1 + ColCfg<N, V>::C - 1) / ColCfg<N, V>::C;
  const bool shared = pencil_shares_fields(blocks, 1);
  const dim3 pen(blocks, shared ? 1 : 3, 1);
  k_r2c_rows<N, V><<<rows, RowCfg<N, V>::T, RowCfg<N, V>::smem, s>>>(in, 0, n, spec, 0, nc, nrows, tw, nullptr);
  constexpr int T = ColCfg<N, V>::T;
  const size_t sm = col_smem<N, V>(1);
  k_cols<N, false, V><<<cols, T, sm, s>>>(spec, 0, nc, ncx2, n3h, (long long)d.n2 * n3h, n3h, tw, nullptr);
  k_pencil1<N, V, true><<<pen, T, col_smem<N, V>(1, true), s>>>(
      spec, 0, nc, shared ? 3 : 1, d, op, 1.f / (float)((double)d.n1 * d.n2 * d.n3), params, SpecParams{}, tw, nullptr);
  k_cols<N, true, V><<<cols, T, sm, s>>>(spec, 0, nc, ncx2, n3h, (long long)d.n2 * n3h, n3h, tw, nullptr);
  k_c2r_rows<N, V><<<rows, RowCfg<N, V>::T, RowCfg<N, V>::smem, s>>>(spec, 0, nc, out, 0, n, nrows, tw, EPI_STORE, nullptr,
                                                           nullptr, 0, nullptr, nullptr);
  return (int)cudaGetLastError();
}

int launch_spectral3_explicit(const float* in, float* out, float2* spec, const SpecParams* params, const Dims& d,
                              int op, const float2* tw, cudaStream_t s) {
  if (!cubic_supported(d) || !aligned16(in)) return (int)cudaErrorInvalidValue;
  int e = 0;
  CB_DISPATCH_N(d.n1, e = (spectral3_explicit_impl<NN, 0>(in, out, spec, params, d, op, tw, s)));
  return e;
}

// ---------------------------------------------------------------------------
// autotuner: CLAIRE plans its transforms by measurement (accfft_plan_dft_3d_r2c
// with ACCFFT_MEASURE, src/RegOpt.cpp:993-994); here the candidates are the
// variants above, timed on the work the solver does with them.
// ---------------------------------------------------------------------------
__global__ void k_tune_fill(float* x, long long len) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x)
    x[i] = __sinf(0.001f * (float)(i % 100003));
}

static std::atomic<bool> g_fft_tuned[9];
static std::mutex g_tune_mutex;

bool fft_tuned(int n) {
  const int k = size_slot(n);
  return k >= 0 && g_fft_tuned[k].load();
}

int fft_autotune_once(int n, int nprob, cudaStream_t s) {
  std::lock_guard<std::mutex> lock(g_tune_mutex);
  if (fft_tuned(n)) return 0;
  int best = 0;
  return fft_autotune(n, nprob, s, &best, nullptr);
}

int fft_autotune(int n, int nprob, cudaStream_t s, int* best, float* ms) {
  int cand[4];
  const int ncand = fft_variant_candidates(n, cand);
  if (!ncand || nprob < 1) return (int)cudaErrorInvalidValue;
  const Dims d{n, n, fft_size_supported(n) ? n : 64};  // 150: column / pencil passes only
  const long long nn = d.n(), nc = d.nc();
  float *in = nullptr, *out = nullptr;
  float2* spec = nullptr;
  SpecParams* par = nullptr;
  int e = 0;
  if (cudaMalloc(&in, sizeof(float) * 3 * nn * nprob) != cudaSuccess ||
      cudaMalloc(&out, sizeof(float) * 3 * nn * nprob) != cudaSuccess ||
      cudaMalloc(&spec, sizeof(float2) * 3 * nc * nprob) != cudaSuccess ||
      cudaMalloc(&par, sizeof(SpecParams) * nprob) != cudaSuccess)
    e = (int)cudaErrorMemoryAllocation;
  std::vector<SpecParams> hp(nprob);
  for (auto& p : hp) {
    p.norm = NORM_H2;
    p.beta0 = 1e-3f;
    p.beta1 = 1e-4f;
    p.beta2 = 1e-4f;
    p.hd = 1.f;
    p.sigma[0] = p.sigma[1] = p.sigma[2] = 1.f;
  }
  if (!e) e = (int)cudaMemcpyAsync(par, hp.data(), sizeof(SpecParams) * nprob, cudaMemcpyHostToDevice, s);
  if (!e) {
    k_tune_fill<<<148 * 4, 256, 0, s>>>(in, 3 * nn * nprob);
    e = (int)cudaGetLastError();
  }
  cudaEvent_t t0 = nullptr, t1 = nullptr;
  if (!e && (cudaEventCreate(&t0) != cudaSuccess || cudaEventCreate(&t1) != cudaSuccess)) e = (int)cudaErrorUnknown;
  const int old = fft_variant(n);
  float best_ms = 0.f;
  int best_v = old;
  auto work = [&]() -> int {
    int r = launch_r2c3d(in, 3 * nn, nn, spec, 3 * nc, 3, nprob, d, nullptr, s);
    if (!r) r = launch_pencil(spec, 3 * nc, nprob, d, OP_REG_INV, par, 3, 3, nullptr, s);
    if (!r) r = launch_c2r3d(spec, 3 * nc, out, 3 * nn, nn, 3, nprob, d, EPI_STORE, nullptr, nullptr, 0, nullptr, s);
    for (int a = 0; a < 3 && !r; ++a)
      r = launch_deriv(in, 3 * nn, nn, out + a * nn, 3 * nn, 3 * nn, 1, nprob, d, a, EPI_STORE, nullptr, 0, nullptr,
                       s);
    return r;
  };
  for (int i = 0; i < ncand && !e; ++i) {
    g_fft_var[size_slot(n)].store(cand[i], std::memory_order_relaxed);
    for (int w = 0; w < 2 && !e; ++w) e = work();
    constexpr int kReps = 5;
    if (!e) e = (int)cudaEventRecord(t0, s);
    for (int r = 0; r < kReps && !e; ++r) e = work();
    if (!e) e = (int)cudaEventRecord(t1, s);
    if (!e) e = (int)cudaEventSynchronize(t1);
    float t = 0.f;
    if (!e) e = (int)cudaEventElapsedTime(&t, t0, t1);
    t /= kReps;
    if (ms) ms[i] = t;
    if (!e && (i == 0 || t < best_ms)) {
      best_ms = t;
      best_v = cand[i];
    }
  }
  g_fft_var[size_slot(n)].store(e ? old : best_v, std::memory_order_relaxed);
  if (!e) g_fft_tuned[size_slot(n)].store(true);
  if (best) *best = e ? old : best_v;
  cudaStreamSynchronize(s);
  if (t0) cudaEventDestroy(t0);
  if (t1) cudaEventDestroy(t1);
  cudaFree(in);
  cudaFree(out);
  cudaFree(spec);
  cudaFree(par);
  return e;
}

}  // namespace cb
