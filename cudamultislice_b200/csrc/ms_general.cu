// ms_general.cu -- slice passes of mixed-radix line lengths (see ms_general.cuh).
#include "ms_general.cuh"

#include <cmath>

#include "ms_slice_impl.cuh"

namespace ms {

namespace {

// ---- compile-time trigonometry (Taylor series in double, |x| <= pi) ----
constexpr double kPi = 3.14159265358979323846;
__host__ __device__ constexpr double ct_sin(double x) {
  double t = x, s = x;
  for (int k = 1; k < 20; ++k) {
    t *= -x * x / ((2 * k) * (2 * k + 1));
    s += t;
  }
  return s;
}
__host__ __device__ constexpr double ct_cos(double x) {
  double t = 1.0, s = 1.0;
  for (int k = 1; k < 20; ++k) {
    t *= -x * x / ((2 * k - 1) * (2 * k));
    s += t;
  }
  return s;
}
// angle -2 pi j / n brought to (-pi, pi]
__host__ __device__ constexpr double ct_angle(int j, int n) {
  const int m = ((j % n) + n) % n;
  return 2 * m <= n ? -2.0 * kPi * m / n : 2.0 * kPi * (n - m) / n;
}

// x exp(-2 pi i J / M): an exact quarter turn and three shears (each of
// determinant exactly 1, so the rotation does not change the norm; see
// fft::twc).
template <int J, int M>
MS_D float2 rot(float2 x) {
  constexpr int j = ((J % M) + M) % M;
  if constexpr (j == 0) {
    return x;
  } else {
    constexpr double a = ct_angle(j, M);  // (-pi, pi]
    constexpr int q = (int)(a / (kPi / 2) + (a > 0 ? 0.5 : -0.5));
    constexpr double r = a - q * (kPi / 2);
    float2 y = x;
    if constexpr (q == 1) y = make_float2(-x.y, x.x);
    else if constexpr (q == 2 || q == -2) y = make_float2(-x.x, -x.y);
    else if constexpr (q == -1) y = make_float2(x.y, -x.x);
    if constexpr (4 * j % M == 0) {
      return y;
    } else {
      constexpr float t = (float)(ct_sin(r / 2) / ct_cos(r / 2)), s = (float)ct_sin(r);
      const float x1 = fmaf(-t, y.y, y.x);
      const float y1 = fmaf(s, x1, y.y);
      return make_float2(fmaf(-t, y1, x1), y1);
    }
  }
}

// c v + acc with the constant c as a sum of two floats: a rounded cosine or
// sine would scale the wave the same way in every transform.
template <int J, int P, bool SINE>
MS_D float fma_trig(float v, float acc) {
  constexpr double c = SINE ? ct_sin(ct_angle(J, P)) : ct_cos(ct_angle(J, P));
  constexpr float hi = (float)c, lo = (float)(c - (double)hi);
  return fmaf(hi, v, fmaf(lo, v, acc));
}

// DFT of an odd prime length from the sums and differences of mirrored inputs:
// X_k = x_0 + sum_j cos(2 pi j k / P) t_j -+ i sum_j sin(2 pi j k / P) s_j.
template <int P, int K, int J>
MS_D void odd_terms(const float2 (&t)[P / 2], const float2 (&s)[P / 2], float2& c, float2& d) {
  c.x = fma_trig<J * K, P, false>(t[J - 1].x, c.x);
  c.y = fma_trig<J * K, P, false>(t[J - 1].y, c.y);
  d.x = fma_trig<J * K, P, true>(s[J - 1].x, d.x);
  d.y = fma_trig<J * K, P, true>(s[J - 1].y, d.y);
  if constexpr (J < P / 2) odd_terms<P, K, J + 1>(t, s, c, d);
}
template <int P, int K = 1>
MS_D void odd_outputs(float2 (&x)[P], float2 x0, const float2 (&t)[P / 2], const float2 (&s)[P / 2]) {
  float2 c = x0, d = make_float2(0.f, 0.f);
  odd_terms<P, K, 1>(t, s, c, d);  // (d carries sin of the negative angle)
  x[K] = make_float2(c.x - d.y, c.y + d.x);
  x[P - K] = make_float2(c.x + d.y, c.y - d.x);
  if constexpr (K < P / 2) odd_outputs<P, K + 1>(x, x0, t, s);
}

template <int R>
MS_D void gen_dft(float2 (&x)[R]);

// R = A B: A-point transforms over stride B, twiddles, B-point transforms.
template <int A, int B, int N2, int K1>
MS_D void comp_twiddle(float2 (&y)[A]) {
  y[K1] = rot<N2 * K1, A * B>(y[K1]);
  if constexpr (K1 + 1 < A) comp_twiddle<A, B, N2, K1 + 1>(y);
}
template <int A, int B, int N2 = 0>
MS_D void comp_inner(float2 (&x)[A * B]) {
  float2 y[A];
#pragma unroll
  for (int i = 0; i < A; ++i) y[i] = x[B * i + N2];
  gen_dft<A>(y);
  comp_twiddle<A, B, N2, 0>(y);
#pragma unroll
  for (int i = 0; i < A; ++i) x[B * i + N2] = y[i];
  if constexpr (N2 + 1 < B) comp_inner<A, B, N2 + 1>(x);
}
template <int A, int B>
MS_D void comp_dft(float2 (&x)[A * B]) {
  comp_inner<A, B>(x);
  float2 o[A * B];
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    float2 z[B];
#pragma unroll
    for (int i = 0; i < B; ++i) z[i] = x[B * k1 + i];
    gen_dft<B>(z);
#pragma unroll
    for (int i = 0; i < B; ++i) o[k1 + A * i] = z[i];
  }
#pragma unroll
  for (int i = 0; i < A * B; ++i) x[i] = o[i];
}

// Natural-order forward DFT of R registers.
template <int R>
MS_D void gen_dft(float2 (&x)[R]) {
  if constexpr (R == 6) comp_dft<3, 2>(x);
  else if constexpr (R == 9) comp_dft<3, 3>(x);
  else if constexpr (R == 10) comp_dft<5, 2>(x);
  else if constexpr (R == 12) comp_dft<3, 4>(x);
  else if constexpr (R == 15) comp_dft<5, 3>(x);
  else if constexpr (R % 2 == 1) {
    float2 t[R / 2], s[R / 2];
    float2 sum = x[0];
#pragma unroll
    for (int j = 1; j <= R / 2; ++j) {
      t[j - 1] = cadd(x[j], x[R - j]);
      s[j - 1] = csub(x[j], x[R - j]);
      sum = cadd(sum, t[j - 1]);
    }
    odd_outputs<R>(x, x[0], t, s);
    x[0] = sum;
  } else {
    float2 y[R];
#pragma unroll
    for (int i = 0; i < R; ++i) y[i] = x[i];
    fft::dft<R, false, true>(y);
#pragma unroll
    for (int i = 0; i < R; ++i) x[i] = y[fft::brev(i, fft::ilog2(R))];
  }
}

// One Stockham pass of radix R over a line of n points at stride cb in shared
// memory (in -> out), threads t of T.
template <int R>
MS_D void gen_pass(const float2* in, float2* out, const float2* tw, int ns, int nb, int step, float inv, int cb, int t,
                   int T) {
  for (int i = t; i < nb; i += T) {
    // (i < 2^12: the quotient's rounding stays below its distance 1/(2 ns) to
    // the next integer)
    const int q = ns == 1 ? i : (int)(((float)i + 0.5f) * inv), k = i - q * ns;
    float2 x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = in[(i + r * nb) * cb];
    if (ns > 1) {
      const int w = k * step;  // (r k step < n)
#pragma unroll
      for (int r = 1; r < R; ++r) x[r] = cmul(x[r], tw[r * w]);
    }
    gen_dft<R>(x);
    const int b = q * ns * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) out[(b + r * ns) * cb] = x[r];
  }
}

// Forward transform of the line(s) in a (b: scratch of the same size); the
// CTA's threads all call it.  On return a points to the result.  Synchronises
// before its first pass's reads and after its last pass's writes.
MS_D void gen_line_fft(const GenPlan& p, float2*& a, float2*& b, const float2* tw, int cb, int t, int T) {
  __syncthreads();
#pragma unroll 1
  for (int k = 0; k < p.npass; ++k) {
    const int ns = p.ns[k], nb = p.nb[k], step = p.step[k];
    const float inv = p.inv[k];
    switch (p.radix[k]) {
      case 2: gen_pass<2>(a, b, tw, ns, nb, step, inv, cb, t, T); break;
      case 3: gen_pass<3>(a, b, tw, ns, nb, step, inv, cb, t, T); break;
      case 4: gen_pass<4>(a, b, tw, ns, nb, step, inv, cb, t, T); break;
      case 5: gen_pass<5>(a, b, tw, ns, nb, step, inv, cb, t, T); break;
      case 6: gen_pass<6>(a, b, tw, ns, nb, step, inv, cb, t, T); break;
      case 7: gen_pass<7>(a, b, tw, ns, nb, step, inv, cb, t, T); break;
      case 8: gen_pass<8>(a, b, tw, ns, nb, step, inv, cb, t, T); break;
      case 9: gen_pass<9>(a, b, tw, ns, nb, step, inv, cb, t, T); break;
      case 10: gen_pass<10>(a, b, tw, ns, nb, step, inv, cb, t, T); break;
      case 11: gen_pass<11>(a, b, tw, ns, nb, step, inv, cb, t, T); break;
      case 12: gen_pass<12>(a, b, tw, ns, nb, step, inv, cb, t, T); break;
      case 13: gen_pass<13>(a, b, tw, ns, nb, step, inv, cb, t, T); break;
      case 15: gen_pass<15>(a, b, tw, ns, nb, step, inv, cb, t, T); break;
      case 16: gen_pass<16>(a, b, tw, ns, nb, step, inv, cb, t, T); break;
    }
    float2* s = a;
    a = b;
    b = s;
    __syncthreads();
  }
}

// Rows: one line per CTA, at most EPT points per thread.
// Bound (600 x 450): the chain of load, six to eight passes of a few hundred
// nanoseconds each, and store; the grid is one to three CTAs per SM.
template <int EPT, int T>
__global__ void __launch_bounds__(T) k_general_rows(const __grid_constant__ GenArgs g, int flags) {
  extern __shared__ float2 smem[];
  const int n = g.nx, t = threadIdx.x;
  float2 *a = smem, *b = smem + n;
  const float2* tw = smem + 2 * n;
  const long long row0 = (long long)blockIdx.x * n;
  pdl_launch_dependents();
  for (int i = t; i < n; i += T) smem[2 * n + i] = g.tw[i];
  pdl_wait();
  float V[EPT];
  if (flags & G_MULT) {
#pragma unroll
    for (int m = 0; m < EPT; ++m) V[m] = t + T * m < n ? g.V[row0 + t + T * m] : 0.0f;
  }
  const bool inv = flags & G_INV;
#pragma unroll
  for (int m = 0; m < EPT; ++m) {
    const int i = t + T * m;
    if (i >= n) break;
    float2 v = make_float2(0.f, 0.f);
    if (!inv) v = g.in[row0 + i];
    else if (i < g.cpos || i >= n - g.cneg) v = cconj(g.in[row0 + i]);  // IFFT(x) = conj FFT(conj x)
    a[i] = v;
  }
  // (one copy of the transform's code: first the inverse, then the forward)
#pragma unroll 1
  for (int it = inv ? 0 : 1; it < (flags & G_FWD ? 2 : 1); ++it) {
    if (it == 1 && (flags & G_MULT)) {
#pragma unroll
      for (int m = 0; m < EPT; ++m) {
        const int i = t + T * m;
        if (i >= n) break;
        float s, c;
        sincos_red(fmul_x(g.sigma, V[m]), &s, &c);
        const float2 v = inv ? cconj(a[i]) : a[i];
        // (contraction written out: one slice per launch pair and a chain of
        // slices round the same way)
        a[i] = make_float2(fmaf(v.x, c, -fmul_x(v.y, s)), fmaf(v.x, s, fmul_x(v.y, c)));
      }
    }
    gen_line_fft(g.plan, a, b, tw, 1, t, T);
  }
  if (flags & G_FWD) {
#pragma unroll
    for (int m = 0; m < EPT; ++m) {
      const int i = t + T * m;
      if (i < n && (i < g.cpos || i >= n - g.cneg)) g.out[row0 + i] = a[i];
    }
  } else {
#pragma unroll
    for (int m = 0; m < EPT; ++m) {
      const int i = t + T * m;
      if (i < n) g.out[row0 + i] = cconj(a[i]);
    }
  }
}

// Columns: CB adjacent columns of the band per CTA, points [row][column].
template <int CB>
__global__ void __launch_bounds__(256) k_general_columns(const __grid_constant__ GenArgs g) {
  extern __shared__ float2 smem[];
  constexpr int T = 256 / CB;
  const int n = g.ny, c = threadIdx.x % CB, t = threadIdx.x / CB;
  float2 *a = smem + c, *b = smem + (size_t)n * CB + c;
  float2* tw = smem + (size_t)2 * n * CB;
  const int u = blockIdx.x * CB + c;
  const bool live = u < g.cpos + g.cneg;
  const int col = !live ? 0 : u < g.cpos ? u : u - g.cpos + g.nx - g.cneg;
  pdl_launch_dependents();
  for (int i = threadIdx.x; i < n; i += 256) tw[i] = g.tw[i];
  const float kx = g.kx[col], kx2 = fmul_x(kx, kx);
  const float2 pxv = g.px[col];
  pdl_wait();
  for (int i = t; i < n; i += T) a[i * CB] = live ? g.in[(long long)i * g.nx + col] : make_float2(0.f, 0.f);
#pragma unroll 1
  for (int it = 0; it < 2; ++it) {
    gen_line_fft(g.plan, a, b, tw, CB, t, T);
    if (it == 1) break;
    for (int i = t; i < n; i += T) {
      float2 v = make_float2(0.f, 0.f);
      if (i < g.rpos || i >= n - g.rneg) {
        const float ky = g.ky[i];
        // CreatePropsKernel (U.cu:419): keep sqrtf(kx^2+ky^2) < kmax
        if (fadd_x(kx2, fmul_x(ky, ky)) < g.k2_lt) {
          v = cmul(cmul(a[i * CB], pxv), g.py[i]);
          // x 1/N, and conjugated for the inverse
          v = make_float2(fmaf(v.x, g.scale, v.x * g.scale_lo), -fmaf(v.y, g.scale, v.y * g.scale_lo));
        }
      }
      a[i * CB] = v;
    }
  }
  if (live)
    for (int i = t; i < n; i += T) g.out[(long long)i * g.nx + col] = cconj(a[i * CB]);
}

template <int EPT, int T>
cudaError_t run_rows(const GenArgs& a, int flags, cudaStream_t s) {
  const size_t smem = (size_t)3 * a.nx * sizeof(float2);
  constexpr size_t most = (size_t)3 * EPT * T * sizeof(float2);
  static unsigned long long done = 0;
  auto kernel = k_general_rows<EPT, T>;
  if (cudaError_t e = set_smem_once(done, kernel, most)) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.ny);
  cfg.blockDim = dim3(T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, a, flags);
}

template <int CB>
cudaError_t run_columns(const GenArgs& a, cudaStream_t s) {
  const size_t smem = (size_t)(2 * CB + 1) * a.ny * sizeof(float2);
  static unsigned long long done = 0;
  auto kernel = k_general_columns<CB>;
  if (cudaError_t e = set_smem_once(done, kernel, (size_t)200 << 10)) return e;
  const int cols = a.cpos + a.cneg;
  return launch_pdl(kernel, dim3((cols + CB - 1) / CB), 256, smem, s, a);
}

}  // namespace

// The factorisation with the shortest chain for 128 threads per line: per pass
// the rounds of butterflies a thread takes times the instructions of one
// (loads, twiddles, index arithmetic and stores included), plus a barrier.
// Small radices that keep all threads busy beat few passes of large ones (600 =
// 15 x 10 x 4 and 450 = 15 x 15 x 2: 12.2 and 13.3 us a pass at 600 x 450).
GenPlan general_plan(int n) {
  GenPlan p;
  if (n < 2 || n > 4096) return p;
  p.n = n;
  static const int kRadix[] = {16, 15, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};
  static const int kCost[] = {330, 520, 680, 330, 500, 330, 260, 150, 230, 150, 140, 75, 70, 45};
  constexpr int kThreads = 128, kBarrier = 60;
  int best = 1 << 30, cur[kGenMaxPass] = {};
  auto search = [&](auto&& self, int rest, int depth, int from, int cost) -> void {
    if (cost >= best) return;
    if (rest == 1) {
      best = cost;
      p.npass = depth;
      for (int i = 0; i < depth; ++i) p.radix[i] = cur[i];
      return;
    }
    if (depth >= kGenMaxPass) return;
    for (int i = from; i < (int)(sizeof(kRadix) / sizeof(int)); ++i)
      if (rest % kRadix[i] == 0) {
        cur[depth] = kRadix[i];
        const int rounds = (n / kRadix[i] + kThreads - 1) / kThreads;
        self(self, rest / kRadix[i], depth + 1, i, cost + rounds * kCost[i] + kBarrier);
      }
  };
  search(search, n, 0, 0, 0);
  for (int k = 0, ns = 1; k < p.npass; ns *= p.radix[k], ++k) {
    p.ns[k] = ns;
    p.nb[k] = n / p.radix[k];
    p.step[k] = p.nb[k] / ns;
    p.inv[k] = 1.0f / (float)ns;
  }
  return p;
}

cudaError_t launch_general_rows(const GenArgs& a, int flags, cudaStream_t s) {
  if (a.plan.n != a.nx || a.plan.npass < 1 || a.ny < 1) return cudaErrorInvalidValue;
  if (flags != G_INV && flags != (G_MULT | G_FWD) && flags != (G_INV | G_MULT | G_FWD)) return cudaErrorInvalidValue;
  if (a.nx <= 512) return run_rows<4, 128>(a, flags, s);
  if (a.nx <= 1024) return run_rows<8, 128>(a, flags, s);
  if (a.nx <= 2048) return run_rows<8, 256>(a, flags, s);
  return run_rows<16, 256>(a, flags, s);
}

// Columns per CTA: eight (64-byte row segments) where that still gives every
// SM a CTA and fits, else four, else two.
cudaError_t launch_general_columns(const GenArgs& a, cudaStream_t s) {
  if (a.plan.n != a.ny || a.plan.npass < 1 || a.cpos + a.cneg < 1) return cudaErrorInvalidValue;
  const int cols = a.cpos + a.cneg;
  auto fits = [&](int cb) { return (size_t)(2 * cb + 1) * a.ny * sizeof(float2) <= (size_t)200 << 10; };
  if (fits(8) && cols >= 8 * 148) return run_columns<8>(a, s);
  if (fits(4) && cols >= 4 * 148) return run_columns<4>(a, s);
  return run_columns<2>(a, s);
}

}  // namespace ms
