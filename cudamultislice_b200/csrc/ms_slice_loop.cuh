// ms_slice_loop.cuh -- the whole conventional slice loop of one instance in
// one persistent cooperative kernel.
//
// The two-pass slice step of ms_slice_impl.cuh (row pass: IFFT_row ->
// x exp(i sigma V) -> FFT_row; column pass: FFT_col -> x P(k)/N -> IFFT_col)
// runs here for all S slices inside a single launch.  Every CTA is resident
// for the whole loop (cooperative launch, one CTA per SM): between the phases
// the CTAs meet at a grid barrier instead of a kernel boundary, so a slice
// costs no launch, ramp-up or drain, the frequency tables stay in shared
// memory, and the next slice's potential rows are prefetched into L2 while
// the column phase runs.
//
// Work split (lines of N points, one warp per line, E = N/32 points per
// thread): row r goes to CTA r % G, warp r / G; column unit u (CW adjacent
// columns of the band's N/2, CW warps interleaved so that every warp access
// covers whole 32-byte sectors) to CTA u % G, group u / G.  A wave of 1024^2
// puts at most 7 rows and 4 columns on one SM per phase.
//
// Grid barrier: a monotonic arrival counter (zeroed before each launch); the
// k-th barrier waits for k * G arrivals.  Each wait is bounded by a time limit
// (default one second, %globaltimer): a CTA that runs out sets the error word
// and returns, and the others see the error word and return too, so a lost
// arrival ends the kernel with an error status instead of a hang.
#pragma once
#include "ms_slice_impl.cuh"

namespace ms {

// v *= exp(i sigma V) over a thread's E points: the polynomial-only sincos
// when every phase of the warp is within a quarter turn of 0 (bit-identical,
// the usual case for slices of a few angstroms), else the reduced one.
template <int E>
MS_D void transmit_line(float2 (&v)[E], float (&vv)[E], float sigma) {
  bool small = true;
#pragma unroll
  for (int j = 0; j < E; ++j) {
    vv[j] = fmul_x(sigma, vv[j]);
    small = small && sincos_small_ok(vv[j]);
  }
  if (__all_sync(0xffffffffu, small)) {
#pragma unroll
    for (int j = 0; j < E; j += 2) {
      float s0, c0, s1, c1;
      sincos_small2(vv[j], vv[j + 1], &s0, &c0, &s1, &c1);
      v[j] = cmul(v[j], make_float2(c0, s0));
      v[j + 1] = cmul(v[j + 1], make_float2(c1, s1));
    }
  } else {
#pragma unroll
    for (int j = 0; j < E; j += 2) {
      float s0, c0, s1, c1;
      sincos_red2(vv[j], vv[j + 1], &s0, &c0, &s1, &c1);
      v[j] = cmul(v[j], make_float2(c0, s0));
      v[j + 1] = cmul(v[j + 1], make_float2(c1, s1));
    }
  }
}

MS_D unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Grid barrier number `epoch` (1, 2, ...) in two halves, so that work which no
// other CTA's result feeds runs between the arrival and the wait.
//
// TIGHT = false: the wait polls with a short sleep, inside full fences; TIGHT =
// true: it polls back to back, checking the clock and the error word every 32
// polls, and starts only when the arrival's own return value shows that others
// are still to come (148 CTAs polling from the start slow the last arrivals:
// 1.24 us a barrier with a release reduction, 1.15 with this).  FENCED: full
// fences around the arrival and after the wait (as cooperative groups' grid
// sync); without them the acquire-release arrival and the acquire load carry
// the ordering (both are cumulative over what the CTA's bar.sync has ordered
// before them).  Measured and left out: arrivals spread over eight counters
// (1.37 us), relaxed polls with a fence after the wait (1.38), one CTA of a
// cluster for two or four (2.1), an arrival per warp (1.9).
template <bool TIGHT, bool FENCED = true>
MS_D unsigned int loop_arrive(const LoopSync& s) {
  __syncthreads();
  unsigned int seen = 0;
  if (threadIdx.x == 0) {
    if constexpr (FENCED || !TIGHT) __threadfence();
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(seen) : "l"(s.count) : "memory");
    ++seen;
  }
  return seen;
}
// `seen`: loop_arrive's result.  Returns false (in every thread of the CTA)
// when the grid must stop: this CTA's wait ran out or another CTA reported an
// error.
template <bool TIGHT, bool FENCED = true>
MS_D bool loop_wait(const LoopSync& s, unsigned int epoch, unsigned int seen) {
  int ok = 1;
  if (threadIdx.x == 0) {
    const unsigned int target = epoch * gridDim.x + s.expect_extra;
    if (seen < target) {
      const unsigned long long t0 = global_ns();
      for (unsigned int it = 0;; ++it) {
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(s.count) : "memory");
        if (v >= target) break;
        if (!TIGHT || (it & 31) == 31) {
          if (*reinterpret_cast<volatile int*>(s.error) != 0) {
            ok = 0;
            break;
          }
          if (global_ns() - t0 > s.limit_ns) {
            atomicExch(s.error, kLoopTimeout);
            ok = 0;
            break;
          }
        }
        if constexpr (!TIGHT) __nanosleep(32);
      }
    }
    if constexpr (FENCED || !TIGHT) __threadfence();
  }
  return __syncthreads_and(ok) != 0;
}
template <bool TIGHT, bool FENCED = true>
MS_D bool loop_barrier(const LoopSync& s, unsigned int epoch) {
  return loop_wait<TIGHT, FENCED>(s, epoch, loop_arrive<TIGHT, FENCED>(s));
}

// PL: rows, PC: columns (the same length; the columns may take more threads
// per line: a CTA has at most four columns of a 1024^2 phase).
template <class PL, class PC, int CW>
struct LoopShape {
  static constexpr int N = PL::N, E = PL::E, P = PL::P;
  static_assert(P == 32 && PC::N == N && (PC::P == 32 || PC::P == 64), "rows of one warp, columns of one or two");
  static constexpr int NT = 256;                 // threads per CTA
  static constexpr int LINES = NT / P;           // rows per CTA per round
  static constexpr int GS = CW * PC::P;          // threads of one column unit
  static constexpr int GROUPS = NT / GS;         // column units per CTA per round
  static_assert(GROUPS >= 1 && NT % GS == 0, "column units must tile the CTA");
  static constexpr int ROW_SLOT = PL::SLOT;
  static constexpr int COL_SLOT = ((N + N / PC::R1 + 15) / 16) * 16 + 16 / CW;
  static constexpr int EXCH = (LINES * ROW_SLOT > GROUPS * CW * COL_SLOT) ? LINES * ROW_SLOT : GROUPS * CW * COL_SLOT;
  // exchange slots, then ky (N floats, padded to float2), py (N float2) and the
  // twiddle tables of rows and columns (one when the plans are the same): the
  // barriers' acquires empty L1, and every phase fetched them from L2 again
  static constexpr int KY = EXCH, PY = KY + (N + 1) / 2, TWR = PY + N;
  static constexpr bool ONE_TW = PL::E == PC::E;
  static constexpr int TWC = ONE_TW ? TWR : TWR + PL::TWSIZE;
  static constexpr size_t SMEM = ((size_t)TWC + PC::TWSIZE) * sizeof(float2);
};

// The transmission exp(i sigma V) of a line's points: the polynomial-only
// sincos when every phase of the warp is within a quarter turn of 0
// (bit-identical, the usual case for slices of a few angstroms), else the
// reduced one.
template <int E>
MS_D void transmission_line(float2 (&tr)[E], const float* __restrict__ V, int t, float sigma) {
  constexpr int P = 32;
  float ph[E];
  bool small = true;
#pragma unroll
  for (int j = 0; j < E; ++j) ph[j] = V[t + P * j];
#pragma unroll
  for (int j = 0; j < E; ++j) {
    ph[j] = fmul_x(sigma, ph[j]);
    small = small && sincos_small_ok(ph[j]);
  }
  if (__all_sync(0xffffffffu, small)) {
#pragma unroll
    for (int j = 0; j < E; j += 2)
      sincos_small2(ph[j], ph[j + 1], &tr[j].y, &tr[j].x, &tr[j + 1].y, &tr[j + 1].x);
  } else {
#pragma unroll
    for (int j = 0; j < E; j += 2)
      sincos_red2(ph[j], ph[j + 1], &tr[j].y, &tr[j].x, &tr[j + 1].y, &tr[j + 1].x);
  }
}

// Row phase of one line: [IFFT_row] -> x t -> FFT_row, in place on the wave's
// band (or from psi0 on the first slice).
template <class PL, bool INV>
MS_D void loop_row(const float2* in, float2* out, const float2 (&tr)[PL::E], int line, int t, float2* sm,
                   const float2* stw) {
  constexpr int NX = PL::N, E = PL::E, P = PL::P;
  const long long row0 = (long long)line * NX;
  float2 v[E];
#pragma unroll
  for (int j = 0; j < E; ++j) v[j] = (!INV || in_band(j, E)) ? in[row0 + t + P * j] : make_float2(0.f, 0.f);
  if constexpr (INV) {
    fft::conj_all(v);
    fft::line_fft<PL, 0, true, false, true>(v, sm, t, stw);
    fft::conj_all(v);
  }
#pragma unroll
  for (int j = 0; j < E; ++j) v[j] = cmul(v[j], tr[j]);
  fft::line_fft<PL, 0, false, true, true>(v, sm, t, stw);
#pragma unroll
  for (int j = 0; j < E; ++j)
    if (in_band(j, E)) out[row0 + t + P * j] = v[j];
}

// Column phase of one unit of CW columns starting at the band's column c0:
// FFT_col -> x P/N (band-limited) -> IFFT_col, in place.
template <class PL, int CW>
MS_D void loop_col(const PassBArgs& b, float2* wave, int c0, int cl, int t, float2* sm,
                   const float* __restrict__ sky, const float2* __restrict__ spy, const float2* stw) {
  constexpr int E = PL::E, P = PL::P, GS = CW * P;
  const int nx = b.nx;
  const int col = band_column(c0, nx) + cl;
  const float2* src = wave + (long long)t * nx + col;
  const int step = P * nx;
  float2 v[E];
#pragma unroll
  for (int j = 0; j < E; ++j) v[j] = src[j * step];
  const ColFactors cf = ColFactors::load<B_PROPAGATE>(b, col);
  fft::line_fft<fft::PaddedPlan<PL>, GS, false, true, true>(v, sm, t, stw);
  col_mid<PL, B_PROPAGATE>(v, b, cf, sky, spy, col, t, 0);
  fft::conj_all(v);
  fft::line_fft<fft::PaddedPlan<PL>, GS, true, false, true>(v, sm, t, stw);
  fft::conj_all(v);
  int ostep;
  asm volatile("mov.b32 %0, %1;" : "=r"(ostep) : "r"(step));
  float2* dst = wave + (long long)t * nx + col;
#pragma unroll
  for (int j = 0; j < E; ++j) dst[j * ostep] = v[j];
}

// Bulk L2 prefetch of the potential rows this CTA's lines read in the next
// row phase (issued before the column phase; one 4-byte-per-point row each).
template <class PL>
MS_D void prefetch_rows(const float* V, int G) {
  constexpr int NX = PL::N, P = PL::P;
  const int li = threadIdx.x / P, lt = threadIdx.x % P;
  const int line = li * G + blockIdx.x;
  if (lt == 0 && line < NX) {
    const float* p = V + (long long)line * NX;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"((unsigned)(NX * sizeof(float)))
                 : "memory");
  }
}

template <class PL, class PC, int CW, bool TIGHT, bool FENCED>
__global__ void __launch_bounds__(256, 1) k_slice_loop(LoopArgs L) {
  using SH = LoopShape<PL, PC, CW>;
  constexpr int N = PL::N, E = PL::E, P = PL::P, GS = SH::GS, GROUPS = SH::GROUPS;
  extern __shared__ float2 smem[];
  float* sky = reinterpret_cast<float*>(smem + SH::KY);
  float2* spy = smem + SH::PY;
  float2 *stwr = smem + SH::TWR, *stwc = smem + SH::TWC;
  for (int i = threadIdx.x; i < N; i += SH::NT) {
    sky[i] = L.b.ky[i];
    spy[i] = L.b.py[i];
  }
  for (int i = threadIdx.x; i < PL::TWSIZE; i += SH::NT) stwr[i] = L.a.tw[i];
  if constexpr (!SH::ONE_TW)
    for (int i = threadIdx.x; i < PC::TWSIZE; i += SH::NT) stwc[i] = L.b.tw[i];
  __syncthreads();
  const int G = gridDim.x;
  const int li = threadIdx.x / P, lt = threadIdx.x % P;  // row line of the CTA, index within it
  // this thread's column-unit coordinates
  const int g = threadIdx.x / GS, gr = threadIdx.x % GS;
  const int cl = gr % CW, t = gr / CW;
  const int line0 = li * G + blockIdx.x;  // this warp's (first) row of every slice
  float2* sm = smem + li * SH::ROW_SLOT;
  unsigned int epoch = 0;
  // the transmission of this warp's row for the coming slice
  float2 tr[E];
  if (line0 < N) transmission_line<E>(tr, L.Vstack + (long long)line0 * N, lt, L.a.sigma);
  for (int s = 0; s < L.S; ++s) {
    const float* V = L.Vstack + (long long)s * L.vstride;
    // ---- row phase ----
    for (int line = line0; line < N; line += SH::LINES * G) {
      if (line != line0) transmission_line<E>(tr, V + (long long)line * N, lt, L.a.sigma);  // (small grids of CTAs)
      if (s == 0)
        loop_row<PL, false>(L.psi0, L.wave, tr, line, lt, sm, stwr);
      else
        loop_row<PL, true>(L.wave, L.wave, tr, line, lt, sm, stwr);
    }
    if (!loop_barrier<TIGHT, FENCED>(L.sync, ++epoch)) return;
    // ---- column phase ----
    const bool more = s + 1 < L.S;
    if (more) prefetch_rows<PL>(V + L.vstride, G);
    for (int u = g * G + blockIdx.x; u < L.b.nx / 2 / CW; u += GROUPS * G)
      loop_col<PC, CW>(L.b, L.wave, u * CW, cl, t, smem + (g * CW + cl) * SH::COL_SLOT, sky, spy, stwc);
    if (!more) return;
    // the next slice's transmission needs no other CTA's columns: it is formed
    // while the arrivals come in
    const unsigned int seen = loop_arrive<TIGHT, FENCED>(L.sync);
    if (line0 < N) transmission_line<E>(tr, V + L.vstride + (long long)line0 * N, lt, L.a.sigma);
    if (!loop_wait<TIGHT, FENCED>(L.sync, ++epoch, seen)) return;
  }
}

// ---------------------------------------------------------------------------
// Finite-difference loop: all steps of MultisliceStep (U.cu:2040-2083) on the
// band-limited potential planes in one cooperative launch, with the two phases
// and barriers of the slice loop.  Every warp keeps its row of psi_{n-1}, and
// every column thread its part of the spectrum FFT2(psi_n), in registers from
// step to step: a step moves the row-frequency band twice and one plane, where
// the per-pass form also wrote and read psi_n, psi_{n-1} and the spectrum.
// One row per warp and one column unit per group: the launch checks that the
// grid of CTAs is large enough.
// us a step, per-pass kernels in a graph against this: 256^2 6.5 and 4.6, 512^2
// 9.9 and 5.9, 1024^2 14.5 and 11.2.
// ---------------------------------------------------------------------------
template <class PL, class PC, int CW>
__global__ void __launch_bounds__(256, 1) k_fd_loop(FdLoopArgs L) {
  using SH = LoopShape<PL, PC, CW>;
  constexpr int N = PL::N, E = PL::E, P = PL::P, EC = PC::E, PPC = PC::P, GS = SH::GS;
  extern __shared__ float2 smem[];
  float* sky = reinterpret_cast<float*>(smem + SH::KY);
  float2 *stwr = smem + SH::TWR, *stwc = smem + SH::TWC;
  for (int i = threadIdx.x; i < N; i += SH::NT) sky[i] = L.b.ky[i];
  for (int i = threadIdx.x; i < PL::TWSIZE; i += SH::NT) stwr[i] = L.a.tw[i];
  if constexpr (!SH::ONE_TW)
    for (int i = threadIdx.x; i < PC::TWSIZE; i += SH::NT) stwc[i] = L.b.tw[i];
  __syncthreads();
  const int G = gridDim.x;
  const int li = threadIdx.x / P, lt = threadIdx.x % P;
  const int line = li * G + blockIdx.x;
  const bool has_row = line < N;
  const long long row0 = (long long)line * N;
  float2* smr = smem + li * SH::ROW_SLOT;
  const int g = threadIdx.x / GS, gr = threadIdx.x % GS;
  const int cl = gr % CW, t = gr / CW, unit = g * G + blockIdx.x;
  const bool has_col = unit < N / 2 / CW;
  const int col = has_col ? band_column(unit * CW, N) + cl : 0;
  float2* smc = smem + (g * CW + cl) * SH::COL_SLOT;
  float2* wcol = L.wave + (long long)t * N + col;
  const float kx = L.b.kx[col], kx2 = fmul_x(kx, kx);
  unsigned int epoch = 0;

  float2 prev[E];      // psi_{n-1} of this warp's row
  float2 spec[EC / 2]; // FFT2(psi_n): this thread's points of its column, band rows
  float V[E];
  // spectrum of the initial wave
  {
    if (has_row) {
      float2 v[E];
#pragma unroll
      for (int j = 0; j < E; ++j) v[j] = L.psi[row0 + lt + P * j];
      fft::line_fft<PL, 0, false, true, true>(v, smr, lt, stwr);
#pragma unroll
      for (int j = 0; j < E; ++j)
        if (in_band(j, E)) L.wave[row0 + lt + P * j] = v[j];
#pragma unroll
      for (int j = 0; j < E; ++j) prev[j] = L.psim[row0 + lt + P * j];
    }
    if (!loop_barrier<true, false>(L.sync, ++epoch)) return;
    if (has_col) {
      float2 v[EC];
#pragma unroll
      for (int j = 0; j < EC; ++j) v[j] = wcol[(long long)j * PPC * N];
      fft::line_fft<fft::PaddedPlan<PC>, GS, false, true, true>(v, smc, t, stwc);
#pragma unroll
      for (int j = 0; j < EC; ++j)
        if (in_band(j, EC)) spec[j < EC / 4 ? j : j - EC / 2] = v[j];
    }
    const unsigned int seen = loop_arrive<true, false>(L.sync);
    if (has_row) {
#pragma unroll
      for (int j = 0; j < E; ++j) V[j] = L.planes[row0 + lt + P * j];
    }
    if (!loop_wait<true, false>(L.sync, ++epoch, seen)) return;
  }
  for (int s = 0; s < L.S; ++s) {
    const bool more = s + 1 < L.S;
    // ---- row phase: psi_n, the three-level update without its Laplacian ----
    if (has_row) {
      float2 v[E];
      if (s == 0) {
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = L.psi[row0 + lt + P * j];
      } else {
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = in_band(j, E) ? L.wave[row0 + lt + P * j] : make_float2(0.f, 0.f);
        fft::conj_all(v);
        fft::line_fft<PL, 0, true, false, true>(v, smr, lt, stwr);
        fft::conj_all(v);
      }
#pragma unroll
      for (int j = 0; j < E; ++j) {
        const float f = 2.0f - L.a.fd_kv * V[j];
        const float2 q = csub(cmul(L.a.fd_rc, cscale(v[j], f)), cmul(L.a.fd_ratio, prev[j]));
        prev[j] = v[j];
        v[j] = q;
      }
      fft::line_fft<PL, 0, false, true, true>(v, smr, lt, stwr);
#pragma unroll
      for (int j = 0; j < E; ++j)
        if (in_band(j, E)) L.wave[row0 + lt + P * j] = v[j];
      if (!more) {
#pragma unroll
        for (int j = 0; j < E; ++j) L.psim[row0 + lt + P * j] = prev[j];
      }
    }
    if (!loop_barrier<true, false>(L.sync, ++epoch)) return;
    // ---- column phase: + rc dz^2 4 pi^2 k^2 FFT2(psi_n), band limit ----
    if (more) prefetch_rows<PL>(L.planes + (long long)(s + 1) * L.pstride, G);
    if (has_col) {
      float2 v[EC];
#pragma unroll
      for (int j = 0; j < EC; ++j) v[j] = wcol[(long long)j * PPC * N];
      fft::line_fft<fft::PaddedPlan<PC>, GS, false, true, true>(v, smc, t, stwc);
#pragma unroll
      for (int j = 0; j < EC; ++j) {
        if (!in_band(j, EC)) {
          v[j] = make_float2(0.f, 0.f);
          continue;
        }
        const int k = j < EC / 4 ? j : j - EC / 2;
        const float ky = sky[t + PPC * j];
        const bool keep = fadd_x(kx2, fmul_x(ky, ky)) < L.b.k2_le;  // sqrt(k^2) <= kmax
        const float k2 = kx * kx + ky * ky;
        const float2 nv = keep ? cadd(v[j], cscale(cmul(L.b.fd_c, spec[k]), k2)) : make_float2(0.f, 0.f);
        spec[k] = nv;
        v[j] = cscale(nv, L.b.scale);
        if (!more) L.b.spec[(long long)col * N + t + PPC * j] = nv;
      }
      fft::conj_all(v);
      fft::line_fft<fft::PaddedPlan<PC>, GS, true, false, true>(v, smc, t, stwc);
      fft::conj_all(v);
#pragma unroll
      for (int j = 0; j < EC; ++j) wcol[(long long)j * PPC * N] = v[j];
    }
    if (!more) return;
    const unsigned int seen = loop_arrive<true, false>(L.sync);
    if (has_row) {
      const float* Vn = L.planes + (long long)(s + 1) * L.pstride + row0;
#pragma unroll
      for (int j = 0; j < E; ++j) V[j] = Vn[lt + P * j];
    }
    if (!loop_wait<true, false>(L.sync, ++epoch, seen)) return;
  }
}

// ---------------------------------------------------------------------------
// Batched loop: the instances of up to two groups (grid sizes N0 >= N1) share
// every phase.  A row phase covers every line of every instance, a column
// phase every column unit of every instance, with grid barriers between them,
// so the barrier cost is shared by B instance-steps and each warp handles
// several lines per phase.  Lines and units are numbered group 0 first, then
// instance by instance, and dealt round-robin over the CTAs' line slots.
// ---------------------------------------------------------------------------

// Row phase of one line of a batched instance: [IFFT_row] -> x t -> FFT_row
// in place, t = exp(i sigma V) from V on the fly or a stored transmission.
template <class PL, bool TC>
MS_D void batch_row(const LoopGroup& G, int s, int inst, int line, int t, float2* sm, bool first) {
  constexpr int NX = PL::N, E = PL::E, P = PL::P;
  const long long nn = (long long)NX * NX;
  float2* w = G.wave + inst * nn + (long long)line * NX;
  const long long q0 = inst * G.inst_stride + (long long)s * G.slice_stride + (long long)line * NX;
  float2 v[E];
#pragma unroll
  for (int j = 0; j < E; ++j) v[j] = (first || in_band(j, E)) ? w[t + P * j] : make_float2(0.f, 0.f);
  if constexpr (!TC) {
    float vv[E];
#pragma unroll
    for (int j = 0; j < E; ++j) vv[j] = G.Vstack[q0 + t + P * j];
    if (!first) {
      fft::conj_all(v);
      fft::line_fft<PL, 0, true>(v, sm, t, G.a.tw);
      fft::conj_all(v);
    }
    transmit_line<E>(v, vv, G.a.sigma);
  } else {
    float2 tc[E];
#pragma unroll
    for (int j = 0; j < E; ++j) tc[j] = G.tstack[q0 + t + P * j];
    if (!first) {
      fft::conj_all(v);
      fft::line_fft<PL, 0, true>(v, sm, t, G.a.tw);
      fft::conj_all(v);
    }
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = cmul(v[j], tc[j]);
  }
  fft::line_fft<PL, 0, false, true>(v, sm, t, G.a.tw);
#pragma unroll
  for (int j = 0; j < E; ++j)
    if (in_band(j, E)) w[t + P * j] = v[j];
}

// Column phase of one unit of a batched instance: FFT_col, then either the
// propagator and IFFT_col (in place), or, on the last slice of a group with a
// detector, the annular sum of |FFT_col|^2 inside the band limit (the last
// propagation only masks: |FFT2(psi_exit)|^2 = |P|^2 |FFT_col|^2), FP64 per
// warp, added to sig[inst] with the scale 1/N.
template <class PL, int CW>
MS_D void batch_col(const LoopGroup& G, int inst, int c0, int cl, int t, float2* sm, const float* __restrict__ sky,
                    const float2* __restrict__ spy, bool detect) {
  constexpr int NY = PL::N, E = PL::E, P = PL::P, GS = CW * P;
  const int nx = NY;
  const long long nn = (long long)NY * NY;
  float2* base = G.wave + inst * nn;
  const int col = band_column(c0, nx) + cl;
  const float2* src = base + (long long)t * nx + col;
  const int step = P * nx;
  float2 v[E];
#pragma unroll
  for (int j = 0; j < E; ++j) v[j] = src[j * step];
  const ColFactors cf = ColFactors::load<B_PROPAGATE>(G.b, col);
  if (detect) {
    fft::line_fft<fft::PaddedPlan<PL>, GS>(v, sm, t, G.b.tw);
    const float kx2 = fmul_x(cf.kx, cf.kx);
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < E; ++j) {
      const float ky = sky[t + P * j];
      const float k2 = fadd_x(kx2, fmul_x(ky, ky));
      const bool keep = k2 < G.b.k2_lt && k2 >= G.b.kin2 && k2 < G.b.kout2;  // sqrt(k^2) < kmax
      if (keep) acc += v[j].x * v[j].x + v[j].y * v[j].y;
    }
    double d = (double)acc;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d += __shfl_down_sync(0xffffffffu, d, o);
    if ((threadIdx.x & 31) == 0 && d != 0.0) atomicAdd(G.sig + inst, d * (double)G.b.scale);
    return;
  }
  fft::line_fft<fft::PaddedPlan<PL>, GS, false, true>(v, sm, t, G.b.tw);
  col_mid<PL, B_PROPAGATE>(v, G.b, cf, sky, spy, col, t, 0);
  fft::conj_all(v);
  fft::line_fft<fft::PaddedPlan<PL>, GS, true>(v, sm, t, G.b.tw);
  fft::conj_all(v);
  int ostep;
  asm volatile("mov.b32 %0, %1;" : "=r"(ostep) : "r"(step));
  float2* dst = base + (long long)t * nx + col;
#pragma unroll
  for (int j = 0; j < E; ++j) dst[j * ostep] = v[j];
}

template <class PL0, class PL1, int CW>
struct BatchShape {
  using A = LoopShape<PL0, PL0, CW>;
  using B = LoopShape<PL1, PL1, CW>;
  static constexpr int NT = 256;
  static constexpr int LINES_ROWS = NT / 32;  // row lines in flight per CTA
  static constexpr int EXCH = A::EXCH > B::EXCH ? A::EXCH : B::EXCH;
  static constexpr int N0 = PL0::N, N1 = PL1::N;
  // exchange slots, then ky0 | ky1 (floats, padded to float2) and py0 | py1
  static constexpr int KY = (N0 + N1 + 1) / 2;
  static constexpr size_t SMEM = ((size_t)EXCH + KY + N0 + N1) * sizeof(float2);
};

// TC: the groups multiply by stored transmissions (tstack) rather than
// forming exp(i sigma V) from Vstack.
template <class PL0, class PL1, int CW, bool TC>
__global__ void __launch_bounds__(256, 1) k_batch_loop(BatchLoopArgs L) {
  using SH = BatchShape<PL0, PL1, CW>;
  using SA = typename SH::A;
  using SB = typename SH::B;
  static_assert(PL0::P == 32 && PL1::P == 32, "batched loop runs one warp per line");
  constexpr int N0 = PL0::N, N1 = PL1::N, GS = CW * 32, GROUPS = SH::NT / GS;
  extern __shared__ float2 smem[];
  float* sky0 = reinterpret_cast<float*>(smem + SH::EXCH);
  float* sky1 = sky0 + N0;
  float2* spy0 = smem + SH::EXCH + SH::KY;
  float2* spy1 = spy0 + N0;
  const LoopGroup& G0 = L.g[0];
  const LoopGroup& G1 = L.g[1];
  const bool has1 = G1.n > 0 && G1.B > 0;
  for (int i = threadIdx.x; i < N0; i += SH::NT) {
    sky0[i] = G0.b.ky[i];
    spy0[i] = G0.b.py[i];
  }
  if (has1)
    for (int i = threadIdx.x; i < N1; i += SH::NT) {
      sky1[i] = G1.b.ky[i];
      spy1[i] = G1.b.py[i];
    }
  __syncthreads();
  const int G = gridDim.x;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int g = threadIdx.x / GS, gr = threadIdx.x % GS;
  const int cl = gr % CW, t = gr / CW;
  // one slot size for both grids: the CTA's column groups may hold units of
  // different grids at the same time (N0 >= N1, so group 0's slots are the larger)
  constexpr int CSLOT = SA::COL_SLOT > SB::COL_SLOT ? SA::COL_SLOT : SB::COL_SLOT;
  constexpr int RSLOT = SA::ROW_SLOT > SB::ROW_SLOT ? SA::ROW_SLOT : SB::ROW_SLOT;
  static_assert(SH::LINES_ROWS * RSLOT <= SH::EXCH && GROUPS * CW * CSLOT <= SH::EXCH, "exchange slots overflow");
  const long long rows0 = (long long)G0.B * N0, rows1 = has1 ? (long long)G1.B * N1 : 0;
  const long long units0 = (long long)G0.B * (N0 / 2 / CW), units1 = has1 ? (long long)G1.B * (N1 / 2 / CW) : 0;
  unsigned int epoch = 0;
  for (int s = 0; s < L.S; ++s) {
    const bool first = s == 0, last = s + 1 == L.S;
    // ---- row phase: every line of every instance ----
    for (long long r = (long long)warp * G + blockIdx.x; r < rows0 + rows1; r += (long long)SA::LINES * G) {
      float2* sm = smem + warp * RSLOT;
      if (r < rows0)
        batch_row<PL0, TC>(G0, s, (int)(r / N0), (int)(r % N0), lane, sm, first);
      else
        batch_row<PL1, TC>(G1, s, (int)((r - rows0) / N1), (int)((r - rows0) % N1), lane, sm, first);
    }
    if (!loop_barrier<true>(L.sync, ++epoch)) return;
    // ---- column phase: every column unit of every instance ----
    for (long long u = (long long)g * G + blockIdx.x; u < units0 + units1; u += (long long)GROUPS * G) {
      float2* sm = smem + (g * CW + cl) * CSLOT;
      if (u < units0) {
        batch_col<PL0, CW>(G0, (int)(u / (N0 / 2 / CW)), (int)(u % (N0 / 2 / CW)) * CW, cl, t, sm, sky0, spy0,
                           last && G0.sig != nullptr);
      } else {
        const long long v = u - units0;
        batch_col<PL1, CW>(G1, (int)(v / (N1 / 2 / CW)), (int)(v % (N1 / 2 / CW)) * CW, cl, t, sm, sky1, spy1,
                           last && G1.sig != nullptr);
      }
    }
    if (!last && !loop_barrier<true>(L.sync, ++epoch)) return;
  }
}

// Variants of the loop kernel: columns of one warp or two (WIDE: twice the
// warps per column, one more exchange), the column unit width CW and the
// barrier form.
constexpr int kLoopVariants = 10;
template <int CW_, bool WIDE_, bool TIGHT_, bool FENCED_>
struct LoopForm {
  static constexpr int CW = CW_;
  static constexpr bool WIDE = WIDE_, TIGHT = TIGHT_, FENCED = FENCED_;
};
template <int V> struct LoopVariant;
template <> struct LoopVariant<0> : LoopForm<4, false, false, true> {};
template <> struct LoopVariant<1> : LoopForm<8, false, false, true> {};
template <> struct LoopVariant<2> : LoopForm<4, false, true, true> {};
template <> struct LoopVariant<3> : LoopForm<8, false, true, true> {};
template <> struct LoopVariant<4> : LoopForm<2, false, true, true> {};
template <> struct LoopVariant<5> : LoopForm<4, true, true, false> {};
template <> struct LoopVariant<6> : LoopForm<2, true, true, false> {};
template <> struct LoopVariant<7> : LoopForm<2, false, true, false> {};
template <> struct LoopVariant<8> : LoopForm<8, false, true, false> {};
template <> struct LoopVariant<9> : LoopForm<4, false, true, false> {};

// FFT plan variant (PlanSel) of the loop per line length: the packed plan with
// one warp per line (rows, and columns of the narrow variants) or two (wide).
template <int N, bool WIDE>
struct LoopPlan;
template <> struct LoopPlan<256, false> { static constexpr int V = 4; };
template <> struct LoopPlan<512, false> { static constexpr int V = 4; };
template <> struct LoopPlan<1024, false> { static constexpr int V = 3; };
template <> struct LoopPlan<256, true> { static constexpr int V = 5; };
template <> struct LoopPlan<512, true> { static constexpr int V = 5; };
template <> struct LoopPlan<1024, true> { static constexpr int V = 4; };

}  // namespace ms
