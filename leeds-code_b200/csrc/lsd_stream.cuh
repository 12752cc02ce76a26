// lsd_stream.cuh -- banded solves streamed through shared memory.
//
// A warp owns 32 consecutive degrees l of one order m (lane = degree) and walks the radial rows of
// their columns; a CTA takes the same 32 degrees of T / 32 orders, so its warps share the factors,
// which depend on l alone.  The rows of a pass -- the lane's own column values and the CTA's
// factor rows -- arrive by 16-byte asynchronous copies in a ring of SvRing::ST stages of SV_B rows, 12
// rows ahead of the arithmetic (8 for KL > 3); rows outside the system arrive as zeros, so that
// every step of a pass does the same work and only its stores are guarded.
//
// Factors in the solve layouts: per (family, block of 32 degrees) the rows -SV_PAD .. NL + SV_PAD - 1
// (zeros outside the system) of
//   L rows  [KL + 1][32]    L(c+1, c) .. L(c+KL, c), then the pivot's offset p(c) - c (an integer's bits)
//   U rows  [2 KL + 2][32]  U(c, c), U(c-1, c) .. U(c-2KL, c), then the reciprocal of U(c, c)
//   Y rows  [2 KL + 1][32]  the entries of row n of the Y band on X(n-KL) .. X(n+KL)
// so that a stage's factors are one contiguous piece.
//
// What bounds a solve is the chain of dependent rows (a row swap and a fused multiply-add each
// way) and, with many columns, the instructions of a row.  So no load stands in the chain (a
// row loaded when it is needed costs 0.7 us per batch of rows) and no division (114 cycles): x / d is
// formed from the stored reciprocal with one correction step (Markstein, IBM J. Res. Dev. 34, 111
// (1990): q = x r, then q + (x - q d) r).  q is off by at most 2^-52 of itself and r by 2^-53, so
// the sum before its rounding is off by 2^-105: the rounded quotient, but for quotients that
// close to a tie, as long as r is a normal number (the factorisation multiplies by the same
// reciprocals) and |x| is above 2^-968, where x - q d is exact.  Sharing the factors between four
// orders takes their traffic from 84 to 21 bytes per column row and pass.  All passes of a column
// run through one copy of the code (a loop over pass descriptors): with a copy per pass the
// short columns of a small run waited for instruction fetches half of their time.
// Five fields of a step (8256 harmonics, N = 129, KL = 3): predictor 0.150 ms, corrector 0.163 ms; one
// thread per harmonic with batches of eight rows loaded when needed 0.367 and 0.355 ms.  At L = 16,
// N = 17: 25 and 30 us (37 and 40).  Five fields at N = 257, KL = 4, 32896 harmonics (operator
// solves) 0.75 ms (1.14).
#pragma once
#include "lsd_common.cuh"

namespace {

constexpr int SV_B = 4;  // rows per ring stage
constexpr int SV_NS = 2;  // column streams of a pass
__host__ __device__ constexpr int sv_pad(int KL) { return 2 * KL + SV_B; }
__host__ __device__ constexpr int sv_rows(int n, int KL) { return n + 2 * sv_pad(KL); }
// ring stages: as many as leave room for two CTAs of 128 threads per SM
template <int KL> struct SvRing { static constexpr int ST = KL <= 3 ? 4 : 3; };
template <int KL>
__host__ __device__ constexpr size_t sv_stage(int T) {
  return sizeof(double2) * SV_NS * SV_B * T + sizeof(double) * (3 * KL + 2) * SV_B * 32;
}
template <int KL>
__host__ __device__ constexpr size_t sv_smem(int T) { return SvRing<KL>::ST * sv_stage<KL>(T); }

// row 0 of (family fam, degree block lb) in the solve layouts, rows of e entries
__host__ __device__ __forceinline__ size_t sv_row0(int fam, int lb, int nlb, int n, int KL, int e) {
  return (((size_t)fam * nlb + lb) * sv_rows(n, KL) + sv_pad(KL)) * e * 32;
}

__device__ __forceinline__ void sv_cp16(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ double2 axpy2(double2 y, double a, double2 x) {  // y + a x
  return make_double2(y.x + a * x.x, y.y + a * x.y);
}
// x / d from r = the rounded 1 / d.  An infinite or NaN x r stays as it is (inf / d = inf; the
// correction would make it NaN); the select costs 0.7 % of a solve, a branch to a division 4 to 10 %.
__device__ __forceinline__ double sv_div(double x, double d, double r) {
  const double q = x * r, e = fma(-q, d, x);
  return fma((__double2hiint(q) & 0x7fffffff) < 0x7ff00000 ? e : 0.0, r, q);
}

// One pass over the N rows of a system, a thread's column (row stride rst) and its CTA's factors.
//  SV_FWD    dgbtrs forward part (LAPACK order) on r(n): for c = 0..N-1 swap rows c and p(c), then
//            x(c+i) -= L(c+i, c) x(c), i <= KL; out(c) = x(c).  r(n) is in0(n), or with diff
//            scale (in0(n) - in1(n)) (tim_nlincorr, timestep.F90:696-715); save(n) = in0(n).
//  SV_FWDY   the same on r(n) + (Y X)(n), X = in0 (tim_multY, timestep.F90:640-670), r = in1; save = r.
//            (With zero L rows: the product alone.)
//  SV_BWD    dtbsv (upper, non-unit, bandwidth 2KL; LAPACK column order) on in0: for c = N-1..0:
//            x(c) = y(c) / U(c, c); x(c-t) -= x(c) U(c-t, c); out(c) = x(c), or with add in1(c) + x(c)
//            (tim_addcorr, timestep.F90:717-737), squares summed.  Keeps x(0), x(N-1).
//  SV_GREEN  d = in0(n) - ca g1(n) - cb g2(n), F the rows [2][32] of the two functions; out as SV_BWD.
// r's boundary rows 0 and N-1 are replaced by (b0, 0) and (bN, 0).  unit: r is (1, 0) at row 0, (0, 1) at
// row N-1, else 0 (the two Green's functions; in0 is not read).
// IC: a system over both cores: rows below brk lie in the first of each pair of arrays, the others
// in the second (whose base is set so that row n is base + n rst); row brk of the right-hand side is 0
// and its result goes to both cores (xb: the first's old value, with add); rot: the first core's r is
// -omega d/dphi of its field, r = (om y, -om x) of X (SV_FWDY) or in0 (diff), om = omega m.
enum SvKind { SV_FWD = 0, SV_FWDY, SV_BWD, SV_GREEN };
struct SvPass {
  int kind, N;
  const double* F;
  const double* Y;
  const double2 *in0, *in1, *in0b, *in1b;
  double2 *save, *saveb, *out, *outb;
  bool diff, add, rot, unit;
  int brk;
  double b0, bN;
  double2 ca, cb, xb;
};
// what a column's passes share
struct SvCta {
  unsigned char* sm;
  int T, tid;
  bool on;      // this thread owns a column
  size_t rst;
  double scale, om;
};
struct SvSums { double ss, ssic; double2 x0, xN; };

// the stage's rows of both streams: rows r0, r0 + dr, ... (SV_B of them)
template <bool IC>
__device__ __forceinline__ void sv_rows_in(const SvCta& k, const SvPass& p, double2* dst, const double2* lo,
                                           const double2* hi, int r0, int dr) {
#pragma unroll
  for (int u = 0; u < SV_B; ++u) {
    const int r = r0 + u * dr;
    const double2* base = IC && r >= p.brk ? hi : lo;
    sv_cp16(dst + u * k.T, base + (ptrdiff_t)r * (ptrdiff_t)k.rst, k.on && (unsigned)r < (unsigned)p.N ? 16 : 0);
  }
}
// n doubles (a multiple of 2) of contiguous factors
__device__ __forceinline__ void sv_factors_in(const SvCta& k, double* dst, const double* src, int n) {
  for (int i = k.tid * 2; i < n; i += k.T * 2) sv_cp16(dst + i, src + i, 16);
}

// The ring around a pass: fill(stage, b) queues batch b's copies, body(stage, b) works on it.
template <int KL, class FILL, class BODY>
__device__ __forceinline__ void sv_ring(const SvCta& k, int nsteps, FILL&& fill, BODY&& body) {
  constexpr int ST = SvRing<KL>::ST;
  const int nb = (nsteps + SV_B - 1) / SV_B;
  const size_t stage = sv_stage<KL>(k.T);
  auto issue = [&](int b) {
    if (b < nb) fill(k.sm + (b % ST) * stage, b);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  __threadfence_block();
  __syncthreads();  // the ring is free; this thread's stores of the last pass are performed
  for (int b = 0; b < ST - 1; ++b) issue(b);
  for (int b = 0; b < nb; ++b) {
    asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
    __syncthreads();
    issue(b + ST - 1);
    body(k.sm + (b % ST) * stage, b);
  }
}

// the result d of row c of a backward or Green's pass
template <bool IC>
__device__ __forceinline__ void sv_result(const SvCta& k, const SvPass& p, SvSums& s, int c, double2 d, double2 old) {
  if (c == 0) s.x0 = d;
  if (c == p.N - 1) s.xN = d;
  if (k.on && (unsigned)c < (unsigned)p.N) {
    double2 v = d;
    const double sq = d.x * d.x + d.y * d.y;
    const bool hi = IC && c >= p.brk;
    if (p.add) {
      v = make_double2(old.x + d.x, old.y + d.y);
      if (IC && !hi && p.brk < p.N) s.ssic = s.ssic + sq;
      else s.ss = s.ss + sq;
    }
    (hi ? p.outb : p.out)[(ptrdiff_t)c * (ptrdiff_t)k.rst] = v;
    if (IC && c == p.brk) {
      if (p.add) {
        v = make_double2(p.xb.x + d.x, p.xb.y + d.y);
        s.ssic = s.ssic + sq;
      }
      p.out[(ptrdiff_t)c * (ptrdiff_t)k.rst] = v;
    }
  }
}

template <int KL, bool Y, bool IC>
__device__ __forceinline__ void sv_forward(const SvCta& k, const SvPass& p) {
  constexpr int LDM = 2 * KL + 1, OFF = Y ? KL : 0, EL = KL + 1;
  const int N = p.N, T = k.T, lane = k.tid & 31;
  const size_t fofs = sizeof(double2) * SV_NS * SV_B * T;
  const bool two = Y ? p.in1 != nullptr || p.in1b != nullptr : p.diff;
  double2 w[KL + 1], xw[LDM];
#pragma unroll
  for (int i = 0; i <= KL; ++i) w[i] = make_double2(0.0, 0.0);
#pragma unroll
  for (int i = 0; i < LDM; ++i) xw[i] = make_double2(0.0, 0.0);
  sv_ring<KL>(
      k, N + KL + OFF,
      [&](unsigned char* st, int b) {
        const int t = b * SV_B;
        double2* sd = (double2*)st + k.tid;
        if (!p.unit) sv_rows_in<IC>(k, p, sd, p.in0, p.in0b, t, 1);
        if (two) sv_rows_in<IC>(k, p, sd + SV_B * T, p.in1, p.in1b, t - OFF, 1);
        double* fd = (double*)(st + fofs);
        sv_factors_in(k, fd, p.F + (ptrdiff_t)(t - OFF - KL) * (EL * 32), SV_B * EL * 32);
        if (Y) sv_factors_in(k, fd + SV_B * EL * 32, p.Y + (ptrdiff_t)(t - OFF) * (LDM * 32), SV_B * LDM * 32);
      },
      [&](const unsigned char* st, int b) {
        const double2* sd = (const double2*)st + k.tid;
        const double* fl = (const double*)(st + fofs) + lane;
        const double* fy = fl + SV_B * EL * 32;
#pragma unroll
        for (int u = 0; u < SV_B; ++u) {
          const int n = b * SV_B + u - OFF, c = n - KL;
          const double2 a = sd[u * T];
          if (Y) {
#pragma unroll
            for (int i = 0; i < LDM - 1; ++i) xw[i] = xw[i + 1];
            xw[LDM - 1] = a;
          }
          double2 r = a;
          if (Y) r = two ? sd[(SV_B + u) * T] : make_double2(0.0, 0.0);
          const bool hi = IC && n >= p.brk;
          if (IC && p.rot && !hi) {
            const double2 x = Y ? xw[KL] : a;
            r = make_double2(k.om * x.y, -(k.om * x.x));
          }
          double2* sv = hi ? p.saveb : p.save;
          if (sv && k.on && (unsigned)n < (unsigned)N) sv[(ptrdiff_t)n * (ptrdiff_t)k.rst] = r;
          if (!Y && p.diff) {
            const double2 q = sd[(SV_B + u) * T];
            r = make_double2(k.scale * (r.x - q.x), k.scale * (r.y - q.y));
          }
          if (Y) {
#pragma unroll
            for (int i = 0; i < LDM; ++i) r = axpy2(r, fy[(u * LDM + i) * 32], xw[i]);
          }
          if (!Y && p.unit) r = make_double2(0.0, 0.0);
          if (n == 0) r = make_double2(!Y && p.unit ? 1.0 : p.b0, 0.0);
          if (n == N - 1) r = !Y && p.unit ? make_double2(0.0, 1.0) : make_double2(p.bN, 0.0);
          if (IC && n == p.brk) r = make_double2(0.0, 0.0);
          w[KL] = r;
          const int pv = *(const int*)(fl + (u * EL + KL) * 32);
          if (__any_sync(0xffffffffu, pv != 0)) {  // rows are seldom swapped
#pragma unroll
            for (int i = 1; i <= KL; ++i)
              if (pv == i) { const double2 x = w[0]; w[0] = w[i]; w[i] = x; }
          }
          const double2 m = make_double2(-w[0].x, -w[0].y);
#pragma unroll
          for (int i = 1; i <= KL; ++i) w[i] = axpy2(w[i], fl[(u * EL + i - 1) * 32], m);
          if (k.on && (unsigned)c < (unsigned)N)
            (IC && c >= p.brk ? p.outb : p.out)[(ptrdiff_t)c * (ptrdiff_t)k.rst] = w[0];
#pragma unroll
          for (int i = 0; i < KL; ++i) w[i] = w[i + 1];
        }
      });
}

template <int KL, bool IC>
__device__ __forceinline__ void sv_backward(const SvCta& k, const SvPass& p, SvSums& s) {
  constexpr int K2 = 2 * KL, EU = K2 + 2;
  const int N = p.N, T = k.T, lane = k.tid & 31;
  const size_t fofs = sizeof(double2) * SV_NS * SV_B * T;
  double2 w[K2 + 1];
#pragma unroll
  for (int i = 0; i <= K2; ++i) w[i] = make_double2(0.0, 0.0);
  sv_ring<KL>(
      k, N + K2,
      [&](unsigned char* st, int b) {
        const int n = N - 1 - b * SV_B;
        double2* sd = (double2*)st + k.tid;
        sv_rows_in<IC>(k, p, sd, p.in0, p.in0b, n, -1);
        if (p.add) sv_rows_in<IC>(k, p, sd + SV_B * T, p.in1, p.in1b, n + K2, -1);
        sv_factors_in(k, (double*)(st + fofs), p.F + (ptrdiff_t)(n + K2 - (SV_B - 1)) * (EU * 32), SV_B * EU * 32);
      },
      [&](const unsigned char* st, int b) {
        const double2* sd = (const double2*)st + k.tid;
        const double* fu = (const double*)(st + fofs) + lane;
#pragma unroll
        for (int u = 0; u < SV_B; ++u) {
          const int c = N - 1 - (b * SV_B + u) + K2;
          const double* f = fu + (SV_B - 1 - u) * EU * 32;
          w[K2] = sd[u * T];
          const double d = f[0], r = f[(K2 + 1) * 32];
          const double2 x = make_double2(sv_div(w[0].x, d, r), sv_div(w[0].y, d, r));
          sv_result<IC>(k, p, s, c, x, p.add ? sd[(SV_B + u) * T] : x);
          const double2 m = make_double2(-x.x, -x.y);
#pragma unroll
          for (int i = 1; i <= K2; ++i) w[i] = axpy2(w[i], f[i * 32], m);
#pragma unroll
          for (int i = 0; i < K2; ++i) w[i] = w[i + 1];
        }
      });
}

template <int KL>
__device__ __forceinline__ void sv_green(const SvCta& k, const SvPass& p, SvSums& s) {
  const int T = k.T, lane = k.tid & 31;
  const size_t fofs = sizeof(double2) * SV_NS * SV_B * T;
  sv_ring<KL>(
      k, p.N,
      [&](unsigned char* st, int b) {
        const int n = b * SV_B;
        double2* sd = (double2*)st + k.tid;
        sv_rows_in<false>(k, p, sd, p.in0, nullptr, n, 1);
        if (p.add) sv_rows_in<false>(k, p, sd + SV_B * T, p.in1, nullptr, n, 1);
        sv_factors_in(k, (double*)(st + fofs), p.F + (size_t)n * 64, SV_B * 64);
      },
      [&](const unsigned char* st, int b) {
        const double2* sd = (const double2*)st + k.tid;
        const double* f = (const double*)(st + fofs) + lane;
#pragma unroll
        for (int u = 0; u < SV_B; ++u) {
          const double g1 = f[u * 64], g2 = f[u * 64 + 32];
          const double2 x = sd[u * T];
          const double2 d = make_double2(x.x - p.ca.x * g1 - p.cb.x * g2, x.y - p.ca.y * g1 - p.cb.y * g2);
          sv_result<false>(k, p, s, b * SV_B + u, d, p.add ? sd[(SV_B + u) * T] : d);
        }
      });
}

// One pass; YP, GP: passes with Y / Green's passes occur
template <int KL, bool YP, bool GP, bool IC>
__device__ __forceinline__ void sv_run(const SvCta& k, const SvPass& p, SvSums& s) {
  if (YP && p.kind == SV_FWDY) sv_forward<KL, true, IC>(k, p);
  else if (p.kind == SV_FWD) sv_forward<KL, false, IC>(k, p);
  else if (p.kind == SV_BWD) sv_backward<KL, IC>(k, p, s);
  else if (GP) sv_green<KL>(k, p, s);
}

}  // namespace
