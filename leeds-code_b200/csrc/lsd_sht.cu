// lsd_sht.cu -- FP64 associated-Legendre contractions on the Gauss half grid.
//
// Synthesis (spectral -> theta-Fourier) restates the _loop_sumth accumulations of
// tra_spec2phys / tra_qst2rtp / tra_grad (transform.fftw3.F90:472-520, 719-818,
// 955-1000): for each m, Y(j, m, parity) += c_lm * table(j, lm), then the north/south
// recombination Y_even +- Y_odd.  Analysis restates the parity fold and Gauss
// quadrature of tra_phys2spec / tra_leg_trans_p2s_native / tra_rtp2qst
// (transform.fftw3.F90:527-602, 825-949).
//
// Data layouts: spectral [n][H] complex (harmonic fastest, the reference's `spec`
// order; the harmonics of an m-counter are contiguous, l ascending from m, so parity
// (l + m) mod 2 alternates along them); theta-Fourier rows folded into even/odd half-grid
// sums: synthesis writes them in half-row pairs for the FFT (four_off:
// [n][h/2][m-counter][E/O][h%2]), analysis reads them counter-major (four_off_a:
// [m-counter][n][h][E/O]); tables [nh][Th2] (the reference's leg_*(Th2, 0:H-1)).
//
// Both directions are real matrix products per (m-counter, parity): M = theta rows
// (synthesis) or harmonics (analysis), K = harmonics or theta rows, columns = (shell, Re / Im
// of the outputs).  They run on the FP64 tensor instruction m8n8k4, whose products and sums
// are IEEE FP64 fused multiply-adds at the card's full FP64 rate (36.8 TF/s here, FFMA code
// 34.1) with a third of the operand reads of a thread-tiled product.
//
// A CTA (4 warps) takes one counter, 48 M rows and 64 columns; warp = (parity, column half),
// a tile of 6 x 4 m8n8 accumulators.  Both parities of a counter share the staged data, since
// every value enters one parity directly and (vector transforms) the other one crosswise:
//   vector  out0 = a0 T1 (other parity) - i a1 T2 (own), out1 = a1 T1 + i a0 T2
//   scalar  out = a T (own parity; the output's label flips for the theta derivative)
// K runs in chunks of 8 + 8 (both parities) through a three-stage ring of asynchronous
// copies (16-byte, 8-byte where an odd Th2 misaligns the tables), three CTAs per SM.  What bounds
// it: the FP64 tensor pipe at large L, the ring's first fill where a counter has few K.
// At lmax 127, Nr 129 (one evaluation: 4 vector syntheses and a gradient, 2 vector and a scalar
// analysis) 0.47 ms at 60 % of the pipe and 0.30 ms at 80 %; thread-tiled products with a theta row
// or a harmonic per thread took 3.37 and 1.40 ms (2.8 and 3.2 TF/s, waiting for their tables).
#include <type_traits>

#include "lsd_common.cuh"

namespace {

constexpr int LG_MT = 6, LG_BM = 8 * LG_MT;  // m8 tiles and M rows of a CTA
constexpr int LG_NT = 4;                     // n8 tiles of a warp (32 columns)
constexpr int LG_STAGES = 3, LG_THREADS = 128;
constexpr int LG_MAXG = 8, LG_MAXCLASS = 4;
// shared-memory strides, chosen so that the 16 lanes of a 128-byte access of a fragment read
// (4 along K x 4 along the other index) fall in distinct banks:
constexpr int LG_DROW = 17;   // complex per staged (shell, field) row: 16 = 8 K x 2 parities
constexpr int LG_AS = 50;     // synthesis: doubles per table row [kk][48 theta]
constexpr int LG_AA = 10;     // analysis: doubles per table row [harmonic][8 theta]
constexpr int LG_DATA = 32 * LG_DROW * 2;           // doubles of a stage's data
constexpr int LG_TAB_S = 16 * LG_AS, LG_TAB_A = 2 * LG_BM * LG_AA;  // ... of one table tile

// Groups of one launch that share tables: vec: two fields per group, tables T1 (other parity)
// and T2 (own); scalar: one field, table tab[0].
struct LegClass {
  int vec, tab[2];
  int flip, rot, scale;  // scalar synthesis: output parity flipped; times i; times 1/r
  int ng;
  unsigned zero;         // analysis: bit g: drop the imaginary part of m = 0
  const cplx* in[2][LG_MAXG];
  cplx* out[2][LG_MAXG];
};
struct LegArgs {
  int N, H, Th2, NM, HB, mtiles;
  int cols[LG_MAXCLASS];  // column blocks of each class
  const int* mstart;
  const int* mlen;
  const int* hm;
  const double* leg;   // 8 tables [t][H][Th2]
  const double* rinv;  // 1/r per shell
  LegClass k[LG_MAXCLASS];
};

__device__ __forceinline__ uint32_t lg_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// asynchronous copies of 16 / 8 bytes; valid = false writes zeros and reads nothing (the address may
// then lie outside the array)
__device__ __forceinline__ void cp16(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(lg_smem(dst)), "l"(src), "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp8(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(lg_smem(dst)), "l"(src), "r"(valid ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

template <bool ANAL, bool VEC>
__device__ __forceinline__ void leg_tile(const LegArgs& a, const LegClass& k, int col, int cm, double* sm) {
  constexpr int NTAB = VEC ? 2 : 1, SH = VEC ? 16 : 32;  // shells of a CTA's 64 columns
  constexpr int TAB = ANAL ? LG_TAB_A : LG_TAB_S, STAGE = LG_DATA + 2 * TAB;
  const int c = cm / a.mtiles, m0 = (cm - c * a.mtiles) * LG_BM;
  const int nsh = k.ng * a.N, s0 = col * SH;
  const int kbeg = a.mstart[c], klen = a.mlen[c], Th2 = a.Th2;
  if (ANAL && 2 * m0 >= klen) return;
  const int tid = threadIdx.x, lane = tid & 31, par = tid >> 6, half = (tid >> 5) & 1;
  const int lk = lane & 3, lq = lane >> 2;
  // M rows of this warp: theta rows m0 .. (synthesis), harmonics par + 2 (m0 ..) (analysis)
  const int mrows = ANAL ? (klen + 1 - par) / 2 - m0 : Th2 - m0;
  const int klast = ANAL ? 2 * Th2 : klen;  // staged values per (shell, field) row
  const int nch = (klast + 15) / 16;
  const int neg = (lq & 3) == 1 || (lq & 3) == 2 ? (int)0x80000000 : 0;  // sign of segment 2's column lq & 3

  // Copies: addresses are formed once, a chunk only advances them (the index arithmetic of a
  // chunk took six integer instructions per matrix instruction).  Data: value e of the staged
  // rows r0 + 8 i.
  const int e = tid & 15;
  const cplx* src[4];
  int live = 0;  // bit i: the row exists
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = (tid >> 4) + 8 * i, s = s0 + (VEC ? row >> 1 : row), f = VEC ? row & 1 : 0;
    const int g = s / a.N, n = s - g * a.N;
    src[i] = k.in[f][s < nsh ? g : 0] + (ANAL ? four_off_a(n, c, 0, 0, a.N, Th2) : (size_t)n * a.H + kbeg) + e;
    live |= (s < nsh ? 1 : 0) << i;
  }
  // Tables: row tr (+ trs i), doubles tj (+ tjs i) of the tile: 16 rows (kk) x 48 theta, 8 threads a row
  // (synthesis), 96 rows (harmonics) x 8 theta, 4 threads a row of 16-byte, 8 of 8-byte copies
  const bool even = (Th2 & 1) == 0;
  const int tw = even ? 2 : 1, tper = ANAL ? 8 / tw : 8;  // doubles a copy, threads a row
  const int tr = tid / tper, tj = (tid & (tper - 1)) * tw;
  const double* tsrc = a.leg + ((size_t)k.tab[0] * a.H + kbeg + (ANAL ? 2 * m0 : 0) + tr) * Th2 + (ANAL ? 0 : m0) + tj;
  const ptrdiff_t t2 = VEC ? (ptrdiff_t)(k.tab[1] - k.tab[0]) * a.H * Th2 : 0;  // T2 - T1
  const int tdst = tr * (ANAL ? LG_AA : LG_AS) + tj;
  auto issue = [&](int ch) {
    if (ch < nch) {
      double* st = sm + (ch % LG_STAGES) * STAGE;
      const bool in = ch * 16 + e < klast;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        cp16(st + 2 * (((tid >> 4) + 8 * i) * LG_DROW + e), src[i] + ch * 16, in && ((live >> i) & 1));
      double* tb = st + LG_DATA + tdst;
      if (ANAL) {
        const double* p = tsrc + ch * 8;
        const bool jin = ch * 8 + tj < Th2;
        const int rest = klen - 2 * m0 - tr;  // rows of this counter from tr on
        if (even) {
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int t = 0; t < NTAB; ++t)
              cp16(tb + t * TAB + 32 * i * LG_AA, p + t * t2 + (ptrdiff_t)(32 * i) * Th2, jin && 32 * i < rest);
        } else {
#pragma unroll
          for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int t = 0; t < NTAB; ++t)
              cp8(tb + t * TAB + 16 * i * LG_AA, p + t * t2 + (ptrdiff_t)(16 * i) * Th2, jin && 16 * i < rest);
        }
      } else {
        const double* p = tsrc + (ptrdiff_t)(ch * 16) * Th2;
        const bool rin = ch * 16 + tr < klen;
        const int rest = Th2 - m0 - tj;
        if (even) {
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int t = 0; t < NTAB; ++t)
              cp16(tb + t * TAB + 16 * i, p + t * t2 + 16 * i, rin && 16 * i < rest);
        } else {
#pragma unroll
          for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int t = 0; t < NTAB; ++t)
              cp8(tb + t * TAB + 8 * i, p + t * t2 + 8 * i, rin && 8 * i < rest);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  double acc[LG_MT][LG_NT][2];
#pragma unroll
  for (int i = 0; i < LG_MT; ++i)
#pragma unroll
    for (int j = 0; j < LG_NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  for (int i = 0; i < LG_STAGES - 1; ++i) issue(i);
  for (int ch = 0; ch < nch; ++ch) {
    asm volatile("cp.async.wait_group %0;" ::"n"(LG_STAGES - 2) : "memory");
    __syncthreads();  // chunk ch has landed for every thread; chunk ch - 1's stage is free
    issue(ch + LG_STAGES - 1);
    const double* st = sm + (ch % LG_STAGES) * STAGE;
    auto multiply = [&](auto full) {  // full: no M tile to leave out
#pragma unroll
      for (int seg = 0; seg < NTAB; ++seg) {
        const int dp = VEC && seg == 0 ? 1 - par : par;  // parity of the data of this segment
        const double* tb = st + LG_DATA + seg * TAB;
#pragma unroll
        for (int q = 0; q < 2; ++q) {  // four K of each parity
          if (ch * 16 + 8 * q >= klast) break;
          const int ki = dp + 2 * (4 * q + lk);
          double b[LG_NT];
#pragma unroll
          for (int j = 0; j < LG_NT; ++j) {
            const int col = half * 32 + j * 8 + lq;
            if (VEC) {  // columns: Re, Im of out0, Re, Im of out1 of a shell
              const int comp = col & 3, f = seg ? 1 - (comp >> 1) : comp >> 1, part = seg ? 1 - (comp & 1) : comp & 1;
              const double x = st[2 * (((col >> 2) * 2 + f) * LG_DROW + ki) + part];
              b[j] = seg ? __hiloint2double(__double2hiint(x) ^ neg, __double2loint(x)) : x;
            } else {
              b[j] = st[2 * ((col >> 1) * LG_DROW + ki) + (col & 1)];
            }
          }
#pragma unroll
          for (int i = 0; i < LG_MT; ++i) {
            if (decltype(full)::value || i * 8 < mrows) {
              const double av = ANAL ? tb[(par + 2 * (i * 8 + lq)) * LG_AA + 4 * q + lk] : tb[ki * LG_AS + i * 8 + lq];
#pragma unroll
              for (int j = 0; j < LG_NT; ++j) dmma(acc[i][j], av, b[j]);
            }
          }
        }
      }
    };
    if (mrows >= LG_BM) multiply(std::true_type());
    else multiply(std::false_type());
  }

  // accumulators: M row lq, columns 2 lk, 2 lk + 1 (Re, Im) of each tile
#pragma unroll
  for (int j = 0; j < LG_NT; ++j) {
    const int col = half * 32 + j * 8 + 2 * lk, s = s0 + (VEC ? col >> 2 : col >> 1);
    if (s >= nsh) continue;
    const int g = s / a.N, n = s - g * a.N;
    cplx* out = k.out[VEC ? (col >> 1) & 1 : 0][g];
    if (ANAL) {
      out += (size_t)n * a.H + kbeg + par;
      const bool zero = ((k.zero >> g) & 1) && a.hm[kbeg] == 0;
#pragma unroll
      for (int i = 0; i < LG_MT; ++i)
        if (i * 8 + lq < mrows) out[2 * (m0 + i * 8 + lq)] = make_double2(acc[i][j][0], zero ? 0.0 : acc[i][j][1]);
    } else {  // theta rows m0 + 8 i + lq: 4 half-row pairs of four_off apart
      const int po = k.flip ? 1 - par : par;
      cplx* o = out + four_off(n, c, po, m0 + lq, a.NM, a.HB);
      const size_t step = (size_t)a.NM * 16;
      const double f = k.scale ? a.rinv[n] : 1.0;
#pragma unroll
      for (int i = 0; i < LG_MT; ++i)
        if (i * 8 + lq < mrows) {
          const double x = acc[i][j][0] * f, y = acc[i][j][1] * f;
          o[i * step] = k.rot ? make_double2(-y, x) : make_double2(x, y);
        }
    }
  }
}

// grid: (counters x M tiles) of every column block of every class, one class after another (a grid
// of the largest class's column blocks for all classes spent 8 % on CTAs without work)
template <bool ANAL>
__global__ void __launch_bounds__(LG_THREADS, 3) k_leg(LegArgs a) {
  extern __shared__ __align__(16) double lg_sm[];
  const int per = a.NM * a.mtiles;
  int col = blockIdx.x / per, z = 0;
  const int cm = blockIdx.x - col * per;
  while (col >= a.cols[z]) col -= a.cols[z++];
  const LegClass& k = a.k[z];
  if (k.vec) leg_tile<ANAL, true>(a, k, col, cm, lg_sm);
  else leg_tile<ANAL, false>(a, k, col, cm, lg_sm);
}

// The classes of a launch: add() opens a class for its tables or joins the open one.
struct LegBuilder {
  LegArgs a{};
  int nc = 0;
  LegClass* find(int vec, int t1, int t2, int flip, int rot, int scale) {
    for (int i = 0; i < nc; ++i) {
      LegClass& k = a.k[i];
      if (k.vec == vec && k.tab[0] == t1 && k.tab[1] == t2 && k.rot == rot && k.ng < LG_MAXG) return &k;
    }
    if (nc == LG_MAXCLASS) return nullptr;
    LegClass& k = a.k[nc++];
    k = LegClass{};
    k.vec = vec; k.tab[0] = t1; k.tab[1] = t2; k.flip = flip; k.rot = rot; k.scale = scale;
    return &k;
  }
  bool add(LegClass* k, const cplx* i0, const cplx* i1, cplx* o0, cplx* o1, bool zero) {
    if (!k) return false;
    k->in[0][k->ng] = i0; k->in[1][k->ng] = i1;
    k->out[0][k->ng] = o0; k->out[1][k->ng] = o1;
    if (zero) k->zero |= 1u << k->ng;
    k->ng++;
    return true;
  }
};

template <bool ANAL>
int launch_leg(lsd_ctx* ctx, LegBuilder& b) {
  if (b.nc == 0) return LSD_OK;
  LegArgs& a = b.a;
  for (int i = 1; i < b.nc; ++i)  // the vector class, whose tiles are the longest, first
    if (a.k[i].vec && !a.k[0].vec) {
      const LegClass t = a.k[0];
      a.k[0] = a.k[i];
      a.k[i] = t;
    }
  a.N = ctx->N; a.H = ctx->H; a.Th2 = ctx->Th2; a.NM = ctx->NM; a.HB = ctx->HB;
  a.mstart = ctx->d_mstart; a.mlen = ctx->d_mlen; a.hm = ctx->d_m; a.leg = ctx->d_leg; a.rinv = ctx->d_rinv;
  int klmax = 0, cols = 0;
  for (int c = 0; c < ctx->NM; ++c) klmax = ctx->mlen[c] > klmax ? ctx->mlen[c] : klmax;
  a.mtiles = ANAL ? ceil_div((klmax + 1) / 2, LG_BM) : ceil_div(ctx->Th2, LG_BM);
  for (int i = 0; i < b.nc; ++i) {
    a.cols[i] = ceil_div(a.k[i].ng * ctx->N, a.k[i].vec ? 16 : 32);
    cols += a.cols[i];
  }
  const size_t smem = sizeof(double) * LG_STAGES * (LG_DATA + 2 * (ANAL ? LG_TAB_A : LG_TAB_S));
  CUDA_TRY(cudaFuncSetAttribute(k_leg<ANAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_leg<ANAL><<<ctx->NM * a.mtiles * cols, LG_THREADS, smem, ctx->stream>>>(a);
  ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return lsd_fail(ctx, LSD_ECUDA, std::string("k_leg: ") + cudaGetErrorString(e));
  return LSD_OK;
}

}  // namespace

int lsd_launch_synth(lsd_ctx* ctx, const SynthGroup* groups, int ngroups) {
  if (lsd_ozaki_use_synth(ctx)) return lsd_ozaki_launch_synth(ctx, groups, ngroups);
  LegBuilder b;
  bool ok = true;
  auto scalar = [&](const cplx* in, cplx* out, int tab, int flip, int rot, int scale) {
    ok = ok && b.add(b.find(0, tab, -1, flip, rot, scale), in, nullptr, out, nullptr, false);
  };
  for (int i = 0; i < ngroups; ++i) {
    const SynthGroup& G = groups[i];
    if (G.kind == SK_VECTOR) {
      scalar(G.in[0], G.out[0], LSD_LEG_P, 0, 0, 0);
      ok = ok && b.add(b.find(1, LSD_LEG_LLP_, LSD_LEG_LLSIN1MP, 0, 0, 0), G.in[1], G.in[2], G.out[1], G.out[2], false);
    } else if (G.kind == SK_SCALAR) {
      scalar(G.in[0], G.out[0], LSD_LEG_P, 0, 0, 0);
    } else {  // gradients: (C/r) dP/dtheta, i (C/r) m P / sin(theta)
      const bool three = G.kind == SK_GRAD3;
      if (three) scalar(G.in[0], G.out[0], LSD_LEG_P, 0, 0, 0);
      scalar(G.in[three ? 1 : 0], G.out[three ? 1 : 0], LSD_LEG_P_, 1, 0, 1);
      scalar(G.in[three ? 1 : 0], G.out[three ? 2 : 1], LSD_LEG_SIN1MP, 0, 1, 1);
    }
  }
  if (!ok) return lsd_fail(ctx, LSD_EARG, "synthesis: too many groups in one launch");
  return launch_leg<false>(ctx, b);
}

int lsd_launch_anal(lsd_ctx* ctx, const AnalGroup* groups, int ngroups) {
  if (lsd_ozaki_use_anal(ctx)) return lsd_ozaki_launch_anal(ctx, groups, ngroups);
  // k_leg has no such limit; longer columns (L > 512) are outside what is tested
  if (ceil_div(ctx->Hr, 32) * 32 > 1024) return lsd_fail(ctx, LSD_EARG, "analysis: folded column longer than 1024 harmonics");
  LegBuilder b;
  bool ok = true;
  for (int i = 0; i < ngroups; ++i) {
    const AnalGroup& G = groups[i];
    const bool vec = G.kind == AK_VECTOR;  // q keeps Im of m = 0 (transform.fftw3.F90:869)
    ok = ok && b.add(b.find(0, LSD_LEG_GWP, -1, 0, 0, 0), G.in[0], nullptr, G.out[0], nullptr, !vec);
    if (vec)
      ok = ok && b.add(b.find(1, LSD_LEG_GWLLP_, LSD_LEG_GWLLSIN1MP, 0, 0, 0), G.in[1], G.in[2], G.out[1], G.out[2], true);
  }
  if (!ok) return lsd_fail(ctx, LSD_EARG, "analysis: too many groups in one launch");
  return launch_leg<true>(ctx, b);
}
