// Device kernels of the pnFAM solver (sm_103a).
//
// One FAM iteration (pnfam_solver.f90:114-209) for a batch of omega points:
//   k_gemm        grouped multi-term FP64 block GEMM, used for the basis
//                 changes dR_qp -> dR_sp (pnfam_solver.f90:144-150) and
//                 dH_sp -> dH_qp (:160-166), and F_sp -> F_qp (:368-381)
//   k_density     fused sum_a phi_a rho_ab + reduction over b into the 28
//                 local densities (pnfam_hamiltonian_blas.f90:124-711)
//   k_meanfield   densities -> field tensor mf(0:4,0:4,s,s') and the pairing
//                 fields (pnfam_hamiltonian_blas.f90:775-1094, 1201-1208)
//   k_hproj       h_ab = 2 sum_r phi_a (mf phi_b), Delta_ab likewise
//                 (pnfam_hamiltonian_blas.f90:1107-1167, 1212-1260)
//   k_green       dR = G o (q dH + F)  (pnfam_solver.f90:169-183, 510-544)
//   k_bro_*       modified Broyden mixing (pnfam_broyden.f90:117-216)
//   k_contract    S = -1/pi sum F dR  (pnfam_type_bbm.f90:393-421)
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "tc.cuh"
#include "pair_arith.cuh"

namespace pnfam {

// ---------------------------------------------------------------------------
// grouped multi-term GEMM
// ---------------------------------------------------------------------------
enum BufId { B_UP = 0, B_VP, B_UN, B_VN, B_STATE, B_T, B_RSP, B_HSP, B_HQP, NBUF };

template <class T>
struct BufDescT {
  T* base;
  long long sp;   // stride between points
  long long spl;  // stride between the Re and Im planes
};
using BufDesc = BufDescT<double>;

struct GemmTerm {
  long long aoff, boff;
  int abuf, bbuf;
  int lda, ldb;
  int tA, tB;          // 0 = as stored, 1 = transposed
  double alpha[2];     // per plane (Re, Im)
};

#define PNFAM_MAXTERM 4
struct GemmTask {
  int M, N, K, nterm;
  GemmTerm t[PNFAM_MAXTERM];
  long long coff;
  int cbuf, ldc;
  int tile0, ntm;      // first tile in the flattened grid, tiles along M
  int mr, nc;          // rows and columns of a tile
};

enum { GT_K = 16, GT_THREADS = 256, GT_R = 8, GT_SIDE = 96 };   // GT_SIDE: most rows or columns of a tile

template <class T>
__device__ __forceinline__ const T* bufptr(const BufDescT<T>* b, int id, int p, int plane, long long off) {
  const BufDescT<T> d = b[id];
  return d.base + (long long)p * d.sp + (long long)plane * d.spl + off;
}

// dst[kk * ld + i] = al * element (x0 + i, k0 + kk) for i < n, kk < kl; kfast: k is
// consecutive in memory (i at stride lds), otherwise i is (k at stride lds)
__device__ __forceinline__ void gemm_stage(const double* __restrict__ src, int lds, bool kfast, int x0, int n, int k0,
                                           int kl, double al, double* __restrict__ dst, int ld) {
  if (kfast) {
    const int kk = threadIdx.x % GT_K;
    if (kk >= kl) return;
    const double* s = src + k0 + kk + (long long)x0 * lds;
    for (int i = threadIdx.x / GT_K; i < n; i += GT_THREADS / GT_K) dst[kk * ld + i] = al * s[(long long)i * lds];
  } else {
    // (i, kk) of element threadIdx.x + 256 j without a division per element
    const int di = GT_THREADS % n, dk = GT_THREADS / n;
    int i = threadIdx.x % n, kk = threadIdx.x / n;
    const double* s = src + x0 + (long long)k0 * lds;
    while (kk < kl) {
      dst[kk * ld + i] = al * s[i + (long long)kk * lds];
      i += di; kk += dk;
      if (i >= n) { i -= n; ++kk; }
    }
  }
}

// C = sum_t alpha_t op(A_t) op(B_t) in FP64 for both planes (Re, Im) of one point.
// The DFMA rate bounds it (a warp's DFMA takes the SM's FP64 pipe 16 cycles, its two
// shared-memory reads 3), so what counts is that no lane works on padding: the mr x nc x 2
// outputs of a tile are dealt to the threads in one row, element e = thread + 256 i (rows
// fastest: reads of the row operand are consecutive, those of the column operand mostly
// one address), K runs over the block's own size, and the ground-state operand is staged
// once for both planes.  Against tiles of 1024 outputs padded in M, N and K: N_sh = 8, 40
// points, 23 against 56 ms per solve, N_sh = 6 11 against 22 us per launch; at N_sh = 16
// (blocks 1 to 81, nine points) 1.04 TFLOP/s (a DGEMM reaches 1.1) against 0.69, and with
// shared products and active quasiparticles only 0.33 ms per point against 1.01.  Every
// output sums over the terms and k in order.  Of the two operands of a term one is the
// point's (two planes), one the ground state's; alpha (+-1) goes into the point's.  grid (tiles, P)
__global__ void __launch_bounds__(GT_THREADS) k_gemm(const GemmTask* __restrict__ tasks,
                                                     const int* __restrict__ tile2task,
                                                     const BufDescT<double>* __restrict__ bufs,
                                                     const int* __restrict__ active) {
  const int p = blockIdx.y;
  if (!active[p]) return;
  const GemmTask& Tk = tasks[tile2task[blockIdx.x]];
  const int lt = blockIdx.x - Tk.tile0;
  const int M = Tk.M, N = Tk.N, K = Tk.K;
  const int m0 = (lt % Tk.ntm) * Tk.mr, n0 = (lt / Tk.ntm) * Tk.nc;
  const int mr = min(Tk.mr, M - m0), nc = min(Tk.nc, N - n0);
  const int ma = mr | 1, nb = nc | 1;          // odd strides: conflict-free transposed stores
  __shared__ double sm[3 * GT_K * (GT_SIDE + 1)];
  const bool pa = Tk.t[0].abuf >= B_STATE;     // the point's operand on the left
  double* As = sm;                             // [2 planes if pa][GT_K][ma]
  double* Bs = sm + (pa ? 2 : 1) * GT_K * ma;  // [2 planes if !pa][GT_K][nb]
  const int total = 2 * mr * nc, w0 = threadIdx.x & ~31;
  double acc[GT_R];
  int ia[GT_R], ib[GT_R];
#pragma unroll
  for (int i = 0; i < GT_R; ++i) {
    const int e = min((int)threadIdx.x + GT_THREADS * i, total - 1);
    const int pl = e >= mr * nc, q = e - pl * mr * nc;
    ia[i] = q % mr + (pa ? pl * GT_K * ma : 0);
    ib[i] = q / mr + (pa ? 0 : pl * GT_K * nb);
    acc[i] = 0.0;
  }
  const int nr = (total - w0 + GT_THREADS - 1) / GT_THREADS;   // this warp's outputs per thread
  for (int it = 0; it < Tk.nterm; ++it) {
    const GemmTerm& tm = Tk.t[it];
    for (int k0 = 0; k0 < K; k0 += GT_K) {
      const int kl = min((int)GT_K, K - k0);
      __syncthreads();
      // op(A) rows, op(B) columns
      for (int pl = 0; pl < (pa ? 2 : 1); ++pl)
        gemm_stage(bufptr(bufs, tm.abuf, p, pl, tm.aoff), tm.lda, tm.tA != 0, m0, mr, k0, kl,
                   pa ? tm.alpha[pl] : 1.0, As + pl * GT_K * ma, ma);
      for (int pl = 0; pl < (pa ? 1 : 2); ++pl)
        gemm_stage(bufptr(bufs, tm.bbuf, p, pl, tm.boff), tm.ldb, tm.tB == 0, n0, nc, k0, kl,
                   pa ? 1.0 : tm.alpha[pl], Bs + pl * GT_K * nb, nb);
      __syncthreads();
#pragma unroll 4
      for (int kk = 0; kk < kl; ++kk) {
        const double *a = As + kk * ma, *b = Bs + kk * nb;
#pragma unroll
        for (int i = 0; i < GT_R; ++i)
          if (i < nr) acc[i] = fma(a[ia[i]], b[ib[i]], acc[i]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < GT_R; ++i) {
    const int e = threadIdx.x + GT_THREADS * i;
    if (e >= total) break;
    const int pl = e >= mr * nc, q = e - pl * mr * nc;
    double* C = const_cast<double*>(bufptr(bufs, Tk.cbuf, p, pl, Tk.coff));
    C[m0 + q % mr + (long long)(n0 + q / mr) * Tk.ldc] = acc[i];
  }
}

// ---------------------------------------------------------------------------
// grouped block GEMM on the tensor cores (FP32 data, 3xTF32 products).
// Every term multiplies a per-point block (state, intermediate, field) by a
// ground-state block (U or V) shared by all points.  The per-point operand is
// put on the M side of the MMA so that the rows of all active points and both
// planes (Re, Im) fill 128-row tiles:
//   case 0 (per-point operand on the left):  D[i][j] = C[i][j],  D = op(P) op(S)
//   case 1 (per-point operand on the right): D[j][i] = C[i][j],  D = op(P)^T op(S)^T
// Rows: (point, plane, i) with i fastest; columns padded to a multiple of 16.
// ---------------------------------------------------------------------------
struct GemmTaskTC {
  int M, N, K, nterm;
  int rcase;              // 0 or 1, as above
  int mrows, ncols, npad; // D rows per (point, plane), D columns, padded columns
  GemmTerm t[PNFAM_MAXTERM];
  long long coff;
  int cbuf, ldc;
  long long bsoff;        // floats: the task's ground-state operand, split and laid out per chunk
};
enum { GTC_K = 16, GTC_PROD = 256, GTC_THREADS = GTC_PROD + 32 };

// two stages sized for the widest padded block (npmax <= 256) of the launch's tasks:
// narrower task lists leave room for more CTAs per SM, so more loads are in flight
__host__ __device__ constexpr size_t gemm_tc_smem_bytes(int npmax = 256) {
  return (size_t)2 * (2 * 128 * GTC_K + 2 * npmax * GTC_K) * sizeof(float);
}

// the B tile of chunk c of a task: B[n][k] = op(S)[k0 + k][n] (case 0) or
// op(S)[n][k0 + k] (case 1), n < ncols, zero elsewhere
__device__ __forceinline__ float4 gemm_tc_b4(const GemmTaskTC& Tk, const BufDescT<float>* bufs, int c, int n, int k4) {
  const int nkc = (Tk.K + GTC_K - 1) / GTC_K;
  const GemmTerm& tm = Tk.t[c / nkc];
  const int k0 = (c % nkc) * GTC_K;
  const bool pa = Tk.rcase == 0;
  const int sbuf = pa ? tm.bbuf : tm.abuf;
  const long long soff = pa ? tm.boff : tm.aoff;
  const int sld = pa ? tm.ldb : tm.lda, str_ = pa ? tm.tB : tm.tA;
  float x[4] = {0.f, 0.f, 0.f, 0.f};
  if (n < Tk.ncols) {
    const float* S = bufs[sbuf].base + soff;
    const bool kfast = pa ? str_ == 0 : str_ != 0;
    const long long sn = kfast ? sld : 1, sk = kfast ? 1 : sld;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = k0 + 4 * k4 + u;
      if (k < Tk.K) x[u] = S[(long long)n * sn + (long long)k * sk];
    }
  }
  return make_float4(x[0], x[1], x[2], x[3]);
}

// the ground-state operand of every chunk of every task, split into TF32 hi and lo
// in the canonical layout, once per operator: gsplit[bsoff + c*npad*2*GTC_K] = hi | lo
// grid (ntasks, most chunks of a task), 256 threads
__global__ void __launch_bounds__(256) k_gemm_bsplit(const GemmTaskTC* __restrict__ tasks,
                                                     const BufDescT<float>* __restrict__ bufs,
                                                     float* __restrict__ gsplit) {
  const GemmTaskTC& Tk = tasks[blockIdx.x];
  const int c = blockIdx.y;
  if (c >= Tk.nterm * ((Tk.K + GTC_K - 1) / GTC_K)) return;
  const int NP = Tk.npad;
  float* dst = gsplit + Tk.bsoff + (long long)c * NP * 2 * GTC_K;
  for (int e = threadIdx.x; e < NP * (GTC_K / 4); e += blockDim.x) {
    const int n = e % NP, k4 = e / NP;
    const int o = tc::cm_off(n, 4 * k4, NP);
    st_split4(dst + o, dst + NP * GTC_K + o, gemm_tc_b4(Tk, bufs, c, n, k4));
  }
}

// grid (ntasks, row tiles of 128); GTC_THREADS threads; dynamic smem gemm_tc_smem_bytes(npmax),
// npmax >= every task's npad
__global__ void __launch_bounds__(GTC_THREADS, 2) k_gemm_tc(const GemmTaskTC* __restrict__ tasks,
                                                            const BufDescT<float>* __restrict__ bufs,
                                                            const float* __restrict__ gsplit,
                                                            const int* __restrict__ actlist, int nact,
                                                            int npmax, int* __restrict__ err) {
  const GemmTaskTC& Tk = tasks[blockIdx.x];
  const int rows_total = 2 * nact * Tk.mrows;
  const int R0 = blockIdx.y * 128;
  if (R0 >= rows_total) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  float* stage_base = reinterpret_cast<float*>(smraw);
  const int stage_floats = 2 * 128 * GTC_K + 2 * npmax * GTC_K;
  __shared__ __align__(8) uint64_t full_bar[2], empty_bar[2];
  __shared__ uint32_t tslot;
  __shared__ volatile int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int NP = Tk.npad, K = Tk.K, mr = Tk.mrows;
  const int nkc = (K + GTC_K - 1) / GTC_K;
  const int nchunk = Tk.nterm * nkc;
  const uint32_t ncols = NP <= 32 ? 32u : NP <= 64 ? 64u : NP <= 128 ? 128u : 256u;
  if (tid == 0) {
    tc::mbar_init(&full_bar[0], GTC_PROD); tc::mbar_init(&full_bar[1], GTC_PROD);
    tc::mbar_init(&empty_bar[0], 1); tc::mbar_init(&empty_bar[1], 1);
    abort_flag = 0;
  }
  if (warp == 0) tc::tmem_alloc(&tslot, ncols);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tslot;
  if (warp < GTC_PROD / 32) {
    // ---------------- producers ----------------
    // A thread stages the same row of every chunk, four k at two places: the row's point,
    // plane and offset are found once, and the elements of the next chunk are loaded while
    // this one waits for its stage (4 divisions and the loads' latency per chunk before;
    // summed over a solve of 56 points at N_sh = 16: 23.1 -> 22.0 ms, over 6 steps of 64
    // points at N_sh = 20: 25.7 -> 23.7 ms).
    constexpr int NI = 128 * (GTC_K / 4) / GTC_PROD;   // float4 items of a thread per chunk
    const bool pa = Tk.rcase == 0;   // which operand of a term is the per-point one
    const int m = tid & 127, R = R0 + m;
    const bool live = R < rows_total;
    const int i = live ? R % mr : 0, rest = live ? R / mr : 0, pl = rest & 1;
    const long long p = actlist[rest >> 1];
    // A[m][k]: row m = (point, plane, i); case 0: op(P)[i][k], case 1: op(P)[k][i]
    float x[NI][4];
    auto fetch = [&](int c) {
      const GemmTerm& tm = Tk.t[c / nkc];
      const int k0 = (c % nkc) * GTC_K;
      const BufDescT<float> d = bufs[pa ? tm.abuf : tm.bbuf];
      const int pld = pa ? tm.lda : tm.ldb;
      const float al = (float)tm.alpha[pl];
      // element (i, k) of op(P) (case 0) or (k, i) of op(P) (case 1): stride in k
      const bool kfast = pa ? tm.tA != 0 : tm.tB == 0;
      const long long si = kfast ? pld : 1, sk = kfast ? 1 : pld;
      const float* P = d.base + p * d.sp + (long long)pl * d.spl + (pa ? tm.aoff : tm.boff) + (long long)i * si;
#pragma unroll
      for (int it = 0; it < NI; ++it)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int k = k0 + 4 * ((tid >> 7) + (GTC_PROD / 128) * it) + u;
          x[it][u] = live && k < K ? al * P[(long long)k * sk] : 0.f;
        }
    };
    int lc0 = -1, lc1 = -1;   // thread 0: last chunk copied into stage 0, stage 1
    if (nchunk > 0) fetch(0);
    for (int c = 0; c < nchunk; ++c) {
      const int st = c & 1;
      if (c >= 2 && !abort_flag && !tc::mbar_wait(&empty_bar[st], ((c >> 1) - 1) & 1)) abort_flag = 1;
      float* sAh = stage_base + st * stage_floats;
      float* sAl = sAh + 128 * GTC_K;
      float* sBh = sAl + 128 * GTC_K;
      bool issued = false;
      if (tid == 0 && !abort_flag) {
        // B: the ground-state operand of this chunk, pre-split (hi then lo, NP x GTC_K
        // each); this thread's arrival on the stage comes with the copy
        const uint32_t bbytes = (uint32_t)NP * GTC_K * 2 * 4;
        tc::mbar_expect_tx(&full_bar[st], bbytes);
        tc::bulk_g2s(sBh, gsplit + Tk.bsoff + (long long)c * NP * 2 * GTC_K, bbytes, &full_bar[st]);
        issued = true;
        if (st == 0) lc0 = c; else lc1 = c;
      }
      if (!abort_flag) {
#pragma unroll
        for (int it = 0; it < NI; ++it) {
          const int o = tc::cm_off(m, 4 * ((tid >> 7) + (GTC_PROD / 128) * it), 128);
          st_split4(sAh + o, sAl + o, make_float4(x[it][0], x[it][1], x[it][2], x[it][3]));
        }
      }
      tc::fence_async_smem();
      if (!issued) tc::mbar_arrive(&full_bar[st]);
      if (c + 1 < nchunk) fetch(c + 1);
    }
    // no copy may still be landing when the memory is reused (the last two chunks
    // are the only ones that can be in flight)
    if (tid == 0) {
      if (lc0 >= 0 && !tc::mbar_wait(&full_bar[0], (lc0 >> 1) & 1)) abort_flag = 1;
      if (lc1 >= 0 && !tc::mbar_wait(&full_bar[1], (lc1 >> 1) & 1)) abort_flag = 1;
    }
  } else if (tid == GTC_PROD) {
    // ---------------- MMA issuer ----------------
    const uint32_t idesc = tc::idesc_tf32(128, NP);
    const uint32_t lboA = (128 / 8) * 128, lboB = (uint32_t)(NP / 8) * 128;
    for (int c = 0; c < nchunk; ++c) {
      const int st = c & 1;
      if (!abort_flag && !tc::mbar_wait(&full_bar[st], (c >> 1) & 1)) abort_flag = 1;
      tc::fence_after();
      if (!abort_flag) {
        const float* sAh = stage_base + st * stage_floats;
        const float* sAl = sAh + 128 * GTC_K;
        const float* sBh = sAl + 128 * GTC_K;
        const float* sBl = sBh + NP * GTC_K;
#pragma unroll
        for (int ks = 0; ks < GTC_K / 8; ++ks) {
          const uint32_t oa = ks * 2 * lboA, ob = ks * 2 * lboB;
          const uint64_t ah = tc::sdesc(tc::smem_u32(sAh) + oa, lboA, 128);
          const uint64_t al = tc::sdesc(tc::smem_u32(sAl) + oa, lboA, 128);
          const uint64_t bh = tc::sdesc(tc::smem_u32(sBh) + ob, lboB, 128);
          const uint64_t bl = tc::sdesc(tc::smem_u32(sBl) + ob, lboB, 128);
          tc::mma_tf32(tmem, ah, bh, idesc, c > 0 || ks > 0);
          tc::mma_tf32(tmem, ah, bl, idesc, true);
          tc::mma_tf32(tmem, al, bh, idesc, true);
        }
      }
      tc::mma_commit(&empty_bar[st]);
    }
  }
  const int last = nchunk - 1;
  bool ok = nchunk == 0 || tc::mbar_wait(&empty_bar[last & 1], (last >> 1) & 1);
  ok = __syncthreads_and(ok && !abort_flag);
  tc::fence_after();
  if (!ok) {
    if (tid == 0) atomicExch(err, 1);
  } else if (warp < 4) {
    const int m = tid, R = R0 + m;
    const bool mine = R < rows_total;
    const int i = mine ? R % mr : 0, rest = mine ? R / mr : 0, pl = rest & 1;
    const int p = mine ? actlist[rest >> 1] : 0;
    const BufDescT<float> d = bufs[Tk.cbuf];
    float* C = d.base + (long long)p * d.sp + (long long)pl * d.spl + Tk.coff;
    for (int n0 = 0; n0 < NP; n0 += 8) {
      float v[8];
      tc::tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)n0, v);
      if (mine) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int n = n0 + u;
          if (n < Tk.ncols) {
            if (Tk.rcase == 0) C[i + (long long)n * Tk.ldc] = v[u];
            else C[n + (long long)i * Tk.ldc] = v[u];
          }
        }
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_free(tmem, ncols);
}

// ---------------------------------------------------------------------------
// basis on device
// ---------------------------------------------------------------------------
template <class T>
struct DevBasisT {
  int nb, dqp, nghl;
  const int* db;
  const int* st;
  const int* nup;
  const signed char* ns;
  const T* phi;          // [5][dqp][nghl]
  const double* wdcori;
  const double* crho;
  const double* cs;
  const double* cpair;
  const double* cspair;
  double sc[12];         // cdrho, ctau, ctj0, ctj1, ctj2, crdj, cds, ct, cj, cgs, cf, csdj
};
using DevBasis = DevBasisT<double>;

enum { ND = 28 };  // complex local densities
// 0 rho 1 tau 2 tjrr 3 tjpr 4 tjzr 5 tjrp 6 tjpp 7 tjzp 8 tjrz 9 tjpz 10 tjzz
// 11 sr 12 sp 13 sz 14 tr 15 tp 16 tz 17 jr 18 jp 19 jz 20 fr 21 fp 22 fz 23 gs
// 24 rb 25 sbr 26 sbp 27 sbz
enum { D_RHO = 0, D_TAU, D_TJRR, D_TJPR, D_TJZR, D_TJRP, D_TJPP, D_TJZP, D_TJRZ, D_TJPZ, D_TJZZ,
       D_SR, D_SP, D_SZ, D_TR, D_TP, D_TZ, D_JR, D_JP, D_JZ, D_FR, D_FP, D_FZ, D_GS,
       D_RB, D_SBR, D_SBP, D_SBZ };

// One density call: rho in structure (rcols, roffs), kappa in (kcols, koffs), both
// [P][2 planes][plane stride] at the given base/offset.
template <class T>
struct DensCallT {
  const T* rho; long long rho_sp, rho_spl;
  const int* rcols; const long long* roffs;
  const T* kap; long long kap_sp, kap_spl;
  const int* kcols; const long long* koffs;
};
using DensCall = DensCallT<double>;

// four consecutive elements from shared memory (16-byte aligned) as 128-bit loads
__device__ __forceinline__ void lds4(const float* p, float (&v)[4]) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void lds4(const double* p, double (&v)[4]) {
  const double2 t0 = reinterpret_cast<const double2*>(p)[0], t1 = reinterpret_cast<const double2*>(p)[1];
  v[0] = t0.x; v[1] = t0.y; v[2] = t1.x; v[3] = t1.y;
}

#define DRT 32   // mesh points per CTA

// b columns per thread: 4 consecutive columns per lane, 8 lanes
template <class T> struct DensTile {
  static constexpr int BT = 4;
  static constexpr int BW = 8 * BT;              // b columns per chunk (8 lanes x BT)
  static constexpr int BWP = BW + 4;             // padded row: conflict-free transposed staging
  static constexpr int AK = sizeof(T) >= 8 ? 16 : 32;  // a rows per chunk
};

template <class T>
__host__ __device__ constexpr size_t density_smem_bytes() {
  return (size_t)(DensTile<T>::AK * DRT * 4 + 2 * DensTile<T>::AK * DensTile<T>::BWP) * sizeof(T);
}

// contributions of one column b at one mesh point from the rows of the SAME spin
// as b (S) or of the OPPOSITE spin (O); P = phi_q(b, r), sg = spin of b,
// sig = +1 if b is spin down (pnfam_hamiltonian_blas.f90:124-711)
template <class T>
__device__ __forceinline__ void dens_same(T (&acc)[2 * ND], const T (&Sr)[4], const T (&Si)[4], const T (&P)[4],
                                          T sg) {
  const T h5 = T(0.5);
#define ACC(k, re, im) { acc[2 * (k)] += (re); acc[2 * (k) + 1] += (im); }
  T xr, xi;
  xr = Sr[0] * P[0]; xi = Si[0] * P[0];
  ACC(D_RHO, xr, xi);
  ACC(D_SZ, sg * xr, sg * xi);
  xr = h5 * (Sr[0] * P[2] + Sr[2] * P[0]); xi = h5 * (Si[0] * P[2] + Si[2] * P[0]);
  ACC(D_JP, xr, xi);
  ACC(D_TJPZ, sg * xr, sg * xi);
  xr = Sr[1] * P[1] + Sr[2] * P[2] + Sr[3] * P[3]; xi = Si[1] * P[1] + Si[2] * P[2] + Si[3] * P[3];
  ACC(D_TAU, xr, xi);
  ACC(D_TZ, sg * xr, sg * xi);
  xr = h5 * (Sr[0] * P[1] - Sr[1] * P[0]); xi = h5 * (Si[0] * P[1] - Si[1] * P[0]);
  ACC(D_JR, -xi, xr);
  ACC(D_TJRZ, -sg * xi, sg * xr);
  xr = h5 * (Sr[0] * P[3] - Sr[3] * P[0]); xi = h5 * (Si[0] * P[3] - Si[3] * P[0]);
  ACC(D_JZ, -xi, xr);
  ACC(D_TJZZ, -sg * xi, sg * xr);
  ACC(D_GS, sg * (Sr[0] * P[3] + Sr[3] * P[0]), sg * (Si[0] * P[3] + Si[3] * P[0]));
  ACC(D_FR, h5 * sg * (Sr[1] * P[3] + Sr[3] * P[1]), h5 * sg * (Si[1] * P[3] + Si[3] * P[1]));
  {
    const T ar = h5 * sg * (Sr[2] * P[3] - Sr[3] * P[2]), ai = h5 * sg * (Si[2] * P[3] - Si[3] * P[2]);
    ACC(D_FP, -ai, ar);
  }
  ACC(D_FZ, sg * Sr[3] * P[3], sg * Si[3] * P[3]);
}

template <class T>
__device__ __forceinline__ void dens_opp(T (&acc)[2 * ND], const T (&Or)[4], const T (&Oi)[4], const T (&P)[4],
                                         T sig) {
  const T h5 = T(0.5);
  T xr, xi;
  ACC(D_GS, sig * (Or[0] * P[2] - Or[2] * P[0]) + (Or[0] * P[1] + Or[1] * P[0]),
      sig * (Oi[0] * P[2] - Oi[2] * P[0]) + (Oi[0] * P[1] + Oi[1] * P[0]));
  ACC(D_FR, Or[1] * P[1] + sig * h5 * (Or[1] * P[2] - Or[2] * P[1]),
      Oi[1] * P[1] + sig * h5 * (Oi[1] * P[2] - Oi[2] * P[1]));
  {
    const T ar = sig * Or[2] * P[2] + h5 * (Or[2] * P[1] - Or[1] * P[2]);
    const T ai = sig * Oi[2] * P[2] + h5 * (Oi[2] * P[1] - Oi[1] * P[2]);
    ACC(D_FP, -ai, ar);
  }
  ACC(D_FZ, h5 * (Or[3] * P[1] + sig * Or[3] * P[2] + Or[1] * P[3] - sig * Or[2] * P[3]),
      h5 * (Oi[3] * P[1] + sig * Oi[3] * P[2] + Oi[1] * P[3] - sig * Oi[2] * P[3]));
  xr = Or[0] * P[0]; xi = Oi[0] * P[0];
  ACC(D_SR, xr, xi);
  ACC(D_SP, -sig * xi, sig * xr);
  xr = h5 * (Or[2] * P[0] + Or[0] * P[2]); xi = h5 * (Oi[2] * P[0] + Oi[0] * P[2]);
  ACC(D_TJPR, xr, xi);
  ACC(D_TJPP, -sig * xi, sig * xr);
  xr = Or[1] * P[1] + Or[2] * P[2] + Or[3] * P[3]; xi = Oi[1] * P[1] + Oi[2] * P[2] + Oi[3] * P[3];
  ACC(D_TR, xr, xi);
  ACC(D_TP, -sig * xi, sig * xr);
  xr = h5 * (Or[0] * P[1] - Or[1] * P[0]); xi = h5 * (Oi[0] * P[1] - Oi[1] * P[0]);
  ACC(D_TJRR, -xi, xr);
  ACC(D_TJRP, -sig * xr, -sig * xi);
  xr = h5 * (Or[0] * P[3] - Or[3] * P[0]); xi = h5 * (Oi[0] * P[3] - Oi[3] * P[0]);
  ACC(D_TJZR, -xi, xr);
  ACC(D_TJZP, -sig * xr, -sig * xi);
}

// W_q(r, b) += sum over the staged rows a of phi_q(a, r) rho(a, b), q < NQ
template <class T, int NH, int NQ, int AK, int BWP>
__device__ __forceinline__ void dens_rows(const T* sphi, const T* srho, int na, int rl, int bl,
                                          T (&W)[NH][4][4][2]) {
  for (int aa = 0; aa < na; ++aa) {
    T f4[4];
    lds4(&sphi[(aa * DRT + rl) * 4], f4);
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      T xr[4], xi[4];
      lds4(&srho[(0 * AK + aa) * BWP + 4 * bl + 32 * h], xr);
      lds4(&srho[(1 * AK + aa) * BWP + 4 * bl + 32 * h], xi);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          W[h][i][q][0] = fma(f4[q], xr[i], W[h][i][q][0]);
          W[h][i][q][1] = fma(f4[q], xi[i], W[h][i][q][1]);
        }
    }
  }
}

// grid (ceil(nghl/DRT), G, P*2 calls); block 256 = DRT mesh points x 8 column lanes.
// Thread (r, lane) owns mesh point r and columns b0 + 4*lane + i + 32*h of each chunk;
// W_q(r, b) = sum_a phi_q(a, r) rho_ab is accumulated over the rows of one spin, then
// folded into the thread's 28 complex densities, which are reduced over the 8 lanes
// at the end.  dpart: [P][2][G][2*ND][nghl]
template <class T>
__global__ void __launch_bounds__(256, sizeof(T) >= 8 ? 1 : 2) k_density(DevBasisT<T> B, DensCallT<T> c0, DensCallT<T> c1, int G,
                                                    T* __restrict__ dpart, const int* __restrict__ active) {
  constexpr int BT = DensTile<T>::BT, NH = BT / 4, BW = DensTile<T>::BW, BWP = DensTile<T>::BWP;
  constexpr int AK = DensTile<T>::AK;
  const int p = blockIdx.z >> 1, call = blockIdx.z & 1;
  if (!active[p]) return;
  const DensCallT<T>& C = call ? c1 : c0;
  const int g = blockIdx.y;
  const int r0 = blockIdx.x * DRT;
  const int rl = threadIdx.x >> 3, bl = threadIdx.x & 7;
  const int nghl = B.nghl;
  const int r = r0 + rl;
  const bool rok = r < nghl;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sphi = reinterpret_cast<T*>(smraw);   // [AK][DRT][4]
  T* srho = sphi + AK * DRT * 4;            // [2 pl][AK][BWP]
  const long long ps = (long long)B.dqp * nghl;
  T acc[2 * ND];
#pragma unroll
  for (int k = 0; k < 2 * ND; ++k) acc[k] = T(0);

  for (int kind = 0; kind < 2; ++kind) {  // 0: normal densities, 1: pairing densities
    const int* cols = kind == 0 ? C.rcols : C.kcols;
    const long long* offs = kind == 0 ? C.roffs : C.koffs;
    const T* base = kind == 0 ? C.rho : C.kap;
    const long long bsp = kind == 0 ? C.rho_sp : C.kap_sp, bspl = kind == 0 ? C.rho_spl : C.kap_spl;
    const int nq = kind == 0 ? 4 : 1;
    for (int ix = g; ix < B.nb; ix += G) {
      const int iy = cols[ix];
      if (iy < 0) continue;
      const int d = B.db[ix], dc = B.db[iy], nu = B.nup[ix];
      const int sa = B.st[ix], sb = B.st[iy];
      const T* mat = base + (long long)p * bsp + offs[ix];
      for (int b0 = 0; b0 < dc; b0 += BW) {
        // this thread's columns: spin (0 outside the block or the mesh) and phi_q(b, r),
        // loaded ahead of the row loop
        T sgb[NH][4], Pb[NH][4][4];
#pragma unroll
        for (int h = 0; h < NH; ++h)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int b = b0 + 4 * bl + i + 32 * h;
            const bool ok = rok && b < dc;
            sgb[h][i] = ok ? (T)B.ns[sb + b] : T(0);
            const long long jb = sb + (ok ? b : 0);
#pragma unroll
            for (int q = 0; q < 4; ++q) Pb[h][i][q] = (ok && q < nq) ? B.phi[q * ps + jb * nghl + r] : T(0);
          }
        for (int s = 0; s < 2; ++s) {  // rows of spin up [0, nu), then spin down [nu, d)
          const int alo = s == 0 ? 0 : nu, ahi = s == 0 ? nu : d;
          if (alo >= ahi) continue;
          T W[NH][4][4][2];
#pragma unroll
          for (int h = 0; h < NH; ++h)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int q = 0; q < 4; ++q) { W[h][i][q][0] = T(0); W[h][i][q][1] = T(0); }
          for (int a0 = alo; a0 < ahi; a0 += AK) {
            const int na = min(AK, ahi - a0);
            __syncthreads();
            for (int e = threadIdx.x; e < AK * DRT; e += blockDim.x) {
              const int rr = e % DRT, aa = e / DRT;
              T v[4] = {T(0), T(0), T(0), T(0)};
              if (aa < na && r0 + rr < nghl) {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                  if (q < nq) v[q] = B.phi[q * ps + (long long)(sa + a0 + aa) * nghl + r0 + rr];
              }
              T* dst = &sphi[(aa * DRT + rr) * 4];
              dst[0] = v[0]; dst[1] = v[1]; dst[2] = v[2]; dst[3] = v[3];
            }
            // 8 consecutive rows x 4 columns per warp: coalesced reads, conflict-free writes
            for (int e = threadIdx.x; e < 2 * AK * BW; e += blockDim.x) {
              const int aa = (e & 7) + 8 * ((e >> 5) % (AK / 8));
              const int bb = ((e >> 3) & 3) + 4 * ((e >> 5) / (AK / 8) % (BW / 4));
              const int pl = e / (AK * BW);
              T v = T(0);
              if (aa < na && b0 + bb < dc) v = mat[(long long)pl * bspl + (a0 + aa) + (long long)(b0 + bb) * d];
              srho[(pl * AK + aa) * BWP + bb] = v;
            }
            __syncthreads();
            if (kind == 0) dens_rows<T, NH, 4, AK, BWP>(sphi, srho, na, rl, bl, W);
            else dens_rows<T, NH, 1, AK, BWP>(sphi, srho, na, rl, bl, W);
          }
          // fold the rows of spin s into the densities
          const T srow = s == 0 ? T(1) : T(-1);
#pragma unroll
          for (int h = 0; h < NH; ++h)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const T sg = sgb[h][i];
              if (sg == T(0)) continue;
              const T sig = sg < T(0) ? T(1) : T(-1);
              T Wr[4], Wi[4], Pq[4];
#pragma unroll
              for (int q = 0; q < 4; ++q) { Wr[q] = W[h][i][q][0]; Wi[q] = W[h][i][q][1]; Pq[q] = Pb[h][i][q]; }
              if (kind == 0) {
                if (sg == srow) dens_same(acc, Wr, Wi, Pq, sg);
                else dens_opp(acc, Wr, Wi, Pq, sig);
              } else {
                const T two = T(2);
                if (sg == srow) {
                  const T xr = two * Wr[0] * Pq[0], xi = two * Wi[0] * Pq[0];
                  ACC(D_SBR, sig * xr, sig * xi);
                  ACC(D_SBP, xi, -xr);
                } else {
                  const T xr = two * Wr[0] * Pq[0], xi = two * Wi[0] * Pq[0];
                  ACC(D_RB, -sg * xr, -sg * xi);
                  ACC(D_SBZ, xr, xi);
                }
              }
            }
        }
      }
    }
  }
#undef ACC
  // reduce over the 8 column lanes (same warp, low 3 bits of the lane)
#pragma unroll
  for (int k = 0; k < 2 * ND; ++k) {
    T v = acc[k];
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    acc[k] = v;
  }
  if (bl == 0 && rok) {
    T* out = dpart + (((long long)p * 2 + call) * G + g) * (2 * ND) * nghl;
#pragma unroll
    for (int k = 0; k < 2 * ND; ++k) out[(long long)k * nghl + r] = acc[k];
  }
}

// ---------------------------------------------------------------------------
// FP64 densities over the whole mesh: a CTA takes 32 mesh points, a warp the columns
// b = warp, warp + 8, ... of the blocks; a lane accumulates W of its point for a column
// over the rows, folds it into its own 28 complex densities (registers), and these are
// summed over the 8 warps at the end (as a tree: the order is part of the result,
// an iteration that amplifies rounding repeats to the last digit).
// Bound by the FP64 pipe.  With 8 lanes of a warp on 8 columns and the rows staged in
// shared memory the pipe was 83 % busy, 40 % of it with columns that a block of 1 ... 25
// does not have and with factors 1/2 that the sums can take along; a warp of one column
// skips what is missing and needs neither staging nor barriers.  40 points at N_sh = 8:
// 11.5 ms before, now 7.7 ms.
// ---------------------------------------------------------------------------

// grid (ceil(nghl/DRT), G, P*2 calls); block 256 = 8 warps x DRT mesh points
// dpart: [P][2][G][2*ND][nghl]
__global__ void __launch_bounds__(256, 1) k_density_fp64(DevBasis B, DensCall c0, DensCall c1, int G,
                                                         double* __restrict__ dpart, const int* __restrict__ active) {
  using T = double;
  const int p = blockIdx.z >> 1, call = blockIdx.z & 1;
  if (!active[p]) return;
  const DensCall& C = call ? c1 : c0;
  const int g = blockIdx.y;
  const int w8 = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int nghl = B.nghl;
  const bool rok = (int)blockIdx.x * DRT + l < nghl;
  const int r = rok ? blockIdx.x * DRT + l : nghl - 1;   // lanes past the mesh repeat its last point
  T al[2 * ND];   // this lane's densities at mesh point r
#pragma unroll
  for (int k = 0; k < 2 * ND; ++k) al[k] = 0;
  const long long ps = (long long)B.dqp * nghl;
  const T h5 = (T)0.5, two = (T)2;

#define ACC(k, re, im) { al[2 * (k)] += (re); al[2 * (k) + 1] += (im); }
// with a factor that is exact: 1/2 or 2, and the sign s
#define ACCF(k, f, re, im) { al[2 * (k)] = fma((f), (re), al[2 * (k)]); al[2 * (k) + 1] = fma((f), (im), al[2 * (k) + 1]); }

  // ---------------- normal densities ----------------
  for (int ix = g; ix < B.nb; ix += G) {
    const int iy = C.rcols[ix];
    if (iy < 0) continue;
    const int d = B.db[ix], dc = B.db[iy], nu = B.nup[ix];
    const T* phi = B.phi + (long long)B.st[ix] * nghl + r;
    const T* rho = C.rho + (long long)p * C.rho_sp + C.roffs[ix];
    for (int b = w8; b < dc; b += 8) {
      const T *cr = rho + (long long)b * d, *ci = cr + C.rho_spl;
      T w[2][4][2];
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int q = 0; q < 4; ++q) { w[s][q][0] = 0; w[s][q][1] = 0; }
#pragma unroll
      for (int s = 0; s < 2; ++s) {   // spin-up rows first
#pragma unroll 4
        for (int a = s ? nu : 0; a < (s ? d : nu); ++a) {
          const T re = cr[a], im = ci[a];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const T f = phi[q * ps + (long long)a * nghl];
            w[s][q][0] = fma(f, re, w[s][q][0]); w[s][q][1] = fma(f, im, w[s][q][1]);
          }
        }
      }
      // contributions of column b at mesh point r
      const int jb = B.st[iy] + b;
      const T P0 = B.phi[0 * ps + (long long)jb * nghl + r];
      const T P1 = B.phi[1 * ps + (long long)jb * nghl + r];
      const T P2 = B.phi[2 * ps + (long long)jb * nghl + r];
      const T P3 = B.phi[3 * ps + (long long)jb * nghl + r];
      const T sg = (T)B.ns[jb];
      const int si = (sg > 0) ? 0 : 1;  // same-spin set of wfa
      // select S (same spin as b) and O (opposite)
      T Sr[4], Si[4], Or[4], Oi[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        Sr[q] = si == 0 ? w[0][q][0] : w[1][q][0]; Si[q] = si == 0 ? w[0][q][1] : w[1][q][1];
        Or[q] = si == 0 ? w[1][q][0] : w[0][q][0]; Oi[q] = si == 0 ? w[1][q][1] : w[0][q][1];
      }
      const T sig = (sg < 0) ? (T)1 : (T)-1;  // +1 if b is spin down
      const T hs = h5 * sg, hg = h5 * sig;
      T xr, xi;
      // diagonal in spin
      xr = Sr[0] * P0; xi = Si[0] * P0;
      ACC(D_RHO, xr, xi);
      ACC(D_SZ, sg * xr, sg * xi);
      xr = Sr[0] * P2 + Sr[2] * P0; xi = Si[0] * P2 + Si[2] * P0;
      ACCF(D_JP, h5, xr, xi);
      ACCF(D_TJPZ, hs, xr, xi);
      xr = Sr[1] * P1 + Sr[2] * P2 + Sr[3] * P3; xi = Si[1] * P1 + Si[2] * P2 + Si[3] * P3;
      ACC(D_TAU, xr, xi);
      ACC(D_TZ, sg * xr, sg * xi);
      xr = Sr[0] * P1 - Sr[1] * P0; xi = Si[0] * P1 - Si[1] * P0;
      ACCF(D_JR, h5, -xi, xr);
      ACCF(D_TJRZ, hs, -xi, xr);
      xr = Sr[0] * P3 - Sr[3] * P0; xi = Si[0] * P3 - Si[3] * P0;
      ACCF(D_JZ, h5, -xi, xr);
      ACCF(D_TJZZ, hs, -xi, xr);
      // gs: diagonal part + off-diagonal parts
      {
        T gr = sg * (Sr[0] * P3 + Sr[3] * P0), gi = sg * (Si[0] * P3 + Si[3] * P0);
        gr += sig * (Or[0] * P2 - Or[2] * P0) + (Or[0] * P1 + Or[1] * P0);
        gi += sig * (Oi[0] * P2 - Oi[2] * P0) + (Oi[0] * P1 + Oi[1] * P0);
        ACC(D_GS, gr, gi);
      }
      {
        T fr = h5 * sg * (Sr[1] * P3 + Sr[3] * P1), fi = h5 * sg * (Si[1] * P3 + Si[3] * P1);
        fr += Or[1] * P1 + sig * h5 * (Or[1] * P2 - Or[2] * P1);
        fi += Oi[1] * P1 + sig * h5 * (Oi[1] * P2 - Oi[2] * P1);
        ACC(D_FR, fr, fi);
      }
      {
        // fp += i*sg*(S2P3 - S3P2)/2 + i*(sig*O2P2 + (O2P1 - O1P2)/2)
        const T ar = h5 * sg * (Sr[2] * P3 - Sr[3] * P2) + sig * Or[2] * P2 + h5 * (Or[2] * P1 - Or[1] * P2);
        const T ai = h5 * sg * (Si[2] * P3 - Si[3] * P2) + sig * Oi[2] * P2 + h5 * (Oi[2] * P1 - Oi[1] * P2);
        ACC(D_FP, -ai, ar);
      }
      {
        T zr = sg * Sr[3] * P3, zi = sg * Si[3] * P3;
        zr += h5 * (Or[3] * P1 + sig * Or[3] * P2 + Or[1] * P3 - sig * Or[2] * P3);
        zi += h5 * (Oi[3] * P1 + sig * Oi[3] * P2 + Oi[1] * P3 - sig * Oi[2] * P3);
        ACC(D_FZ, zr, zi);
      }
      // not diagonal in spin
      xr = Or[0] * P0; xi = Oi[0] * P0;
      ACC(D_SR, xr, xi);
      ACC(D_SP, -sig * xi, sig * xr);
      xr = Or[2] * P0 + Or[0] * P2; xi = Oi[2] * P0 + Oi[0] * P2;
      ACCF(D_TJPR, h5, xr, xi);
      ACCF(D_TJPP, hg, -xi, xr);
      xr = Or[1] * P1 + Or[2] * P2 + Or[3] * P3; xi = Oi[1] * P1 + Oi[2] * P2 + Oi[3] * P3;
      ACC(D_TR, xr, xi);
      ACC(D_TP, -sig * xi, sig * xr);
      xr = Or[0] * P1 - Or[1] * P0; xi = Oi[0] * P1 - Oi[1] * P0;
      ACCF(D_TJRR, h5, -xi, xr);
      ACCF(D_TJRP, hg, -xr, -xi);
      xr = Or[0] * P3 - Or[3] * P0; xi = Oi[0] * P3 - Oi[3] * P0;
      ACCF(D_TJZR, h5, -xi, xr);
      ACCF(D_TJZP, hg, -xr, -xi);
    }
  }
  // ---------------- pairing densities ----------------
  for (int ix = g; ix < B.nb; ix += G) {
    const int iy = C.kcols[ix];
    if (iy < 0) continue;
    const int d = B.db[ix], dc = B.db[iy], nu = B.nup[ix];
    const T* phi = B.phi + (long long)B.st[ix] * nghl + r;
    const T* kap = C.kap + (long long)p * C.kap_sp + C.koffs[ix];
    for (int b = w8; b < dc; b += 8) {
      const T *cr = kap + (long long)b * d, *ci = cr + C.kap_spl;
      T w[2][2] = {{0, 0}, {0, 0}};
#pragma unroll
      for (int s = 0; s < 2; ++s) {
#pragma unroll 4
        for (int a = s ? nu : 0; a < (s ? d : nu); ++a) {
          const T f = phi[(long long)a * nghl];
          w[s][0] = fma(f, cr[a], w[s][0]); w[s][1] = fma(f, ci[a], w[s][1]);
        }
      }
      const int jb = B.st[iy] + b;
      const T P0 = B.phi[(long long)jb * nghl + r];
      const T sg = (T)B.ns[jb];
      const int si = (sg > 0) ? 0 : 1;
      const T Sr = si == 0 ? w[0][0] : w[1][0], Si = si == 0 ? w[0][1] : w[1][1];
      const T Or = si == 0 ? w[1][0] : w[0][0], Oi = si == 0 ? w[1][1] : w[0][1];
      const T sig = (sg < 0) ? (T)1 : (T)-1;
      T xr = two * Or * P0, xi = two * Oi * P0;
      ACC(D_RB, -sg * xr, -sg * xi);
      ACC(D_SBZ, xr, xi);
      xr = two * Sr * P0; xi = two * Si * P0;
      ACC(D_SBR, sig * xr, sig * xi);
      ACC(D_SBP, xi, -xr);
    }
  }
#undef ACC
#undef ACCF
  // over the warps, DSUM densities at a time
  constexpr int DSUM = 8;
  __shared__ T red[DSUM][8][DRT];
  T* out = dpart + (((long long)p * 2 + call) * G + g) * (2 * ND) * nghl;
#pragma unroll
  for (int k0 = 0; k0 < 2 * ND; k0 += DSUM) {
    if (k0) __syncthreads();
#pragma unroll
    for (int k = 0; k < DSUM; ++k) red[k][w8][l] = al[k0 + k];
    __syncthreads();
    T v[8];   // warp w8 sums density k0 + w8
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = red[w8][i][l];
    if (rok) out[(long long)(k0 + w8) * nghl + r] = ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]));
  }
}

// ---------------------------------------------------------------------------
// fold of W_q(r, b) = sum_a phi_q(a, r) rho_ab into the 28 local densities, one
// component q at a time (the terms of pnfam_hamiltonian_blas.f90:124-711 that
// contain W_q), for the tensor-core density kernel
// ---------------------------------------------------------------------------
// the terms of the density formulas that contain W_q of rows with the SAME spin as b
template <int Q>
__device__ __forceinline__ void fold_same(float (&acc)[2 * ND], float wr, float wi, const float (&P)[4], float sg) {
  const float h5 = 0.5f;
#define A_(k, re, im) { acc[2 * (k)] += (re); acc[2 * (k) + 1] += (im); }
  if (Q == 0) {
    A_(D_RHO, wr * P[0], wi * P[0]);
    A_(D_SZ, sg * wr * P[0], sg * wi * P[0]);
    A_(D_JP, h5 * wr * P[2], h5 * wi * P[2]);
    A_(D_TJPZ, sg * h5 * wr * P[2], sg * h5 * wi * P[2]);
    A_(D_JR, -h5 * wi * P[1], h5 * wr * P[1]);
    A_(D_TJRZ, -sg * h5 * wi * P[1], sg * h5 * wr * P[1]);
    A_(D_JZ, -h5 * wi * P[3], h5 * wr * P[3]);
    A_(D_TJZZ, -sg * h5 * wi * P[3], sg * h5 * wr * P[3]);
    A_(D_GS, sg * wr * P[3], sg * wi * P[3]);
  } else if (Q == 1) {
    A_(D_TAU, wr * P[1], wi * P[1]);
    A_(D_TZ, sg * wr * P[1], sg * wi * P[1]);
    A_(D_JR, h5 * wi * P[0], -h5 * wr * P[0]);
    A_(D_TJRZ, sg * h5 * wi * P[0], -sg * h5 * wr * P[0]);
    A_(D_FR, h5 * sg * wr * P[3], h5 * sg * wi * P[3]);
  } else if (Q == 2) {
    A_(D_JP, h5 * wr * P[0], h5 * wi * P[0]);
    A_(D_TJPZ, sg * h5 * wr * P[0], sg * h5 * wi * P[0]);
    A_(D_TAU, wr * P[2], wi * P[2]);
    A_(D_TZ, sg * wr * P[2], sg * wi * P[2]);
    A_(D_FP, -h5 * sg * wi * P[3], h5 * sg * wr * P[3]);
  } else {
    A_(D_TAU, wr * P[3], wi * P[3]);
    A_(D_TZ, sg * wr * P[3], sg * wi * P[3]);
    A_(D_JZ, h5 * wi * P[0], -h5 * wr * P[0]);
    A_(D_TJZZ, sg * h5 * wi * P[0], -sg * h5 * wr * P[0]);
    A_(D_GS, sg * wr * P[0], sg * wi * P[0]);
    A_(D_FR, h5 * sg * wr * P[1], h5 * sg * wi * P[1]);
    A_(D_FP, h5 * sg * wi * P[2], -h5 * sg * wr * P[2]);
    A_(D_FZ, sg * wr * P[3], sg * wi * P[3]);
  }
}

// the terms that contain W_q of rows with the OPPOSITE spin to b (sig = +1 if b is spin down)
template <int Q>
__device__ __forceinline__ void fold_opp(float (&acc)[2 * ND], float wr, float wi, const float (&P)[4], float sig) {
  const float h5 = 0.5f;
  if (Q == 0) {
    A_(D_GS, sig * wr * P[2] + wr * P[1], sig * wi * P[2] + wi * P[1]);
    A_(D_SR, wr * P[0], wi * P[0]);
    A_(D_SP, -sig * wi * P[0], sig * wr * P[0]);
    A_(D_TJPR, h5 * wr * P[2], h5 * wi * P[2]);
    A_(D_TJPP, -sig * h5 * wi * P[2], sig * h5 * wr * P[2]);
    A_(D_TJRR, -h5 * wi * P[1], h5 * wr * P[1]);
    A_(D_TJRP, -sig * h5 * wr * P[1], -sig * h5 * wi * P[1]);
    A_(D_TJZR, -h5 * wi * P[3], h5 * wr * P[3]);
    A_(D_TJZP, -sig * h5 * wr * P[3], -sig * h5 * wi * P[3]);
  } else if (Q == 1) {
    A_(D_GS, wr * P[0], wi * P[0]);
    A_(D_FR, wr * P[1] + sig * h5 * wr * P[2], wi * P[1] + sig * h5 * wi * P[2]);
    A_(D_FP, h5 * wi * P[2], -h5 * wr * P[2]);
    A_(D_FZ, h5 * wr * P[3], h5 * wi * P[3]);
    A_(D_TR, wr * P[1], wi * P[1]);
    A_(D_TP, -sig * wi * P[1], sig * wr * P[1]);
    A_(D_TJRR, h5 * wi * P[0], -h5 * wr * P[0]);
    A_(D_TJRP, sig * h5 * wr * P[0], sig * h5 * wi * P[0]);
  } else if (Q == 2) {
    A_(D_GS, -sig * wr * P[0], -sig * wi * P[0]);
    A_(D_FR, -sig * h5 * wr * P[1], -sig * h5 * wi * P[1]);
    A_(D_FP, -(sig * wi * P[2] + h5 * wi * P[1]), sig * wr * P[2] + h5 * wr * P[1]);
    A_(D_FZ, -sig * h5 * wr * P[3], -sig * h5 * wi * P[3]);
    A_(D_TJPR, h5 * wr * P[0], h5 * wi * P[0]);
    A_(D_TJPP, -sig * h5 * wi * P[0], sig * h5 * wr * P[0]);
    A_(D_TR, wr * P[2], wi * P[2]);
    A_(D_TP, -sig * wi * P[2], sig * wr * P[2]);
  } else {
    A_(D_FZ, h5 * (wr * P[1] + sig * wr * P[2]), h5 * (wi * P[1] + sig * wi * P[2]));
    A_(D_TR, wr * P[3], wi * P[3]);
    A_(D_TP, -sig * wi * P[3], sig * wr * P[3]);
    A_(D_TJZR, h5 * wi * P[0], -h5 * wr * P[0]);
    A_(D_TJZP, sig * h5 * wr * P[0], sig * h5 * wi * P[0]);
  }
}
#undef A_

struct DensTCArgs {
  const float* rho; long long rho_sp, rho_spl;   // as DensCallT, per call
  const int* rcols; const long long* roffs;
  const float* kap; long long kap_sp, kap_spl;
  const int* kcols; const long long* koffs;
};

// ---------------------------------------------------------------------------
// densities on the tensor cores with operands moved by the bulk-copy engine.
// A unit is (kind, block row ix, spin s of its rows, columns [b0, b0 + nc) of the
// block iy = cols[ix]), nc <= 64:
//   W[m][n] = sum_{a in s} phi_q(a, r) rho(a, b; pl),  m = q*32 + l (r = r0 + l),
//                                                     n = pl*nc + (b - b0)
// with K (the rows a of spin s) in chunks of 8.  Both operands are split into TF32
// high parts and remainders ahead of the kernel and laid out in the canonical
// K-major core-matrix order: A (phi) once per ground state for every (ix, s, chunk,
// 32-point mesh tile), B (rho of every active point) by k_dens_bsplit in each
// evaluation.  In the kernel one thread copies A and B chunks into a ring of
// DTC2_NS shared-memory stages (cp.async.bulk, completion on an mbarrier), one
// thread issues the 3xTF32 MMAs into one of two 128-column TMEM accumulators,
// and eight warps fold the finished accumulator (warp w: component q = w % 4, half
// of the columns; sums per row spin and column spin, turned into the 28 local
// densities at the end) while the other one fills.  dpart: [P][2][G][2*ND][nghl]
// ---------------------------------------------------------------------------
enum { DTC2_NS = 4, DTC2_FOLD = 256, DTC2_THREADS = DTC2_FOLD + 64, DTC2_MAXNC = 64 };
enum { DTC2_ACH = 2 * 128 * 8,                   // floats of one A chunk (hi, lo)
       DTC2_STAGE = DTC2_ACH + 2 * 128 * 8 };    // floats of one stage (A chunk, B chunk with npad <= 128)

struct DUnitTC {
  int kind, ix, iy, s;    // rows of block ix of spin s (0 up, 1 down), columns of block iy
  int b0, nc, npad, nk;   // columns [b0, b0 + nc), N = 2*nc padded to 16, K chunks of 8
  int achunk, nub;        // first A chunk of (ix, s); spin-up columns of block iy
  long long boff;         // floats: first B chunk of the unit within a point's B buffer
};
struct DBChunkTC {        // one B chunk: rows [a0, min(a0 + 8, ahi)) of a unit's columns
  int call, kind, ix, a0, ahi, b0, nc, npad;
  long long dst;          // floats within a point's B buffer
};
struct DAChunkTC { int ix, a0, ahi, pad_; };

__host__ __device__ constexpr size_t density_tc2_smem_bytes() {
  // the stage ring, then the column basis functions [64 b][32 r][4 q]; the
  // end-of-CTA reduction buffer [8 warps][2*ND][32] reuses the same memory
  return (size_t)(DTC2_NS * DTC2_STAGE + DTC2_MAXNC * 32 * 4) * sizeof(float);
}
static_assert(8 * 2 * ND * 32 <= DTC2_NS * DTC2_STAGE + DTC2_MAXNC * 32 * 4, "reduction buffer");

// A chunks (once per ground state): aphi[rt][chunk][hi | lo][128 x 8], rows m = q*32 + l
// grid (nachunk, ceil(nghl/32)), 256 threads
__global__ void __launch_bounds__(256) k_dens_asplit(DevBasisT<float> B, const DAChunkTC* __restrict__ chunks,
                                                     int nachunk, float* __restrict__ aphi) {
  const DAChunkTC ch = chunks[blockIdx.x];
  const int r0 = blockIdx.y * 32, nghl = B.nghl;
  const long long ps = (long long)B.dqp * nghl;
  float* dst = aphi + ((long long)blockIdx.y * nachunk + blockIdx.x) * DTC2_ACH;
  const int m = threadIdx.x & 127, k4 = threadIdx.x >> 7;
  const int q = m >> 5, r = r0 + (m & 31);
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (r < nghl) {
    const int a = ch.a0 + 4 * k4;
    const float* src = B.phi + q * ps + (long long)(B.st[ch.ix] + a) * nghl + r;
    if (a < ch.ahi) v.x = src[0];
    if (a + 1 < ch.ahi) v.y = src[nghl];
    if (a + 2 < ch.ahi) v.z = src[2 * nghl];
    if (a + 3 < ch.ahi) v.w = src[3 * nghl];
  }
  const int o = tc::cm_off(m, 4 * k4, 128);
  st_split4(dst + o, dst + 128 * 8 + o, v);
}

// B chunks of the listed points: bsplit[p][chunk.dst + (hi | lo)][npad x 8], rows n = pl*nc + b
// grid (nbchunk, nact), 256 threads
__global__ void __launch_bounds__(256) k_dens_bsplit(DevBasisT<float> B, DensTCArgs c0, DensTCArgs c1,
                                                     const DBChunkTC* __restrict__ chunks,
                                                     const int* __restrict__ actlist, float* __restrict__ bsplit,
                                                     long long bstride) {
  const DBChunkTC ch = chunks[blockIdx.x];
  const int p = actlist[blockIdx.y];
  const DensTCArgs& C = ch.call ? c1 : c0;
  const float* base = ch.kind == 0 ? C.rho : C.kap;
  const long long bsp = ch.kind == 0 ? C.rho_sp : C.kap_sp, bspl = ch.kind == 0 ? C.rho_spl : C.kap_spl;
  const long long off = (ch.kind == 0 ? C.roffs : C.koffs)[ch.ix];
  const float* mat = base + (long long)p * bsp + off;
  const int d = B.db[ch.ix];
  float* dst = bsplit + (long long)p * bstride + ch.dst;
  for (int e = threadIdx.x; e < 2 * ch.npad; e += blockDim.x) {
    const int n = e >> 1, k4 = e & 1;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (n < 2 * ch.nc) {
      const int pl = n >= ch.nc ? 1 : 0, b = n - pl * ch.nc;
      const int a = ch.a0 + 4 * k4;
      const float* src = mat + (long long)pl * bspl + (long long)(ch.b0 + b) * d + a;
      if (a < ch.ahi) v.x = src[0];
      if (a + 1 < ch.ahi) v.y = src[1];
      if (a + 2 < ch.ahi) v.z = src[2];
      if (a + 3 < ch.ahi) v.w = src[3];
    }
    const int o = tc::cm_off(n, 4 * k4, ch.npad);
    st_split4(dst + o, dst + ch.npad * 8 + o, v);
  }
}

// Every term of the density formulas is a fixed combination of the sums
//   T[s][up][q'] = sum over the columns b of spin up (1) or down (0) and the rows a
//                  of spin s of W_q(r, b) * phi_q'(b, r)   (re and im of W)
// so a fold warp accumulates only these sums per column (8 FMAs) and turns them
// into the 28 densities once, at the end (dtc2_densities).
// sum_unit: the columns [8*c8lo, 8*c8hi) of one unit (re of W at TMEM column b, im at
// nc + b); columns b < nupl are spin up.  KIND 1 (pairing): q' = 0 only.
template <int KIND, int NQ>
__device__ __forceinline__ void sum_unit(float (&T)[2][NQ][2], uint32_t lane_base, const float* sPb, int lane,
                                         int nc, int nupl, int c8lo, int c8hi, bool skip) {
  for (int c8 = c8lo; c8 < c8hi; ++c8) {
    float wre[8], wim[8];
    tc::tmem_ld8x2(lane_base + (uint32_t)(8 * c8), lane_base + (uint32_t)(nc + 8 * c8), wre, wim);
    if (skip) continue;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int b = 8 * c8 + i;
      if (b >= nc) break;
      const float4 pv = *reinterpret_cast<const float4*>(&sPb[(b * 32 + lane) * 4]);
      const float P[4] = {pv.x, pv.y, pv.z, pv.w};
      if (b < nupl) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          T[1][q][0] = fmaf(wre[i], P[q], T[1][q][0]);
          T[1][q][1] = fmaf(wim[i], P[q], T[1][q][1]);
        }
      } else {
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          T[0][q][0] = fmaf(wre[i], P[q], T[0][q][0]);
          T[0][q][1] = fmaf(wim[i], P[q], T[0][q][1]);
        }
      }
    }
  }
}

// the 28 densities of a fold warp of component Q from its sums: T0 (normal
// densities) and T1 (pairing densities, component 0) per row spin s and column spin
// up.  fold_same / fold_opp are linear in (wr, wi) * P, so a sum is folded as
// (wr, wi, P) = (1, 0, Re sums) plus (0, 1, Im sums).
template <int Q>
__device__ __forceinline__ void dtc2_densities(float (&acc)[2 * ND], const float (&T0)[2][2][4][2],
                                               const float (&T1)[2][2][1][2]) {
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int up = 0; up < 2; ++up) {
      const bool same = (up == 1) == (s == 0);
      const float sg = up ? 1.f : -1.f, sig = -sg;
      const float Pre[4] = {T0[s][up][0][0], T0[s][up][1][0], T0[s][up][2][0], T0[s][up][3][0]};
      const float Pim[4] = {T0[s][up][0][1], T0[s][up][1][1], T0[s][up][2][1], T0[s][up][3][1]};
      if (same) {
        fold_same<Q>(acc, 1.f, 0.f, Pre, sg);
        fold_same<Q>(acc, 0.f, 1.f, Pim, sg);
      } else {
        fold_opp<Q>(acc, 1.f, 0.f, Pre, sig);
        fold_opp<Q>(acc, 0.f, 1.f, Pim, sig);
      }
      if (Q == 0) {
        const float xr = 2.f * T1[s][up][0][0], xi = 2.f * T1[s][up][0][1];
        if (same) {
          acc[2 * D_SBR] += sig * xr; acc[2 * D_SBR + 1] += sig * xi;
          acc[2 * D_SBP] += xi; acc[2 * D_SBP + 1] += -xr;
        } else {
          acc[2 * D_RB] += -sg * xr; acc[2 * D_RB + 1] += -sg * xi;
          acc[2 * D_SBZ] += xr; acc[2 * D_SBZ + 1] += xi;
        }
      }
    }
}

// grid (ceil(nghl/32), G, 2*nact); DTC2_THREADS threads; dynamic smem density_tc2_smem_bytes().
// A CTA takes the units of its call with ix % G == g for its mesh tile and point.
__global__ void __launch_bounds__(DTC2_THREADS, 2) k_density_tc2(
    DevBasisT<float> B, const DUnitTC* __restrict__ units0, int nunit0, const DUnitTC* __restrict__ units1,
    int nunit1, const float* __restrict__ aphi, int nachunk, const float* __restrict__ bsplit, long long bstride,
    int G, const int* __restrict__ actlist, float* __restrict__ dpart, int* __restrict__ err) {
  const int p = actlist[blockIdx.z >> 1], call = blockIdx.z & 1;
  const DUnitTC* units = call ? units1 : units0;
  const int nunit = call ? nunit1 : nunit0;
  const int g = blockIdx.y, rt = blockIdx.x, r0 = rt * 32;
  const int nghl = B.nghl;
  const long long ps = (long long)B.dqp * nghl;
  extern __shared__ __align__(16) unsigned char smraw[];
  float* stages = reinterpret_cast<float*>(smraw);
  float* sPb = stages + DTC2_NS * DTC2_STAGE;
  __shared__ __align__(8) uint64_t full_bar[DTC2_NS], empty_bar[DTC2_NS], accf_bar[2], acce_bar[2];
  __shared__ uint32_t tslot;
  __shared__ volatile int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < DTC2_NS; ++i) { tc::mbar_init(&full_bar[i], 1); tc::mbar_init(&empty_bar[i], 1); }
    for (int j = 0; j < 2; ++j) { tc::mbar_init(&accf_bar[j], 1); tc::mbar_init(&acce_bar[j], DTC2_FOLD); }
    abort_flag = 0;
  }
  if (warp == 0) tc::tmem_alloc(&tslot, 256);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tslot;
  const int q = warp & 3, half = warp >> 2;
  float T0[2][2][4][2], T1[2][2][1][2];   // fold warps: [row spin s][column spin up][q'][re, im]
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int k = 0; k < 4; ++k) T0[a][b][k][c] = 0.f;
        T1[a][b][0][c] = 0.f;
      }
  if (warp < DTC2_FOLD / 32) {
    // ---------------- fold warps ----------------
    int u = 0, skind = -1, siy = -1, sb0 = -1;
    for (int i = 0; i < nunit; ++i) {
      const DUnitTC U = units[i];
      if (U.ix % G != g) continue;
      const int j = u & 1;
      if (U.kind != skind || U.iy != siy || U.b0 != sb0) {
        // column basis functions of the unit's columns, once per column range
        asm volatile("bar.sync 1, %0;" ::"r"(DTC2_FOLD) : "memory");   // previous fold done with sPb
        const int sb = B.st[U.iy] + U.b0;
        for (int e = tid; e < U.nc * 32; e += DTC2_FOLD) {
          const int b = e >> 5, l = e & 31, r = r0 + l;
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
          if (r < nghl) {
            const float* src = B.phi + (long long)(sb + b) * nghl + r;
            v.x = src[0];
            if (U.kind == 0) { v.y = src[ps]; v.z = src[2 * ps]; v.w = src[3 * ps]; }
          }
          *reinterpret_cast<float4*>(&sPb[(b * 32 + l) * 4]) = v;
        }
        asm volatile("bar.sync 1, %0;" ::"r"(DTC2_FOLD) : "memory");
        skind = U.kind; siy = U.iy; sb0 = U.b0;
      }
      if (!abort_flag && !tc::mbar_wait(&accf_bar[j], (u >> 1) & 1)) abort_flag = 1;
      tc::fence_after();
      // pairing units: only the warps of component 0 read their rows
      if (U.kind == 0 || q == 0) {
        const int nb8 = (U.nc + 7) / 8;
        const int c8lo = half == 0 ? 0 : (nb8 + 1) / 2, c8hi = half == 0 ? (nb8 + 1) / 2 : nb8;
        const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(128 * j);
        const bool skip = abort_flag || r0 + lane >= nghl;
        const int nupl = U.nub - U.b0;
        if (U.kind == 0) {
          if (U.s == 0) sum_unit<0, 4>(T0[0], lane_base, sPb, lane, U.nc, nupl, c8lo, c8hi, skip);
          else sum_unit<0, 4>(T0[1], lane_base, sPb, lane, U.nc, nupl, c8lo, c8hi, skip);
        } else {
          if (U.s == 0) sum_unit<1, 1>(T1[0], lane_base, sPb, lane, U.nc, nupl, c8lo, c8hi, skip);
          else sum_unit<1, 1>(T1[1], lane_base, sPb, lane, U.nc, nupl, c8lo, c8hi, skip);
        }
      }
      tc::fence_before();
      tc::mbar_arrive(&acce_bar[j]);   // accumulator j free for the unit after next
      ++u;
    }
  } else if (tid == DTC2_FOLD) {
    // ---------------- MMA issuer ----------------
    int cc = 0, u = 0;
    for (int i = 0; i < nunit; ++i) {
      const DUnitTC U = units[i];
      if (U.ix % G != g) continue;
      const int j = u & 1;
      if (u >= 2 && !abort_flag && !tc::mbar_wait(&acce_bar[j], ((u >> 1) - 1) & 1)) abort_flag = 1;
      tc::fence_after();
      const uint32_t idesc = tc::idesc_tf32(128, U.npad);
      const uint32_t lboA = (128 / 8) * 128, lboB = (uint32_t)(U.npad / 8) * 128;
      const uint32_t acc_t = tmem + (uint32_t)(128 * j);
      for (int kc = 0; kc < U.nk; ++kc, ++cc) {
        const int st = cc % DTC2_NS;
        if (!abort_flag && !tc::mbar_wait(&full_bar[st], (cc / DTC2_NS) & 1)) abort_flag = 1;
        tc::fence_after();
        if (!abort_flag) {
          const float* sAh = stages + st * DTC2_STAGE;
          const float* sAl = sAh + 128 * 8;
          const float* sBh = sAh + DTC2_ACH;
          const float* sBl = sBh + U.npad * 8;
          const uint64_t ah = tc::sdesc(tc::smem_u32(sAh), lboA, 128);
          const uint64_t al = tc::sdesc(tc::smem_u32(sAl), lboA, 128);
          const uint64_t bh = tc::sdesc(tc::smem_u32(sBh), lboB, 128);
          const uint64_t bl = tc::sdesc(tc::smem_u32(sBl), lboB, 128);
          tc::mma_tf32(acc_t, ah, bh, idesc, kc > 0);
          tc::mma_tf32(acc_t, ah, bl, idesc, true);
          tc::mma_tf32(acc_t, al, bh, idesc, true);
        }
        tc::mma_commit(&empty_bar[st]);
      }
      tc::mma_commit(&accf_bar[j]);   // W of this unit complete
      ++u;
    }
    // nothing may be in flight when the tensor memory is released
    if (u > 0 && !tc::mbar_wait(&accf_bar[(u - 1) & 1], ((u - 1) >> 1) & 1)) abort_flag = 1;
  } else if (tid == DTC2_FOLD + 32) {
    // ---------------- bulk-copy producer ----------------
    const float* asrc = aphi + (long long)rt * nachunk * DTC2_ACH;
    const float* bsrc = bsplit + (long long)p * bstride;
    int cc = 0;   // chunks issued, in order
    for (int i = 0; i < nunit && !abort_flag; ++i) {
      const DUnitTC U = units[i];
      if (U.ix % G != g) continue;
      const uint32_t bbytes = (uint32_t)U.npad * 64;
      for (int kc = 0; kc < U.nk; ++kc) {
        const int st = cc % DTC2_NS;
        if (cc >= DTC2_NS && !abort_flag && !tc::mbar_wait(&empty_bar[st], ((cc / DTC2_NS) - 1) & 1)) abort_flag = 1;
        if (abort_flag) break;
        float* sA = stages + st * DTC2_STAGE;
        tc::mbar_expect_tx(&full_bar[st], (uint32_t)(DTC2_ACH * 4) + bbytes);
        tc::bulk_g2s(sA, asrc + (long long)(U.achunk + kc) * DTC2_ACH, DTC2_ACH * 4, &full_bar[st]);
        tc::bulk_g2s(sA + DTC2_ACH, bsrc + U.boff + (long long)kc * 16 * U.npad, bbytes, &full_bar[st]);
        ++cc;
      }
    }
    // no copy of this CTA may still be landing when the memory is reused: the last
    // DTC2_NS chunks issued are the only ones that can be in flight
    for (int k = cc > DTC2_NS ? cc - DTC2_NS : 0; k < cc; ++k)
      if (!tc::mbar_wait(&full_bar[k % DTC2_NS], (k / DTC2_NS) & 1)) abort_flag = 1;
  }
  // all folds done: each fold warp's densities from its sums, then the sum of the 8 warps
  tc::fence_before();
  const bool ok = __syncthreads_and(!abort_flag);
  float* red = stages;   // [8][2*ND][32]; the stages are no longer in use
  if (warp < 8) {
    float acc[2 * ND];
#pragma unroll
    for (int k = 0; k < 2 * ND; ++k) acc[k] = 0.f;
    switch (q) {
      case 0: dtc2_densities<0>(acc, T0, T1); break;
      case 1: dtc2_densities<1>(acc, T0, T1); break;
      case 2: dtc2_densities<2>(acc, T0, T1); break;
      default: dtc2_densities<3>(acc, T0, T1); break;
    }
#pragma unroll
    for (int k = 0; k < 2 * ND; ++k) red[(warp * 2 * ND + k) * 32 + lane] = acc[k];
  }
  __syncthreads();
  if (!ok) {
    if (tid == 0) atomicExch(err, 1);
  } else {
    float* out = dpart + (((long long)p * 2 + call) * G + g) * (2 * ND) * nghl;
    for (int e = tid; e < 2 * ND * 32; e += blockDim.x) {
      const int k = e / 32, l = e % 32;
      if (r0 + l >= nghl) continue;
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) v += red[(w * 2 * ND + k) * 32 + l];
      out[(long long)k * nghl + r0 + l] = v;
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_free(tmem, 256);
}

// ---------------------------------------------------------------------------
// mean field: mf slot (iy, iz, sa, sb) = ((iy*5 + iz)*2 + (sa<0))*2 + (sb<0);
// pairing fields at 100 + (sa<0)*2 + (sb<0)
// mf: [P][2][NMF][2][nghl]
// ---------------------------------------------------------------------------
enum { NMF = 104 };
__host__ __device__ __forceinline__ int mfslot(int iy, int iz, int sa, int sb) {
  return ((iy * 5 + iz) * 2 + (sa < 0 ? 1 : 0)) * 2 + (sb < 0 ? 1 : 0);
}

// complex arithmetic of the mean field in the evaluation's precision S (FP64 for the
// FP64 form and the anchors, FP32 for the increment evaluations of the mixed form)
template <class S> struct cplxT { S r, i; };
template <class S> __device__ __forceinline__ cplxT<S> cmk(S r, S i) { cplxT<S> c; c.r = r; c.i = i; return c; }
template <class S> __device__ __forceinline__ cplxT<S> cadd(cplxT<S> a, cplxT<S> b) { return cmk<S>(a.r + b.r, a.i + b.i); }
template <class S> __device__ __forceinline__ cplxT<S> csc(S s, cplxT<S> a) { return cmk<S>(s * a.r, s * a.i); }

template <class T>
__global__ void __launch_bounds__(128) k_meanfield(DevBasisT<T> B, int G, const T* __restrict__ dpart,
                                                   T* __restrict__ mfout, const int* __restrict__ active) {
  using S = T;
  using C = cplxT<S>;
  const int p = blockIdx.y >> 1, call = blockIdx.y & 1;
  if (!active[p]) return;
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const int nghl = B.nghl;
  if (r >= nghl) return;
  C d[ND];
  const T* dp = dpart + ((long long)p * 2 + call) * G * (2 * ND) * nghl;
  const S wd = B.wdcori[r];
  for (int k = 0; k < ND; ++k) {
    S sr = S(0.0), si = S(0.0);
    for (int g = 0; g < G; ++g) {
      sr += (S)dp[((long long)g * 2 * ND + 2 * k) * nghl + r];
      si += (S)dp[((long long)g * 2 * ND + 2 * k + 1) * nghl + r];
    }
    d[k] = cmk<S>(sr * wd, si * wd);
  }
  const S crho = B.crho[r], cs = B.cs[r], cpair = B.cpair[r], cspair = B.cspair[r];
  const S cdrho = B.sc[0], ctau = B.sc[1], ctj0 = B.sc[2], ctj1 = B.sc[3], ctj2 = B.sc[4], crdj = B.sc[5];
  const S cds = B.sc[6], ct = B.sc[7], cj = B.sc[8], cgs = B.sc[9], cf = B.sc[10], csdj = B.sc[11];
  C mf[NMF];
  for (int k = 0; k < NMF; ++k) mf[k] = cmk<S>(S(0.0), S(0.0));
#define M_(iy, iz, sa, sb) mf[mfslot(iy, iz, sa, sb)]
#define ADD(iy, iz, sa, sb, sym, v) M_(iy, iz, sa, sb) = cadd<S>(M_(iy, iz, sa, sb), csc<S>(sym, v))
  const C rho = d[D_RHO], tau = d[D_TAU], tjrr = d[D_TJRR], tjpr = d[D_TJPR], tjzr = d[D_TJZR];
  const C tjrp = d[D_TJRP], tjpp = d[D_TJPP], tjzp = d[D_TJZP], tjrz = d[D_TJRZ], tjpz = d[D_TJPZ];
  const C tjzz = d[D_TJZZ], sr = d[D_SR], sp = d[D_SP], sz = d[D_SZ], tr = d[D_TR], tp = d[D_TP];
  const C tz = d[D_TZ], jr = d[D_JR], jp = d[D_JP], jz = d[D_JZ], fr = d[D_FR], fp = d[D_FP];
  const C fz = d[D_FZ], gs = d[D_GS];
  const C t0 = csc<S>(ctj0, cadd<S>(cadd<S>(tjrr, tjpp), tjzz));
  const C t1a = csc<S>(ctj1, cadd<S>(tjzr, csc<S>(-S(1.0), tjrz)));
  const C t1b = csc<S>(ctj1, cadd<S>(tjpz, csc<S>(-S(1.0), tjzp)));
  const C t2a = csc<S>(ctj2, cadd<S>(tjrz, tjzr));
  const C t2b = csc<S>(ctj2, cadd<S>(tjpz, tjzp));
  C aux;
  // diagonal in spin (pnfam_hamiltonian_blas.f90:783-905)
  M_(0, 0, 1, 1) = cadd<S>(csc<S>(S(2.0) * crho, rho), csc<S>(ctau, tau));
  M_(0, 0, -1, -1) = M_(0, 0, 1, 1);
  aux = cadd<S>(cadd<S>(csc<S>(S(2.0) * cs, sz), csc<S>(ct, tz)), csc<S>(cf, fz));
  ADD(0, 0, 1, 1, S(1.0), aux); ADD(0, 0, -1, -1, -S(1.0), aux);

  M_(0, 1, 1, 1) = csc<S>(-crdj, cadd<S>(tjpz, csc<S>(-S(1.0), tjzp)));
  M_(0, 1, -1, -1) = M_(0, 1, 1, 1);
  aux = csc<S>(-csdj, jp);
  ADD(0, 1, 1, 1, S(1.0), aux); ADD(0, 1, -1, -1, -S(1.0), aux);
  M_(1, 0, 1, 1) = M_(0, 1, 1, 1);
  M_(1, 0, -1, -1) = M_(0, 1, -1, -1);
  aux = cmk<S>(-t1a.i + S(0.5) * t2a.i, t1a.r - S(0.5) * t2a.r);
  ADD(0, 1, 1, 1, S(1.0), aux); ADD(0, 1, -1, -1, -S(1.0), aux);
  ADD(1, 0, 1, 1, -S(1.0), aux); ADD(1, 0, -1, -1, S(1.0), aux);
  aux = cmk<S>(cj * jr.i, -cj * jr.r);
  ADD(0, 1, 1, 1, S(1.0), aux); ADD(0, 1, -1, -1, S(1.0), aux);
  ADD(1, 0, 1, 1, -S(1.0), aux); ADD(1, 0, -1, -1, -S(1.0), aux);

  M_(0, 2, 1, 1) = csc<S>(cj, jp);
  M_(0, 2, -1, -1) = M_(0, 2, 1, 1);
  aux = cadd<S>(t1b, csc<S>(S(0.5), t2b));
  ADD(0, 2, 1, 1, S(1.0), aux); ADD(0, 2, -1, -1, -S(1.0), aux);
  M_(2, 0, 1, 1) = M_(0, 2, 1, 1);
  M_(2, 0, -1, -1) = M_(0, 2, -1, -1);
  aux = cmk<S>(-csdj * jr.i, csdj * jr.r);
  ADD(0, 2, 1, 1, S(1.0), aux); ADD(0, 2, -1, -1, -S(1.0), aux);
  ADD(2, 0, 1, 1, -S(1.0), aux); ADD(2, 0, -1, -1, S(1.0), aux);
  aux = cmk<S>(crdj * (tjzr.i - tjrz.i), -crdj * (tjzr.r - tjrz.r));
  ADD(0, 2, 1, 1, S(1.0), aux); ADD(0, 2, -1, -1, S(1.0), aux);
  ADD(2, 0, 1, 1, -S(1.0), aux); ADD(2, 0, -1, -1, -S(1.0), aux);

  M_(0, 3, 1, 1) = csc<S>(-crdj, cadd<S>(tjrp, csc<S>(-S(1.0), tjpr)));
  M_(0, 3, -1, -1) = M_(0, 3, 1, 1);
  aux = csc<S>(S(2.0) * cgs, gs);
  ADD(0, 3, 1, 1, S(1.0), aux); ADD(0, 3, -1, -1, -S(1.0), aux);
  M_(3, 0, 1, 1) = M_(0, 3, 1, 1);
  M_(3, 0, -1, -1) = M_(0, 3, -1, -1);
  aux = cmk<S>(t0.i - ctj2 * (tjrr.i + tjpp.i - S(2.0) * tjzz.i) / S(3.0),
            -t0.r + ctj2 * (tjrr.r + tjpp.r - S(2.0) * tjzz.r) / S(3.0));
  ADD(0, 3, 1, 1, S(1.0), aux); ADD(0, 3, -1, -1, -S(1.0), aux);
  ADD(3, 0, 1, 1, -S(1.0), aux); ADD(3, 0, -1, -1, S(1.0), aux);
  aux = cmk<S>(cj * jz.i, -cj * jz.r);
  ADD(0, 3, 1, 1, S(1.0), aux); ADD(0, 3, -1, -1, S(1.0), aux);
  ADD(3, 0, 1, 1, -S(1.0), aux); ADD(3, 0, -1, -1, -S(1.0), aux);

  M_(0, 4, 1, 1) = csc<S>(S(2.0) * cdrho, rho);
  M_(0, 4, -1, -1) = M_(0, 4, 1, 1);
  aux = csc<S>(S(2.0) * cds, sz);
  ADD(0, 4, 1, 1, S(1.0), aux); ADD(0, 4, -1, -1, -S(1.0), aux);
  M_(4, 0, 1, 1) = M_(0, 4, 1, 1);
  M_(4, 0, -1, -1) = M_(0, 4, -1, -1);

  M_(1, 2, 1, 1) = csc<S>(csdj, sz);
  M_(1, 2, -1, -1) = M_(1, 2, 1, 1);
  aux = csc<S>(crdj, rho);
  ADD(1, 2, 1, 1, S(1.0), aux); ADD(1, 2, -1, -1, -S(1.0), aux);
  M_(2, 1, 1, 1) = M_(1, 2, 1, 1);
  M_(2, 1, -1, -1) = M_(1, 2, -1, -1);

  M_(1, 3, 1, 1) = csc<S>(S(0.5) * cf, sr);
  M_(1, 3, -1, -1) = csc<S>(-S(1.0), M_(1, 3, 1, 1));
  M_(3, 1, 1, 1) = M_(1, 3, 1, 1);
  M_(3, 1, -1, -1) = M_(1, 3, -1, -1);
  aux = cmk<S>(-csdj * sp.i, csdj * sp.r);
  ADD(1, 3, 1, 1, S(1.0), aux); ADD(1, 3, -1, -1, S(1.0), aux);
  ADD(3, 1, 1, 1, -S(1.0), aux); ADD(3, 1, -1, -1, -S(1.0), aux);

  M_(2, 3, 1, 1) = csc<S>(-csdj, sr);
  M_(2, 3, -1, -1) = M_(2, 3, 1, 1);
  aux = cmk<S>(S(0.5) * cf * sp.i, -S(0.5) * cf * sp.r);
  ADD(2, 3, 1, 1, S(1.0), aux); ADD(2, 3, -1, -1, -S(1.0), aux);
  M_(3, 2, 1, 1) = M_(2, 3, -1, -1);
  M_(3, 2, -1, -1) = M_(2, 3, 1, 1);

  M_(1, 1, 1, 1) = csc<S>(S(4.0) * cdrho + ctau, rho);
  M_(1, 1, -1, -1) = M_(1, 1, 1, 1);
  aux = csc<S>(S(4.0) * cds + ct, sz);
  ADD(1, 1, 1, 1, S(1.0), aux); ADD(1, 1, -1, -1, -S(1.0), aux);
  M_(2, 2, 1, 1) = M_(1, 1, 1, 1);
  M_(2, 2, -1, -1) = M_(1, 1, -1, -1);
  M_(3, 3, 1, 1) = M_(1, 1, 1, 1);
  M_(3, 3, -1, -1) = M_(1, 1, -1, -1);
  aux = csc<S>(cf, sz);
  ADD(3, 3, 1, 1, S(1.0), aux); ADD(3, 3, -1, -1, -S(1.0), aux);

  // not diagonal in spin (pnfam_hamiltonian_blas.f90:908-1094)
  M_(0, 0, 1, -1) = cadd<S>(cadd<S>(csc<S>(S(2.0) * cs, sr), csc<S>(ct, tr)), csc<S>(cf, fr));
  M_(0, 0, -1, 1) = M_(0, 0, 1, -1);
  aux = cmk<S>(S(2.0) * cs * sp.i + ct * tp.i + cf * fp.i, -S(2.0) * cs * sp.r - ct * tp.r - cf * fp.r);
  ADD(0, 0, 1, -1, S(1.0), aux); ADD(0, 0, -1, 1, -S(1.0), aux);

  M_(0, 1, 1, -1) = csc<S>(S(2.0) * cgs, gs);
  M_(0, 1, -1, 1) = M_(0, 1, 1, -1);
  aux = cmk<S>(csdj * jz.i, -csdj * jz.r);
  ADD(0, 1, 1, -1, S(1.0), aux); ADD(0, 1, -1, 1, -S(1.0), aux);
  M_(1, 0, 1, -1) = M_(0, 1, 1, -1);
  M_(1, 0, -1, 1) = M_(0, 1, -1, 1);
  M_(0, 2, 1, -1) = M_(0, 1, 1, -1);
  M_(2, 0, -1, 1) = M_(1, 0, -1, 1);
  M_(2, 0, 1, -1) = csc<S>(-S(1.0), M_(0, 2, 1, -1));
  M_(0, 2, -1, 1) = csc<S>(-S(1.0), M_(2, 0, -1, 1));
  aux = csc<S>(-ctj1, cadd<S>(tjrp, csc<S>(-S(1.0), tjpr)));
  ADD(0, 1, 1, -1, S(1.0), aux); ADD(0, 1, -1, 1, -S(1.0), aux); ADD(1, 0, 1, -1, -S(1.0), aux); ADD(1, 0, -1, 1, S(1.0), aux);
  ADD(0, 2, 1, -1, S(1.0), aux); ADD(0, 2, -1, 1, S(1.0), aux); ADD(2, 0, 1, -1, S(1.0), aux); ADD(2, 0, -1, 1, S(1.0), aux);
  aux = cmk<S>(t0.i, -t0.r);
  ADD(0, 1, 1, -1, S(1.0), aux); ADD(0, 1, -1, 1, S(1.0), aux); ADD(1, 0, 1, -1, -S(1.0), aux); ADD(1, 0, -1, 1, -S(1.0), aux);
  ADD(0, 2, 1, -1, S(1.0), aux); ADD(0, 2, -1, 1, -S(1.0), aux); ADD(2, 0, 1, -1, S(1.0), aux); ADD(2, 0, -1, 1, -S(1.0), aux);
  aux = csc<S>(-S(0.5) * ctj2, cadd<S>(tjrp, tjpr));
  ADD(0, 1, 1, -1, S(1.0), aux); ADD(0, 1, -1, 1, -S(1.0), aux); ADD(1, 0, 1, -1, -S(1.0), aux); ADD(1, 0, -1, 1, S(1.0), aux);
  ADD(0, 2, 1, -1, -S(1.0), aux); ADD(0, 2, -1, 1, -S(1.0), aux); ADD(2, 0, 1, -1, -S(1.0), aux); ADD(2, 0, -1, 1, -S(1.0), aux);
  aux = cmk<S>(-ctj2 * (-S(2.0) * tjrr.i + tjpp.i + tjzz.i) / S(3.0), ctj2 * (-S(2.0) * tjrr.r + tjpp.r + tjzz.r) / S(3.0));
  ADD(0, 1, 1, -1, S(1.0), aux); ADD(0, 1, -1, 1, S(1.0), aux); ADD(1, 0, 1, -1, -S(1.0), aux); ADD(1, 0, -1, 1, -S(1.0), aux);
  aux = cmk<S>(-ctj2 * (tjrr.i - S(2.0) * tjpp.i + tjzz.i) / S(3.0), ctj2 * (tjrr.r - S(2.0) * tjpp.r + tjzz.r) / S(3.0));
  ADD(0, 2, 1, -1, S(1.0), aux); ADD(0, 2, -1, 1, -S(1.0), aux); ADD(2, 0, 1, -1, S(1.0), aux); ADD(2, 0, -1, 1, -S(1.0), aux);

  M_(0, 3, 1, -1) = csc<S>(csdj, jp);
  M_(0, 3, -1, 1) = M_(0, 3, 1, -1);
  aux = cmk<S>(-csdj * jr.i, csdj * jr.r);
  ADD(0, 3, 1, -1, S(1.0), aux); ADD(0, 3, -1, 1, -S(1.0), aux);
  M_(3, 0, 1, -1) = M_(0, 3, 1, -1);
  M_(3, 0, -1, 1) = M_(0, 3, -1, 1);
  aux = cmk<S>(t1a.i + S(0.5) * t2a.i, -t1a.r - S(0.5) * t2a.r);
  ADD(0, 3, 1, -1, S(1.0), aux); ADD(0, 3, -1, 1, S(1.0), aux); ADD(3, 0, 1, -1, -S(1.0), aux); ADD(3, 0, -1, 1, -S(1.0), aux);
  aux = cadd<S>(t1b, csc<S>(-S(0.5), t2b));
  ADD(0, 3, 1, -1, S(1.0), aux); ADD(0, 3, -1, 1, -S(1.0), aux); ADD(3, 0, 1, -1, -S(1.0), aux); ADD(3, 0, -1, 1, S(1.0), aux);

  M_(0, 4, 1, -1) = csc<S>(S(2.0) * cds, sr);
  M_(0, 4, -1, 1) = M_(0, 4, 1, -1);
  aux = cmk<S>(S(2.0) * cds * sp.i, -S(2.0) * cds * sp.r);
  ADD(0, 4, 1, -1, S(1.0), aux); ADD(0, 4, -1, 1, -S(1.0), aux);
  M_(4, 0, 1, -1) = M_(0, 4, 1, -1);
  M_(4, 0, -1, 1) = M_(0, 4, -1, 1);

  M_(1, 2, 1, -1) = cmk<S>(-S(0.5) * cf * sp.i, S(0.5) * cf * sp.r);
  M_(1, 2, -1, 1) = M_(1, 2, 1, -1);
  aux = csc<S>(S(0.5) * cf, sr);
  ADD(1, 2, 1, -1, S(1.0), aux); ADD(1, 2, -1, 1, -S(1.0), aux);
  M_(2, 1, 1, -1) = csc<S>(-S(1.0), M_(1, 2, 1, -1));
  M_(2, 1, -1, 1) = csc<S>(-S(1.0), M_(1, 2, -1, 1));

  M_(1, 3, 1, -1) = csc<S>(S(0.5) * cf, sz);
  M_(1, 3, -1, 1) = M_(1, 3, 1, -1);
  aux = csc<S>(crdj, rho);
  ADD(1, 3, 1, -1, S(1.0), aux); ADD(1, 3, -1, 1, -S(1.0), aux);
  M_(3, 1, 1, -1) = M_(1, 3, -1, 1);
  M_(3, 1, -1, 1) = M_(1, 3, 1, -1);
  M_(3, 2, 1, -1) = M_(3, 1, 1, -1);
  M_(2, 3, -1, 1) = M_(1, 3, -1, 1);
  M_(2, 3, 1, -1) = csc<S>(-S(1.0), M_(1, 3, 1, -1));
  M_(3, 2, -1, 1) = csc<S>(-S(1.0), M_(3, 1, -1, 1));

  M_(3, 3, 1, -1) = csc<S>(ct + S(4.0) * cds, sr);
  M_(3, 3, -1, 1) = M_(3, 3, 1, -1);
  aux = cmk<S>((ct + S(4.0) * cds) * sp.i, -(ct + S(4.0) * cds) * sp.r);
  ADD(3, 3, 1, -1, S(1.0), aux); ADD(3, 3, -1, 1, -S(1.0), aux);
  M_(1, 1, 1, -1) = M_(3, 3, 1, -1);
  M_(1, 1, -1, 1) = M_(3, 3, -1, 1);
  aux = csc<S>(cf, sr);
  ADD(1, 1, 1, -1, S(1.0), aux); ADD(1, 1, -1, 1, S(1.0), aux);
  M_(2, 2, 1, -1) = M_(3, 3, 1, -1);
  M_(2, 2, -1, 1) = M_(3, 3, -1, 1);
  aux = cmk<S>(cf * sp.i, -cf * sp.r);
  ADD(2, 2, 1, -1, S(1.0), aux); ADD(2, 2, -1, 1, -S(1.0), aux);
#undef ADD
#undef M_
  // pairing fields (pnfam_hamiltonian_blas.f90:1201-1208): index (sa, sb)
  const C rb = d[D_RB], sbr = d[D_SBR], sbp = d[D_SBP], sbz = d[D_SBZ];
  mf[100] = cmk<S>(cspair * (sbr.r + sbp.i), cspair * (sbr.i - sbp.r));        // a+ b+
  mf[101] = cmk<S>(cpair * rb.r - cspair * sbz.r, cpair * rb.i - cspair * sbz.i); // a+ b-
  mf[102] = cmk<S>(-cpair * rb.r - cspair * sbz.r, -cpair * rb.i - cspair * sbz.i); // a- b+
  mf[103] = cmk<S>(cspair * (-sbr.r + sbp.i), cspair * (-sbr.i - sbp.r));      // a- b-
  T* out = mfout + ((long long)p * 2 + call) * NMF * 2 * nghl;
  for (int k = 0; k < NMF; ++k) {
    out[((long long)k * 2) * nghl + r] = (T)mf[k].r;
    out[((long long)k * 2 + 1) * nghl + r] = (T)mf[k].i;
  }
}

// ---------------------------------------------------------------------------
// field projection: out_ab = 2 sum_r sum_iy phi_iy(a,r) hpsi(iy)(r,b)
// ---------------------------------------------------------------------------
// part of an output block of the FP64 projection: na rows (of one spin) from state ja on,
// nb columns from state jb on; output element (a, b) at off + a + b*ld of the quadrants
struct HPiece {
  int ja, na, jb, nb;
  long long off;
  int ld, item0;   // first output of the piece in its group
};
// pieces with the same field tensor that one CTA computes: at most HP_ITEMS outputs, one
// per thread
enum { HP_PIECES = 4, HP_ITEMS = 256, HP_ROWS = 64, HP_TAB = 128, HRC = 16 };
struct HGroup {
  int call;        // 0: pn, 1: np
  int sa;          // spin of the rows (+1/-1)
  int mode;        // 0: mean field (5 components), 1: pairing (1 component)
  int hr;          // mesh points per chunk: 16 or 8
  int np, nrow, ncol, nitem;
  HPiece piece[HP_PIECES];
};
// dynamic shared memory of a group: row functions, field tensor (18 component pairs: the
// others vanish, see k_meanfield), hpsi; the padding keeps 16-byte reads of different
// rows or columns on different banks
__host__ __device__ constexpr size_t hproj_fp64_smem(int hr, int mode, int nrow, int ncol) {
  return sizeof(double) * (mode == 0 ? 5 * nrow * (hr + 2) + 18 * 4 * hr + 5 * ncol * (2 * hr + 2)
                                     : nrow * (hr + 2) + 4 * hr + ncol * (2 * hr + 2));
}
// groups are filled up to the first figure (5 CTAs on an SM); a single piece stays below
// the second: 64 rows and 4 columns, or 8 and 32
constexpr size_t HP_SMEM_FILL = 44 * 1024, HP_SMEM_MAX = 64 * 1024;

// FP64 field projection.  Per chunk of mesh points a CTA stages the row functions and the
// field tensor, forms hpsi of its columns and adds each thread's output:
//   out_ab = 2 sum_r sum_iy phi_iy(a, r) hpsi(iy)(r, b)
// over the chunks, in each over the components, in each over the points (this order and the
// chunk length of a block pair are part of the result: an iteration that amplifies
// rounding repeats to the last digit).
// Bound by the FP64 pipe (one warp instruction per 16 cycles of an SM), so the outputs are
// dealt to the threads in one row over several block pairs: with tiles of 32 x 32, 64 x 16 or
// 128 x 8 outputs, 2 x 2 per thread, the small blocks of N_sh = 8 left most warps without
// rows (46 % of the pipe, 23 of 33 cycles per instruction at barriers) and formed hpsi with
// the 7 vanishing pairs of the field tensor: 40 points there 20.2 ms, now 5.5 ms.
// grid (ngroups, P); 256 threads; dynamic smem: the largest hproj_fp64_smem of the groups
template <int HR>
__device__ __forceinline__ void hproj_fp64_group(const DevBasis& B, const HGroup& g, const double* __restrict__ mfp,
                                                 double* __restrict__ out, long long nxy, double* sm, const int* srow,
                                                 const int* scol, int row, int col, long long off) {
  constexpr int SA = HR + 2, SH = 2 * HR + 2;
  const int nghl = B.nghl, nc = g.mode == 0 ? 5 : 1, nrow = g.nrow, ncol = g.ncol, tid = threadIdx.x;
  const long long ps = (long long)B.dqp * nghl;
  double* sA = sm;                      // [nc][nrow][SA]
  double* sM = sA + nc * nrow * SA;     // [18 or 1][2 sb][2 re/im][HR]
  double* sH = sM + (g.mode == 0 ? 18 : 1) * 4 * HR;   // [nc][ncol][2 re/im][HR], a column SH apart
  double ar = 0.0, ai = 0.0;
  for (int r0 = 0; r0 < nghl; r0 += HR) {
    const int nr = min(HR, nghl - r0);
    __syncthreads();
    for (int q = 0; q < nc; ++q)
      for (int e = tid; e < nrow * HR; e += 256) {
        const int rr = e % HR, a = e / HR;
        sA[(q * nrow + a) * SA + rr] = rr < nr ? B.phi[q * ps + (long long)srow[a] * nghl + r0 + rr] : 0.0;
      }
    for (int e = tid; e < (g.mode == 0 ? 18 : 1) * 4 * HR; e += 256) {
      const int rr = e % HR, m = e / HR, pair = m >> 2, sb = (m >> 1) & 1, ri = m & 1;
      int slot;
      if (g.mode == 0) {
        const int iy = pair < 16 ? pair >> 2 : pair == 16 ? 0 : 4, iz = pair < 16 ? pair & 3 : pair == 16 ? 4 : 0;
        slot = mfslot(iy, iz, g.sa, sb == 0 ? 1 : -1);
      } else {
        slot = 100 + (g.sa < 0 ? 2 : 0) + sb;
      }
      sM[e] = rr < nr ? mfp[((long long)slot * 2 + ri) * nghl + r0 + rr] : 0.0;
    }
    __syncthreads();
    // hpsi(iy, b, r) = sum_iz mf(iy, iz, sa, s_b)(r) phi_iz(b, r)
    for (int e = tid; e < ncol * HR; e += 256) {
      const int rr = e % HR, b = e / HR, jb = scol[b];
      const double* f = B.phi + (long long)jb * nghl + r0 + rr;
      const double* m = sM + (B.ns[jb] > 0 ? 0 : 2 * HR) + rr;
      double* h = sH + b * SH + rr;
      if (g.mode == 0) {
        double p[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) p[q] = rr < nr ? f[q * ps] : 0.0;
#pragma unroll
        for (int iy = 0; iy < 5; ++iy) {
          double hr = 0.0, hi = 0.0;
#pragma unroll
          for (int iz = 0; iz < 5; ++iz) {
            if (iz == 4 ? iy != 0 : iy == 4 && iz != 0) continue;   // vanishes
            const int pair = iz == 4 ? 16 : iy == 4 ? 17 : iy * 4 + iz;
            hr = fma(m[pair * 4 * HR], p[iz], hr);
            hi = fma(m[pair * 4 * HR + HR], p[iz], hi);
          }
          h[iy * ncol * SH] = hr;
          h[iy * ncol * SH + HR] = hi;
        }
      } else {
        const double p = rr < nr ? f[0] : 0.0;
        h[0] = m[0] * p;
        h[HR] = m[HR] * p;
      }
    }
    __syncthreads();
    if (row >= 0)
      for (int q = 0; q < nc; ++q) {
        const double2* a = reinterpret_cast<const double2*>(sA + (q * nrow + row) * SA);
        const double2* h = reinterpret_cast<const double2*>(sH + (q * ncol + col) * SH);
#pragma unroll
        for (int i = 0; i < HR / 2; ++i) {
          const double2 x = a[i], u = h[i], v = h[HR / 2 + i];
          ar = fma(x.x, u.x, ar); ai = fma(x.x, v.x, ai);
          ar = fma(x.y, u.y, ar); ai = fma(x.y, v.y, ai);
        }
      }
  }
  if (row >= 0) {
    out[off] = 2.0 * ar;
    out[4 * nxy + off] = 2.0 * ai;
  }
}

__global__ void __launch_bounds__(256) k_hproj_fp64(DevBasis B, const HGroup* __restrict__ groups,
                                                    const double* __restrict__ mf, double* __restrict__ hsp,
                                                    long long nxy, const int* __restrict__ active) {
  const int p = blockIdx.y;
  if (!active[p]) return;
  const HGroup& g = groups[blockIdx.x];
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ int srow[HP_TAB], scol[HP_TAB];   // states of the rows and columns
  int row = -1, col = 0, r0 = 0, c0 = 0;
  long long off = 0;
  for (int k = 0; k < g.np; ++k) {
    const HPiece& q = g.piece[k];
    for (int a = threadIdx.x; a < q.na; a += 256) srow[r0 + a] = q.ja + a;
    for (int b = threadIdx.x; b < q.nb; b += 256) scol[c0 + b] = q.jb + b;
    const int i = (int)threadIdx.x - q.item0;
    if (i >= 0 && i < q.na * q.nb) {
      const int a = i % q.na, b = i / q.na;
      row = r0 + a;
      col = c0 + b;
      off = q.off + a + (long long)b * q.ld;
    }
    r0 += q.na;
    c0 += q.nb;
  }
  const double* mfp = mf + ((long long)p * 2 + g.call) * NMF * 2 * B.nghl;
  double* out = hsp + (long long)p * 8 * nxy;
  double* sm = reinterpret_cast<double*>(smraw);
  if (g.hr == 8) hproj_fp64_group<8>(B, g, mfp, out, nxy, sm, srow, scol, row, col, off);
  else hproj_fp64_group<HRC>(B, g, mfp, out, nxy, sm, srow, scol, row, col, off);
}

// ---------------------------------------------------------------------------
// field projection on the tensor cores (FP32 data, 3xTF32 products).
// One CTA computes, for one (block pair, spin segment of the rows) and up to pg
// points, D[m][n] = sum_k hpsi[k][m] phi[k][n] with
//   m = pl*64 + j, j = (point in the group)*nbc + b   (rows: Re, then Im of hpsi)
//   n = a (the rows of the output block, N padded to np)
//   k = (q, r), 32 mesh points of one component q per chunk.
// Warps 0-7 produce the A operand of a chunk (hpsi generated from the field
// tensor and the column basis functions) into one of two shared-memory stages;
// the B operand (the row basis functions, constant: split into TF32 hi and lo once
// per operator in the canonical layout) is copied in by the bulk-copy engine.
// Warp 8 issues the MMAs of a chunk as soon as its stage is full and releases the
// stage through tcgen05.commit, so operand production and tensor-core work
// overlap.  D accumulates in tensor memory and out_ab = 2 D.
// ---------------------------------------------------------------------------
struct HTaskTC {
  int ix, iy, a0, na, b0, nbc, sa, mode, call, outq;
  int np;          // N of the MMA: na rounded up to 16
  int pg;          // points per CTA (pg * nbc <= 64)
  long long ooff;
  long long tphi;  // floats: the pre-split row basis functions of rows a0..a0+na of block ix
};
enum { HTC_K = 32, HTC_MAXB = 64, HTC_MAXN = 128, HTC_MAXPG = 8, HTC_PROD = 256, HTC_THREADS = HTC_PROD + 32 };
// pre-split B operand of one row tile (rows a0..a0+na of block ix): for component q
// and mesh chunk rc (32 points), [hi | lo][np x 32] at off + (q * nrc + rc) * 64 * np
struct HPTile { int ix, a0, na, np; long long off; };

// grid (ntiles, 5 * nrc), 256 threads
__global__ void __launch_bounds__(256) k_hproj_bsplit(DevBasisT<float> B, const HPTile* __restrict__ tiles, int nrc,
                                                      float* __restrict__ hphi) {
  const HPTile t = tiles[blockIdx.x];
  const int q = blockIdx.y / nrc, r0 = (blockIdx.y % nrc) * HTC_K;
  const int nghl = B.nghl;
  const long long ps = (long long)B.dqp * nghl;
  float* dst = hphi + t.off + (long long)blockIdx.y * 64 * t.np;
  const int ja0 = B.st[t.ix] + t.a0;
  for (int e = threadIdx.x; e < t.np * 8; e += blockDim.x) {
    const int n = e % t.np, r4 = e / t.np;
    const float4 v = ld_row4(B.phi + q * ps + (long long)(ja0 + n) * nghl, r0 + 4 * r4, nghl, n < t.na);
    const int o = tc::cm_off(n, 4 * r4, t.np);
    st_split4(dst + o, dst + 32 * t.np + o, v);
  }
}

// dynamic shared memory for tiles of at most npmax output rows: two stages of
// A (128 x 32, hi and lo) and B (npmax x 32, hi and lo), then the field tensor
// of the current chunk [pg][2 sb][5 iz][2 re/im][32 r]
__host__ __device__ constexpr size_t hproj_tc_smem_bytes(int npmax) {
  return (size_t)(2 * (2 * 128 * HTC_K + 2 * npmax * HTC_K) + HTC_MAXPG * 2 * 5 * 2 * HTC_K) * sizeof(float);
}

// grid (ntasks, point groups); HTC_THREADS threads; dynamic smem hproj_tc_smem_bytes(npmax)
// actlist[nact]: the points to evaluate; err: set to 1 if a wait on the tensor
// cores gave up (the CTA then writes nothing)
__global__ void __launch_bounds__(HTC_THREADS, 2) k_hproj_tc(DevBasisT<float> B, const HTaskTC* __restrict__ tasks,
                                                             const int* __restrict__ actlist, int nact, int npmax,
                                                             const float* __restrict__ mf,
                                                             const float* __restrict__ hphi, float* __restrict__ hsp,
                                                             long long nxy, int* __restrict__ err) {
  const HTaskTC Th = tasks[blockIdx.x];
  const int g0 = blockIdx.y * Th.pg;
  if (g0 >= nact) return;
  const int npg = min(Th.pg, nact - g0);
  extern __shared__ __align__(16) unsigned char smraw[];
  float* stage_base = reinterpret_cast<float*>(smraw);
  const int stage_floats = 2 * 128 * HTC_K + 2 * npmax * HTC_K;
  float* sMF = stage_base + 2 * stage_floats;   // [pg][2 sb][5 iz][2 re/im][32 r]
  __shared__ __align__(8) uint64_t full_bar[2], empty_bar[2];
  __shared__ uint32_t tslot;
  __shared__ volatile int abort_flag;
  __shared__ signed char sns[HTC_MAXB];
  __shared__ int spt[HTC_MAXPG];
  const int tid = threadIdx.x, warp = tid >> 5;
  const int nbc = Th.nbc, NP = Th.np, nj = npg * nbc;
  const int nghl = B.nghl;
  const long long ps = (long long)B.dqp * nghl;
  const int jb0 = B.st[Th.iy] + Th.b0;
  const int nc = Th.mode == 0 ? 5 : 1;
  const int nrc = (nghl + HTC_K - 1) / HTC_K;   // chunks per component
  const int nchunk = nc * nrc;
  const uint32_t ncols = NP <= 32 ? 32u : NP <= 64 ? 64u : NP <= 128 ? 128u : 256u;
  if (tid < HTC_MAXB) sns[tid] = tid < nbc ? B.ns[jb0 + tid] : (signed char)1;
  if (tid < HTC_MAXPG) spt[tid] = tid < npg ? actlist[g0 + tid] : 0;
  if (tid == 0) {
    tc::mbar_init(&full_bar[0], HTC_PROD); tc::mbar_init(&full_bar[1], HTC_PROD);
    tc::mbar_init(&empty_bar[0], 1); tc::mbar_init(&empty_bar[1], 1);
    abort_flag = 0;
  }
  if (warp == 0) tc::tmem_alloc(&tslot, ncols);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tslot;
  const float* mfbase = mf + (long long)Th.call * NMF * 2 * nghl;
  if (warp < HTC_PROD / 32) {
    // ---------------- producers ----------------
    // chunks in mesh-point-major order: the column basis functions phi_iz(b, r) of a
    // thread's two A items stay in registers for the nc components of one r range.
    // Everything that does not depend on the chunk is computed once: the hpsi row
    // (point, column), spin and shared-memory offsets of the two A items.
    float4 fz[2][5];
    int a_m[2], a_row[2], a_ore[2], a_oim[2];   // a_row < 0: no hpsi row
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      const int e = tid + it * HTC_PROD;
      const int j = e % HTC_MAXB, r4 = e / HTC_MAXB;
      const int pi = j < nj ? j / nbc : 0, b = j < nj ? j % nbc : 0;
      const int sbi = sns[b] > 0 ? 0 : 1;
      a_m[it] = (((pi * 2 + sbi) * 5) * 2) * HTC_K + 4 * r4;
      a_row[it] = j < nj ? jb0 + b : -1;
      a_ore[it] = tc::cm_off(j, 4 * r4, 128);
      a_oim[it] = tc::cm_off(64 + j, 4 * r4, 128);
    }
    int lc0 = -1, lc1 = -1;   // thread 0: last chunk copied into stage 0, stage 1
    for (int c = 0; c < nchunk; ++c) {
      const int st = c & 1;
      if (c >= 2 && !abort_flag && !tc::mbar_wait(&empty_bar[st], ((c >> 1) - 1) & 1)) abort_flag = 1;
      float* sAh = stage_base + st * stage_floats;
      float* sAl = sAh + 128 * HTC_K;
      float* sBh = sAl + 128 * HTC_K;
      const int q = c % nc, r0 = (c / nc) * HTC_K;
      bool issued = false;
      if (tid == 0 && !abort_flag) {
        // B: the row basis functions phi_q(a, r) of this chunk, pre-split (hi then lo,
        // NP x 32 each); this thread's arrival on the stage comes with the copy
        const uint32_t bbytes = (uint32_t)NP * HTC_K * 2 * 4;
        tc::mbar_expect_tx(&full_bar[st], bbytes);
        tc::bulk_g2s(sBh, hphi + Th.tphi + (long long)(q * nrc + c / nc) * 64 * NP, bbytes, &full_bar[st]);
        issued = true;
        if (st == 0) lc0 = c; else lc1 = c;
      }
      // the field tensor of this chunk (component q, mesh points r0..r0+31) of every
      // point of the group, shared by all rows; the barriers keep one chunk's copy
      // from being overwritten while another chunk's rows are generated
      asm volatile("bar.sync 1, %0;" ::"r"(HTC_PROD) : "memory");
      for (int e = tid; e < npg * 2 * 5 * 2 * 8; e += HTC_PROD) {
        const int r4 = e & 7, ri = (e >> 3) & 1, iz = (e >> 4) % 5, sbi = (e / 80) & 1, pi = e / 160;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (iz < nc) {
          const int sb = sbi == 0 ? 1 : -1;
          const int slot = Th.mode == 0 ? mfslot(q, iz, Th.sa, sb) : 100 + (Th.sa < 0 ? 2 : 0) + sbi;
          const float* mp = mfbase + (long long)spt[pi] * 2 * NMF * 2 * nghl;
          v = ld_row4(mp + ((long long)slot * 2 + ri) * nghl, r0 + 4 * r4, nghl, true);
        }
        *reinterpret_cast<float4*>(&sMF[((((pi * 2 + sbi) * 5 + iz) * 2 + ri) * HTC_K) + 4 * r4]) = v;
      }
      asm volatile("bar.sync 1, %0;" ::"r"(HTC_PROD) : "memory");
      if (!abort_flag) {
        // A: hpsi rows, Re at j, Im at 64 + j, four mesh points per item
#pragma unroll
        for (int it = 0; it < 2; ++it) {
          const int r = r0 + 4 * ((tid + it * HTC_PROD) / HTC_MAXB);
          float4 hr = make_float4(0.f, 0.f, 0.f, 0.f), hi = hr;
          if (a_row[it] >= 0) {
            if (q == 0) {
#pragma unroll
              for (int iz = 0; iz < 5; ++iz)
                if (iz < nc) fz[it][iz] = ld_row4(B.phi + iz * ps + (long long)a_row[it] * nghl, r, nghl, true);
            }
            const float* m = &sMF[a_m[it]];
#pragma unroll
            for (int iz = 0; iz < 5; ++iz)
              if (iz < nc) {
                fma4(hr, *reinterpret_cast<const float4*>(m + (iz * 2 + 0) * HTC_K), fz[it][iz]);
                fma4(hi, *reinterpret_cast<const float4*>(m + (iz * 2 + 1) * HTC_K), fz[it][iz]);
              }
          }
          st_split4(sAh + a_ore[it], sAl + a_ore[it], hr);
          st_split4(sAh + a_oim[it], sAl + a_oim[it], hi);
        }
      }
      tc::fence_async_smem();
      if (!issued) tc::mbar_arrive(&full_bar[st]);
    }
    // no copy may still be landing when the memory is reused (the last two chunks
    // are the only ones that can be in flight)
    if (tid == 0) {
      if (lc0 >= 0 && !tc::mbar_wait(&full_bar[0], (lc0 >> 1) & 1)) abort_flag = 1;
      if (lc1 >= 0 && !tc::mbar_wait(&full_bar[1], (lc1 >> 1) & 1)) abort_flag = 1;
    }
  } else if (tid == HTC_PROD) {
    // ---------------- MMA issuer (one thread of warp 8) ----------------
    const uint32_t idesc = tc::idesc_tf32(128, NP);
    const uint32_t lboA = (128 / 8) * 128, lboB = (uint32_t)(NP / 8) * 128;
    for (int c = 0; c < nchunk; ++c) {
      const int st = c & 1;
      if (!abort_flag && !tc::mbar_wait(&full_bar[st], (c >> 1) & 1)) abort_flag = 1;
      tc::fence_after();
      if (!abort_flag) {
        const float* sAh = stage_base + st * stage_floats;
        const float* sAl = sAh + 128 * HTC_K;
        const float* sBh = sAl + 128 * HTC_K;
        const float* sBl = sBh + NP * HTC_K;
#pragma unroll
        for (int ks = 0; ks < HTC_K / 8; ++ks) {
          const uint32_t oa = ks * 2 * lboA, ob = ks * 2 * lboB;
          const uint64_t ah = tc::sdesc(tc::smem_u32(sAh) + oa, lboA, 128);
          const uint64_t al = tc::sdesc(tc::smem_u32(sAl) + oa, lboA, 128);
          const uint64_t bh = tc::sdesc(tc::smem_u32(sBh) + ob, lboB, 128);
          const uint64_t bl = tc::sdesc(tc::smem_u32(sBl) + ob, lboB, 128);
          tc::mma_tf32(tmem, ah, bh, idesc, c > 0 || ks > 0);
          tc::mma_tf32(tmem, ah, bl, idesc, true);
          tc::mma_tf32(tmem, al, bh, idesc, true);
        }
      }
      tc::mma_commit(&empty_bar[st]);   // stage free (and, for the last chunk, D complete)
    }
  }
  // every MMA issued before the last commit has completed once its phase flips
  const int last = nchunk - 1;
  bool ok = tc::mbar_wait(&empty_bar[last & 1], (last >> 1) & 1);
  ok = __syncthreads_and(ok && !abort_flag);
  tc::fence_after();
  if (!ok) {
    if (tid == 0) atomicExch(err, 1);
  } else if (warp < 4) {
    // epilogue: lane m of TMEM = row m; every lane of the warp takes part in the loads
    const int m = tid, pl = m >> 6, j = m & 63;
    const bool mine = j < nj;
    const int pi = mine ? j / nbc : 0, b = mine ? j % nbc : 0;
    const int ld = B.db[Th.ix];
    float* out = hsp + ((long long)spt[pi] * 2 + pl) * 4 * nxy + (long long)Th.outq * nxy + Th.ooff +
                 (long long)(Th.b0 + b) * ld + Th.a0;
    for (int n0 = 0; n0 < NP; n0 += 8) {
      float v[8];
      tc::tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)n0, v);
      if (mine) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (n0 + i < Th.na) out[n0 + i] = 2.f * v[i];
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_free(tmem, ncols);
}

// ---------------------------------------------------------------------------
// Green's function update: vout = G o (q*H + F); layout [P][Re X|Y[|P|Q], Im ...]
// ---------------------------------------------------------------------------
// the Green's function of the points flagged in mask, once per point (omega is fixed):
// G = -1/(E1 + E2 -/+ w) on X (quadrant 0, -w) and Y (1, +w) and, in the statistical
// FAM (nq = 4), G = -1/(E1 - E2 -/+ w) on P (2) and Q (3) (pnfam_solver.f90:420-442),
// times the occupation factor 1 - f1 - f2 (X, Y) or f2 - f1 (P, Q) (:445-458), which
// the reference applies to G o H; gfn: [P][Re | Im][nq*nxy]
__global__ void k_green_prep(long long nxy, int nq, const int* __restrict__ erow, const int* __restrict__ ecol,
                             const double* __restrict__ E1, const double* __restrict__ E2,
                             const double* __restrict__ f1, const double* __restrict__ f2,
                             const double* __restrict__ wre, const double* __restrict__ wim,
                             double* __restrict__ gfn, const int* __restrict__ mask) {
  const int p = blockIdx.y;
  if (!mask[p]) return;
  const long long n2 = nq * nxy;
  const double wr = wre[p], wi = wim[p];
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n2; e += (long long)gridDim.x * blockDim.x) {
    const int q = (int)(e / nxy);
    const double sgn = (q & 1) ? 1.0 : -1.0;
    const double c2 = q < 2 ? 1.0 : -1.0;
    const int r = erow[e], k = ecol[e];
    const double dr = E1[r] + c2 * E2[k] + sgn * wr, di = sgn * wi;
    const double den = dr * dr + di * di;
    double gr = -dr / den, gi = di / den;
    if (f1) {
      const double t = q < 2 ? (-f1[r] - f2[k]) + 1.0 : (-f1[r] + f2[k]) + 0.0;
      gr *= t; gi *= t;
    }
    gfn[(long long)p * 2 * n2 + e] = gr;
    gfn[(long long)p * 2 * n2 + n2 + e] = gi;
  }
}

// vout = G o (q*H + F), G from k_green_prep (FP64 form; the mixed form: k_bro_step2)
__global__ void k_green(long long nxy, int nq, const double* __restrict__ hqp, const double* __restrict__ fqp,
                        const double* __restrict__ gfn, double quench, double* __restrict__ vout,
                        const int* __restrict__ active, const int* __restrict__ zeroh) {
  const int p = blockIdx.y;
  if (!active[p]) return;
  const long long n2 = nq * nxy;
  const bool useh = hqp && !zeroh[p];  // zeroh: H = 0 (the field of X = 0)
  const long long o = (long long)p * 2 * n2;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n2; e += (long long)gridDim.x * blockDim.x) {
    double hr = 0.0, hi = 0.0;
    if (useh) { hr = quench * hqp[o + e]; hi = quench * hqp[o + n2 + e]; }
    hr += fqp[e];
    const double gr = gfn[o + e], gi = gfn[o + n2 + e];
    vout[o + e] = gr * hr - gi * hi;
    vout[o + n2 + e] = gr * hi + gi * hr;
  }
}

// ---------------------------------------------------------------------------
// Broyden mixing on device (pnfam_broyden.f90:117-216), one independent
// history per point: itp[p] is the point's own Broyden iteration number and
// modep[p] what the step does (BRO_* below)
// ---------------------------------------------------------------------------
enum { BRO_BROYDEN = 0, BRO_LINEAR = 1, BRO_NOMIX = 2 };
struct BroState {
  int N;            // vector length (2*nq*nxy: Re and Im of the QP quadrants)
  int M;            // history size
  double alpha;
  double* vin;      // [P][N]
  double* vout;     // [P][N]
  double* df;       // [P][M][N]
  double* dv;       // [P][M][N]: u = dv + alpha*df for finished columns, raw vin in column inext
  double* part;     // [P][nchunk][NPART] block partials
  int nchunk;
  const int* itp;   // [P] Broyden iteration of each point
  const int* modep; // [P] BRO_*
};
// block partials, [P][BRO_NPART][nchunk] so that their reduction reads consecutive
// chunks: j = 0: max|vout|, 1: |df_ipos|^2, 2 + k: df_k . df_ipos, 66 + k: df_k . vout
enum { BRO_NPART = 2 + 2 * 64 };
__device__ __forceinline__ long long bro_part(int nchunk, int p, int j) { return ((long long)p * BRO_NPART + j) * nchunk; }
enum { BRO_CHUNK = 1024 };          // elements per CTA of the Broyden kernels (4 per thread)

// history slots of Broyden iteration `it` (Fortran integer division truncates
// toward zero, as C++ does): iter_used columns in use, ipos the column updated
// this step, inext the column written at the end (0-based)
__host__ __device__ __forceinline__ void bro_slots(int it, int M, int& iter_used, int& ipos, int& inext) {
  iter_used = it - 1 < M ? it - 1 : M;
  ipos = it - 1 - ((it - 2) / M) * M - 1;
  inext = it - ((it - 1) / M) * M - 1;
}

__device__ __forceinline__ double block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0) for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += sh[i];
  return s;  // valid in thread 0
}
__device__ __forceinline__ double block_max(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0) for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s = fmax(s, sh[i]);
  return s;
}

// vout -= vin; max|vout|; history column ipos: df = vout - df, dv = vin - dv, |df|^2
__global__ void __launch_bounds__(256) k_bro_diff(BroState S, const int* __restrict__ active) {
  const int p = blockIdx.y;
  if (!active[p]) return;
  __shared__ double sh[32];
  const int it = S.itp[p], mode = S.modep[p];
  int iu, ipos, inext;
  bro_slots(it, S.M, iu, ipos, inext);
  const bool upd = mode == BRO_BROYDEN && it >= 2;
  double* vo = S.vout + (long long)p * S.N;
  const double* vi = S.vin + (long long)p * S.N;
  double* df = upd ? S.df + ((long long)p * S.M + ipos) * S.N : nullptr;
  double* dv = upd ? S.dv + ((long long)p * S.M + ipos) * S.N : nullptr;
  double mx = 0.0, nn = 0.0;
  const int e0 = blockIdx.x * BRO_CHUNK, e1 = min(S.N, e0 + BRO_CHUNK);
  for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
    const double v = vo[e] - vi[e];
    vo[e] = v;
    mx = fmax(mx, fabs(v));
    if (upd) {
      const double f = v - df[e];
      df[e] = f;
      dv[e] = vi[e] - dv[e];
      nn = fma(f, f, nn);
    }
  }
  const double m = block_max(mx, sh);
  const double s = block_sum(nn, sh);
  if (threadIdx.x == 0) {
    S.part[bro_part(S.nchunk, p, 0) + blockIdx.x] = m;
    S.part[bro_part(S.nchunk, p, 1) + blockIdx.x] = s;
  }
}

// normalise column ipos by 1/|df_ipos| (and finish its u column) and form the dots
// dd[k] = df_k . df_ipos and wk[k] = df_k . vout for k < iter_used.
// A CTA covers BRO_CHUNK elements: the normalised df_ipos and vout of its chunk
// are staged in shared memory, then each warp takes whole columns (k = warp,
// warp + 8, ...), every lane streaming its share of the column with many loads
// in flight, and one shuffle reduction per column.
__global__ void __launch_bounds__(256) k_bro_dots(BroState S, const double* __restrict__ norm,
                                                  const int* __restrict__ active) {
  const int p = blockIdx.y;
  if (!active[p]) return;
  const int it = S.itp[p], mode = S.modep[p];
  if (mode != BRO_BROYDEN || it < 1) return;
  int iu, ipos, inext;
  bro_slots(it, S.M, iu, ipos, inext);
  const bool upd = it >= 2;
  __shared__ double sf[BRO_CHUNK], sv[BRO_CHUNK];
  const double* vo = S.vout + (long long)p * S.N;
  double* dfp = S.df + (long long)p * S.M * S.N;
  double* dvp = S.dv + (long long)p * S.M * S.N;
  const long long base = (long long)blockIdx.x * BRO_CHUNK;
  const int len = (int)min((long long)BRO_CHUNK, (long long)S.N - base);
  const double sc = upd ? norm[p] : 0.0;
  for (int i = threadIdx.x; i < BRO_CHUNK; i += blockDim.x) {
    double f = 0.0, v = 0.0;
    if (i < len) {
      const long long e = base + i;
      if (upd) {
        f = dfp[(long long)ipos * S.N + e] * sc;
        dfp[(long long)ipos * S.N + e] = f;
        // the finished dv column is kept as u = dv + alpha*df, the only combination
        // of the two that the update reads
        dvp[(long long)ipos * S.N + e] = fma(S.alpha, f, dvp[(long long)ipos * S.N + e] * sc);
      }
      v = vo[e];
    }
    sf[i] = f;
    sv[i] = v;
  }
  __syncthreads();
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  double* pt = S.part + bro_part(S.nchunk, p, 0) + blockIdx.x;
  for (int k = w; k < iu; k += 8) {
    double a = 0.0, b = 0.0;
    if (k == ipos && upd) {  // column ipos itself: its normalised values are in shared memory
      for (int j = l; j < len; j += 32) {
        const double f = sf[j];
        a = fma(f, f, a);
        b = fma(f, sv[j], b);
      }
    } else {
      const double* fk = dfp + (long long)k * S.N + base;
      if (len == BRO_CHUNK) {  // 16 loads of each lane in flight at a time
        for (int h = 0; h < BRO_CHUNK; h += 16 * 32) {
          double fv[16];
#pragma unroll
          for (int u = 0; u < 16; ++u) fv[u] = __ldcs(fk + h + u * 32 + l);
#pragma unroll
          for (int u = 0; u < 16; ++u) {
            a = fma(fv[u], sf[h + u * 32 + l], a);
            b = fma(fv[u], sv[h + u * 32 + l], b);
          }
        }
      } else {
        for (int j = l; j < len; j += 32) {
          const double f = fk[j];
          a = fma(f, sf[j], a);
          b = fma(f, sv[j], b);
        }
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (l == 0) { pt[(long long)(2 + k) * S.nchunk] = a; pt[(long long)(2 + 64 + k) * S.nchunk] = b; }
  }
}

// one CTA (256 threads) per point: reduce partials; stage 0: si and 1/|df_ipos|;
// stage 1: maintain beta (M x M) and solve beta*gamma = work.  beta is the Gram
// matrix of the unit vectors df_k plus w0^2 on the diagonal, symmetric positive
// definite (the reference factorises it with DSYTRF/DSYTRI, pnfam_broyden.f90:190-206):
// here L D L^T without pivoting, one barrier per column, then two triangular solves
// by one warp
// cs (mixed form, BroState2): the dots are those of unnormalised columns and are made
// here; stage 2 is both stages in one launch
__global__ void __launch_bounds__(256) k_bro_solve(BroState S, int stage, double w0, double* __restrict__ si,
                                                   double* __restrict__ norm, double* __restrict__ beta,
                                                   double* __restrict__ gamma, const int* __restrict__ active,
                                                   double* __restrict__ cs = nullptr) {
  const int p = blockIdx.x;
  if (!active[p]) return;
  const double* pt = S.part + bro_part(S.nchunk, p, 0);
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  __shared__ double red[8][2];
  __shared__ double scale[2];   // of the columns and the residual (k_bro_step2), of the update
  const int it = S.itp[p], mode = S.modep[p];
  int n, ipos, inext;
  bro_slots(it, S.M, n, ipos, inext);
  if (stage != 1) {
    double m = 0.0, s = 0.0;
    for (int c = tid; c < S.nchunk; c += blockDim.x) { m = fmax(m, pt[c]); s += pt[S.nchunk + c]; }
    for (int o = 16; o > 0; o >>= 1) {
      m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
      s += __shfl_xor_sync(0xffffffffu, s, o);
    }
    if (l == 0) { red[w][0] = m; red[w][1] = s; }
    __syncthreads();
    if (tid == 0) {
      double mm = 0.0, ss = 0.0;
      for (int i = 0; i < 8; ++i) { mm = fmax(mm, red[i][0]); ss += red[i][1]; }
      norm[p] = ss > 0.0 ? 1.0 / sqrt(ss) : 0.0;
      if (cs && mode == BRO_BROYDEN && it >= 2) {
        scale[0] = scalbn(1.0, -pair_scale(si[p]));
        scale[1] = scalbn(1.0, pair_scale(mm));
        cs[(long long)p * S.M + ipos] = norm[p] * scale[0];
      }
      si[p] = mm;
    }
    if (stage == 0) return;
    __syncthreads();
  }
  if (mode != BRO_BROYDEN || it < 1) return;
  __shared__ double A[64][65];
  __shared__ double x[64];
  __shared__ double dinv[2];   // 1/D of the current and the next column
  const int M = S.M;
  double* bp = beta + (long long)p * M * M;
  for (int k = w; k < n; k += 8) {   // one warp per k: sum the chunk partials
    double dd = 0.0, wk = 0.0;
    const double* pd = pt + (long long)(2 + k) * S.nchunk;
    const double* pw = pt + (long long)(2 + 64 + k) * S.nchunk;
#pragma unroll 4
    for (int c = l; c < S.nchunk; c += 32) { dd += pd[c]; wk += pw[c]; }
    for (int o = 16; o > 0; o >>= 1) {
      dd += __shfl_xor_sync(0xffffffffu, dd, o);
      wk += __shfl_xor_sync(0xffffffffu, wk, o);
    }
    if (l == 0) {
      if (cs) {
        const double ck = cs[(long long)p * M + k];
        dd *= ck * cs[(long long)p * M + ipos];
        wk *= ck * scale[0];
      }
      if (k != ipos) { bp[k * M + ipos] = dd; bp[ipos * M + k] = dd; }
      x[k] = wk;
    }
  }
  __syncthreads();
  for (int k = tid; k < n; k += blockDim.x) bp[k * M + k] = w0 * w0 + 1.0;
  __syncthreads();
  for (int e = tid; e < n * n; e += blockDim.x) A[e / n][e % n] = bp[(e / n) * M + (e % n)];
  if (tid == 0 && n > 0) dinv[0] = 1.0 / A[0][0];
  __syncthreads();
  // L D L^T in place: D on the diagonal, L[r][c] (r > c) in the upper triangle A[c][r]
  for (int c = 0; c < n; ++c) {
    const double di = dinv[c & 1];
    for (int r = c + 1 + w; r < n; r += 8) {
      const double lr = A[r][c] * di;
      for (int j = c + 1 + l; j <= r; j += 32) A[r][j] -= lr * A[j][c];
      if (l == 0) A[c][r] = lr;
      // the next pivot is final as soon as its own update is done (warp 0, lane 0)
      if (r == c + 1 && l == 0) dinv[(c + 1) & 1] = 1.0 / A[r][r];
    }
    __syncthreads();
  }
  // L y = work, y /= D, L^T gamma = y (columns in turn, one warp)
  if (tid < 32) {
    for (int c = 0; c < n; ++c) {
      const double yc = x[c];
      for (int r = c + 1 + tid; r < n; r += 32) x[r] -= A[c][r] * yc;
      __syncwarp();
    }
    for (int r = tid; r < n; r += 32) x[r] /= A[r][r];
    __syncwarp();
    for (int c = n - 1; c >= 0; --c) {
      const double gc = x[c];
      for (int r = tid; r < c; r += 32) x[r] -= A[r][c] * gc;
      __syncwarp();
    }
    for (int k = tid; k < n; k += 32) gamma[(long long)p * 64 + k] = cs ? x[k] * cs[(long long)p * M + k] * scale[1] : x[k];
  }
}

// BRO_BROYDEN: curv = alpha*vout - sum_i gamma_i u_i  (u_i = dv_i + alpha df_i);
//              df[inext] = vout; dv[inext] = vin; vin += curv
// BRO_LINEAR:  vin += alpha*vout;  BRO_NOMIX: vin += vout
__global__ void __launch_bounds__(256) k_bro_update(BroState S, const double* __restrict__ gamma,
                                                    const int* __restrict__ active) {
  const int p = blockIdx.y;
  if (!active[p]) return;
  const int it = S.itp[p], mode = S.modep[p];
  int iu, ipos, inext;
  bro_slots(it, S.M, iu, ipos, inext);
  if (mode != BRO_BROYDEN) iu = 0;
  double* vi = S.vin + (long long)p * S.N;
  const double* vo = S.vout + (long long)p * S.N;
  __shared__ double g[64];
  if (mode == BRO_BROYDEN && (int)threadIdx.x < iu) g[threadIdx.x] = gamma[(long long)p * 64 + threadIdx.x];
  __syncthreads();
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < S.N; e += (long long)gridDim.x * blockDim.x) {
    const double v = vo[e];
    if (mode == BRO_NOMIX) { vi[e] += v; continue; }
    if (mode == BRO_LINEAR) { vi[e] += S.alpha * v; continue; }
    double c = S.alpha * v;
    const double* up = S.dv + (long long)p * S.M * S.N;
    for (int k = 0; k < iu; ++k) c -= g[k] * up[(long long)k * S.N + e];
    const double old = vi[e];
    S.df[((long long)p * S.M + inext) * S.N + e] = v;
    S.dv[((long long)p * S.M + inext) * S.N + e] = old;
    vi[e] = old + c;
  }
}

// ---------------------------------------------------------------------------
// Broyden of the mixed form.  The history columns df_k and u_k are kept as pairs
// of floats (hi + lo, about 48 significant bits) and every product with them is
// formed in pair arithmetic on the FP32 cores, which GB300 runs at dozens of times
// its FP64 rate; the residuals of this and the previous step and the vectors themselves
// stay FP64, so the secant pairs are formed before any rounding, and the small solve
// is FP64 (k_bro_solve).  Same steps as k_bro_diff / k_bro_dots /
// k_bro_update.
// ---------------------------------------------------------------------------
struct BroState2 {
  int N;              // vector length (2*nq*nxy, a multiple of 4)
  int M;              // history size
  double alpha;
  double* vin;        // [P][N]
  double* v0;         // [P][N] this step's residual vout - vin and the previous step's by
  double* v1;         // [P][N] turns: of iteration it in v0 (even) or v1 (odd)
  double* lastv;      // [P][N] vin of the previous step
  float2* df;         // [P][M][N] columns 2^s (res - previous res), s of k_bro_step2
  float2* u;          // [P][M][N] columns 2^s (vin - lastv + alpha (res - previous res))
  double* cs;         // [P][M] 2^-s / |res - previous res| of a column: what normalises it
  double* part;       // [P][BRO_NPART][nchunk]
  int nchunk;
  const int* itp;
  const int* modep;
  __device__ double* res(int it) const { return it & 1 ? v1 : v0; }
  __device__ const double* prev(int it) const { return it & 1 ? v0 : v1; }
};

// The Green's function update (as k_green) and the start of the Broyden step of a mixed-
// form slot: vout = G o (q*H + F) or, on an increment evaluation, G o (q*H32) + g(X_a);
// the residual vout - vin and its maximum; its difference f to the previous step's, |f|^2,
// the new columns df and u, and the dots df_k . df_ipos and df_k . res with every column.
// An anchor evaluation (anch) leaves X_a = vin and g(X_a) = vout.
// grid (nchunk, P): a CTA takes BRO_CHUNK / 2 complex elements, two per thread, keeps f
// and the residual as pairs in shared memory and then gives each warp a column in turn.
// The columns are stored before their norm is known, scaled by the power of two that
// brings the previous residual's maximum (si) to 1; cs carries the norm.
// Bound by FP64 (8 operations per element) in the first iterations and by the reads of the
// columns later.  As separate passes with FP64 conversions, sums and normalisation (Green's
// function, copies, differences, dots) these took 1.2, 2.0 and 3.6 ms for 64 points at N_sh =
// 20 with 3 columns; in this form 3.2 ms.  With 35 to 55 columns (24 points, N_sh = 16) it reads
// at 4.5-5.4 TB/s.  k_bro_update2 there 1.5 -> 1.16 ms and 6.2 TB/s, k_to_f32 0.78 -> 0.53 ms.
__global__ void __launch_bounds__(256, 4) k_bro_step2(BroState2 S, const double* __restrict__ hqp,
                                                      const float* __restrict__ hqp32, const double* __restrict__ fqp,
                                                      const double* __restrict__ gfn, double quench,
                                                      const int* __restrict__ active, const int* __restrict__ corr,
                                                      const int* __restrict__ anch, const int* __restrict__ zeroh,
                                                      const double* __restrict__ si, double* __restrict__ xsave,
                                                      double* __restrict__ radd) {
  const int p = blockIdx.y;
  if (!active[p]) return;
  constexpr int HC = BRO_CHUNK / 2;
  __shared__ float4 sf[2][HC / 2], sv[2][HC / 2];   // [Re, Im][pairs of elements]
  __shared__ double sn[256];
  __shared__ unsigned long long sm[8];
  const int it = S.itp[p], mode = S.modep[p], n2 = S.N / 2;
  int iu, ipos, inext;
  bro_slots(it, S.M, iu, ipos, inext);
  const bool upd = mode == BRO_BROYDEN && it >= 2;
  const bool cstep = corr[p] != 0, useh = hqp && !zeroh[p], an = anch[p] != 0;
  const long long o = (long long)p * S.N;
  const int t = threadIdx.x, w = t >> 5, l = t & 31;
  const int e0 = blockIdx.x * HC, e = e0 + 2 * t;   // n2 is even: both elements or none
  const int s = upd ? pair_scale(si[p]) : 0;
  float2* dfp = S.df + (long long)p * S.M * S.N;
  unsigned long long mx = 0;
  double nn = 0.0;
  float4 f4[2], v4[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) f4[c] = v4[c] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (e < n2) {
    auto ld2 = [](const double* q) { return *reinterpret_cast<const double2*>(q); };
    auto st2 = [](double* q, double a, double b) { *reinterpret_cast<double2*>(q) = make_double2(a, b); };
    double h[2][2] = {{0.0, 0.0}, {0.0, 0.0}};   // [Re, Im][element]
    if (useh) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (cstep) {
          const float2 q = *reinterpret_cast<const float2*>(hqp32 + o + (c ? n2 : 0) + e);
          h[c][0] = f64_of(q.x);
          h[c][1] = f64_of(q.y);
        } else {
          const double2 q = ld2(hqp + o + (c ? n2 : 0) + e);
          h[c][0] = q.x;
          h[c][1] = q.y;
        }
        if (quench != 1.0) { h[c][0] *= quench; h[c][1] *= quench; }
      }
    }
    if (!cstep) {
      const double2 q = ld2(fqp + e);
      h[0][0] += q.x;
      h[0][1] += q.y;
    }
    const double2 gr = ld2(gfn + o + e), gi = ld2(gfn + o + n2 + e);
    double v[2][2];
    v[0][0] = gr.x * h[0][0] - gi.x * h[1][0];
    v[1][0] = gr.x * h[1][0] + gi.x * h[0][0];
    v[0][1] = gr.y * h[0][1] - gi.y * h[1][1];
    v[1][1] = gr.y * h[1][1] + gi.y * h[0][1];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const long long q = o + (c ? n2 : 0) + e;
      if (cstep) {
        const double2 ra = ld2(radd + q);
        v[c][0] += ra.x;
        v[c][1] += ra.y;
      }
      const double2 x = ld2(S.vin + q);
      if (an) {
        st2(xsave + q, x.x, x.y);
        st2(radd + q, v[c][0], v[c][1]);
      }
      const double r0 = v[c][0] - x.x, r1 = v[c][1] - x.y;
      st2(S.res(it) + q, r0, r1);
      mx = abs_max(abs_max(mx, r0), r1);
      if (upd) {
        const double2 pr = ld2(S.prev(it) + q), lv = ld2(S.lastv + q);
        const double d0 = r0 - pr.x, d1 = r1 - pr.y;
        nn = fma(d0, d0, nn);
        nn = fma(d1, d1, nn);
        const float2 a = pair_split(d0, s), b = pair_split(d1, s);
        f4[c] = make_float4(a.x, a.y, b.x, b.y);
        const long long cq = (long long)ipos * S.N + (c ? n2 : 0) + e;
        *reinterpret_cast<float4*>(dfp + cq) = f4[c];
        const float2 ua = pair_split(fma(S.alpha, d0, x.x - lv.x), s), ub = pair_split(fma(S.alpha, d1, x.y - lv.y), s);
        *reinterpret_cast<float4*>(S.u + (long long)p * S.M * S.N + cq) = make_float4(ua.x, ua.y, ub.x, ub.y);
        const float2 va = pair_split(r0, s), vb = pair_split(r1, s);
        v4[c] = make_float4(va.x, va.y, vb.x, vb.y);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) { sf[c][t] = f4[c]; sv[c][t] = v4[c]; }
  sn[t] = nn;
  mx = warp_abs_max(mx);
  if (l == 0) sm[w] = mx;
  __syncthreads();
  double* pt = S.part + bro_part(S.nchunk, p, 0) + blockIdx.x;
  if (w == 7) {   // few FP64 sums: one warp adds the threads' values
    double q = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) q += sn[32 * i + l];
    for (int i = 16; i > 0; i >>= 1) q += __shfl_xor_sync(0xffffffffu, q, i);
    const unsigned long long m = warp_abs_max(l < 8 ? sm[l] : 0ULL);
    if (l == 0) { pt[0] = __longlong_as_double((long long)m); pt[S.nchunk] = q; }
  }
  if (!upd) return;
  const int half = max(0, min(HC, n2 - e0)) / 2;   // pairs of elements of this CTA, each of Re and Im
  for (int k = w; k < iu; k += 8) {
    float2 a = make_float2(0.f, 0.f), b = a;
    auto add = [&](float4 x, float4 f, float4 v) {
      pair_fma(a, make_float2(x.x, x.y), make_float2(f.x, f.y));
      pair_fma(b, make_float2(x.x, x.y), make_float2(v.x, v.y));
      pair_fma(a, make_float2(x.z, x.w), make_float2(f.z, f.w));
      pair_fma(b, make_float2(x.z, x.w), make_float2(v.z, v.w));
    };
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (k == ipos) {   // the new column itself
        for (int j = l; j < half; j += 32) add(sf[c][j], sf[c][j], sv[c][j]);
        continue;
      }
      const float4* fk = reinterpret_cast<const float4*>(dfp + (long long)k * S.N + (c ? n2 : 0) + e0);
      if (half == HC / 2) {
        float4 x[HC / 64];
#pragma unroll
        for (int i = 0; i < HC / 64; ++i) x[i] = __ldcs(fk + l + 32 * i);
#pragma unroll
        for (int i = 0; i < HC / 64; ++i) add(x[i], sf[c][l + 32 * i], sv[c][l + 32 * i]);
      } else {
        for (int j = l; j < half; j += 32) add(__ldcs(fk + j), sf[c][j], sv[c][j]);
      }
    }
    const double sum = pair_warp_sums(a, b, l);
    if ((l & 15) == 0) pt[(long long)(2 + (l ? 64 : 0) + k) * S.nchunk] = sum;
  }
}

// BRO_BROYDEN: vin += alpha*res - sum_k gamma_k u_k; lastv = vin.  gamma holds the
// columns' factors and the scale of the residual (k_bro_solve)
// BRO_LINEAR:  vin += alpha*res;  BRO_NOMIX: vin += res
__global__ void __launch_bounds__(256) k_bro_update2(BroState2 S, const double* __restrict__ gamma,
                                                     const double* __restrict__ si, const int* __restrict__ active) {
  const int p = blockIdx.y;
  if (!active[p]) return;
  const int it = S.itp[p], mode = S.modep[p];
  int iu, ipos, inext;
  bro_slots(it, S.M, iu, ipos, inext);
  if (mode != BRO_BROYDEN) iu = 0;
  const long long o = (long long)p * S.N;
  __shared__ float2 g[64];
  if (mode == BRO_BROYDEN && (int)threadIdx.x < iu) g[threadIdx.x] = pair_split(gamma[(long long)p * 64 + threadIdx.x]);
  __syncthreads();
  const int s = pair_scale(si[p]);
  const int e = 2 * (blockIdx.x * 256 + threadIdx.x);   // N is even
  if (e >= S.N) return;
  const float2* up = S.u + (long long)p * S.M * S.N + e;
  const double2 v = *reinterpret_cast<const double2*>(S.res(it) + o + e);
  double2* vin = reinterpret_cast<double2*>(S.vin + o + e);
  const double2 old = *vin;
  if (mode == BRO_NOMIX) { *vin = make_double2(old.x + v.x, old.y + v.y); return; }
  if (mode == BRO_LINEAR) { *vin = make_double2(old.x + S.alpha * v.x, old.y + S.alpha * v.y); return; }
  float2 a = make_float2(0.f, 0.f), b = a;
#pragma unroll 8
  for (int k = 0; k < iu; ++k) {
    const float4 x = __ldcs(reinterpret_cast<const float4*>(up + (long long)k * S.N));
    pair_fma(a, make_float2(x.x, x.y), g[k]);
    pair_fma(b, make_float2(x.z, x.w), g[k]);
  }
  *reinterpret_cast<double2*>(S.lastv + o + e) = old;
  *vin = make_double2(old.x + (S.alpha * v.x - pair_value(a, -s)), old.y + (S.alpha * v.y - pair_value(b, -s)));
}

// dst = 0 for the points with mask[p], [P][n] layout
__global__ void k_zero(double* __restrict__ dst, long long n, const int* __restrict__ mask) {
  const int p = blockIdx.y;
  if (!mask[p]) return;
  double* d = dst + (long long)p * n;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
    d[e] = 0.0;
}

// out[k][e] = in[k][idx[e]]; grid (ceil(n / 256), rows)
__global__ void __launch_bounds__(256) k_gather(const double* __restrict__ in, long long ld, const int* __restrict__ idx,
                                                long long n, double* __restrict__ out) {
  const long long e = blockIdx.x * 256LL + threadIdx.x;
  if (e < n) out[blockIdx.y * n + e] = in[blockIdx.y * ld + idx[e]];
}

// S_k = -1/pi * (F_k . Re, F_k . Im) for the operator (k=0) and cross terms
// fops: [nops][nq*nxy]; part: [P][nchunk][2*nops].  grid (nchunk, P)
// Bound by the chain of loads and sums of a CTA: a chunk is two elements per thread (up to
// 64 chunks; with one chunk per 4096 elements 16 us for one point at N_sh = 6 and 73 us for
// five with cross terms in the statistical FAM, now 5.6 and 10.5), and the operators meet at
// one barrier.
__global__ void __launch_bounds__(256) k_contract(long long nxy, int nq, int nops, const double* __restrict__ fops,
                                                  const double* __restrict__ vin, int nchunk,
                                                  double* __restrict__ part, const int* __restrict__ active) {
  const int p = blockIdx.y;
  if (!active[p]) return;
  constexpr int KB = 8;
  __shared__ double sh[8][2 * KB];
  const int t = threadIdx.x, w = t >> 5;
  const long long n2 = nq * nxy;
  const double* v = vin + (long long)p * 2 * n2;
  const long long chunk = (n2 + nchunk - 1) / nchunk;
  const long long e0 = blockIdx.x * chunk, e1 = min(n2, e0 + chunk);
  for (int k0 = 0; k0 < nops; k0 += KB) {
    const int nk = min(KB, nops - k0);
    if (k0) __syncthreads();
    for (int k = 0; k < nk; ++k) {
      double a = 0.0, b = 0.0;
#pragma unroll 2
      for (long long e = e0 + t; e < e1; e += 256) {
        const double f = fops[(k0 + k) * n2 + e];
        a = fma(f, v[e], a);
        b = fma(f, v[n2 + e], b);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
      }
      if ((t & 31) == 0) { sh[w][2 * k] = a; sh[w][2 * k + 1] = b; }
    }
    __syncthreads();
    if (t < 2 * nk) {
      double s = 0.0;
#pragma unroll
      for (int i = 0; i < 8; ++i) s += sh[i][t];
      part[((long long)p * nchunk + blockIdx.x) * 2 * nops + 2 * k0 + t] = s;
    }
  }
}

}  // namespace pnfam

namespace pnfam {
// per-point precision conversions: out[p*n + e] = in[p*n + e] for points with act[p]
// (act == nullptr: all points)
// out = (float)(in - sub), sub optional; with dmax, dmax[p] = max(dmax[p], max|in - sub|)
// (dmax as the bit pattern of a non-negative double, which orders like the integer)
__global__ void __launch_bounds__(256) k_to_f32(const double* __restrict__ in, float* __restrict__ out, long long n,
                                                int P, long long ld, const int* __restrict__ act,
                                                const double* __restrict__ sub = nullptr,
                                                unsigned long long* __restrict__ dmax = nullptr) {
  const int p = blockIdx.y;
  if (act && !act[p]) return;
  unsigned long long m = 0;
#pragma unroll 4
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const double v = sub ? in[p * ld + e] - sub[p * ld + e] : in[p * ld + e];
    m = abs_max(m, v);
    out[p * ld + e] = f32_of(v);
  }
  if (dmax) {   // one atomic per block
    __shared__ unsigned long long wm[8];
    m = warp_abs_max(m);
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
      m = warp_abs_max(threadIdx.x < 8 ? wm[threadIdx.x] : 0ULL);
      if (threadIdx.x == 0) atomicMax(dmax + p, m);
    }
  }
}
__global__ void k_to_f64(const float* __restrict__ in, double* __restrict__ out, long long n, long long ld,
                         const int* __restrict__ act) {
  const int p = blockIdx.y;
  if (act && !act[p]) return;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
    out[p * ld + e] = (double)in[p * ld + e];
}

// the four densities of calc_hamiltonian_z ([4][nxy] complex: rho_pn, kappa+, rho_np, kappa-)
// into the planes and quadrants of point 0 ([2 re/im][4]: rho_pn, kappa+, kappa-, rho_np), and
// its slot flags; k_merge_z: the fields back.  grid (ceil(nxy/256), 4)
template <class T>
__global__ void __launch_bounds__(256) k_split_z(long long nxy, const double2* __restrict__ z, T* __restrict__ rsp,
                                                 int* __restrict__ active, int* __restrict__ actlist) {
  const int k = blockIdx.y, q = k < 2 ? k : 5 - k;
  const long long i = blockIdx.x * 256LL + threadIdx.x;
  if (k == 0 && i == 0) {
    active[0] = 1;
    if (actlist) actlist[0] = 0;
  }
  if (i >= nxy) return;
  const double2 v = z[k * nxy + i];
  rsp[q * nxy + i] = (T)v.x;
  rsp[(4 + q) * nxy + i] = (T)v.y;
}
template <class T>
__global__ void __launch_bounds__(256) k_merge_z(long long nxy, const T* __restrict__ hsp, double2* __restrict__ z) {
  const int k = blockIdx.y, q = k < 2 ? k : 5 - k;
  const long long i = blockIdx.x * 256LL + threadIdx.x;
  if (i < nxy) z[k * nxy + i] = make_double2((double)hsp[q * nxy + i], (double)hsp[(4 + q) * nxy + i]);
}
}  // namespace pnfam
