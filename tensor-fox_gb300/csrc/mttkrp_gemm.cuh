// MTTKRPs T_(G) KR as GEMMs: what the FP32 and FP64 kernels share.
//
// The rows are a group of modes G = [g0, g1): one mode, or the first or the last
// modes merged.  The other modes are split into an inner group F, contiguous in
// memory beside the rows, whose Khatri-Rao block KR_F (dF x R) is formed once in
// global memory (L2-resident), and the outer rest O:
//   M[d, r] = sum_o KR_O[o, r] (sum_f T[d, o, f] KR_F[f, r]).
// So the inner loop is a plain GEMM whose operands both arrive by cp.async, and
// every dF steps, in FP32 at the latest after a chain's length, the sums are
// scaled by KR_O's row and folded into a second set (none in FP64 when F holds
// every other mode; FP32 then adds chunk by chunk).  Forming Khatri-Rao rows in
// the loop instead cost as many instructions as the FMAs.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "tfx_common.cuh"

namespace tfx {

struct CpDims {
  int L, R;
  int d[TFX_MAX_ORDER];
  int off[TFX_MAX_ORDER];
};

namespace mg {

constexpr int BK = 32;  // contraction steps a chunk

// What the GEMM walks: nO outer positions of dF inner steps each.
struct Walk {
  long long D;               // rows
  int dF, nc;                // inner steps; chunks of BK an outer position
  long long nO, Q1, sP, sQ;  // outer position o starts at (o / Q1) * sP + (o % Q1) * sQ
  long long sD;              // row stride (1 for the last modes)
  int ldp, vec;              // columns of a result row, 16-byte copies
};

struct Plan {
  Walk w;
  int TN, WM, nblk, ks, f0, f1, g0, g1;
  long long tilesM;
  bool last, fold;
  long long rowsF;
  size_t krF_bytes, krO_bytes, part_bytes;
  size_t total() const { return krF_bytes + krO_bytes + part_bytes; }
};

// The launch for the rows [g0, g1) of element size es.
// Columns: blocks of at most 64, all as narrow as a multiple of 8 (FP32: lanes
// hold column pairs) or 4 (FP64) allows: R = 50 takes 56, R = 100 2 x 56.
// Rows: FP32 128, 64 or 32 a CTA, the largest whose padding stays within 1/8
// of the least; FP64 32, its warps past the last row idle.
// F: every other mode if they lie together and the block stays within 8 MB;
// else the one beside the rows, and those next to it while the chunks' padding
// is above 1/8 and the block within 4096 rows.  Where that still pads every
// chunk to four times its steps or more, every other mode if they lie together
// and the block stays within 64 MB (10 x 200000 x 3 at R = 8, the first mode:
// chunks of 3 steps took 339 us in FP32 and 458 in FP64; so 58 and 183).
// Splits: one wave of the resident CTAs, in FP32 at least 4 chunks each.
inline Plan plan(int es, const CpDims& sh, int g0, int g1, int sms) {
  Plan p;
  const int L = sh.L, R = sh.R;
  const bool f32 = es == 4;
  p.g0 = g0;
  p.g1 = g1;
  p.nblk = (R + 63) / 64;
  const int per = (R + p.nblk - 1) / p.nblk;
  p.TN = f32 ? 2 * ((per + 7) / 8) : (per + 3) / 4;
  const int BN = 4 * p.TN;
  p.w.ldp = p.nblk * BN;
  long long P = 1, D = 1, Q = 1;
  for (int m = 0; m < g0; ++m) P *= sh.d[m];
  for (int m = g0; m < g1; ++m) D *= sh.d[m];
  for (int m = g1; m < L; ++m) Q *= sh.d[m];
  p.w.D = D;
  p.last = Q == 1;
  const int lo = p.last ? 0 : g1, hi = p.last ? g0 : L;  // the modes F may take
  const long long K = p.last ? P : Q;
  const bool together = p.last || P == 1;
  long long dF = K;
  p.f0 = lo;
  if (!together || K * p.w.ldp * es > (8LL << 20)) {
    p.f0 = hi - 1;
    dF = sh.d[hi - 1];
    while (p.f0 > lo && ((dF + BK - 1) / BK * BK - dF) * 8 > dF && dF * sh.d[p.f0 - 1] <= 4096) dF *= sh.d[--p.f0];
    if (together && (dF + BK - 1) / BK * BK >= 4 * dF && K * p.w.ldp * es <= (64LL << 20)) {
      p.f0 = lo;
      dF = K;
    }
  }
  p.f1 = hi;
  p.w.dF = (int)dF;
  p.w.nc = (int)((dF + BK - 1) / BK);
  p.rowsF = (long long)p.w.nc * BK;
  p.w.nO = P * Q / dF;
  // some mode is outside, if only of size 1: its factor's row scales all the same
  p.fold = L - (g1 - g0) - (p.f1 - p.f0) > 0;
  p.w.Q1 = p.last ? 1 : Q / dF;
  p.w.sP = p.last ? dF * D : D * Q;
  p.w.sQ = dF;
  p.w.sD = Q;
  p.w.vec = 0;
  p.WM = 1;
  if (f32) {
    const long long least = (D + 31) / 32 * 32;
    for (int wm = 2; wm <= 4; wm *= 2)
      if ((D + 32 * wm - 1) / (32 * wm) * (32 * wm) * 8 <= least * 9) p.WM = wm;
  }
  p.tilesM = (D + 32 * p.WM - 1) / (32 * p.WM);
  const long long nch = p.w.nO * p.w.nc, slots = (long long)sms * (f32 ? (p.TN > 8 ? 2 : 3) : (p.TN > 8 ? 4 : 6));
  long long ks = std::max<long long>(1, slots / (p.tilesM * p.nblk));
  ks = std::max<long long>(1, std::min(ks, f32 ? nch / 4 : nch));
  p.ks = (int)std::min<long long>(ks, 32768);
  p.krF_bytes = (size_t)((p.rowsF * p.w.ldp * es + 255) & ~255LL);
  p.krO_bytes = (size_t)((p.w.nO * p.w.ldp * es + 255) & ~255LL);
  p.part_bytes = ((size_t)p.ks * D * p.w.ldp * es + 255) & ~(size_t)255;
  return p;
}

// part[split][D][ldp]; krF[block][rowsF][BN], krO[nO][ldp]
cudaError_t gemm_f32(const Plan& p, const float* T, const float* krF, const float* krO, float* part, cudaStream_t st);
cudaError_t gemm_f64(const Plan& p, const double* T, const double* krF, const double* krO, double* part,
                     cudaStream_t st);

// Where a product goes: element (d, r) at p[d * sd + r * sr], r < R; sd = 0: the
// padded rows [D][ldp] of a group that is contracted further.
template <class T>
struct Out {
  T* p;
  long long sd, sr;
};

// The sum over the ks partials part[.][D][ldp], compensated in FP32: 32 outputs
// a CTA, the partials dealt to SG groups of threads whose sums are added in a
// fixed order.
constexpr int SG = 16;

template <class T>
__device__ __forceinline__ void put(const Out<T>& out, long long e, int ldp, int R, T v) {
  if (out.sd == 0) {
    out.p[e] = v;
    return;
  }
  const long long d = e / ldp;
  const int r = (int)(e - d * ldp);
  if (r < R) out.p[d * out.sd + r * out.sr] = v;
}

template <class T>
__global__ void __launch_bounds__(32 * SG) k_sum(const T* __restrict__ part, long long D, int R, int ldp, int ks,
                                                 Out<T> out) {
  __shared__ T hi[SG][32], lo[SG][32];
  const long long n = D * ldp;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const long long e = (long long)blockIdx.x * 32 + x;
  Acc<T> s;
  if (e < n) {
#pragma unroll 8
    for (int k = y; k < ks; k += SG) s.add(__ldcs(part + (size_t)k * n + e));
  }
  hi[y][x] = s.hi_or_v();
  lo[y][x] = s.lo_or_0();
  __syncthreads();
  if (y == 0 && e < n) {
    Acc<T> t;
#pragma unroll
    for (int j = 0; j < SG; ++j) {
      t.add(hi[j][x]);
      if (sizeof(T) == 4) t.add(lo[j][x]);
    }
    put(out, e, ldp, R, (T)t.value());
  }
}

// The same for few partials: one output a thread.
template <class T>
__global__ void __launch_bounds__(256) k_sum_few(const T* __restrict__ part, long long D, int R, int ldp, int ks,
                                                 Out<T> out) {
  const long long n = D * ldp, e = (long long)blockIdx.x * 256 + threadIdx.x;
  if (e >= n) return;
  Acc<T> s;
#pragma unroll 4
  for (int k = 0; k < ks; ++k) s.add(__ldcs(part + (size_t)k * n + e));
  put(out, e, ldp, R, (T)s.value());
}

// KR_F as [column block][nF rows padded to chunks][BN] (zeros in the padding)
// and KR_O as [nO][ldp], from the flat column-major factors: modes [f0, f1)
// are F, the others but [g0, g1) are O, both with the last mode fastest.  I:
// 32-bit indices where the element count fits (64-bit divisions took 3x the
// time).
template <class T, class I>
__global__ void __launch_bounds__(256) k_kr(const T* __restrict__ W, const __grid_constant__ CpDims sh, int g0, int g1,
                                            int f0, int f1, I dF, I rowsF, I nO, int BN, int ldp, T* __restrict__ krF,
                                            T* __restrict__ krO) {
  const I e = (I)blockIdx.x * blockDim.x + threadIdx.x;
  const I nF = rowsF * (I)ldp;
  if (e >= nF + nO * (I)ldp) return;
  const bool isF = e < nF;
  const I w = isF ? e : e - nF;
  const I row = w / (I)ldp;
  const int r = (int)(w - row * (I)ldp);
  T v = T(0);
  if (r < sh.R && (!isF || row < dF)) {
    v = T(1);
    I rem = row;
    for (int m = isF ? f1 - 1 : sh.L - 1; m >= (isF ? f0 : 0); --m) {
      if (!isF && ((m >= g0 && m < g1) || (m >= f0 && m < f1))) continue;
      const I q = rem / (I)sh.d[m];
      v *= W[sh.off[m] + (long long)r * sh.d[m] + (long long)(rem - q * (I)sh.d[m])];
      rem = q;
    }
  }
  if (isF) krF[((size_t)(r / BN) * rowsF + row) * BN + r % BN] = v;
  else krO[(size_t)row * ldp + r] = v;
}

inline cudaError_t gemm(const Plan& p, const float* T, const float* krF, const float* krO, float* part,
                        cudaStream_t st) {
  return gemm_f32(p, T, krF, krO, part, st);
}
inline cudaError_t gemm(const Plan& p, const double* T, const double* krF, const double* krO, double* part,
                        cudaStream_t st) {
  return gemm_f64(p, T, krF, krO, part, st);
}

// One product.  scratch: 16-byte aligned, p.total() bytes.  *launches counts the
// kernels.
template <class T>
inline cudaError_t run(Plan p, const T* X, const T* W, const CpDims& sh, Out<T> out, void* scratch,
                       cudaStream_t st, int* launches) {
  constexpr int PV = 16 / sizeof(T);  // values a 16-byte copy
  const long long ext = p.last ? p.w.D : p.w.dF;
  p.w.vec = ((uintptr_t)X & 15) == 0 && ext % PV == 0 && (p.last || p.w.sD % PV == 0);
  T* krF = (T*)scratch;
  T* krO = (T*)((char*)scratch + p.krF_bytes);
  T* part = (T*)((char*)scratch + p.krF_bytes + p.krO_bytes);
  const int BN = 4 * p.TN;
  const long long nkr = (p.rowsF + p.w.nO) * p.w.ldp;
  const unsigned kb = (unsigned)((nkr + 255) / 256);
  if (nkr < (1LL << 31))
    k_kr<T, unsigned><<<kb, 256, 0, st>>>(W, sh, p.g0, p.g1, p.f0, p.f1, (unsigned)p.w.dF, (unsigned)p.rowsF,
                                          (unsigned)p.w.nO, BN, p.w.ldp, krF, krO);
  else
    k_kr<T, unsigned long long><<<kb, 256, 0, st>>>(W, sh, p.g0, p.g1, p.f0, p.f1, p.w.dF, p.rowsF, p.w.nO, BN,
                                                    p.w.ldp, krF, krO);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const bool direct = out.sd == 0 && p.ks == 1;
  if ((e = gemm(p, X, krF, krO, direct ? out.p : part, st)) != cudaSuccess) return e;
  *launches += direct ? 2 : 3;
  if (direct) return cudaSuccess;
  const long long n = p.w.D * p.w.ldp;
  // one thread an output where those fill the chip or the partials are few
  // (147456 outputs of 2 partials: 12 us dealt to groups, 3 us this way)
  if (p.ks <= 8 || n >= (1 << 20)) {
    const unsigned sb = (unsigned)((n + 255) / 256);
    k_sum_few<T><<<sb, 256, 0, st>>>(part, p.w.D, sh.R, p.w.ldp, p.ks, out);
    return cudaGetLastError();
  }
  const unsigned sb = (unsigned)((n + 31) / 32);
  k_sum<T><<<sb, 32 * SG, 0, st>>>(part, p.w.D, sh.R, p.w.ldp, p.ks, out);
  return cudaGetLastError();
}

// Where the MTTKRPs of every mode go: p[m] (null: not wanted) d_m x R,
// column-major or (rows) row-major.
struct Outs {
  void* p[TFX_MAX_ORDER];
  int rows;
};

// The MTTKRPs of every mode in out.p (mttkrp.cu); scratch as
// tfx_mttkrp_all_scratch_bytes().
int all_modes(int dtype, const void* T, const CpDims& sh, const void* W, const Outs& out, void* scratch,
              size_t scratch_bytes, cudaStream_t st);

}  // namespace mg
}  // namespace tfx
