// FP32 MTTKRP T_(l) KR_l on the FP32 pipes, any order and mode with d_l > 16.
//
// The product is a GEMM: rows d (mode l), contraction over the other modes,
// columns r.  What bounds it is the FP32 FMA rate (2 R flop for each 4-byte
// tensor value: at R = 50 the FMAs need 2.3x the time of reading the tensor).
// FP32 entry points stay on FP32 FMAs: the tensor cores' accumulation
// truncates (tcgen05 3xTF32 is 2.7e-5 off at 512^3, this kernel 6e-8).
//
// The other modes are split into an inner group F, whose Khatri-Rao block KR_F
// (dF x R) is formed once in global memory (L2-resident), and the outer rest O:
//   M[d, r] = sum_o KR_O[o, r] (sum_f T[d, o, f] KR_F[f, r]).
// So the inner loop is a plain GEMM whose operands both arrive by cp.async,
// and every dF steps the sums are scaled by KR_O's row and folded into a second
// set (no fold when F holds every other mode).  Forming Khatri-Rao rows in the
// loop instead cost as many instructions as the FMAs.
//
// A CTA has four warps: WM along the rows (32 rows each) and 4 / WM along the
// k of a 32-step chunk.  A lane holds 4 rows x TN columns, fma.rn.f32x2 taking
// two columns at a time: at TN = 14 a k step is 28 FMA instructions, 4 register
// pairs and 4.5 shared-memory reads, all reads one wavefront.  Copies are 16
// bytes where the contiguous extent is a multiple of 4 and the base aligned, 4
// bytes otherwise.  Partials of the splits are summed in compensated FP32.
#pragma once
#include <stdint.h>

namespace tfx {
namespace mf32 {

constexpr int BK = 32, NT = 128, AST = BK + 4, STAGES = 3;

__device__ __forceinline__ void cp16(void* s, const float* g, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp4(void* s, const float* g, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g),
               "r"(bytes)
               : "memory");
}
typedef unsigned long long f2;  // two floats in a register pair
__device__ __forceinline__ f2 pack2(float a, float b) {
  f2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float2 unpack2(f2 v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ void fma2(f2& c, f2 a, f2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }

// What the main kernel walks: nO outer positions of dF inner steps each.
struct Walk {
  int D, dF, nc;             // rows; inner steps; chunks of BK an outer position
  long long nO, Q1, sP, sQ;  // outer position o starts at (o / Q1) * sP + (o % Q1) * sQ
  long long sD;              // row stride (1 for the last mode)
  int ldp, vec;
};

template <int TN, int WM, bool LAST, bool FOLD>
struct Cfg {
  static constexpr int BM = 32 * WM, BN = 4 * TN;
  static constexpr int WK = 4 / WM, KW = BK / WK;
  static constexpr int CTAS = TN > 8 ? 2 : 3;
  static constexpr int ASZ = LAST ? BK * BM : BM * AST;
  static constexpr int STG = ASZ + BK * BN + BN;  // A, KR_F rows, KR_O row
  static constexpr size_t SMEM = (size_t)STAGES * STG * 4;
};

// part[split][D][ldp], column block blockIdx.z; krF[block][nc * BK][BN], krO[nO][ldp]
template <int TN, int WM, bool LAST, bool FOLD>
__global__ void __launch_bounds__(NT, Cfg<TN, WM, LAST, FOLD>::CTAS)
    k_mttkrp_f32(const float* __restrict__ Tt, const float* __restrict__ krF, const float* __restrict__ krO,
                 const __grid_constant__ Walk wk_, float* __restrict__ part, int R) {
  using C = Cfg<TN, WM, LAST, FOLD>;
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp % WM, wk = warp / WM;
  const int lm = lane >> 2, ln = lane & 3;
  const int D = wk_.D, dF = wk_.dF, nc = wk_.nc;
  const int m0 = blockIdx.x * C::BM;
  const bool full = m0 + C::BM <= D, vec = wk_.vec != 0;
  const long long nch = wk_.nO * nc;
  const long long cb = nch * blockIdx.y / gridDim.y, ce = nch * (blockIdx.y + 1) / gridDim.y;
  krF += (size_t)blockIdx.z * nc * BK * C::BN;
  krO += (size_t)blockIdx.z * C::BN;

  // the next chunk to load: outer position, chunk within it, the position's base
  long long lo = cb / nc;
  int lc = (int)(cb - lo * nc);
  const float* base = Tt;
  auto rebase = [&]() {
    const long long p = lo / wk_.Q1, q = lo - p * wk_.Q1;
    base = Tt + p * wk_.sP + q * wk_.sQ;
  };
  rebase();
  auto load = [&](int s) {
    float* A = sm + s * C::STG;
    float* B = A + C::ASZ;
    const int f0 = lc * BK;
    if (LAST) {  // k rows of BM consecutive values
      const float* g0 = base + (long long)f0 * D + m0;
      if (vec) {
        constexpr int PR = C::BM / 4;
        const int m = (tid % PR) * 4, kr = tid / PR;
        const int rb = m0 + m < D ? 16 : 0;
        const float* g = rb ? g0 + m : Tt;
#pragma unroll
        for (int u = 0; u < BK * PR / NT; ++u) {
          const int k = kr + u * (NT / PR);
          const int nb = f0 + k < dF ? rb : 0;
          cp16(A + k * C::BM + m, nb ? g + (long long)k * D : Tt, nb);
        }
      } else {
        const int m = tid % C::BM, kr = tid / C::BM;
        const int rb = m0 + m < D ? 4 : 0;
        const float* g = rb ? g0 + m : Tt;
#pragma unroll 8
        for (int u = 0; u < BK * C::BM / NT; ++u) {
          const int k = kr + u * (NT / C::BM);
          const int nb = f0 + k < dF ? rb : 0;
          cp4(A + k * C::BM + m, nb ? g + (long long)k * D : Tt, nb);
        }
      }
    } else if (vec) {
      const int kk = (tid & 7) * 4, m = tid >> 3;
      const int kb = f0 + kk < dF ? 16 : 0;
      const float* g = (kb ? base + f0 + kk : Tt) + (m0 + (full ? m : 0)) * wk_.sD;
      float* a = A + m * AST + kk;
      if (full) {
#pragma unroll
        for (int u = 0; u < C::BM / 16; ++u) cp16(a + 16 * u * AST, g + 16 * u * wk_.sD, kb);
      } else {
#pragma unroll
        for (int u = 0; u < C::BM / 16; ++u) {
          const bool ok = m0 + m + 16 * u < D;
          cp16(a + 16 * u * AST, ok ? g + (m + 16 * u) * wk_.sD : Tt, ok ? kb : 0);
        }
      }
    } else {
      const int kb = f0 + lane < dF ? 4 : 0;
      const float* g = (kb ? base + f0 + lane : Tt) + (m0 + (full ? warp : 0)) * wk_.sD;
      float* a = A + warp * AST + lane;
      if (full) {
#pragma unroll
        for (int u = 0; u < C::BM / 4; ++u) cp4(a + 4 * u * AST, g + 4 * u * wk_.sD, kb);
      } else {
#pragma unroll 8
        for (int u = 0; u < C::BM / 4; ++u) {
          const bool ok = m0 + warp + 4 * u < D;
          cp4(a + 4 * u * AST, ok ? g + (warp + 4 * u) * wk_.sD : Tt, ok ? kb : 0);
        }
      }
    }
    const float* b = krF + (size_t)f0 * C::BN + 4 * tid;
#pragma unroll
    for (int u = 0; u < (BK * C::BN / 4 + NT - 1) / NT; ++u)
      if (BK * C::BN / 4 % NT == 0 || tid + NT * u < BK * C::BN / 4) cp16(B + 4 * (tid + NT * u), b + 4 * NT * u, 16);
    if (FOLD && tid < C::BN / 4) cp16(B + BK * C::BN + 4 * tid, krO + lo * wk_.ldp + 4 * tid, 16);
    if (++lc == nc) {
      lc = 0;
      ++lo;
      rebase();
    }
  };

  f2 acc[4][TN / 2], sum[4][FOLD ? TN / 2 : 1];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) {
      acc[i][j] = 0ull;
      if (FOLD) sum[i][j] = 0ull;
    }

#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (cb + s < ce) load(s);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  int cc = (int)(cb % nc), stage = 0;  // the chunk being multiplied
  for (long long c = cb; c < ce; ++c) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncthreads();  // chunk c is there; everyone is done with chunk c - 1
    if (c + STAGES - 1 < ce) load(stage == 0 ? STAGES - 1 : stage - 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const float* A = sm + stage * C::STG;
    const float* B = A + C::ASZ + wk * C::KW * C::BN;
#pragma unroll 2
    for (int k4 = 0; k4 < C::KW; k4 += 4) {
      float a[4][4];  // [row][k]
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(
            LAST ? A + (wk * C::KW + k4 + i) * C::BM + wm * 32 + 4 * lm
                 : A + (wm * 32 + 8 * i + lm) * AST + wk * C::KW + k4);
        if (LAST) {
          a[0][i] = x.x; a[1][i] = x.y; a[2][i] = x.z; a[3][i] = x.w;
        } else {
          a[i][0] = x.x; a[i][1] = x.y; a[i][2] = x.z; a[i][3] = x.w;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float* bp = B + (k4 + u) * C::BN;
        f2 bv[TN / 2];
#pragma unroll
        for (int g = 0; g < TN / 4; ++g) {
          const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(bp + 16 * g + 4 * ln);
          bv[2 * g] = x.x;
          bv[2 * g + 1] = x.y;
        }
        if (TN % 4) bv[TN / 2 - 1] = *reinterpret_cast<const f2*>(bp + 16 * (TN / 4) + 2 * ln);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const f2 ad = pack2(a[i][u], a[i][u]);
#pragma unroll
          for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], ad, bv[j]);
        }
      }
    }
    if (FOLD && (++cc == nc || c + 1 == ce)) {
      if (cc == nc) cc = 0;
      const float* sp = A + C::ASZ + BK * C::BN;
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) {
        const f2 s = *reinterpret_cast<const f2*>(sp + (j < 2 * (TN / 4) ? 16 * (j >> 1) + 4 * ln + 2 * (j & 1)
                                                                          : 16 * (TN / 4) + 2 * ln));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          fma2(sum[i][j], acc[i][j], s);
          acc[i][j] = 0ull;
        }
      }
    }
    if (++stage == STAGES) stage = 0;
  }
  if (FOLD)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) acc[i][j] = sum[i][j];
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  if (C::WK > 1) {  // the k groups' sums, in order, into group 0
    __syncthreads();
    f2* red = reinterpret_cast<f2*>(sm);
    constexpr int PT = 32 * WM;  // threads a group
    if (wk > 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) red[((wk - 1) * 2 * TN + i * (TN / 2) + j) * PT + tid % PT] = acc[i][j];
    }
    __syncthreads();
    if (wk > 0) return;
#pragma unroll
    for (int q = 1; q < C::WK; ++q)
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) {
          const float2 x = unpack2(acc[i][j]), y = unpack2(red[((q - 1) * 2 * TN + i * (TN / 2) + j) * PT + tid]);
          acc[i][j] = pack2(x.x + y.x, x.y + y.y);
        }
  }
  float* out = part + (size_t)blockIdx.y * D * wk_.ldp + blockIdx.z * C::BN;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = m0 + wm * 32 + (LAST ? 4 * lm + i : 8 * i + lm);
    if (row >= D) continue;
    float* o = out + (size_t)row * wk_.ldp;
#pragma unroll
    for (int j = 0; j < TN / 2; ++j)
      *reinterpret_cast<f2*>(o + (j < 2 * (TN / 4) ? 16 * (j >> 1) + 4 * ln + 2 * (j & 1) : 16 * (TN / 4) + 2 * ln)) =
          acc[i][j];
  }
}

// out[r * D + d] = sum over the ks partials of part[.][d][ldp], compensated:
// 32 outputs a CTA, the partials dealt to SG groups of threads whose sums are
// added in a fixed order.
constexpr int SG = 16;

__global__ void __launch_bounds__(32 * SG) k_mttkrp_sum(const float* __restrict__ part, int D, int R, int ldp, int ks,
                                                        float* __restrict__ out) {
  __shared__ float2 red[SG][32];
  const long long n = (long long)D * ldp;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const long long e = (long long)blockIdx.x * 32 + x;
  Acc<float> s;
  if (e < n) {
#pragma unroll 8
    for (int k = y; k < ks; k += SG) s.add(__ldcs(part + (size_t)k * n + e));
  }
  red[y][x] = make_float2(s.hi, s.lo);
  __syncthreads();
  if (y == 0 && e < n) {
    Acc<float> t;
#pragma unroll
    for (int j = 0; j < SG; ++j) t.add2(red[j][x].x, red[j][x].y);
    const long long d = e / ldp;
    const int r = (int)(e - d * ldp);
    if (r < R) out[(size_t)r * D + d] = t.hi + t.lo;
  }
}

// KR_F as [column block][nF rows padded to chunks][BN] (zeros in the padding)
// and KR_O as [nO][ldp], from the flat column-major factors: modes [f0, f1)
// are F, the others but l are O, both with the last mode fastest.  I: 32-bit
// indices where the element count fits (64-bit divisions took 3x the time).
template <class I>
__global__ void __launch_bounds__(256) k_mttkrp_kr(const float* __restrict__ W, const __grid_constant__ CpDims sh,
                                                   int l, int f0, int f1, I dF, I rowsF, I nO, int BN, int ldp,
                                                   float* __restrict__ krF, float* __restrict__ krO) {
  const I e = (I)blockIdx.x * blockDim.x + threadIdx.x;
  const I nF = rowsF * (I)ldp;
  if (e >= nF + nO * (I)ldp) return;
  const bool isF = e < nF;
  const I w = isF ? e : e - nF;
  const I row = w / (I)ldp;
  const int r = (int)(w - row * (I)ldp);
  float v = 0.f;
  if (r < sh.R && (!isF || row < dF)) {
    v = 1.f;
    I rem = row;
    for (int m = isF ? f1 - 1 : sh.L - 1; m >= (isF ? f0 : 0); --m) {
      if (!isF && (m == l || (m >= f0 && m < f1))) continue;
      const I q = rem / (I)sh.d[m];
      v *= W[sh.off[m] + (long long)r * sh.d[m] + (long long)(rem - q * (I)sh.d[m])];
      rem = q;
    }
  }
  if (isF) krF[((size_t)(r / BN) * rowsF + row) * BN + r % BN] = v;
  else krO[(size_t)row * ldp + r] = v;
}

// The launch.  Columns: blocks of at most 64, all as narrow as a multiple of 8
// allows (R = 50: 56, R = 100: 2 x 56).  Rows: 128, 64 or 32 a CTA, the
// largest whose padding stays within 1/8 of the least.  F: every other mode if
// they can be (l the first or the last mode) and the block stays within 8 MB;
// else the last one, and those before it while the chunks' padding is above
// 1/8 and the block within 4096 rows.  Splits: one wave of the resident CTAs,
// at least 4 chunks each, and without a fold at most 2048 k each (a longer
// FP32 chain loses digits).
struct Plan {
  Walk w;
  int TN, WM, tilesM, nblk, ks, f0, f1;
  bool last, fold;
  long long rowsF;
  size_t krF_bytes, krO_bytes, part_bytes;
  size_t total() const { return krF_bytes + krO_bytes + part_bytes; }
};

inline Plan plan(const CpDims& sh, int l, int sms) {
  Plan p;
  const int L = sh.L, D = sh.d[l], R = sh.R;
  p.nblk = (R + 63) / 64;
  const int BN = 8 * (((R + p.nblk - 1) / p.nblk + 7) / 8);
  p.TN = BN / 4;
  p.w.ldp = p.nblk * BN;
  p.w.D = D;
  long long P = 1, Q = 1;
  for (int m = 0; m < l; ++m) P *= sh.d[m];
  for (int m = l + 1; m < L; ++m) Q *= sh.d[m];
  p.last = Q == 1;
  const int lo = p.last ? 0 : l + 1, hi = p.last ? l : L;  // the modes F may take
  const long long K = p.last ? P : Q;
  long long dF;
  if ((p.last || P == 1) && K * p.w.ldp * 4 <= (8LL << 20)) {
    p.f0 = lo;
    dF = K;
  } else {
    p.f0 = hi - 1;
    dF = sh.d[hi - 1];
    while (p.f0 > lo && ((dF + BK - 1) / BK * BK - dF) * 8 > dF && dF * sh.d[p.f0 - 1] <= 4096) dF *= sh.d[--p.f0];
  }
  p.f1 = hi;
  p.w.dF = (int)dF;
  p.w.nc = (int)((dF + BK - 1) / BK);
  p.rowsF = (long long)p.w.nc * BK;
  p.w.nO = P * Q / dF;
  p.fold = p.w.nO > 1;
  p.w.Q1 = p.last ? 1 : Q / dF;
  p.w.sP = p.last ? dF * D : (long long)D * Q;
  p.w.sQ = dF;
  p.w.sD = Q;
  p.WM = 1;
  const int least = (D + 31) / 32 * 32;
  for (int wm = 2; wm <= 4; wm *= 2) {
    const int padded = (D + 32 * wm - 1) / (32 * wm) * (32 * wm);
    if ((long long)padded * 8 <= (long long)least * 9) p.WM = wm;
  }
  p.tilesM = (D + 32 * p.WM - 1) / (32 * p.WM);
  const long long nch = p.w.nO * p.w.nc, slots = (long long)sms * (p.TN > 8 ? 2 : 3);
  long long ks = std::max<long long>(1, slots / ((long long)p.tilesM * p.nblk));
  while (!p.fold && nch * BK / ks > 2048) ks *= 2;
  ks = std::max<long long>(1, std::min(ks, nch / 4));
  p.ks = (int)std::min<long long>(ks, 32768);
  p.krF_bytes = (size_t)((p.rowsF * p.w.ldp * 4 + 255) & ~255LL);
  p.krO_bytes = (size_t)((p.w.nO * p.w.ldp * 4 + 255) & ~255LL);
  p.part_bytes = (size_t)p.ks * D * p.w.ldp * 4;
  return p;
}

template <int TN, int WM, bool LAST, bool FOLD>
static cudaError_t launch(const Plan& p, const float* T, const float* krF, const float* krO, float* part, int R,
                          cudaStream_t st) {
  const size_t smb = Cfg<TN, WM, LAST, FOLD>::SMEM;
  cudaError_t e =
      cudaFuncSetAttribute(k_mttkrp_f32<TN, WM, LAST, FOLD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smb);
  if (e != cudaSuccess) return e;
  k_mttkrp_f32<TN, WM, LAST, FOLD><<<dim3(p.tilesM, p.ks, p.nblk), NT, smb, st>>>(T, krF, krO, p.w, part, R);
  return cudaGetLastError();
}

template <int TN, int WM>
static cudaError_t launch2(const Plan& p, const float* T, const float* krF, const float* krO, float* part, int R,
                           cudaStream_t st) {
  if (p.last) return p.fold ? launch<TN, WM, true, true>(p, T, krF, krO, part, R, st)
                            : launch<TN, WM, true, false>(p, T, krF, krO, part, R, st);
  return p.fold ? launch<TN, WM, false, true>(p, T, krF, krO, part, R, st)
                : launch<TN, WM, false, false>(p, T, krF, krO, part, R, st);
}

template <int TN>
static cudaError_t launch1(const Plan& p, const float* T, const float* krF, const float* krO, float* part, int R,
                           cudaStream_t st) {
  if (p.WM == 4) return launch2<TN, 4>(p, T, krF, krO, part, R, st);
  if (p.WM == 2) return launch2<TN, 2>(p, T, krF, krO, part, R, st);
  return launch2<TN, 1>(p, T, krF, krO, part, R, st);
}

// scratch: 256-byte aligned, plan(...).total() bytes
inline cudaError_t run(Plan p, const float* T, const float* W, const CpDims& sh, int l, float* out, void* scratch,
                       cudaStream_t st) {
  const int ext = p.last ? p.w.D : p.w.dF;
  p.w.vec = ((uintptr_t)T & 15) == 0 && ext % 4 == 0 && (p.last || p.w.sD % 4 == 0);
  float* krF = (float*)scratch;
  float* krO = (float*)((char*)scratch + p.krF_bytes);
  float* part = (float*)((char*)scratch + p.krF_bytes + p.krO_bytes);
  const int BN = 4 * p.TN, R = sh.R;
  const long long nkr = (p.rowsF + p.w.nO) * p.w.ldp;
  const unsigned kb = (unsigned)((nkr + 255) / 256);
  if (nkr < (1LL << 31))
    k_mttkrp_kr<unsigned><<<kb, 256, 0, st>>>(W, sh, l, p.f0, p.f1, (unsigned)p.w.dF, (unsigned)p.rowsF,
                                              (unsigned)p.w.nO, BN, p.w.ldp, krF, krO);
  else
    k_mttkrp_kr<unsigned long long><<<kb, 256, 0, st>>>(W, sh, l, p.f0, p.f1, p.w.dF, p.rowsF, p.w.nO, BN, p.w.ldp,
                                                        krF, krO);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  switch (p.TN) {
    case 2: e = launch1<2>(p, T, krF, krO, part, R, st); break;
    case 4: e = launch1<4>(p, T, krF, krO, part, R, st); break;
    case 6: e = launch1<6>(p, T, krF, krO, part, R, st); break;
    case 8: e = launch1<8>(p, T, krF, krO, part, R, st); break;
    case 10: e = launch1<10>(p, T, krF, krO, part, R, st); break;
    case 12: e = launch1<12>(p, T, krF, krO, part, R, st); break;
    case 14: e = launch1<14>(p, T, krF, krO, part, R, st); break;
    default: e = launch1<16>(p, T, krF, krO, part, R, st); break;
  }
  if (e != cudaSuccess) return e;
  k_mttkrp_sum<<<(unsigned)(((long long)p.w.D * p.w.ldp + 31) / 32), 32 * SG, 0, st>>>(part, p.w.D, R, p.w.ldp, p.ks,
                                                                                      out);
  return cudaGetLastError();
}

}  // namespace mf32
}  // namespace tfx
