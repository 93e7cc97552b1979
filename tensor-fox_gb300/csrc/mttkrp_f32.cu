// FP32 MTTKRP GEMM on the FP32 pipes.
//
// What bounds it is the FP32 FMA rate (2 R flop for each 4-byte tensor value: at
// R = 50 the FMAs need 2.3x the time of reading the tensor).  FP32 entry points
// stay on FP32 FMAs: the tensor cores' accumulation truncates (tcgen05 3xTF32
// is 2.7e-5 off at 512^3, this kernel 4e-8).
//
// A CTA has four warps: WM along the rows (32 rows each) and 4 / WM along the
// k of a 32-step chunk.  A lane holds 4 rows x TN columns, fma.rn.f32x2 taking
// two columns at a time: at TN = 14 a k step is 28 FMA instructions, 4 register
// pairs and 4.5 shared-memory reads, all reads one wavefront.  Copies are 16
// bytes where the contiguous extent is a multiple of 4 and the base aligned, 4
// bytes otherwise, three stages deep.
//
// 512^3 at R = 50, a mode: 296 us (256 for the last one, whose rows lie
// together) = 45 (52) TFLOP/s (two steps of four k unrolled 310 and 270, one 323
// and 288, eight as here); 2253 us with 4 x 4 thread tiles and Khatri-Rao rows formed in
// the loop.  Also measured: the same tiles with the rows formed in the loop 508
// us (a quarter of the stalls on the factor loads), with the next chunk's
// loaded ahead 545 us (60% more instructions).
#include "mttkrp_gemm.cuh"

namespace tfx {
namespace mg {

constexpr int NT = 128, AST = BK + 4, STAGES = 3;

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
__device__ __forceinline__ void add2(f2& c, f2 a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(c) : "l"(a)); }
__device__ __forceinline__ void fma2(f2& c, f2 a, f2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }

template <int TN, int WM, bool LAST, bool FOLD>
struct Cfg {
  static constexpr int BM = 32 * WM, BN = 4 * TN;
  static constexpr int WK = 4 / WM, KW = BK / WK;
  static constexpr int CTAS = TN > 8 ? 2 : 3;
  // chunks a chain: 512 steps a lane, and 32 where the rows are few, so that long
  // contractions of short modes are summed in chains no longer than theirs
  static constexpr int FC = WM == 1 ? 4 : 512 / KW;
  static constexpr int ASZ = LAST ? BK * BM : BM * AST;
  static constexpr int STG = ASZ + BK * BN + BN;  // A, KR_F rows, KR_O row
  static constexpr size_t SMEM = (size_t)STAGES * STG * 4;
};

// part[split][D][ldp], column block blockIdx.z; krF[block][nc * BK][BN], krO[nO][ldp]
template <int TN, int WM, bool LAST, bool FOLD>
__global__ void __launch_bounds__(NT, Cfg<TN, WM, LAST, FOLD>::CTAS)
    k_mttkrp_f32(const float* __restrict__ Tt, const float* __restrict__ krF, const float* __restrict__ krO,
                 const __grid_constant__ Walk wk_, float* __restrict__ part) {
  using C = Cfg<TN, WM, LAST, FOLD>;
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp % WM, wk = warp / WM;
  const int lm = lane >> 2, ln = lane & 3;
  const long long D = wk_.D, m0 = (long long)blockIdx.x * C::BM;
  const int dF = wk_.dF, nc = wk_.nc;
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

  f2 acc[4][TN / 2], sum[4][TN / 2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) {
      acc[i][j] = 0ull;
      sum[i][j] = 0ull;
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
#pragma unroll 8
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
    if (!FOLD) {  // a chunk's sums into the total: 32-step chains
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) {
          add2(sum[i][j], acc[i][j]);
          acc[i][j] = 0ull;
        }
    } else if (++cc == nc || c + 1 == ce || cc % C::FC == 0) {
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
    const long long row = m0 + wm * 32 + (LAST ? 4 * lm + i : 8 * i + lm);
    if (row >= D) continue;
    float* o = out + (size_t)row * wk_.ldp;
#pragma unroll
    for (int j = 0; j < TN / 2; ++j)
      *reinterpret_cast<f2*>(o + (j < 2 * (TN / 4) ? 16 * (j >> 1) + 4 * ln + 2 * (j & 1) : 16 * (TN / 4) + 2 * ln)) =
          acc[i][j];
  }
}

template <int TN, int WM, bool LAST, bool FOLD>
static cudaError_t launch(const Plan& p, const float* T, const float* krF, const float* krO, float* part,
                          cudaStream_t st) {
  const size_t smb = Cfg<TN, WM, LAST, FOLD>::SMEM;
  cudaError_t e =
      cudaFuncSetAttribute(k_mttkrp_f32<TN, WM, LAST, FOLD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smb);
  if (e != cudaSuccess) return e;
  k_mttkrp_f32<TN, WM, LAST, FOLD><<<dim3((unsigned)p.tilesM, p.ks, p.nblk), NT, smb, st>>>(T, krF, krO, p.w, part);
  return cudaGetLastError();
}

template <int TN, int WM>
static cudaError_t launch2(const Plan& p, const float* T, const float* krF, const float* krO, float* part,
                           cudaStream_t st) {
  if (p.last) return p.fold ? launch<TN, WM, true, true>(p, T, krF, krO, part, st)
                            : launch<TN, WM, true, false>(p, T, krF, krO, part, st);
  return p.fold ? launch<TN, WM, false, true>(p, T, krF, krO, part, st)
                : launch<TN, WM, false, false>(p, T, krF, krO, part, st);
}

template <int TN>
static cudaError_t launch1(const Plan& p, const float* T, const float* krF, const float* krO, float* part,
                           cudaStream_t st) {
  if (p.WM == 4) return launch2<TN, 4>(p, T, krF, krO, part, st);
  if (p.WM == 2) return launch2<TN, 2>(p, T, krF, krO, part, st);
  return launch2<TN, 1>(p, T, krF, krO, part, st);
}

cudaError_t gemm_f32(const Plan& p, const float* T, const float* krF, const float* krO, float* part, cudaStream_t st) {
  switch (p.TN) {
    case 2: return launch1<2>(p, T, krF, krO, part, st);
    case 4: return launch1<4>(p, T, krF, krO, part, st);
    case 6: return launch1<6>(p, T, krF, krO, part, st);
    case 8: return launch1<8>(p, T, krF, krO, part, st);
    case 10: return launch1<10>(p, T, krF, krO, part, st);
    case 12: return launch1<12>(p, T, krF, krO, part, st);
    case 14: return launch1<14>(p, T, krF, krO, part, st);
    default: return launch1<16>(p, T, krF, krO, part, st);
  }
}

}  // namespace mg
}  // namespace tfx
