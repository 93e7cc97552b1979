// FP64 MTTKRP GEMM.
//
// What bounds it is the FP64 pipe (1.2 TFLOP/s measured, two FMAs a cycle and
// SM), so the split wastes none of them: a warp holds 8 rows x 4 TN columns, one
// output a lane and column group, TN = ceil(R / 4); chunks run to the last valid
// step and warps past the last row idle (the strips are dealt to the warps in
// turn, split by split, so that the SM's quarters share them evenly).  Shared
// memory is read once or twice per FMA, which takes 16 cycles of the SM.
#include "mttkrp_gemm.cuh"

namespace tfx {
namespace mg {

constexpr int DNT = 128, DBM = 32, DAST = BK + 2;

__device__ __forceinline__ void dcp16(void* s, const double* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g)
               : "memory");
}
__device__ __forceinline__ void dcp8(void* s, const double* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g)
               : "memory");
}

template <int TN, bool LAST>
struct DCfg {
  static constexpr int BN = 4 * TN;
  static constexpr int ASZ = LAST ? BK * DBM : DBM * DAST;
  static constexpr int STG = ASZ + BK * BN + BN;  // A, KR_F rows, KR_O row
  static constexpr size_t SMEM = (size_t)2 * STG * 8;
};

template <int TN, bool LAST, bool FOLD>
__global__ void __launch_bounds__(DNT, TN > 8 ? 4 : 6)
    k_mttkrp_f64(const double* __restrict__ Tt, const double* __restrict__ krF, const double* __restrict__ krO,
                 const __grid_constant__ Walk wk_, double* __restrict__ part) {
  using C = DCfg<TN, LAST>;
  extern __shared__ __align__(16) double dsm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lm = lane >> 2, ln = lane & 3;
  const int strip = (warp + blockIdx.y) & 3;
  const long long D = wk_.D, m0 = (long long)blockIdx.x * DBM;
  const int dF = wk_.dF, nc = wk_.nc;
  const bool vec = wk_.vec != 0, on = m0 + 8 * strip < D;
  const long long nch = wk_.nO * nc;
  const long long cb = nch * blockIdx.y / gridDim.y, ce = nch * (blockIdx.y + 1) / gridDim.y;
  krF += (size_t)blockIdx.z * nc * BK * C::BN;
  krO += (size_t)blockIdx.z * C::BN;

  long long lo = cb / nc;  // the next chunk to load
  int lc = (int)(cb - lo * nc);
  const double* base = Tt;
  auto rebase = [&]() {
    const long long p = lo / wk_.Q1, q = lo - p * wk_.Q1;
    base = Tt + p * wk_.sP + q * wk_.sQ;
  };
  rebase();
  // steps past dF and rows past D are neither loaded nor used
  auto load = [&](int s) {
    double* A = dsm + s * C::STG;
    double* B = A + C::ASZ;
    const int f0 = lc * BK;
    if (LAST) {
      const int m = vec ? (tid & 15) * 2 : lane, kr = vec ? tid >> 4 : warp;
      if (m0 + m < D) {
        const double* g = base + (long long)f0 * D + m0 + m;
        if (vec) {
#pragma unroll
          for (int k = 0; k < BK; k += 8)
            if (f0 + kr + k < dF) dcp16(A + (kr + k) * DBM + m, g + (long long)(kr + k) * D);
        } else {
#pragma unroll
          for (int k = 0; k < BK; k += 4)
            if (f0 + kr + k < dF) dcp8(A + (kr + k) * DBM + m, g + (long long)(kr + k) * D);
        }
      }
    } else {
      const int k = vec ? (tid & 15) * 2 : lane, mr = vec ? tid >> 4 : warp;
      if (f0 + k < dF) {
        const double* g = base + f0 + k + m0 * wk_.sD;
        if (vec) {
#pragma unroll
          for (int m = 0; m < DBM; m += 8)
            if (m0 + mr + m < D) dcp16(A + (mr + m) * DAST + k, g + (mr + m) * wk_.sD);
        } else {
#pragma unroll
          for (int m = 0; m < DBM; m += 4)
            if (m0 + mr + m < D) dcp8(A + (mr + m) * DAST + k, g + (mr + m) * wk_.sD);
        }
      }
    }
    const double* b = krF + (size_t)f0 * C::BN;
    for (int e = tid; e < BK * C::BN / 2; e += DNT) dcp16(B + 2 * e, b + 2 * e);
    if (FOLD && tid < C::BN / 2) dcp16(B + BK * C::BN + 2 * tid, krO + lo * wk_.ldp + 2 * tid);
    if (++lc == nc) {
      lc = 0;
      ++lo;
      rebase();
    }
  };

  double acc[TN], sum[FOLD ? TN : 1];
#pragma unroll
  for (int g = 0; g < TN; ++g) {
    acc[g] = 0.0;
    if (FOLD) sum[g] = 0.0;
  }
  if (cb < ce) load(0);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  int cc = (int)(cb % nc);
  for (long long c = cb; c < ce; ++c) {
    const int s = (int)((c - cb) & 1);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();  // chunk c is there; everyone is done with chunk c - 1
    if (c + 1 < ce) load(s ^ 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const double* A = dsm + s * C::STG;
    const double* B = A + C::ASZ + ln;
    const int kc = min(BK, dF - cc * BK);
    if (on) {
#pragma unroll 4
      for (int k = 0; k < kc; ++k) {
        const double a = LAST ? A[k * DBM + 8 * strip + lm] : A[(8 * strip + lm) * DAST + k];
#pragma unroll
        for (int g = 0; g < TN; ++g) acc[g] = fma(a, B[k * C::BN + 4 * g], acc[g]);
      }
    }
    if (++cc == nc) cc = 0;
    if (FOLD && (cc == 0 || c + 1 == ce)) {
      const double* sp = A + C::ASZ + BK * C::BN + ln;
#pragma unroll
      for (int g = 0; g < TN; ++g) {
        sum[g] = fma(acc[g], sp[4 * g], sum[g]);
        acc[g] = 0.0;
      }
    }
  }
  const long long row = m0 + 8 * strip + lm;
  if (row >= D) return;
  double* o = part + ((size_t)blockIdx.y * D + row) * wk_.ldp + blockIdx.z * C::BN + ln;
#pragma unroll
  for (int g = 0; g < TN; ++g) o[4 * g] = FOLD ? sum[g] : acc[g];
}

template <int TN, bool LAST, bool FOLD>
static cudaError_t dlaunch(const Plan& p, const double* T, const double* krF, const double* krO, double* part,
                           cudaStream_t st) {
  const size_t smb = DCfg<TN, LAST>::SMEM;
  cudaError_t e = cudaFuncSetAttribute(k_mttkrp_f64<TN, LAST, FOLD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smb);
  if (e != cudaSuccess) return e;
  k_mttkrp_f64<TN, LAST, FOLD><<<dim3((unsigned)p.tilesM, p.ks, p.nblk), DNT, smb, st>>>(T, krF, krO, p.w, part);
  return cudaGetLastError();
}

template <int TN>
static cudaError_t dlaunch1(const Plan& p, const double* T, const double* krF, const double* krO, double* part,
                            cudaStream_t st) {
  if (p.last) return p.fold ? dlaunch<TN, true, true>(p, T, krF, krO, part, st)
                            : dlaunch<TN, true, false>(p, T, krF, krO, part, st);
  return p.fold ? dlaunch<TN, false, true>(p, T, krF, krO, part, st)
                : dlaunch<TN, false, false>(p, T, krF, krO, part, st);
}

cudaError_t gemm_f64(const Plan& p, const double* T, const double* krF, const double* krO, double* part,
                     cudaStream_t st) {
  switch (p.TN) {
    case 1: return dlaunch1<1>(p, T, krF, krO, part, st);
    case 2: return dlaunch1<2>(p, T, krF, krO, part, st);
    case 3: return dlaunch1<3>(p, T, krF, krO, part, st);
    case 4: return dlaunch1<4>(p, T, krF, krO, part, st);
    case 5: return dlaunch1<5>(p, T, krF, krO, part, st);
    case 6: return dlaunch1<6>(p, T, krF, krO, part, st);
    case 7: return dlaunch1<7>(p, T, krF, krO, part, st);
    case 8: return dlaunch1<8>(p, T, krF, krO, part, st);
    case 9: return dlaunch1<9>(p, T, krF, krO, part, st);
    case 10: return dlaunch1<10>(p, T, krF, krO, part, st);
    case 11: return dlaunch1<11>(p, T, krF, krO, part, st);
    case 12: return dlaunch1<12>(p, T, krF, krO, part, st);
    case 13: return dlaunch1<13>(p, T, krF, krO, part, st);
    case 14: return dlaunch1<14>(p, T, krF, krO, part, st);
    case 15: return dlaunch1<15>(p, T, krF, krO, part, st);
    default: return dlaunch1<16>(p, T, krF, krO, part, st);
  }
}

}  // namespace mg
}  // namespace tfx
