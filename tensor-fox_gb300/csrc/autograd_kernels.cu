// Kernels of the differentiable CP layer (forward: reconstruction / fit loss;
// backward: MTTKRP).
//
//   tfx_cp_full    the dense tensor [[W_0, ..., W_{L-1}]] (Conversion.py:52-79 cpd2tens)
//   tfx_cp_wp1     W_l P1_l with P1_l = o_{m != l} W_m^T W_m for every mode
//                  (GaussNewton.py:520-548, :424)
// Factors use the flat column-major layout; the output of tfx_cp_wp1 is (d_l x R)
// column-major.  The MTTKRPs are in mttkrp.cu.
#include <math.h>

#include <algorithm>

#include "tfx_capi_internal.h"
#include "tfx_common.cuh"
#include "mttkrp_gemm.cuh"

namespace tfx {

template <class T, int TS>
__global__ void __launch_bounds__(TFX_THREADS) k_cp_full(const T* __restrict__ W, CpDims sh, T* __restrict__ out) {
  using TL = Tile<TS, TS>;
  __shared__ T sA[TFX_BK * TL::LDA];
  __shared__ T sB[TFX_BK * TL::LDB];
  __shared__ int sIdx[TL::BN * TFX_MAX_ORDER];
  const int L = sh.L, R = sh.R, d0 = sh.d[0];
  long long Q0 = 1;
  for (int l = 1; l < L; ++l) Q0 *= sh.d[l];
  const int tm_ = (d0 + TL::BM - 1) / TL::BM;
  const long long ntiles = (long long)tm_ * ((Q0 + TL::BN - 1) / TL::BN);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int m0 = (int)(t % tm_) * TL::BM;
    const long long q0 = (t / tm_) * TL::BN;
    if (tid < TL::BN) {
      long long q = q0 + tid;
      if (q < Q0)
        for (int l = L - 1; l >= 1; --l) {
          sIdx[tid * TFX_MAX_ORDER + l] = (int)(q % sh.d[l]);
          q /= sh.d[l];
        }
    }
    __syncthreads();
    T acc[TS][TS];
    tile_zero<T, TS, TS>(acc);
    for (int k0 = 0; k0 < R; k0 += TFX_BK) {
      const int kc = min(TFX_BK, R - k0);
      for (int e = tid; e < TFX_BK * TL::BM; e += TFX_THREADS) {
        const int kk = e / TL::BM, mm = e - kk * TL::BM;
        sA[kk * TL::LDA + mm] = (kk < kc && m0 + mm < d0) ? W[sh.off[0] + (k0 + kk) * d0 + m0 + mm] : T(0);
      }
      for (int e = tid; e < TFX_BK * TL::BN; e += TFX_THREADS) {
        const int kk = e / TL::BN, nn = e - kk * TL::BN;
        T v = T(0);
        if (kk < kc && q0 + nn < Q0) {
          v = T(1);
          for (int l = L - 1; l >= 1; --l) v *= W[sh.off[l] + (k0 + kk) * sh.d[l] + sIdx[nn * TFX_MAX_ORDER + l]];
        }
        sB[kk * TL::LDB + nn] = v;
      }
      __syncthreads();
      tile_fma<T, TS, TS>(sA, sB, acc, kc);
      __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < TS; ++u)
#pragma unroll
      for (int v = 0; v < TS; ++v) {
        const int m = m0 + ty + 16 * u;
        const long long q = q0 + tx + 16 * v;
        if (m < d0 && q < Q0) out[(long long)m * Q0 + q] = acc[u][v];
      }
  }
}

// The factors as a caller has them (any strides) into the flat column-major
// layout: tiles of 1024 entries through shared memory, read along whichever
// stride is the shorter.  A tile has 2^LC columns, the fewest that hold R (up to
// 32): with 32 x 32 tiles 27 of 32 lanes idled at R = 5 (1000000 x 5 and 2 x 5, FP32:
// 17 us, 58 that way).
struct PackArgs {
  const void* p[TFX_MAX_ORDER];
  long long rs[TFX_MAX_ORDER], cs[TFX_MAX_ORDER];
};

template <class T, int LC>
__global__ void __launch_bounds__(256) k_pack(const __grid_constant__ PackArgs a, const __grid_constant__ CpDims sh,
                                              T* __restrict__ out) {
  constexpr int TC = 1 << LC, TR = 1024 >> LC, ST = TR + (32 >> LC);
  __shared__ T tile[TC * ST];  // [column][row]; the pad keeps a warp's rows and columns on their own banks
  const int R = sh.R, nr = (R - 1) / TC + 1;
  int t = blockIdx.x, m = 0;
  while (t >= ((sh.d[m] - 1) / TR + 1) * nr) t -= ((sh.d[m++] - 1) / TR + 1) * nr;
  const int i0 = t / nr * TR, r0 = t % nr * TC, d = sh.d[m];
  const T* w = (const T*)a.p[m];
  const long long rs = a.rs[m], cs = a.cs[m];
  const bool along_r = cs <= rs;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int e = threadIdx.x + 256 * u;
    const int i = along_r ? e >> LC : e % TR, r = along_r ? e & (TC - 1) : e / TR;
    if (i < d - i0 && r0 + r < R) tile[r * ST + i] = w[(long long)(i0 + i) * rs + (r0 + r) * cs];
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int e = threadIdx.x + 256 * u, i = e % TR, r = e / TR;
    if (i < d - i0 && r0 + r < R) out[sh.off[m] + (long long)(r0 + r) * d + i0 + i] = tile[r * ST + i];
  }
}

// Gramians of every mode, G_m = W_m^T W_m (FP64, compensated sums of the
// working-type products).  A CTA takes a 16 x 16 block on or above the diagonal
// of one Gramian: 32 rows of its 32 columns at a time through shared memory
// (coalesced), four groups of threads a quarter of the rows each, added in
// order.  512 rows, R = 50: 17 us, 67 with one thread an entry walking two columns.
// Rows past the end and warps past the rank are left out: the FP64 pipe takes as
// long for zeros (4 x 4 x 4, R = 3, FP64 with the product below: 7 us, 15 with them).
template <class T>
__global__ void __launch_bounds__(1024) k_cp_grams(const T* __restrict__ W, CpDims sh, double* __restrict__ gram) {
  __shared__ T sa[16][129], sb[16][129];
  __shared__ double red[3][256];
  const int R = sh.R, RR = R * R, nb = (R + 15) / 16;
  int t = blockIdx.x, ba = 0;
  while (t >= nb - ba) {
    t -= nb - ba;
    ++ba;
  }
  const int a0 = ba * 16, b0 = (ba + t) * 16, m = blockIdx.y, d = sh.d[m];
  const int tid = threadIdx.x, z = tid >> 8, a = (tid >> 4) & 15, b = tid & 15;
  const bool on = a0 + (a & ~1) < R;  // a warp has two values of a
  const T* w = W + sh.off[m];
  Acc<T> s[2];
  for (int i0 = 0; i0 < d; i0 += 128) {
    __syncthreads();
    for (int e = tid; e < 32 * 128; e += 1024) {
      const int c = e >> 7, i = e & 127, col = c < 16 ? a0 + c : b0 + c - 16;
      const T v = (col < R && i0 + i < d) ? w[(long long)col * d + i0 + i] : T(0);
      if (c < 16) sa[c][i] = v;
      else sb[c - 16][i] = v;
    }
    __syncthreads();
    const int n = on ? min(32, d - i0 - 32 * z) : 0;
    const T *pa = sa[a] + 32 * z, *pb = sb[b] + 32 * z;
    if (n == 32) {
#pragma unroll 4
      for (int i = 0; i < 32; i += 2) {
        s[0].fma_(pa[i], pb[i]);
        s[1].fma_(pa[i + 1], pb[i + 1]);
      }
    } else {
      for (int i = 0; i < n; i += 2) {  // an odd end takes one zero
        s[0].fma_(pa[i], pb[i]);
        s[1].fma_(pa[i + 1], pb[i + 1]);
      }
    }
  }
  double v = s[0].value() + s[1].value();
  if (z > 0) red[z - 1][tid & 255] = v;
  __syncthreads();
  if (z == 0 && a0 + a < R && b0 + b < R && a0 + a <= b0 + b) {
    v = ((v + red[0][tid]) + red[1][tid]) + red[2][tid];
    gram[(size_t)m * RR + (a0 + a) * R + b0 + b] = v;
    gram[(size_t)m * RR + (b0 + b) * R + a0 + a] = v;
  }
}

static unsigned gram_blocks(int R) {
  const unsigned nb = (R + 15) / 16;
  return nb * (nb + 1) / 2;
}

// out_l = scale (W_l P1_l - M_l) [times *gl], P1_l = o_{m != l} G_m (ascending
// m, FP64, rounded to the working type in shared memory); M == nullptr means
// M_l = 0; M and out in the same layout.  Grid (ceil(max d / 16), L), 16 rows per
// CTA; four accumulators a thread, whose compensated chains overlap.
template <class T>
__global__ void __launch_bounds__(TFX_THREADS) k_cp_wp1(const T* __restrict__ W, const __grid_constant__ CpDims sh,
                                                        const double* __restrict__ gram, const T* __restrict__ M,
                                                        T scale, const T* __restrict__ gl,
                                                        const __grid_constant__ mg::Outs out) {
  extern __shared__ __align__(16) char smem[];
  T* sP = (T*)smem;          // [R][R]
  const int l = blockIdx.y, L = sh.L, R = sh.R, RR = R * R, tid = threadIdx.x;
  T* sW = sP + RR;           // [R][16]
  T* o = (T*)out.p[l];
  const int dl = sh.d[l], r0 = blockIdx.x * 16;
  if (r0 >= dl || !o) return;
#pragma unroll 4
  for (int e = tid; e < RR; e += TFX_THREADS) {
    double p = 1.0;
    for (int m = 0; m < L; ++m)
      if (m != l) p *= gram[(size_t)m * RR + e];
    sP[e] = (T)p;
  }
  for (int e = tid; e < 16 * R; e += TFX_THREADS) {
    const int q = e >> 4, i = e & 15;
    sW[e] = r0 + i < dl ? W[sh.off[l] + (long long)q * dl + r0 + i] : T(0);
  }
  __syncthreads();
  for (int e = tid; e < 16 * R; e += TFX_THREADS) {
    const int i = out.rows ? e / R : e & 15, r = out.rows ? e - i * R : e >> 4;
    if (r0 + i >= dl) continue;
    Acc<T> s[4];
    int q = 0;
    for (; q + 4 <= R; q += 4)
#pragma unroll
      for (int u = 0; u < 4; ++u) s[u].fma_(sW[(q + u) * 16 + i], sP[(q + u) * R + r]);
    for (; q < R; ++q) s[0].fma_(sW[q * 16 + i], sP[q * R + r]);
#pragma unroll
    for (int u = 1; u < 4; ++u) {
      s[0].add(s[u].hi_or_v());
      if (sizeof(T) == 4) s[0].add((T)s[u].lo_or_0());
    }
    const size_t at = out.rows ? (size_t)(r0 + i) * R + r : (size_t)r * dl + r0 + i;
    if (M) s[0].add(-M[sh.off[l] + at]);
    T v = scale * (T)s[0].value();
    if (gl) v *= *gl;
    o[at] = v;
  }
}

}  // namespace tfx

using namespace tfx;

extern "C" size_t tfx_mttkrp_all_scratch_bytes(int dtype, int L, const int* dims, int R);

// the FP32 model on register-tiled column pairs (dense_kernels.cu); -1 where the
// 64 x 64 tiles here are the faster form
int tfx_cp_full_f32(int L, const int* dims, int R, const float* W, float* out, cudaStream_t st);

static int nsm() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n < 1) n = 1;
  }
  return n;
}

static int cpdims(CpDims& sh, int L, const int* dims, int R) {
  if (L < 2 || L > TFX_MAX_ORDER || !dims || R < 1) return 1;
  sh.L = L;
  sh.R = R;
  int s = 0;
  for (int l = 0; l < L; ++l) {
    if (dims[l] < 1) return 1;
    sh.d[l] = dims[l];
    sh.off[l] = R * s;
    s += dims[l];
  }
  return 0;
}

static int done(const char* w) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return tfx_set_cuda_error(e, w);
  tfx_count_launch(1);
  return TFX_STATUS_OK;
}

static size_t al256(size_t v) { return (v + 255) & ~(size_t)255; }

extern "C" int tfx_cp_full(int dtype, int L, const int* dims, int R, const void* W, void* out, void* stream) {
  CpDims sh;
  if (cpdims(sh, L, dims, R) || !W || !out) return tfx_set_error(TFX_STATUS_ERR_ARG, "cp_full args");
  if (dtype == TFX_F32) {
    const int r = tfx_cp_full_f32(L, dims, R, (const float*)W, (float*)out, (cudaStream_t)stream);
    if (r >= 0) return r;
  }
  long long Q0 = 1;
  for (int l = 1; l < L; ++l) Q0 *= dims[l];
  const long long tiles = ((dims[0] + 63) / 64) * ((Q0 + 63) / 64);
  const int blocks = (int)std::max<long long>(1, std::min<long long>(tiles, 8LL * nsm()));
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == TFX_F32) k_cp_full<float, 4><<<blocks, TFX_THREADS, 0, st>>>((const float*)W, sh, (float*)out);
  else k_cp_full<double, 4><<<blocks, TFX_THREADS, 0, st>>>((const double*)W, sh, (double*)out);
  return done("cp_full");
}

template <class T>
static void launch_pack(int lc, unsigned g, const PackArgs& a, const CpDims& sh, T* out, cudaStream_t st) {
  switch (lc) {
    case 0: k_pack<T, 0><<<g, 256, 0, st>>>(a, sh, out); break;
    case 1: k_pack<T, 1><<<g, 256, 0, st>>>(a, sh, out); break;
    case 2: k_pack<T, 2><<<g, 256, 0, st>>>(a, sh, out); break;
    case 3: k_pack<T, 3><<<g, 256, 0, st>>>(a, sh, out); break;
    case 4: k_pack<T, 4><<<g, 256, 0, st>>>(a, sh, out); break;
    default: k_pack<T, 5><<<g, 256, 0, st>>>(a, sh, out); break;
  }
}

extern "C" int tfx_factors_pack(int dtype, int L, const int* dims, int R, const void* const* W, const long long* rs,
                                const long long* cs, void* out, void* stream) {
  CpDims sh;
  if (cpdims(sh, L, dims, R) || !W || !rs || !cs || !out) return tfx_set_error(TFX_STATUS_ERR_ARG, "factors_pack args");
  PackArgs a;
  int lc = 0;
  while (lc < 5 && (1 << lc) < R) ++lc;
  const int tc = 1 << lc, tr = 1024 >> lc;
  long long nb = 0;
  for (int l = 0; l < L; ++l) {
    if (!W[l]) return tfx_set_error(TFX_STATUS_ERR_ARG, "factors_pack pointer");
    a.p[l] = W[l];
    a.rs[l] = rs[l];
    a.cs[l] = cs[l];
    nb += (long long)((dims[l] - 1) / tr + 1) * ((R - 1) / tc + 1);
  }
  const unsigned g = (unsigned)nb;
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == TFX_F64) launch_pack<double>(lc, g, a, sh, (double*)out, st);
  else launch_pack<float>(lc, g, a, sh, (float*)out, st);
  return done("factors_pack");
}

// Gramians, then scale (W_l P1_l - M_l) [*gl] for every mode
static int grams_and_wp1(int dtype, const CpDims& sh, const void* W, double* gram, const void* M, double scale,
                         const void* gl, const mg::Outs& out, cudaStream_t st, const char* where) {
  const int L = sh.L, R = sh.R;
  const size_t es = dtype == TFX_F64 ? 8 : 4;
  if ((size_t)R * R * es > 200 * 1024) return tfx_set_error(TFX_STATUS_ERR_UNSUPPORTED, where);
  const size_t smb = (size_t)R * (R + 16) * es;
  cudaError_t e = dtype == TFX_F32
                      ? cudaFuncSetAttribute(k_cp_wp1<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smb)
                      : cudaFuncSetAttribute(k_cp_wp1<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smb);
  if (e != cudaSuccess) return tfx_set_cuda_error(e, "cp_wp1 attribute");
  int maxd = 0;
  for (int l = 0; l < L; ++l) maxd = std::max(maxd, sh.d[l]);
  const dim3 gb(gram_blocks(R), L), grid((maxd + 15) / 16, L);
  if (dtype == TFX_F32) {
    k_cp_grams<float><<<gb, 1024, 0, st>>>((const float*)W, sh, gram);
    k_cp_wp1<float><<<grid, TFX_THREADS, smb, st>>>((const float*)W, sh, gram, (const float*)M, (float)scale,
                                                    (const float*)gl, out);
  } else {
    k_cp_grams<double><<<gb, 1024, 0, st>>>((const double*)W, sh, gram);
    k_cp_wp1<double><<<grid, TFX_THREADS, smb, st>>>((const double*)W, sh, gram, (const double*)M, scale,
                                                     (const double*)gl, out);
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return tfx_set_cuda_error(e, "cp_wp1");
  tfx_count_launch(2);
  return TFX_STATUS_OK;
}

// a flat vector's blocks
static mg::Outs flat_outs(const CpDims& sh, void* out, size_t es, int rows) {
  mg::Outs o = {};
  o.rows = rows;
  for (int l = 0; l < sh.L; ++l) o.p[l] = (char*)out + (size_t)sh.off[l] * es;
  return o;
}

extern "C" size_t tfx_cp_wp1_scratch_bytes(int L, int R) { return (size_t)L * R * R * 8; }

extern "C" int tfx_cp_wp1(int dtype, int L, const int* dims, int R, const void* W, void* out, void* scratch,
                          void* stream) {
  CpDims sh;
  if (cpdims(sh, L, dims, R) || !W || !out || !scratch) return tfx_set_error(TFX_STATUS_ERR_ARG, "cp_wp1 args");
  return grams_and_wp1(dtype, sh, W, (double*)scratch, nullptr, 1.0, nullptr,
                       flat_outs(sh, out, dtype == TFX_F64 ? 8 : 4, 0), (cudaStream_t)stream,
                       "cp_wp1: rank too large");
}

// grad_l = 2 (W_l P1_l - T_(l) KR_l) for every mode: the gradient of
// ||T - [[W]]||^2 (twice GaussNewton.py:401-427's g).  Scratch: the Gramians, the
// MTTKRPs and what those need.
struct FitGradLayout {
  size_t gram, M, mtt, mtt_bytes, total;
};
static FitGradLayout fit_grad_layout(int dtype, int L, const int* dims, int R) {
  const size_t es = dtype == TFX_F64 ? 8 : 4;
  long long nx = 0;
  for (int l = 0; l < L; ++l) nx += (long long)dims[l] * R;
  const size_t mtt = tfx_mttkrp_all_scratch_bytes(dtype, L, dims, R);
  FitGradLayout y;
  y.gram = 0;
  y.M = al256((size_t)L * R * R * 8);
  y.mtt = y.M + al256((size_t)nx * es);
  y.mtt_bytes = mtt;
  y.total = y.mtt + al256(mtt);
  return y;
}

extern "C" size_t tfx_cp_fit_grad_scratch_bytes(int dtype, int L, const int* dims, int R) {
  CpDims sh;
  if (cpdims(sh, L, dims, R)) return 0;
  return fit_grad_layout(dtype, L, dims, R).total;
}

static int fit_grad(int dtype, const void* T, const CpDims& sh, const void* W, const void* gl, const mg::Outs& out,
                    void* scratch, size_t scratch_bytes, cudaStream_t st) {
  const FitGradLayout y = fit_grad_layout(dtype, sh.L, sh.d, sh.R);
  if (scratch_bytes < y.total) return tfx_set_error(TFX_STATUS_ERR_ARG, "cp_fit_grad scratch too small");
  const size_t es = dtype == TFX_F64 ? 8 : 4;
  if ((size_t)sh.R * sh.R * es > 200 * 1024)
    return tfx_set_error(TFX_STATUS_ERR_UNSUPPORTED, "cp_fit_grad: rank too large");
  char* sc = (char*)scratch;
  mg::Outs M = flat_outs(sh, sc + y.M, es, out.rows);
  for (int l = 0; l < sh.L; ++l)
    if (!out.p[l]) M.p[l] = nullptr;
  if (int r = mg::all_modes(dtype, T, sh, W, M, sc + y.mtt, y.mtt_bytes, st)) return r;
  return grams_and_wp1(dtype, sh, W, (double*)(sc + y.gram), sc + y.M, 2.0, gl, out, st,
                       "cp_fit_grad: rank too large");
}

extern "C" int tfx_cp_fit_grad(int dtype, const void* T, int L, const int* dims, int R, const void* W, void* grad,
                               void* scratch, size_t scratch_bytes, void* stream) {
  CpDims sh;
  if (cpdims(sh, L, dims, R) || !T || !W || !grad || !scratch) return tfx_set_error(TFX_STATUS_ERR_ARG, "cp_fit_grad args");
  return fit_grad(dtype, T, sh, W, nullptr, flat_outs(sh, grad, dtype == TFX_F64 ? 8 : 4, 0), scratch, scratch_bytes,
                  (cudaStream_t)stream);
}

extern "C" int tfx_cp_fit_backward(int dtype, const void* T, int L, const int* dims, int R, const void* W,
                                   const void* gl, void* const* grads, void* scratch, size_t scratch_bytes,
                                   void* stream) {
  CpDims sh;
  if (cpdims(sh, L, dims, R) || !T || !W || !gl || !grads || !scratch)
    return tfx_set_error(TFX_STATUS_ERR_ARG, "cp_fit_backward args");
  mg::Outs o = {};
  o.rows = 1;
  for (int l = 0; l < L; ++l) o.p[l] = grads[l];
  return fit_grad(dtype, T, sh, W, gl, o, scratch, scratch_bytes, (cudaStream_t)stream);
}
