// MTTKRPs of a dense tensor (GaussNewton.py:401-427, the product at 411-423):
//
//   tfx_mttkrp      M_l = T_(l) (KR of the other factors), one mode
//   tfx_mttkrp_all  every mode at once
//
// Both are made of GEMMs whose rows are a group of modes (mttkrp_gemm.cuh): the
// product X_G[g, r] = sum over the modes outside G, and for a group of several
// modes the small contractions that take X_G to each of them,
//   M_m[i, r] = sum_{g: g_m = i} X_G[g, r] prod_{o in G, o != m} W_o[g_o, r].
// For every mode at once the modes are cut in two halves and the tensor is read
// twice instead of L times; a single short mode takes the first or the last
// modes as its group, so that its GEMM has rows enough.  Which group, and
// whether the halves beat the modes one by one, is decided by the estimate in
// gemm_us / modes_us.
#include <algorithm>

#include "mttkrp_gemm.cuh"
#include "tfx_capi_internal.h"

namespace tfx {

// Any shape with a scratch of one D x R partial or more: 64 x 64 tiles, the
// Khatri-Rao rows generated in shared memory.  Callers whose scratch is below
// what the GEMM asks for come here.
template <class T, int TS>
__global__ void __launch_bounds__(TFX_THREADS) k_mttkrp(const T* __restrict__ Tt, const T* __restrict__ W, CpDims sh,
                                                        int l, int ksplit, T* __restrict__ part) {
  using TL = Tile<TS, TS>;
  __shared__ T sA[TFX_BK * TL::LDA];
  __shared__ T sB[TFX_BK * TL::LDB];
  __shared__ long long sBase[TFX_BK];
  __shared__ int sIdx[TFX_BK * TFX_MAX_ORDER];
  const int L = sh.L, R = sh.R, D = sh.d[l];
  long long P = 1, Q = 1;
  for (int m = 0; m < l; ++m) P *= sh.d[m];
  for (int m = l + 1; m < L; ++m) Q *= sh.d[m];
  const int tilesM = (D + TL::BM - 1) / TL::BM;
  const int m0 = (blockIdx.x % tilesM) * TL::BM;
  const int n0 = (blockIdx.x / tilesM) * TL::BN;
  const long long K = P * Q;
  const long long kb = K * blockIdx.y / ksplit, ke = K * (blockIdx.y + 1) / ksplit;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  T acc[TS][TS];
  tile_zero<T, TS, TS>(acc);
  for (long long k0 = kb; k0 < ke; k0 += TFX_BK) {
    const int kc = (int)min((long long)TFX_BK, ke - k0);
    if (tid < kc) {
      // k = p*Q + q; p and q decompose into the indices of the other modes
      long long k = k0 + tid, q = k % Q, p = k / Q, base = 0, stride = 1;
      for (int m = L - 1; m > l; --m) {
        const long long im = q % sh.d[m];
        q /= sh.d[m];
        sIdx[tid * TFX_MAX_ORDER + m] = (int)im;
        base += im * stride;
        stride *= sh.d[m];
      }
      stride *= D;
      for (int m = l - 1; m >= 0; --m) {
        const long long im = p % sh.d[m];
        p /= sh.d[m];
        sIdx[tid * TFX_MAX_ORDER + m] = (int)im;
        base += im * stride;
        stride *= sh.d[m];
      }
      sBase[tid] = base;
    }
    __syncthreads();
    for (int e = tid; e < TFX_BK * TL::BM; e += TFX_THREADS) {
      int kk, mm;
      if (Q > 1) {
        mm = e / TFX_BK;
        kk = e - mm * TFX_BK;
      } else {
        kk = e / TL::BM;
        mm = e - kk * TL::BM;
      }
      sA[kk * TL::LDA + mm] = (kk < kc && m0 + mm < D) ? __ldg(Tt + sBase[kk] + (long long)(m0 + mm) * Q) : T(0);
    }
    for (int e = tid; e < TFX_BK * TL::BN; e += TFX_THREADS) {
      const int kk = e / TL::BN, nn = e - kk * TL::BN;
      T v = T(0);
      if (kk < kc && n0 + nn < R) {
        v = T(1);
        for (int m = L - 1; m >= 0; --m)
          if (m != l) v *= W[sh.off[m] + (n0 + nn) * sh.d[m] + sIdx[kk * TFX_MAX_ORDER + m]];
      }
      sB[kk * TL::LDB + nn] = v;
    }
    __syncthreads();
    tile_fma<T, TS, TS>(sA, sB, acc, kc);
    __syncthreads();
  }
  T* out = part + (size_t)blockIdx.y * D * R;
#pragma unroll
  for (int u = 0; u < TS; ++u)
#pragma unroll
    for (int v = 0; v < TS; ++v) {
      const int i = m0 + ty + 16 * u, r = n0 + tx + 16 * v;
      if (i < D && r < R) out[(size_t)r * D + i] = acc[u][v];
    }
}

template <class T>
__global__ void k_sum_parts(const T* __restrict__ part, long long n, int ks, T* __restrict__ out) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    Acc<T> s;
    for (int k = 0; k < ks; ++k) s.add(part[(size_t)k * n + i]);
    out[i] = (T)s.value();
  }
}

namespace mg {

// For every mode m of the group (or the one asked for) the Khatri-Rao rows of
// the group's other modes, [D / d_m][ldp], one after the other.
template <class T>
__global__ void __launch_bounds__(256) k_others(const T* __restrict__ W, const __grid_constant__ CpDims sh, int g0,
                                                int g1, int only, unsigned D, int ldp, T* __restrict__ kr) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned row = (unsigned)(e / ldp);
  const int r = (int)(e - (long long)row * ldp);
  int m = only >= 0 ? only : g0;
  if (only < 0)
    while (m < g1 && row >= D / sh.d[m]) row -= D / sh.d[m++];
  if (m >= g1 || row >= D / sh.d[m]) return;
  T v = T(0);
  if (r < sh.R) {
    v = T(1);
    unsigned rem = row;
    for (int o = g1 - 1; o >= g0; --o) {
      if (o == m) continue;
      const unsigned q = rem / (unsigned)sh.d[o];
      v *= W[sh.off[o] + (long long)r * sh.d[o] + (rem - q * sh.d[o])];
      rem = q;
    }
  }
  kr[e] = v;
}

// M_m of every mode m of the group from X_G: a CTA takes one index i of one mode
// and 32 columns, its MY rows of threads the positions j of the other modes in
// turn, summed in compensated FP32 and in a fixed order.  Bound by reading X
// from L2 once per mode (two coalesced reads a product): 46 us for both modes of
// a 512 x 512 group at R = 50; 131 us when every position was taken apart by
// divisions.
constexpr int MY = 16;

template <class T>
__global__ void __launch_bounds__(32 * MY) k_modes(const T* __restrict__ X, const T* __restrict__ kr,
                                                   const __grid_constant__ CpDims sh, int g0, int g1, int only,
                                                   unsigned D, int ldp, const __grid_constant__ Outs out) {
  __shared__ T hi[MY][32], lo[MY][32];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int c = blockIdx.y * 32 + x;
  unsigned i = blockIdx.x;
  int m = only >= 0 ? only : g0;
  const T* kp = kr + c;
  if (only < 0)
    while (i >= (unsigned)sh.d[m]) {
      kp += (size_t)(D / sh.d[m]) * ldp;
      i -= sh.d[m++];
    }
  T* o = (T*)out.p[m];
  if (!o) return;
  const unsigned dm = sh.d[m], n = D / dm;
  unsigned inner = 1;
  for (int q = m + 1; q < g1; ++q) inner *= sh.d[q];
  Acc<T> s;
  if (c < ldp) {
    if (inner == n || inner == 1) {  // the first or the last mode: a fixed stride
      const size_t step = (size_t)(inner == 1 ? dm : 1) * ldp;
      const T* xp = X + (size_t)(inner == 1 ? i : i * n) * ldp + c;
#pragma unroll 8
      for (unsigned j = y; j < n; j += MY) s.add(xp[j * step] * kp[(size_t)j * ldp]);
    } else {
#pragma unroll 8
      for (unsigned j = y; j < n; j += MY) {
        const unsigned h = j / inner;
        s.add(X[((size_t)(h * dm + i) * inner + (j - h * inner)) * ldp + c] * kp[(size_t)j * ldp]);
      }
    }
  }
  hi[y][x] = s.hi_or_v();
  lo[y][x] = s.lo_or_0();
  __syncthreads();
  if (y == 0 && c < sh.R) {
    Acc<T> t;
#pragma unroll
    for (int q = 0; q < MY; ++q) {
      t.add(hi[q][x]);
      if (sizeof(T) == 4) t.add(lo[q][x]);
    }
    o[out.rows ? (size_t)i * sh.R + c : (size_t)c * dm + i] = (T)t.value();
  }
}

// One group's work: the GEMM, and for several modes the contractions.
struct Group {
  Plan p;
  size_t x_bytes, w_bytes;
  double us;
  size_t total() const { return p.total() + x_bytes + w_bytes; }
};

// Microseconds of the GEMM and of the contractions, from the rates measured on
// GB300 (40 and 0.9 TFLOP/s on padded work; Khatri-Rao blocks written at 1 TB/s,
// partials and X read at 2 TB/s; about 3 us a launch).  The contractions' CTAs, one
// an index and 32 columns, take 1.5 us each however few their positions, 608 at a
// time: beyond a few thousand they count (39 x 51351 x 4 at R = 14, the middle mode
// from the last two 164 us, by itself 78).
static double gemm_us(const Plan& p, int es, double N) {
  const double dp = es == 4 ? (double)p.tilesM * 32 * p.WM : (double)((p.w.D + 7) / 8 * 8);
  const double flop = 2.0 * N / p.w.D * dp * ((double)p.rowsF / p.w.dF) * p.w.ldp;
  return 8.0 + flop / (es == 4 ? 40e6 : 0.9e6) + (double)(p.rowsF + p.w.nO) * p.w.ldp * es / 1e6 +
         (p.ks > 1 ? (double)p.ks * p.w.D * p.w.ldp * es / 2e6 : 0.0);
}

static Group group(int es, const CpDims& sh, int g0, int g1, int only, int sms) {
  Group g;
  g.p = plan(es, sh, g0, g1, sms);
  double N = 1.0;
  for (int m = 0; m < sh.L; ++m) N *= sh.d[m];
  g.us = gemm_us(g.p, es, N);
  g.x_bytes = g.w_bytes = 0;
  if (g1 - g0 > 1) {
    const long long D = g.p.w.D;
    long long rows = 0, idx = 0, least = D;
    for (int m = g0; m < g1; ++m)
      if (only < 0 || only == m) {
        rows += D / sh.d[m];
        idx += sh.d[m];
        least = std::min<long long>(least, sh.d[m]);
      }
    const double per = (double)D * g.p.w.ldp * es, steps = (double)(D / least) / MY;
    const double ctas = (double)idx * ((g.p.w.ldp + 31) / 32);
    g.us += 6.0 + ((only < 0 ? g1 - g0 : 1) + 1) * per / 2e6 + 0.1 * steps + std::max(0.0, ctas - 4096.0) * (1.5 / 608);
    if (D > 0x7fffffffLL / g.p.w.ldp) g.us = 1e30;
    g.x_bytes = (size_t)((D * g.p.w.ldp * es + 255) & ~255LL);
    g.w_bytes = (size_t)((rows * g.p.w.ldp * es + 255) & ~255LL);
  }
  return g;
}

// the group of one mode: the mode alone, or the first or the last modes with it
static Group best_single(int es, const CpDims& sh, int l, int sms) {
  Group best = group(es, sh, l, l + 1, l, sms);
  for (int g1 = l + 1; g1 < sh.L; ++g1)
    if (g1 > 1) {
      const Group g = group(es, sh, 0, g1, l, sms);
      if (g.us < best.us) best = g;
    }
  for (int g0 = 1; g0 <= l; ++g0)
    if (sh.L - g0 > 1) {
      const Group g = group(es, sh, g0, sh.L, l, sms);
      if (g.us < best.us) best = g;
    }
  return best;
}

// where the modes are cut in two halves; 0: mode by mode
static int best_cut(int es, const CpDims& sh, int sms) {
  double one = 0.0, least = 1e30;
  int cut = 0;
  for (int l = 0; l < sh.L; ++l) one += group(es, sh, l, l + 1, l, sms).us;
  for (int s = 1; s < sh.L; ++s) {
    const double t = group(es, sh, 0, s, -1, sms).us + group(es, sh, s, sh.L, -1, sms).us;
    if (t < least) {
      least = t;
      cut = s;
    }
  }
  return least < one ? cut : 0;
}

// the group's modes (only >= 0: that one) into out
template <class T>
static cudaError_t run_group(const Group& g, const T* X, const T* W, const CpDims& sh, int only, const Outs& out,
                             char* scratch, cudaStream_t st, int* launches) {
  const int g0 = g.p.g0, g1 = g.p.g1;
  bool any = false;
  for (int m = g0; m < g1; ++m) any = any || (out.p[m] && (only < 0 || only == m));
  if (!any) return cudaSuccess;
  if (g1 - g0 == 1) {
    const Out<T> o = {(T*)out.p[g0], out.rows ? sh.R : 1, out.rows ? 1 : sh.d[g0]};
    return run<T>(g.p, X, W, sh, o, scratch, st, launches);
  }
  T* XG = (T*)(scratch + g.p.total());
  T* kr = (T*)(scratch + g.p.total() + g.x_bytes);
  cudaError_t e = run<T>(g.p, X, W, sh, Out<T>{XG, 0, 0}, scratch, st, launches);
  if (e != cudaSuccess) return e;
  const unsigned D = (unsigned)g.p.w.D;
  long long rows = 0, idx = 0;
  for (int m = g0; m < g1; ++m)
    if (only < 0 || only == m) {
      rows += D / sh.d[m];
      idx += sh.d[m];
    }
  const int ldp = g.p.w.ldp;
  k_others<T><<<(unsigned)((rows * ldp + 255) / 256), 256, 0, st>>>(W, sh, g0, g1, only, D, ldp, kr);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  k_modes<T><<<dim3((unsigned)idx, (unsigned)((ldp + 31) / 32)), 32 * MY, 0, st>>>(XG, kr, sh, g0, g1, only, D, ldp,
                                                                                   out);
  *launches += 2;
  return cudaGetLastError();
}

static cudaError_t run_group(int dtype, const Group& g, const void* X, const void* W, const CpDims& sh, int only,
                             const Outs& out, void* scratch, cudaStream_t st, int* launches) {
  if (dtype == TFX_F64)
    return run_group<double>(g, (const double*)X, (const double*)W, sh, only, out, (char*)scratch, st, launches);
  return run_group<float>(g, (const float*)X, (const float*)W, sh, only, out, (char*)scratch, st, launches);
}

}  // namespace mg
}  // namespace tfx

using namespace tfx;

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

// splits of the general kernel
static int mttkrp_splits(long long K, int D, int R, int dtype) {
  const long long tiles = (long long)((D + 63) / 64) * ((R + 63) / 64);
  long long ks = (4LL * nsm() + tiles - 1) / tiles;
  ks = std::min<long long>(ks, std::max<long long>(1, K / (dtype == TFX_F64 ? 32 : 128)));
  return (int)std::max<long long>(1, std::min<long long>(ks, 128));
}

extern "C" size_t tfx_mttkrp_scratch_bytes(int dtype, int L, const int* dims, int R, int mode) {
  CpDims sh;
  if (cpdims(sh, L, dims, R) || mode < 0 || mode >= L) return 0;
  return mg::best_single(dtype == TFX_F64 ? 8 : 4, sh, mode, nsm()).total();
}

extern "C" int tfx_mttkrp(int dtype, const void* T, int L, const int* dims, int R, const void* W, int mode, void* out,
                          void* scratch, size_t scratch_bytes, void* stream) {
  CpDims sh;
  if (cpdims(sh, L, dims, R) || !T || !W || !out || !scratch || mode < 0 || mode >= L)
    return tfx_set_error(TFX_STATUS_ERR_ARG, "mttkrp args");
  const size_t es = dtype == TFX_F64 ? 8 : 4;
  cudaStream_t st = (cudaStream_t)stream;
  const mg::Group g = mg::best_single((int)es, sh, mode, nsm());
  if (g.total() <= scratch_bytes && ((uintptr_t)scratch & 15) == 0) {
    int nl = 0;
    mg::Outs o = {};
    o.p[mode] = out;
    const cudaError_t e = mg::run_group(dtype, g, T, W, sh, mode, o, scratch, st, &nl);
    if (e != cudaSuccess) return tfx_set_cuda_error(e, "mttkrp");
    tfx_count_launch(nl);
    return TFX_STATUS_OK;
  }
  // a smaller scratch: the general kernel, as many splits as fit
  long long K = 1;
  for (int m = 0; m < L; ++m)
    if (m != mode) K *= dims[m];
  const int D = dims[mode];
  int ks = mttkrp_splits(K, D, R, dtype);
  ks = (int)std::min<size_t>((size_t)ks, scratch_bytes / ((size_t)D * R * es));
  if (ks < 1) return tfx_set_error(TFX_STATUS_ERR_ARG, "mttkrp scratch too small");
  const dim3 grid(((D + 63) / 64) * ((R + 63) / 64), ks);
  const long long n = (long long)D * R;
  const int rb = (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, 4LL * nsm()));
  if (dtype == TFX_F32) {
    k_mttkrp<float, 4><<<grid, TFX_THREADS, 0, st>>>((const float*)T, (const float*)W, sh, mode, ks, (float*)scratch);
    k_sum_parts<float><<<rb, 256, 0, st>>>((const float*)scratch, n, ks, (float*)out);
  } else {
    k_mttkrp<double, 4><<<grid, TFX_THREADS, 0, st>>>((const double*)T, (const double*)W, sh, mode, ks,
                                                      (double*)scratch);
    k_sum_parts<double><<<rb, 256, 0, st>>>((const double*)scratch, n, ks, (double*)out);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return tfx_set_cuda_error(e, "mttkrp");
  tfx_count_launch(2);
  return TFX_STATUS_OK;
}

extern "C" size_t tfx_mttkrp_all_scratch_bytes(int dtype, int L, const int* dims, int R) {
  CpDims sh;
  if (cpdims(sh, L, dims, R)) return 0;
  const int es = dtype == TFX_F64 ? 8 : 4, s = mg::best_cut(es, sh, nsm());
  size_t n = 0;
  if (s == 0)
    for (int l = 0; l < L; ++l) n = std::max(n, mg::best_single(es, sh, l, nsm()).total());
  else
    n = std::max(mg::group(es, sh, 0, s, -1, nsm()).total(), mg::group(es, sh, s, L, -1, nsm()).total());
  return n + 256;  // to align within
}

int tfx::mg::all_modes(int dtype, const void* T, const CpDims& sh, const void* W, const Outs& out, void* scratch,
                       size_t scratch_bytes, cudaStream_t st) {
  const int es = dtype == TFX_F64 ? 8 : 4, s = best_cut(es, sh, nsm());
  const size_t skip = (256 - ((uintptr_t)scratch & 255)) & 255;
  scratch_bytes = scratch_bytes > skip ? scratch_bytes - skip : 0;
  scratch = (char*)scratch + skip;
  int nl = 0;
  for (int h = 0; h < (s ? 2 : sh.L); ++h) {  // two halves, or mode by mode
    const Group g = s ? group(es, sh, h ? s : 0, h ? sh.L : s, -1, nsm()) : best_single(es, sh, h, nsm());
    if (g.total() > scratch_bytes) return tfx_set_error(TFX_STATUS_ERR_ARG, "mttkrp_all scratch too small");
    const cudaError_t e = run_group(dtype, g, T, W, sh, s ? -1 : h, out, scratch, st, &nl);
    if (e != cudaSuccess) return tfx_set_cuda_error(e, "mttkrp_all");
  }
  tfx_count_launch(nl);
  return TFX_STATUS_OK;
}

extern "C" int tfx_mttkrp_all(int dtype, const void* T, int L, const int* dims, int R, const void* W, void* const* out,
                              int row_major, void* scratch, size_t scratch_bytes, void* stream) {
  CpDims sh;
  if (cpdims(sh, L, dims, R) || !T || !W || !out || !scratch)
    return tfx_set_error(TFX_STATUS_ERR_ARG, "mttkrp_all args");
  mg::Outs o = {};
  o.rows = row_major;
  for (int l = 0; l < L; ++l) o.p[l] = out[l];
  return mg::all_modes(dtype, T, sh, W, o, scratch, scratch_bytes, (cudaStream_t)stream);
}
