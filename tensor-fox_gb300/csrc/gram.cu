// The Gram S_(l) S_(l)^T of a C-order tensor viewed as (P, D, Q), in the working
// precision (tfx_mode_gram; Compression.py:192-237: the Gram route replaces the
// randomized SVD's streaming passes over the unfolding):
//   G[i, j] = sum_k A(i, k) A(j, k), A(i, k) = S[p D Q + i Q + q], k = p Q + q.
//
// Upper tiles only, split over k; partials summed in FP64 and mirrored by
// k_gram_sum.
#include <algorithm>

#include "tfx_capi_internal.h"
#include "tfx_common.cuh"

namespace tfx {
namespace gram {

constexpr int BK = 32, NT = 128;
typedef unsigned long long f2;  // two floats in a register pair

template <int BYTES>
__device__ __forceinline__ void cp(void* s, const void* g, bool ok) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g),
                 "r"(ok ? 16 : 0)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g),
                 "r"(ok ? BYTES : 0), "n"(BYTES)
                 : "memory");
}
__device__ __forceinline__ void fma2(f2& c, f2 a, f2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }
__device__ __forceinline__ void add2(f2& c, f2 a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(c) : "l"(a)); }
__device__ __forceinline__ f2 dup2(float a) {
  f2 d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(a));
  return d;
}
__device__ __forceinline__ float2 unpack2(f2 v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}

// tile pair index -> (bi, bj), bi <= bj
__device__ __forceinline__ void tile_pair(int t, int nt, int& bi, int& bj) {
  bi = 0;
  while (t >= nt - bi) {
    t -= nt - bi;
    ++bi;
  }
  bj = bi + t;
}

// One thread's part in bringing the rows [r0, r0 + ROWS) of successive chunks
// by cp.async.  LAST (Q == 1): [k][ROWS] (a k's rows lie together); else
// [row][ST].  Copies of 16 bytes (VEC) or of one element; rows past D and steps
// past K are zero.  The source pointer is carried from chunk to chunk: the index
// arithmetic of a fresh one cost a third of the instructions of the FP32 kernel.
template <class T, int ROWS, int ST, bool LAST, bool VEC>
struct Loader {
  static constexpr int PV = VEC ? 16 / (int)sizeof(T) : 1, CB = VEC ? 16 : (int)sizeof(T);
  // threads along the contiguous direction, and the copies a thread makes
  static constexpr int TX = LAST ? ROWS / PV : BK / PV, NU = ROWS * BK / PV / NT, TY = NT / TX;
  const T* S;    // a valid address for the copies that bring zeros
  const T* g;    // this thread's first source of the next chunk
  long long k, q, Q, K, stride, jump;
  int live;      // LAST: whether the row is inside; else how many of its rows are
  int dst;

  __device__ __forceinline__ void init(const T* S_, long long c, int r0, int D, long long Q_, long long K_) {
    S = S_;
    Q = Q_;
    K = K_;
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    if (LAST) {
      const int m = tx * PV;
      k = c * BK + ty;
      g = S + k * D + r0 + m;
      stride = D;
      live = r0 + m < D ? 1 : 0;
      dst = ty * ROWS + m;
    } else {
      k = c * BK + tx * PV;
      const long long p = k / Q;
      q = k - p * Q;
      g = S + p * D * Q + q + (long long)(r0 + ty) * Q;
      stride = Q;
      jump = (long long)(D - 1) * Q;
      live = D - r0 - ty <= 0 ? 0 : min(NU, (D - r0 - ty + TY - 1) / TY);
      dst = ty * ST + tx * PV;
    }
  }
  __device__ __forceinline__ void load(T* buf) {
    T* d = buf + dst;
    if (LAST) {
      if (live && k + BK - TY < K) {
#pragma unroll
        for (int u = 0; u < NU; ++u) cp<CB>(d + u * TY * ROWS, g + (long long)u * TY * stride, true);
      } else {
#pragma unroll 4
        for (int u = 0; u < NU; ++u) {
          const bool ok = live && k + u * TY < K;
          cp<CB>(d + u * TY * ROWS, ok ? g + (long long)u * TY * stride : S, ok);
        }
      }
      g += BK * stride;
    } else {
      if (live == NU && k < K) {
#pragma unroll
        for (int u = 0; u < NU; ++u) cp<CB>(d + u * TY * ST, g + (long long)u * TY * stride, true);
      } else {
#pragma unroll 4
        for (int u = 0; u < NU; ++u) {
          const bool ok = u < live && k < K;
          cp<CB>(d + u * TY * ST, ok ? g + (long long)u * TY * stride : S, ok);
        }
      }
      g += BK;
      q += BK;
      while (q >= Q) {
        q -= Q;
        g += jump;
      }
    }
    k += BK;
  }
};

// ---------------------------------------------------------------------------
// FP32: bound by the FP32 FMA rate.  64 x 64 tiles: two warps of 32 rows, and
// two that take the other half of each chunk's k; a lane holds 8 x 8 outputs.
// For K-contiguous rows (not the last mode) fma.rn.f32x2 takes two k at once:
// both operands are register pairs as they lie in shared memory, no moves, 16
// one-wavefront reads for 128 FMA instructions.  For the last mode, whose rows
// lie together, it takes two columns.  512 x 262144: 1.66 ms = 41 TFLOP/s on the
// upper triangle (1.79 with two steps unrolled; 6.3 with 4 x 4 thread tiles on scalar
// reads; 2.11 with each chunk's source addresses formed afresh).
// ---------------------------------------------------------------------------
constexpr int FST = BK + 4, FSTAGES = 3;
template <bool LAST>
constexpr int fsz() {
  return LAST ? BK * 64 : 64 * FST;
}

template <bool LAST, bool VEC>
__global__ void __launch_bounds__(NT, 2) k_gram_f32(const float* __restrict__ S, int D, long long Q, long long K,
                                                    float* __restrict__ part) {
  constexpr int SZ = fsz<LAST>();
  extern __shared__ __align__(16) float gsm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp & 1, wk = warp >> 1, lm = lane >> 3, ln = lane & 7;
  int bi, bj;
  tile_pair(blockIdx.x, (D + 63) / 64, bi, bj);
  const int i0 = bi * 64, j0 = bj * 64;
  const bool diag = bi == bj;
  const long long nch = (K + BK - 1) / BK;
  const long long cb = nch * blockIdx.y / gridDim.y, ce = nch * (blockIdx.y + 1) / gridDim.y;
  Loader<float, 64, FST, LAST, VEC> la, lb;
  la.init(S, cb, i0, D, Q, K);
  lb.init(S, cb, j0, D, Q, K);
  auto load = [&](int s) {
    la.load(gsm + s * 2 * SZ);
    if (!diag) lb.load(gsm + s * 2 * SZ + SZ);
  };
  // LAST: pairs of columns, 8 rows x 4 pairs, and a second set into which they
  // are added every 512 steps of a lane (its chain would be half the split; that
  // of a pair of k is a quarter); else pairs of k, 8 x 8
  constexpr int FC = 32;  // chunks
  f2 acc[8][LAST ? 4 : 8], sum[8][LAST ? 4 : 1];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < (LAST ? 4 : 8); ++j) {
      acc[i][j] = 0ull;
      if (LAST) sum[i][j & 3] = 0ull;
    }
  auto fold = [&]() {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        add2(sum[i][LAST ? j : 0], acc[i][j]);
        acc[i][j] = 0ull;
      }
  };
  int left = FC;
#pragma unroll
  for (int s = 0; s < FSTAGES - 1; ++s) {
    if (cb + s < ce) load(s);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  int stage = 0;
  for (long long c = cb; c < ce; ++c) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(FSTAGES - 2) : "memory");
    __syncthreads();  // chunk c is there; everyone is done with chunk c - 1
    if (c + FSTAGES - 1 < ce) load(stage == 0 ? FSTAGES - 1 : stage - 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const float* A = gsm + stage * 2 * SZ;
    const float* B = diag ? A : A + SZ;
    if (LAST) {
      const float* ap = A + wk * 16 * 64 + wm * 32 + 4 * lm;
      const float* bp = B + wk * 16 * 64 + 4 * ln;
#pragma unroll 4
      for (int k = 0; k < 16; ++k) {
        const float4 a0 = *reinterpret_cast<const float4*>(ap + k * 64);
        const float4 a1 = *reinterpret_cast<const float4*>(ap + k * 64 + 16);
        const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(bp + k * 64);
        const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(bp + k * 64 + 32);
        const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const f2 a = dup2(av[i]);
          fma2(acc[i][0], a, b0.x);
          fma2(acc[i][1], a, b0.y);
          fma2(acc[i][2], a, b1.x);
          fma2(acc[i][3], a, b1.y);
        }
      }
      if (--left == 0) {
        fold();
        left = FC;
      }
    } else {
      const float* ap = A + (wm * 32 + lm) * FST + wk * 16;
      const float* bp = B + ln * FST + wk * 16;
#pragma unroll 1
      for (int k4 = 0; k4 < 16; k4 += 4) {
        ulonglong2 a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(ap + 4 * i * FST + k4);
#pragma unroll
        for (int j = 0; j < (LAST ? 4 : 8); ++j) {
          const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(bp + 8 * j * FST + k4);
#pragma unroll
          for (int i = 0; i < 8; ++i) fma2(acc[i][j], a[i].x, b.x);
#pragma unroll
          for (int i = 0; i < 8; ++i) fma2(acc[i][j], a[i].y, b.y);
        }
      }
    }
    if (++stage == FSTAGES) stage = 0;
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  if (LAST) fold();
  // the second k half's sums into the first's
  float v[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < (LAST ? 4 : 8); ++j) {
      const float2 t = unpack2(LAST ? sum[i][j & 3] : acc[i][j]);
      if (LAST) {
        v[i][2 * (j & 3)] = t.x;
        v[i][2 * (j & 3) + 1] = t.y;
      } else {
        v[i][j] = t.x + t.y;
      }
    }
  __syncthreads();
  if (wk == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) gsm[(i * 8 + j) * 64 + (tid & 63)] = v[i][j];
  }
  __syncthreads();
  if (wk == 1) return;
  float* out = part + (size_t)blockIdx.y * D * D;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = i0 + wm * 32 + (LAST ? 16 * (i >> 2) + 4 * lm + (i & 3) : 4 * i + lm);
    if (r >= D) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int cidx = j0 + (LAST ? 32 * (j >> 2) + 4 * ln + (j & 3) : 8 * j + ln);
      if (cidx < D) out[(size_t)r * D + cidx] = v[i][j] + gsm[(i * 8 + j) * 64 + tid];
    }
  }
}

// ---------------------------------------------------------------------------
// FP64: bound by the FP64 pipe, so no work outside the upper triangle: 32 x 32
// tiles, a warp 8 rows x 32 columns as 8 groups of 4, of which it multiplies
// those that reach the diagonal and lie inside the matrix.  150 x 18330: 0.44
// ms = 0.95 TFLOP/s on the upper triangle; 0.91 ms with 64 x 64 tiles.
// ---------------------------------------------------------------------------
constexpr int DST = BK + 2;
template <bool LAST>
constexpr int dsz() {
  return LAST ? BK * 32 : 32 * DST;
}

template <bool LAST, bool VEC>
__global__ void __launch_bounds__(NT, 5) k_gram_f64(const double* __restrict__ S, int D, long long Q, long long K,
                                                    double* __restrict__ part) {
  constexpr int SZ = dsz<LAST>();
  extern __shared__ __align__(16) double gdm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lm = lane >> 2, ln = lane & 3;
  int bi, bj;
  tile_pair(blockIdx.x, (D + 31) / 32, bi, bj);
  const int i0 = bi * 32, j0 = bj * 32;
  const bool diag = bi == bj;
  const int strip = (warp + blockIdx.y) & 3;  // dealt in turn, so that the SM's quarters share the idle ones
  const int r = i0 + 8 * strip;
  const int glo = diag ? 2 * strip : 0, ghi = r < D ? min(8, (D - j0 + 3) / 4) : 0;
  const long long nch = (K + BK - 1) / BK;
  const long long cb = nch * blockIdx.y / gridDim.y, ce = nch * (blockIdx.y + 1) / gridDim.y;
  Loader<double, 32, DST, LAST, VEC> la, lb;
  la.init(S, cb, i0, D, Q, K);
  lb.init(S, cb, j0, D, Q, K);
  auto load = [&](int s) {
    la.load(gdm + s * 2 * SZ);
    if (!diag) lb.load(gdm + s * 2 * SZ + SZ);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  double acc[8];
#pragma unroll
  for (int g = 0; g < 8; ++g) acc[g] = 0.0;
  if (cb < ce) load(0);
  for (long long c = cb; c < ce; ++c) {
    const int s = (int)((c - cb) & 1);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    if (c + 1 < ce) load(s ^ 1);
    const double* A = gdm + s * 2 * SZ;
    const double* B = diag ? A : A + SZ;
    const int kc = (int)min((long long)BK, K - c * BK);
    // four steps at a time under one branch a pair of groups: an FMA that is only
    // predicated off still takes its turn on the pipe (the chunk's tail is zero)
    for (int k = 0; k < kc; k += 4) {
      double a[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) a[u] = LAST ? A[(k + u) * 32 + 8 * strip + lm] : A[(8 * strip + lm) * DST + k + u];
#pragma unroll
      for (int g = 0; g < 8; g += 2) {
        if (g < glo || g >= ghi) continue;
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int h = g; h < g + 2; ++h)
            acc[h] = fma(a[u], LAST ? B[(k + u) * 32 + 4 * h + ln] : B[(4 * h + ln) * DST + k + u], acc[h]);
      }
    }
  }
  const int row = r + lm;
  if (row >= D) return;
  double* out = part + (size_t)blockIdx.y * D * D + (size_t)row * D + j0;
#pragma unroll
  for (int g = 0; g < 8; ++g)
    if (g >= glo && g < ghi && j0 + 4 * g + ln < D) out[4 * g + ln] = acc[g];
}

// G = the sum of the ks partials' upper triangle, in FP64, and its mirror.  A
// CTA takes 8 rows x 32 columns of a 32 x 32 block on or above the diagonal, four
// groups of threads a quarter of the partials each, added in order.
template <class T>
__global__ void __launch_bounds__(1024) k_gram_sum(const T* __restrict__ part, int D, int ks, T* __restrict__ G) {
  __shared__ double red[3][8][32];
  int bi, bj;
  tile_pair(blockIdx.x >> 2, (D + 31) / 32, bi, bj);
  const int x = threadIdx.x & 31, y = (threadIdx.x >> 5) & 7, z = threadIdx.x >> 8;
  const long long n = (long long)D * D;
  const int i = bi * 32 + 8 * (blockIdx.x & 3) + y, j = bj * 32 + x;
  const bool on = i < D && j < D && i <= j;
  double s = 0.0;
  if (on) {
    const T* p = part + (size_t)i * D + j;
#pragma unroll 8
    for (int k = ks * z / 4; k < ks * (z + 1) / 4; ++k) s += (double)__ldcs(p + (size_t)k * n);
  }
  if (z > 0) red[z - 1][y][x] = s;
  __syncthreads();
  if (z == 0 && on) {
    s = ((s + red[0][y][x]) + red[1][y][x]) + red[2][y][x];
    G[(size_t)i * D + j] = (T)s;
    if (j > i) G[(size_t)j * D + i] = (T)s;
  }
}

static int sms() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n < 1) n = 1;
  }
  return n;
}

static long long tiles(int dtype, int D) {
  const long long nt = dtype == TFX_F64 ? (D + 31) / 32 : (D + 63) / 64;
  return nt * (nt + 1) / 2;
}

// Splits: whole waves of the resident CTAs (2 a SM in FP32, 5 in FP64), at
// least 2 (FP32) or 1 (FP64) chunks each; in FP32 a second wave where a quarter of
// the split, a lane's chain but in the last mode's form, is above 4096; in FP64 at
// least 4 while the tiles are within 16 waves, so that the SMs' shares of them
// come out even (1805 x 1464: 1081 tiles 4.63 ms in one split, 3.28 in four; 3000 x
// 1250 4.65 and 4.02, 5000 x 900 3.74 and 3.58).
static long long splits(int dtype, long long K, int D) {
  const long long t = tiles(dtype, D), slots = (long long)sms() * (dtype == TFX_F64 ? 5 : 2);
  long long ks = std::max<long long>(1, slots / t);
  if (dtype != TFX_F64 && K / ks > 4 * 4096) ks = std::max<long long>(ks, 2 * slots / t);
  if (dtype == TFX_F64 && t <= 16 * slots) ks = std::max<long long>(ks, 4);
  ks = std::min(ks, std::max<long long>(1, K / (BK * (dtype == TFX_F64 ? 1 : 2))));
  return std::min<long long>(ks, 1024);
}

template <bool LAST, bool VEC>
static cudaError_t launch_f32(dim3 grid, const void* S, int D, long long Q, long long K, void* part, cudaStream_t st) {
  const int sm = FSTAGES * 2 * 4 * fsz<LAST>();
  cudaError_t e = cudaFuncSetAttribute(k_gram_f32<LAST, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  if (e != cudaSuccess) return e;
  k_gram_f32<LAST, VEC><<<grid, NT, sm, st>>>((const float*)S, D, Q, K, (float*)part);
  return cudaGetLastError();
}

template <bool LAST, bool VEC>
static cudaError_t launch_f64(dim3 grid, const void* S, int D, long long Q, long long K, void* part, cudaStream_t st) {
  k_gram_f64<LAST, VEC><<<grid, NT, 2 * 2 * 8 * dsz<LAST>(), st>>>((const double*)S, D, Q, K, (double*)part);
  return cudaGetLastError();
}

}  // namespace gram
}  // namespace tfx

using namespace tfx;

extern "C" size_t tfx_mode_gram_scratch_bytes(int dtype, long long P, int D, long long Q) {
  return (size_t)gram::splits(dtype, P * Q, D) * D * D * (dtype == TFX_F64 ? 8 : 4);
}

extern "C" int tfx_mode_gram(int dtype, const void* S, long long P, int D, long long Q, void* G, void* scratch,
                             size_t scratch_bytes, void* stream) {
  if (!S || !G || !scratch || P < 1 || D < 1 || Q < 1) return tfx_set_error(TFX_STATUS_ERR_ARG, "mode_gram args");
  const size_t es = dtype == TFX_F64 ? 8 : 4;
  const long long K = P * Q;
  const int ks = (int)std::min<long long>(gram::splits(dtype, K, D), (long long)(scratch_bytes / ((size_t)D * D * es)));
  if (ks < 1) return tfx_set_error(TFX_STATUS_ERR_ARG, "mode_gram scratch too small");
  cudaStream_t st = (cudaStream_t)stream;
  const dim3 grid((unsigned)gram::tiles(dtype, D), (unsigned)ks);
  const bool last = Q == 1;
  const int vec = ((uintptr_t)S & 15) == 0 && (last ? D : Q) % (16 / (long long)es) == 0;
  const unsigned nb = (unsigned)(4 * gram::tiles(TFX_F64, D));
  cudaError_t e;
  if (dtype == TFX_F32) {
    e = last ? (vec ? gram::launch_f32<true, true>(grid, S, D, Q, K, scratch, st)
                    : gram::launch_f32<true, false>(grid, S, D, Q, K, scratch, st))
             : (vec ? gram::launch_f32<false, true>(grid, S, D, Q, K, scratch, st)
                    : gram::launch_f32<false, false>(grid, S, D, Q, K, scratch, st));
    if (e != cudaSuccess) return tfx_set_cuda_error(e, "mode_gram");
    gram::k_gram_sum<float><<<nb, 1024, 0, st>>>((const float*)scratch, D, ks, (float*)G);
  } else {
    e = last ? (vec ? gram::launch_f64<true, true>(grid, S, D, Q, K, scratch, st)
                    : gram::launch_f64<true, false>(grid, S, D, Q, K, scratch, st))
             : (vec ? gram::launch_f64<false, true>(grid, S, D, Q, K, scratch, st)
                    : gram::launch_f64<false, false>(grid, S, D, Q, K, scratch, st));
    if (e != cudaSuccess) return tfx_set_cuda_error(e, "mode_gram");
    gram::k_gram_sum<double><<<nb, 1024, 0, st>>>((const double*)scratch, D, ks, (double*)G);
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return tfx_set_cuda_error(e, "gram_sum");
  tfx_count_launch(2);
  return TFX_STATUS_OK;
}
