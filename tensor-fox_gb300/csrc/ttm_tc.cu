// Mode product with U^T on the 5th-generation tensor cores, 3xTF32 with FP32
// accumulation (precision 'mixed'):
//
//   out[p, j, q] = sum_d U[d, j] T[p, d, q]
//
// the MLSVD's truncation step (Compression.py:152-156, where the sequential
// method forms U_l^T S_(l) as Sigma V^T, and :170-173 with
// MultilinearAlgebra.py:72-105 multilin_mult for the classic one).  The
// contraction index d is the strided one in memory (T[p, d, q] has q
// contiguous), so the tensor is the A operand with M = q and K = d; U^T (n x D,
// n <= 64) is the B operand.
// Both are split x = x_hi + x_lo (x_hi: 13 low mantissa bits cleared, exact
// in TF32) and the product is A_hi B_hi + A_hi B_lo + A_lo B_hi, so the core
// keeps FP32 accuracy (a single TF32 pass moved the headline CPD's final
// error by 1%).
//
// A persistent CTA takes 256-wide q tiles, two halves of 128 rows.  Per tile
// the D axis runs in chunks of 32:
//   * warp 0 (producer) brings each chunk's 32 x 256 tensor tile and the
//     chunk's 64 x 32 block of U^T (K-major SWIZZLE_128B) by TMA into a
//     four-stage ring (a stage is refilled once the converters read it);
//   * warps 2-9 (converters), four to a half, take one row q a thread: its 32
//     values, split hi / lo, go to the thread's lane of tensor memory (one
//     column a d: the transposition costs nothing), and together they split
//     the U^T block in place of layout into a two-stage ring of shared memory;
//   * warp 1 issues tcgen05.mma kind::tf32 (M = 128, N = 64, K = 8; A from
//     tensor memory), three per K step and half, and commits each operand stage
//     back to the converters;
//   * warps 10-13 read a finished tile's accumulators (tcgen05.ld) and store
//     out[p, j, q0 + row] for j < n while the next tile's products go to the
//     other pair of accumulators.
// Tensor memory: 4 accumulators and 2 x 2 operands (hi | lo) of 64 columns.
// With A staged in shared memory as well the chunk of 128 rows moved 1340
// wavefronts of 128 bytes (A written and read three times, B read three times)
// and shared memory bound the kernel (512^3, n 50: 230 us, 2.5 TB/s).  From
// tensor memory it takes 165 us (3.6 TB/s; 107 without any product): an
// instruction takes about 117 cycles whether N is 32 or 64, three a K step.  Two
// (A_hi with both parts of B at N = 128) ran in 148 us, but the separate sum of
// the small terms moved the core by 1e-5 of its norm.
// Every wait is bounded; a wait that runs out sets *err, the CTA stops, waits
// (bounded) for its copies and products in flight and frees TMEM.
#include <cuda.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "tfx_capi_internal.h"
#include "tfx_common.cuh"

namespace tfx {
int ttm_tc_narrow(const float* S, long long P, int D, long long Q, const float* Ut, int n, float* out, int* err,
                  cudaStream_t st);

namespace ttc {

constexpr int BM = 128, BQ = 2 * BM, BD = 32, NJ = 64, NCW = 8, NEW = 4, NT = 64 + 32 * (NCW + NEW);
constexpr int TST = 4, AST = 2, DMAX = 8192, TMEM_COLS = 512;
// tensor memory columns: accumulators [buffer][half], then operands [stage][half] of BD hi and BD lo
constexpr uint32_t TM_ACC = 0, TM_A = 2 * 2 * NJ;
constexpr uint32_t SPIN = 1u << 26;
constexpr uint32_t TTILE = BD * BQ * 4;      // one tensor tile, bytes
constexpr uint32_t BCHUNK = NJ * BD * 4;     // one chunk of U^T, bytes

__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(bar)), "r"(count));
}

__device__ __forceinline__ void expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(su32(bar)) : "memory");
}

__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity) {
  return mbar_wait_bounded(su32(bar), parity, SPIN);
}

__device__ __forceinline__ void tma_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          su32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(su32(bar))
      : "memory");
}

__device__ __forceinline__ void tma_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          su32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(su32(bar))
      : "memory");
}

// K-major SWIZZLE_128B operand: row r (32 fp32 of K) is 128 bytes, 8-row
// groups 1024 bytes apart, 16-byte chunk c stored at c ^ (r % 8)
__device__ __forceinline__ uint64_t desc(const void* tile) {
  const uint64_t a = su32(tile);
  uint64_t d = 0;
  d |= (a >> 4) & 0x3FFFull;          // start address
  d |= (uint64_t)1 << 16;             // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;   // stride byte offset: 8-row groups
  d |= (uint64_t)1 << 46;             // descriptor version
  d |= (uint64_t)2 << 61;             // SWIZZLE_128B
  return d;
}

// D = F32, A = B = TF32, both K-major, M = 128, N = 64
__host__ __device__ constexpr uint32_t idesc() {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(NJ >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

// A from tensor memory (128 lanes, a column a K step), B from shared memory
__device__ __forceinline__ void mma(uint32_t tmem, uint32_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem),
      "r"(a), "l"(b), "r"(idesc()), "r"(acc)
      : "memory");
}

__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(bar))
               : "memory");
}

// 32 columns of the warp's lanes
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
      "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
      "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]),
      "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}

__device__ __forceinline__ float hi13(float x) { return __uint_as_float(__float_as_uint(x) & 0xFFFFE000u); }

struct Smem {
  alignas(1024) unsigned char t[TST][TTILE];           // tensor tiles [32 d][256 q]
  alignas(1024) unsigned char u[TST][BCHUNK];          // U^T blocks, 64 rows j x 32 d (swizzled)
  alignas(1024) unsigned char bhi[AST][BCHUNK];
  alignas(1024) unsigned char blo[AST][BCHUNK];
  alignas(8) uint64_t tfull[TST];
  alignas(8) uint64_t tfree[TST];
  alignas(8) uint64_t afull[AST];
  alignas(8) uint64_t afree[AST];
  alignas(8) uint64_t accfull[2];
  alignas(8) uint64_t accfree[2];
  uint32_t tmem;
  int abort;
  int tissued;    // chunks whose tensor copies the producer issued
  int tconsumed;  // chunks the converters took from the ring
  int missued;    // chunks whose products were issued
};

struct Shape {
  int D, n, dchunks;
  long long P, Q;
  int qtiles;
};

__global__ void __launch_bounds__(NT, 1)
    k_ttm_tc(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap umap, Shape sh,
             float* __restrict__ out, int* err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  Smem& S = *reinterpret_cast<Smem*>((((uintptr_t)smem_raw) + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int DC = sh.dchunks;
  const long long ntiles = sh.P * sh.qtiles;
  // this CTA's tiles: blockIdx.x, blockIdx.x + gridDim.x, ...
  const int mytiles = ntiles > blockIdx.x ? (int)((ntiles - 1 - blockIdx.x) / gridDim.x + 1) : 0;
  const int nchunk = mytiles * DC;
  if (tid == 0) {
    for (int s = 0; s < TST; ++s) {
      mbar_init(&S.tfull[s], 1);
      mbar_init(&S.tfree[s], NCW);
    }
    for (int s = 0; s < AST; ++s) {
      mbar_init(&S.afull[s], NCW);
      mbar_init(&S.afree[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&S.accfull[s], 1);
      mbar_init(&S.accfree[s], NEW);
    }
    S.abort = 0;
    S.tissued = 0;
    S.tconsumed = 0;
    S.missued = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&S.tmem)),
                 "n"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = S.tmem;
  auto tile_of = [&](int local, long long& p, long long& q0) {
    const long long t = blockIdx.x + (long long)local * gridDim.x;
    p = t / sh.qtiles;
    q0 = (t - p * sh.qtiles) * BQ;
  };
  if (warp == 0) {
    // producer: every chunk's tensor tile and U^T block
    if (lane == 0 && nchunk > 0) {
      for (int g = 0; g < nchunk; ++g) {
        const int s = g % TST;
        if (g >= TST && !wait_bar(&S.tfree[s], (uint32_t)(g / TST - 1) & 1u)) {
          atomicExch(err, 4);
          S.abort = 1;
        }
        if (*(volatile int*)&S.abort) break;
        long long p, q0;
        tile_of(g / DC, p, q0);
        const int c = g - (g / DC) * DC;
        expect_tx(&S.tfull[s], TTILE + BCHUNK);
        tma_3d(S.t[s], &tmap, &S.tfull[s], (int)q0, c * BD, (int)p);
        tma_2d(S.u[s], &umap, &S.tfull[s], c * BD, 0);
        S.tissued = g + 1;
      }
    }
  } else if (warp == 1) {
    // MMA issuer
    if (lane == 0 && nchunk > 0) {
      for (int g = 0; g < nchunk && !*(volatile int*)&S.abort; ++g) {
        const int as = g % AST, c = g % DC, tl = g / DC;
        if (!wait_bar(&S.afull[as], (uint32_t)(g / AST) & 1u)) {
          atomicExch(err, 6);
          S.abort = 1;
          break;
        }
        const int ab = tl & 1;
        if (c == 0 && tl > 1 && !wait_bar(&S.accfree[ab], (uint32_t)(tl / 2 - 1) & 1u)) {
          atomicExch(err, 7);
          S.abort = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t bh = desc(S.bhi[as]), bl = desc(S.blo[as]);
        long long p, q0;
        tile_of(tl, p, q0);
        const int nh = q0 + BM < sh.Q ? 2 : 1;  // a half past the end has no rows
        for (int hf = 0; hf < nh; ++hf) {
          const uint32_t acc = tmem + TM_ACC + (uint32_t)(ab * 2 + hf) * NJ;
          const uint32_t ah = tmem + TM_A + (uint32_t)(as * 2 + hf) * 2 * BD, al = ah + BD;
#pragma unroll
          for (int pass = 0; pass < 3; ++pass) {
            // hi*hi, hi*lo, lo*hi
            const uint32_t da = pass == 2 ? al : ah;
            const uint64_t db = pass == 1 ? bl : bh;
#pragma unroll
            for (int kk = 0; kk < BD / 8; ++kk)
              mma(acc, da + (uint32_t)(kk * 8), db + (uint64_t)(kk * 2), (c > 0 || pass > 0 || kk > 0) ? 1u : 0u);
          }
        }
        commit(&S.afree[as]);
        if (c == DC - 1) commit(&S.accfull[ab]);
        S.missued = g + 1;
      }
    }
  } else if (warp < 2 + NCW) {
    // converters (warps 2-9)
    const int cw = warp - 2, hf = cw >> 2;
    const uint32_t lanes = (uint32_t)(32 * (warp & 3));  // the lanes of tensor memory this warp reaches
    const int qr = hf * BM + (int)lanes + lane;          // the row it converts
    for (int g = 0; g < nchunk; ++g) {
      const int s = g % TST, as = g % AST;
      if (!wait_bar(&S.tfull[s], (uint32_t)(g / TST) & 1u)) {
        if (lane == 0) {
          atomicExch(err, 1);
          S.abort = 1;
        }
      }
      if (g >= AST && !wait_bar(&S.afree[as], (uint32_t)(g / AST - 1) & 1u)) {
        if (lane == 0) {
          atomicExch(err, 2);
          S.abort = 1;
        }
      }
      if (__any_sync(0xffffffffu, *(volatile int*)&S.abort)) break;  // the whole warp: what follows is warp-wide
      if (warp == 2 && lane == 0) S.tconsumed = g + 1;
      long long p, q0;
      tile_of(g / DC, p, q0);
      // U^T block: element-wise, the layout stays (the MMA reads hi and lo
      // with the same descriptor form)
      {
        const float4* u4 = reinterpret_cast<const float4*>(S.u[s]);
        float4* bh4 = reinterpret_cast<float4*>(S.bhi[as]);
        float4* bl4 = reinterpret_cast<float4*>(S.blo[as]);
#pragma unroll
        for (int e = 0; e < (int)(BCHUNK / 16) / (32 * NCW); ++e) {
          const float4 v = u4[e * 32 * NCW + cw * 32 + lane];
          float4 h, lo;
          h.x = hi13(v.x); lo.x = v.x - h.x;
          h.y = hi13(v.y); lo.y = v.y - h.y;
          h.z = hi13(v.z); lo.z = v.z - h.z;
          h.w = hi13(v.w); lo.w = v.w - h.w;
          bh4[e * 32 * NCW + cw * 32 + lane] = h;
          bl4[e * 32 * NCW + cw * 32 + lane] = lo;
        }
      }
      if (q0 + hf * BM < sh.Q) {  // uniform: the half has rows
        const float* tt = reinterpret_cast<const float*>(S.t[s]) + qr;
        uint32_t h[32], lo[32];
#pragma unroll
        for (int d = 0; d < BD; ++d) {
          const float v = tt[d * BQ], vh = hi13(v);
          h[d] = __float_as_uint(vh);
          lo[d] = __float_as_uint(v - vh);
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");  // the operand's products were waited for
        const uint32_t ta = tmem + (lanes << 16) + TM_A + (uint32_t)(as * 2 + hf) * 2 * BD;
        tmem_st32(ta, h);
        tmem_st32(ta + BD, lo);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      }
      // the operands are visible to the tensor core; the tensor stage goes
      // back to the producer, the operand to the MMA warp
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        arrive(&S.tfree[s]);
        arrive(&S.afull[as]);
      }
    }
  } else {
    // epilogue (warps 10-13): a tile's accumulators, rows q0 + hf * 128 + erow, columns j
    const uint32_t lanes = (uint32_t)(32 * (warp & 3));
    const int erow = (int)lanes + lane;
    for (int tl = 0; tl < mytiles; ++tl) {
      const int ab = tl & 1;
      if (!wait_bar(&S.accfull[ab], (uint32_t)(tl / 2) & 1u)) {
        if (lane == 0) {
          atomicExch(err, 3);
          S.abort = 1;
        }
      }
      if (__any_sync(0xffffffffu, *(volatile int*)&S.abort)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      long long p, q0;
      tile_of(tl, p, q0);
      for (int hf = 0; hf < 2; ++hf) {
        if (q0 + hf * BM >= sh.Q) break;
        const long long q = q0 + hf * BM + erow;
        float* orow = out + (size_t)p * sh.n * sh.Q + q;
#pragma unroll 1
        for (int cc = 0; cc < NJ && cc < sh.n; cc += 32) {
          uint32_t v[32];
          const uint32_t taddr = tmem + (lanes << 16) + TM_ACC + (uint32_t)(ab * 2 + hf) * NJ + (uint32_t)cc;
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
              "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
              : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
              : "r"(taddr));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (q < sh.Q)
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (cc + j < sh.n) orow[(size_t)(cc + j) * sh.Q] = __uint_as_float(v[j]);
          __syncwarp();
        }
      }
      // every read of the accumulators is done before their next products
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) arrive(&S.accfree[ab]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // after an abort: every issued copy lands and every issued product finishes
  // (bounded waits) before the CTA frees TMEM and exits
  if (tid == 0 && *(volatile int*)&S.abort) {
    const int issued = S.tissued, consumed = S.tconsumed, mi = S.missued;
    for (int g = consumed; g < issued; ++g) wait_bar(&S.tfull[g % TST], (uint32_t)(g / TST) & 1u);
    if (mi > 0) wait_bar(&S.afree[(mi - 1) % AST], (uint32_t)((mi - 1) / AST) & 1u);
  }
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM_COLS) : "memory");
}

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                             const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                             CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeFn)p;
  }
  return fn;
}

static int sms() {
  int dev = 0, n = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n < 1 ? 1 : n;
}

}  // namespace ttc
}  // namespace tfx

using namespace tfx;

extern "C" int tfx_ttm_tc_supported(long long P, int D, long long Q, int n) {
  return P >= 1 && P <= 0x7fffffffLL && D >= ttc::BD && D <= ttc::DMAX && D % ttc::BD == 0 && n >= 1 &&
         n <= ttc::NJ && Q >= ttc::BM && Q % 4 == 0 && Q <= 0x7fffffffLL;
}

// S: (P, D, Q) C-order FP32, 16-byte aligned; Ut: n x D row-major (U^T),
// 16-byte aligned; out: (P, n, Q).  err: device int, set non-zero when a
// bounded wait ran out (the caller raises on it).
extern "C" int tfx_ttm_tc(const float* S, long long P, int D, long long Q, const float* Ut, int n, float* out,
                          int* err, void* stream) {
  if (!S || !Ut || !out || !err) return tfx_set_error(TFX_STATUS_ERR_ARG, "ttm_tc args");
  if (!tfx_ttm_tc_supported(P, D, Q, n))
    return tfx_set_error(TFX_STATUS_ERR_UNSUPPORTED, "ttm_tc: D % 32 == 0, n <= 64, Q >= 128, Q % 4 == 0");
  if (((uintptr_t)S & 15) != 0 || ((uintptr_t)Ut & 15) != 0)
    return tfx_set_error(TFX_STATUS_ERR_ARG, "ttm_tc needs 16-byte aligned operands");
  // 128-wide tiles in one round of the SMs, or one chunk a tile: ttm_tc_narrow.cu
  // (both sides measured there); beyond it 256-wide tiles (P 50, D 512, Q 512, n
  // 50: 29 us, 35 there; P 1, D 64, Q 40000, n 10: 10.9 and 12.2)
  if (P * ((Q + ttc::BM - 1) / ttc::BM) <= ttc::sms() || D < 2 * ttc::BD)
    return ttm_tc_narrow(S, P, D, Q, Ut, n, out, err, (cudaStream_t)stream);
  ttc::EncodeFn enc = ttc::encode_fn();
  if (!enc) return tfx_set_error(TFX_STATUS_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled unavailable");
  CUtensorMap tmap, umap;
  {
    const cuuint64_t gdim[3] = {(cuuint64_t)Q, (cuuint64_t)D, (cuuint64_t)P};
    const cuuint64_t gstride[2] = {(cuuint64_t)Q * 4, (cuuint64_t)Q * D * 4};
    const cuuint32_t box[3] = {ttc::BQ, ttc::BD, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(&tmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void*)S, gdim, gstride, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return tfx_set_error(TFX_STATUS_ERR_ARG, "ttm_tc tensor map encoding failed");
  }
  {
    const cuuint64_t gdim[2] = {(cuuint64_t)D, (cuuint64_t)n};
    const cuuint64_t gstride[1] = {(cuuint64_t)D * 4};
    const cuuint32_t box[2] = {ttc::BD, ttc::NJ};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(&umap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)Ut, gdim, gstride, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return tfx_set_error(TFX_STATUS_ERR_ARG, "ttm_tc U map encoding failed");
  }
  ttc::Shape sh;
  sh.D = D;
  sh.n = n;
  sh.dchunks = D / ttc::BD;
  sh.P = P;
  sh.Q = Q;
  sh.qtiles = (int)((Q + ttc::BQ - 1) / ttc::BQ);
  const long long ntiles = P * sh.qtiles;
  const int grid = (int)std::max<long long>(1, std::min<long long>(ntiles, ttc::sms()));
  cudaStream_t st = (cudaStream_t)stream;
  const size_t sm = sizeof(ttc::Smem) + 1024;
  cudaError_t e = cudaFuncSetAttribute(ttc::k_ttm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return tfx_set_cuda_error(e, "ttm_tc smem");
  ttc::k_ttm_tc<<<grid, ttc::NT, sm, st>>>(tmap, umap, sh, out, err);
  e = cudaGetLastError();
  if (e != cudaSuccess) return tfx_set_cuda_error(e, "ttm_tc launch");
  tfx_count_launch(1);
  return TFX_STATUS_OK;
}
