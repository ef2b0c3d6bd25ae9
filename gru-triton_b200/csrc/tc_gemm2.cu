// The product of tc_gemm.cu for large problems: persistent pairs of CTAs (cta_group::2).
//
// A pair of CTAs on neighbouring SMs computes 256 x 256 tiles.  Each CTA holds its 128 rows of A, half of
// B (128 of the 256 columns) and its 128 x 256 part of the accumulator; one tcgen05.mma reads both shared
// memories.  What bounds the single-CTA kernel at two planes per operand: a 64-deep k-block is 96 KB, so two
// stages fill shared memory and every refill exposes its latency, the 96 KB per 1536 cycles of products are
// more than an SM draws from L2, and the result tile leaves while the tensor cores idle (10 K
// cycles beside 25 K of products at K = 1024).  Here a k-block is 64 KB per CTA (three stages), and the epilogue
// warps scale and store tile i while the products of tile i + 1 run.
//
// As there, the fp32 accumulator of the tensor core truncates, so sums are built in chunks of at most 32 steps
// in one of two tensor-memory buffers and added to register totals with round-to-nearest.

#include <cstring>
#include <map>
#include <mutex>
#include <type_traits>
#include <utility>

#include "tc_common.cuh"
#include "tc_gemm.cuh"

namespace b200gru {
namespace tc {

__device__ int g_tc2_status;

namespace {

constexpr int BM = 128;                      // rows of A per CTA
constexpr int BN = 256;                      // columns of the pair's tile
constexpr int BH = 128;                      // rows of B per CTA
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + 32 * EPI_WARPS;
constexpr int MAX_STAGES = 8;
constexpr int RING = 192 * 1024;
constexpr int TR_LD = 20;                    // floats per row of a warp's 32 x 16 transpose buffer
constexpr int TR_BYTES = EPI_WARPS * 32 * TR_LD * 4;

struct Params {
  int M, N;
  int tiles_m, tiles_n, splits, tiles;       // 256-row and 256-column tiles, K slices, all of them
  int kb_total, kb_per_split;
  int a_planes, b_planes, npairs;
  int pa[TC_MAX_PAIRS], pb[TC_MAX_PAIRS];
  int stages, chunk_kb, accumulate;
  unsigned ab_format;
  float alpha;
  const float* row_scale;
  const float* col_scale;
  const float* bias;
  float* C;
  long long ldc, split_stride;
};

__device__ __forceinline__ uint32_t cta_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t at_leader(uint32_t addr) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
// Tile load into this CTA whose bytes are counted on a barrier of the pair's leader.
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
template <bool I8>
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  if (I8) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
  } else {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
  }
}
// The barrier at this offset of both CTAs receives an arrival once the products issued so far are done.
__device__ __forceinline__ void commit_pair(uint32_t bar) {
  const uint16_t mask = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(mask) : "memory");
}
__device__ __forceinline__ void arrive_at_leader(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(at_leader(bar)) : "memory");
}

template <bool I8, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(THREADS, 1)
tc_gemm2_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const Params p) {
  constexpr int ES = I8 ? 1 : 2;
  constexpr int BK = I8 ? 128 : 64;                       // 128 bytes of K, or 64 k rows
  constexpr int UMMA_K = 32 / ES;
  constexpr int PLANE = BM * 128;                         // 16 KB: a plane of A or of a half of B
  static_assert(!(I8 && (A_MN || B_MN)), "int8 operands are K-major here");
  constexpr int NC = BN / 2;                              // accumulator columns per epilogue thread
  typedef typename std::conditional<I8, int, float>::type AccT;
  const uint32_t IDESC = umma_idesc(I8, A_MN, B_MN, 2 * BM, BN, p.ab_format);

  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) unsigned long long bar_full[MAX_STAGES], bar_empty[MAX_STAGES];
  __shared__ __align__(8) unsigned long long bar_acc_full[2], bar_acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int dead;

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const uint32_t rank = cta_rank();
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int stage_bytes = (p.a_planes + p.b_planes) * PLANE;
  volatile int* deadp = &dead;
  int* status = &g_tc2_status;
  pdl_launch_dependents();

  if (threadIdx.x == 0) {
    dead = (*reinterpret_cast<volatile int*>(status) != 0) ? 1 : 0;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&bar_acc_full[b]), 1);
      mbar_init(smem_u32(&bar_acc_empty[b]), 2 * EPI_WARPS);
    }
    mbar_fence_init();
    tma_prefetch_map(&tmA);
    tma_prefetch_map(&tmB);
  }
  if (warp == 1) tmem_alloc_pair(smem_u32(&tmem_slot), 2 * BN);
  tc_fence_before();
  __syncthreads();
  pair_sync();                                            // barriers of both CTAs exist
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_wait();

  // tile index -> K slice, row panel, column panel (columns fastest: neighbours share the rows of A)
  auto locate = [&](int t, int& m0, int& n0, int& z, int& kb0, int& nkb) {
    n0 = (t % p.tiles_n) * BN;
    const int r = t / p.tiles_n;
    m0 = (r % p.tiles_m) * 2 * BM + (int)rank * BM;
    z = r / p.tiles_m;
    kb0 = z * p.kb_per_split;
    nkb = max(0, min(p.kb_total, kb0 + p.kb_per_split) - kb0);
  };

  if (warp == 0) {
    // ---- loader: own rows of A and own half of B; the leader's barrier counts the bytes of both CTAs
    bool alive = __all_sync(0xffffffffu, *deadp == 0);
    int s = 0;
    uint32_t parity = 1;                                  // the first round finds every stage free
    bool first = true;
    for (int t = pair; t < p.tiles && alive; t += npairs) {
      int m0, n0, z, kb0, nkb;
      locate(t, m0, n0, z, kb0, nkb);
      n0 += (int)rank * BH;
      for (int i = 0; i < nkb; ++i) {
        if (!first) alive = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_empty[s]), parity, deadp, status));
        if (!alive) break;
        if (elect_one()) {
          const uint32_t full = at_leader(smem_u32(&bar_full[s]));
          if (rank == 0) mbar_expect_tx(smem_u32(&bar_full[s]), 2u * (uint32_t)stage_bytes);
          const uint32_t st = smem_u32(smem) + (uint32_t)(s * stage_bytes);
          const int kb = kb0 + i;
          for (int pl = 0; pl < p.a_planes; ++pl) {
            const uint32_t dst = st + (uint32_t)(pl * PLANE);
            if (A_MN) {
              tma_load_pair(dst, &tmA, m0, kb * 64, pl, full);
              tma_load_pair(dst + 8192, &tmA, m0 + 64, kb * 64, pl, full);
            } else {
              tma_load_pair(dst, &tmA, kb * BK, m0, pl, full);
            }
          }
          const uint32_t sb = st + (uint32_t)(p.a_planes * PLANE);
          for (int pl = 0; pl < p.b_planes; ++pl) {
            const uint32_t dst = sb + (uint32_t)(pl * PLANE);
            if (B_MN) {
              tma_load_pair(dst, &tmB, n0, kb * 64, pl, full);
              tma_load_pair(dst + 8192, &tmB, n0 + 64, kb * 64, pl, full);
            } else {
              tma_load_pair(dst, &tmB, kb * BK, n0, pl, full);
            }
          }
        }
        __syncwarp();
        if (++s == p.stages) { s = 0; parity ^= 1u; first = false; }
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // ---- issuer of the pair
      constexpr uint64_t A_STEP = (A_MN ? UMMA_K * 128 : 32) >> 4, B_STEP = (B_MN ? UMMA_K * 128 : 32) >> 4;
      const uint64_t da0 = A_MN ? umma_smem_desc(smem_u32(smem), 8192, 1024) : umma_smem_desc(smem_u32(smem), 16, 1024);
      const uint64_t db0 = B_MN ? umma_smem_desc(smem_u32(smem), 8192, 1024) : umma_smem_desc(smem_u32(smem), 16, 1024);
      const uint32_t b_off = (uint32_t)(p.a_planes * PLANE) >> 4;
      bool alive = __all_sync(0xffffffffu, *deadp == 0);
      int s = 0, c = 0;                                   // ring stage, chunks so far
      uint32_t parity = 0;
      for (int t = pair; t < p.tiles && alive; t += npairs) {
        int m0, n0, z, kb0, nkb;
        locate(t, m0, n0, z, kb0, nkb);
        for (int i0 = 0; i0 < nkb && alive; i0 += p.chunk_kb, ++c) {
          const int buf = c & 1;
          if (c >= 2) alive = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_acc_empty[buf]), ((c >> 1) - 1) & 1, deadp, status));
          if (!alive) break;
          tc_fence_after();
          const uint32_t tacc = tmem + (uint32_t)(buf * BN);
          const int i1 = min(nkb, i0 + p.chunk_kb);
          for (int i = i0; i < i1; ++i) {
            alive = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_full[s]), parity, deadp, status));
            if (!alive) break;
            tc_fence_after();
            if (elect_one()) {
              const uint32_t st = (uint32_t)(s * stage_bytes) >> 4;
              for (int q = 0; q < p.npairs; ++q) {
                const uint64_t da = da0 + st + (uint32_t)(p.pa[q] * (PLANE >> 4));
                const uint64_t db = db0 + st + b_off + (uint32_t)(p.pb[q] * (PLANE >> 4));
                const uint32_t more = (i > i0 || q > 0) ? 1u : 0u;
#pragma unroll
                for (int kk = 0; kk < BK / UMMA_K; ++kk)
                  umma_pair<I8>(tacc, da + kk * A_STEP, db + kk * B_STEP, IDESC, kk > 0 ? 1u : more);
              }
              commit_pair(smem_u32(&bar_empty[s]));
              if (i == i1 - 1) commit_pair(smem_u32(&bar_acc_full[buf]));
            }
            __syncwarp();
            if (++s == p.stages) { s = 0; parity ^= 1u; }
          }
        }
      }
    }
  } else {
    // ---- epilogue: warp w reads lanes 32 (w % 4) .. of this CTA's accumulator, one half of the columns
    const int q = warp & 3, half = (warp - 2) >> 2;
    float* tr = reinterpret_cast<float*>(smem + p.stages * stage_bytes) + (warp - 2) * 32 * TR_LD;
    int c = 0;
    bool ok = __all_sync(0xffffffffu, *deadp == 0);
    for (int t = pair; t < p.tiles && ok; t += npairs) {
      int m0, n0, z, kb0, nkb;
      locate(t, m0, n0, z, kb0, nkb);
      AccT acc[NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) acc[j] = (AccT)0;
      for (int i0 = 0; i0 < nkb; i0 += p.chunk_kb, ++c) {
        const int buf = c & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_acc_full[buf]), (c >> 1) & 1, deadp, status));
        if (!ok) break;
        tc_fence_after();
        const uint32_t tsrc = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN + half * NC);
#pragma unroll
        for (int c0 = 0; c0 < NC; c0 += 32) {
          uint32_t v[32];
          tmem_ld32(tsrc + (uint32_t)c0, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            if (I8) acc[c0 + j] += (AccT)(int)v[j];
            else acc[c0 + j] += (AccT)__uint_as_float(v[j]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_at_leader(smem_u32(&bar_acc_empty[buf]));
      }
      if (!ok) break;
      // store 16 columns at a time through the warp's transpose buffer: 64 contiguous bytes of eight rows per instruction
      const int row_base = m0 + q * 32, col_base = n0 + half * NC;
      const int rsub = lane >> 2, csub = (lane & 3) * 4;
      float rs[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int m = row_base + k * 8 + rsub;
        rs[k] = p.alpha * ((p.row_scale != nullptr && m < p.M) ? __ldg(p.row_scale + m) : 1.0f);
      }
      float* cbase = p.C + (size_t)z * p.split_stride;
#pragma unroll
      for (int j = 0; j < NC; j += 16) {
        const int n = col_base + j + csub;
        if (col_base + j < p.N) {                          // warp-uniform
          __syncwarp();
#pragma unroll
          for (int e = 0; e < 16; e += 4)
            *reinterpret_cast<float4*>(tr + lane * TR_LD + e) =
                make_float4((float)acc[j + e], (float)acc[j + e + 1], (float)acc[j + e + 2], (float)acc[j + e + 3]);
          __syncwarp();
          if (n < p.N) {                                   // N % 4 == 0
            float4 cs = make_float4(1.f, 1.f, 1.f, 1.f), bs = make_float4(0.f, 0.f, 0.f, 0.f);
            if (p.col_scale != nullptr) { cs.x = __ldg(p.col_scale + n); cs.y = __ldg(p.col_scale + n + 1); cs.z = __ldg(p.col_scale + n + 2); cs.w = __ldg(p.col_scale + n + 3); }
            if (p.bias != nullptr) { bs.x = __ldg(p.bias + n); bs.y = __ldg(p.bias + n + 1); bs.z = __ldg(p.bias + n + 2); bs.w = __ldg(p.bias + n + 3); }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int m = row_base + k * 8 + rsub;
              if (m < p.M) {
                const float4 v = *reinterpret_cast<const float4*>(tr + (k * 8 + rsub) * TR_LD + csub);
                float4 o = make_float4(v.x * rs[k], v.y * rs[k], v.z * rs[k], v.w * rs[k]);
                if (p.col_scale != nullptr) { o.x *= cs.x; o.y *= cs.y; o.z *= cs.z; o.w *= cs.w; }
                if (p.bias != nullptr) { o.x += bs.x; o.y += bs.y; o.z += bs.z; o.w += bs.w; }
                float4* dst = reinterpret_cast<float4*>(cbase + (size_t)m * p.ldc + n);
                if (p.accumulate) { const float4 old = *dst; o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w; }
                *dst = o;
              }
            }
          }
        }
      }
    }
  }

  if (warp == 0 && lane == 0 && *deadp) {                 // a CTA that gave up: let tile copies in flight land
    const long long start = clock64();
    while (clock64() - start < (1ll << 18)) {
    }
  }
  tc_fence_before();
  __syncthreads();
  pair_sync();                                            // nobody leaves while the other may still signal it
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc_pair(tmem, 2 * BN);
  }
}

// Pairs of CTAs the device runs at once; 0 when they cannot be launched.
int pairs_on_device(const void* fn, size_t smem) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, int> cache;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_pair(dev, fn);
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  int n = 0;
  if (allow_dynamic_smem(fn, smem) == B200GRU_OK) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
  }
  cache[key] = n;
  return n;
}

template <bool I8, bool A_MN, bool B_MN>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const Params& p, cudaStream_t st) {
  auto kernel = tc_gemm2_kernel<I8, A_MN, B_MN>;
  const size_t smem = (size_t)RING + TR_BYTES + 1024;
  const int pairs = pairs_on_device(reinterpret_cast<const void*>(kernel), smem);
  if (pairs <= 0) return B200GRU_UNSUPPORTED;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * (p.tiles < pairs ? p.tiles : pairs)));
  cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = B200GRU_PDL_ALLOWED;
  cfg.attrs = at; cfg.numAttrs = 2;
  cudaLaunchKernelEx(&cfg, kernel, ta, tb, p);
  note_launch();
  return check_launch("tc_gemm2_kernel");
}

}  // namespace

int launch_tc_gemm_pairs(const TcGemm& g, cudaStream_t st) {
  const bool i8 = g.kind == TC_KIND_I8;
  const int es = i8 ? 1 : 2, bk = tc_gemm_kblock(g);
  Params p;
  memset(&p, 0, sizeof(p));
  p.M = g.M; p.N = g.N;
  p.splits = g.split_k < 1 ? 1 : g.split_k;
  p.tiles_m = cdiv(g.M, 2 * BM); p.tiles_n = cdiv(g.N, BN);
  const long long tiles = (long long)p.tiles_m * p.tiles_n * p.splits;
  if (tiles > 0x7fffffff) return B200GRU_UNSUPPORTED;
  p.tiles = (int)tiles;
  p.kb_total = cdiv(g.K, bk);
  p.kb_per_split = cdiv(p.kb_total, p.splits);
  p.a_planes = g.a_planes; p.b_planes = g.b_planes; p.npairs = g.npairs;
  for (int q = 0; q < g.npairs; ++q) { p.pa[q] = g.pa[q]; p.pb[q] = g.pb[q]; }
  const int stage = (g.a_planes + g.b_planes) * BM * 128;
  p.stages = RING / stage;
  if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
  if (p.stages < 2) return B200GRU_UNSUPPORTED;
  if (g.chunk_kb > 0) p.chunk_kb = g.chunk_kb;
  else if (i8) p.chunk_kb = p.kb_per_split;
  else p.chunk_kb = (32 / (4 * g.npairs)) > 0 ? 32 / (4 * g.npairs) : 1;
  p.accumulate = g.accumulate;
  p.ab_format = (g.kind == TC_KIND_F16) ? 0u : 1u;
  p.alpha = g.alpha; p.row_scale = g.row_scale; p.col_scale = g.col_scale; p.bias = g.bias;
  p.C = g.C; p.ldc = g.ldc; p.split_stride = g.split_stride;

  const CUtensorMapDataType dt = i8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                    : (g.kind == TC_KIND_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16);
  alignas(64) CUtensorMap ta, tb;
  int rc;
  const unsigned long long a_pl = g.a_planes > 1 ? (unsigned long long)g.a_plane_stride * es : (unsigned long long)(g.a_mn ? g.K : g.M) * g.lda * es;
  const unsigned long long b_pl = g.b_planes > 1 ? (unsigned long long)g.b_plane_stride * es : (unsigned long long)(g.b_mn ? g.K : g.N) * g.ldb * es;
  if (g.a_mn) rc = make_tensor_map_3d(&ta, dt, g.A, g.M, g.K, g.a_planes, (unsigned long long)g.lda * es, a_pl, 64, 64);
  else rc = make_tensor_map_3d(&ta, dt, g.A, g.K, g.M, g.a_planes, (unsigned long long)g.lda * es, a_pl, bk, BM);
  if (rc) return rc;
  if (g.b_mn) rc = make_tensor_map_3d(&tb, dt, g.B, g.N, g.K, g.b_planes, (unsigned long long)g.ldb * es, b_pl, 64, 64);
  else rc = make_tensor_map_3d(&tb, dt, g.B, g.K, g.N, g.b_planes, (unsigned long long)g.ldb * es, b_pl, bk, BH);
  if (rc) return rc;
  if (i8) return launch<true, false, false>(ta, tb, p, st);
  if (!g.a_mn && !g.b_mn) return launch<false, false, false>(ta, tb, p, st);
  if (!g.a_mn && g.b_mn) return launch<false, false, true>(ta, tb, p, st);
  if (g.a_mn && !g.b_mn) return launch<false, true, false>(ta, tb, p, st);
  return launch<false, true, true>(ta, tb, p, st);
}

int tc2_read_status(int reset) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_tc2_status, sizeof(int)) != cudaSuccess) return -1;
  if (reset && v != 0) {
    const int z = 0;
    cudaMemcpyToSymbol(g_tc2_status, &z, sizeof(int));
  }
  return v;
}

}  // namespace tc
}  // namespace b200gru
