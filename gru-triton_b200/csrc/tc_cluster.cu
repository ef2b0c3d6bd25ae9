// Dense and block-diagonal scans with blocks of at most 512 units on the tensor cores, all T steps in
// one launch.
//
// A thread-block cluster of C <= 16 CTAs owns one (hidden block, batch tile) problem.  CTA `rank` owns
// 32 hidden units and keeps their 96 weight rows on chip for the whole scan as two fp16 planes (rows
// scaled by a power of two, 22 significant bits: hi = RN16(w s), lo = RN16(w s - hi)): hi in tensor
// memory as the A operand of tcgen05.mma, lo in shared memory.  Weights that are int8 codes are one
// exact plane, and so is a state on an int8 grid; an unquantised state is two planes.  The batch rows
// are the N dimension, so a step costs the same number of instructions for 5 rows as for 48.
//
//   forward   D[96 rows (gate, unit)][rows] = W_own . h^T over all k: every CTA needs the whole h_{t-1};
//             the new slab of 32 units goes to every peer's operand buffer with one bulk copy per peer
//   backward  D[k][rows] = W_own^T . dgh_own: a partial sum for every position k; the 32 positions of
//             rank r go to r's receive buffer (bulk copies: st.async stores kept every later load and store of the SM
//             waiting behind them), r adds the C partials in rank order
//
// The fp32 accumulator of the tensor core truncates.  Forward: the leading products (hi x hi) are summed in
// accumulators of at most 8 steps (16 where the state is on an int8 grid), the small cross products in one of their own,
// and all are added with round-to-nearest (two of 16 steps: the gradient of b_r at H = 512 was off by 5.4e-7 of 64 bits, 4.5e-7 with four;
// 5.0e-7 with FP32 FMAs).  Backward: one accumulator per tile, the 12 small products first and the 6 leading ones
// on top of them (6.7e-7 -> 5.4e-7).  Integer codes are exact in one (|sum| < 2^24).
//
// What bounds a step: the exchange.  A CTA receives C slabs at about 15 bytes per cycle over the cluster
// network (measured; 1300 cycles for the smallest slabs), the products take 12 to 26 cycles per
// instruction with A in tensor memory (42 and more from shared memory) and hide behind the arrival of the slabs,
// the gate phase and its barriers about 1200 cycles.
// The FP32 cluster kernels of block_scan.cu do the same with FMAs: a cluster then holds only 5 or 6 rows
// at H = 512, and a batch of 256 takes seven waves.
//
// Reference: src/gru_qat/triton_kernels/scan.py:120-184 (forward), 389-616 (backward).

#include <cooperative_groups.h>

#include <cstring>
#include <map>
#include <mutex>
#include <utility>

#include "tc_cluster.cuh"
#include "tc_common.cuh"

namespace cg = cooperative_groups;

namespace b200gru {
namespace tcc {

__device__ int g_tcc_status;

namespace {

using namespace tc;

constexpr int NW = 16;                       // compute warps
constexpr int NT = 32 * (NW + 1);            // and one warp that issues the products
constexpr int ROWS_A = 3 * UNITS;            // weight rows of a CTA
constexpr int LO_BLOCK = ROWS_A * 128;       // 64 k of the lo plane, 128-byte rows
constexpr int TMEM_COLS = 512;               // hi planes from column 0, lo planes behind them, accumulators at the end
constexpr int MAX_N = 48;

// 64-byte swizzle, K-major: rows of 64 bytes (32 fp16 k), 8-row groups `sbo` bytes apart.
__device__ __forceinline__ uint64_t desc_sw64(uint32_t saddr, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3fffu);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(sbo >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;
  return d;
}
__device__ __forceinline__ uint32_t sw64(uint32_t row, uint32_t byte) {        // offset of `byte` (0..63) of `row`
  return row * 64 + ((((byte >> 4) ^ (row >> 1)) & 3) << 4) + (byte & 15);
}
__device__ __forceinline__ uint32_t sw128(uint32_t row, uint32_t byte) {       // the same for 128-byte rows
  return row * 128 + ((((byte >> 4) ^ row) & 7) << 4) + (byte & 15);
}

// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
               ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// The barrier at this shared-memory offset of every CTA in `mask` receives an arrival.
__device__ __forceinline__ void umma_commit_cluster(uint32_t bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(mask) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float (&v)[4]) {
  uint32_t u[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]) : "r"(taddr) : "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(u[i]);
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void bulk_to_peer(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "r"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t load_at_peer(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void store_at_peer(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void arrive_at_peer(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait (see tc::mbar_wait) on a barrier that other CTAs of the cluster signal.
__device__ __forceinline__ bool try_wait_cluster(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
               "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool wait_cluster(uint32_t bar, uint32_t parity, volatile int* dead, int* status) {
  if (try_wait_cluster(bar, parity)) return true;
  const long long start = clock64();
  while (*dead == 0) {
    if (try_wait_cluster(bar, parity)) return true;
    if (clock64() - start > WAIT_BUDGET_CYCLES) {
      *dead = 1;
      atomicExch(status, 1);
    }
  }
  return false;
}
// Giving up.  A wait that runs out marks its CTA dead, and every later wait of the CTA that would have to wait returns
// false at once.  The barrier of all warps in every step carries that along (bar_all_any): all warps learn of it at the same
// point and leave the time loop together.  Nothing is committed or copied to a peer, and no byte expected, on a wait that
// failed.  (Products may be issued: they read and write this CTA's own memory.)
// The end of both kernels: a CTA that gave up tells its whole cluster, and then every CTA of it stays long enough
// for products and copies in flight to land before any of them leaves.
__device__ __forceinline__ void leave_together(const cg::cluster_group& cluster, int C, volatile int* dead, int* peer_gave_up) {
  tc_fence_before();
  __syncthreads();                     // `dead` is final
  if (threadIdx.x < C && *dead != 0) store_at_peer(map_to_rank(smem_u32(peer_gave_up), threadIdx.x), 1);
  cluster.sync();                      // no copy or arrival starts behind this, and none is under way unless somebody gave up
  if (*reinterpret_cast<volatile int*>(peer_gave_up) != 0) {
    const long long start = clock64();
    while (clock64() - start < (1ll << 18)) {
    }
    cluster.sync();
  }
}
// The 16 compute warps / all 17 warps.
__device__ __forceinline__ void bar_compute() { asm volatile("bar.sync 1, %0;" ::"n"(32 * NW) : "memory"); }
__device__ __forceinline__ bool bar_all_any(bool gave_up) {       // whether any thread of the CTA gave up
  uint32_t any;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.or.pred p, 2, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(any) : "r"((uint32_t)gave_up), "n"(NT) : "memory");
  return __any_sync(0xffffffffu, any != 0);                // (a vote, so that the compiler knows the warp stays together)
}

__device__ __forceinline__ float warp_max(float v) {              // v >= 0 (or NaN, which counts as largest)
  return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
}
__device__ __forceinline__ void split2(float x, __half* hi, __half* lo) {
  *hi = __float2half_rn(x);
  *lo = __float2half_rn(x - __half2float(*hi));
}
__device__ __forceinline__ uint32_t pack2(__half a, __half b) {
  return (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16);
}
__device__ __forceinline__ float h_code(float h, const Quant& q) { return fminf(fmaxf(fq_code(h, q), q.qmin), q.qmax); }

size_t align1k(size_t x) { return (x + 1023) / 1024 * 1024; }

// Shared memory of the forward kernel (offsets from a 1024-byte aligned base).
struct FwdLayout { size_t lo, hbuf, stg, S, total; };
FwdLayout fwd_layout(int CS, int N, int pw, int ph) {
  FwdLayout l;
  l.lo = 0;
  l.hbuf = pw == 2 ? align1k((size_t)(CS / 2) * LO_BLOCK) : 0;
  const size_t slab = (size_t)ph * N * 64;
  l.stg = l.hbuf + CS * slab;
  l.S = l.stg + slab;
  // the products read 128 rows of a lo block: what lies beyond must be mapped
  size_t end = l.S + (size_t)ROWS_A * (N + 1) * sizeof(float);
  const size_t staged_w = l.hbuf + (size_t)ROWS_A * (CS * 64 + 16);         // hi rows on their way to tensor memory
  if (staged_w > end) end = staged_w;
  if (end < l.hbuf + 4096) end = l.hbuf + 4096;
  l.total = end + 1024;                                                      // base alignment
  return l;
}

// Shared memory of the backward kernel.  The blocks (tile, gate) of the lo plane that fit between the hi plane and
// the accumulators live in tensor memory, 16 columns each.
__host__ __device__ constexpr int lo_blocks_tmem(int tiles, int N) {
  return (TMEM_COLS - tiles * (48 + N)) / 16 < 3 * tiles ? (TMEM_COLS - tiles * (48 + N)) / 16 : 3 * tiles;
}
struct BwdLayout { size_t lo, bop, recv, total; };
BwdLayout bwd_layout(int C, int tiles, int N, int rows, int pw) {
  BwdLayout l;
  l.lo = 0;
  l.bop = pw == 2 ? (size_t)(3 * tiles - lo_blocks_tmem(tiles, N)) * 128 * 64 : 0;
  l.recv = l.bop + (size_t)2 * 3 * N * 64;
  l.total = l.recv + (size_t)2 * C * ((rows + 3) / 4) * 512 + 1024;           // received and staged partial sums
  return l;
}

}  // namespace

// ---------------------------------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------------------------------
template <int N, int CS, int PW, int PH>
__global__ void __launch_bounds__(NT, 1) tcc_fwd_kernel(const Args a) {
  constexpr int RPW = N / NW;                              // batch rows per compute warp
  constexpr bool EXACT = PW == 1 && PH == 1;
  // accumulators of the leading products: eight steps each at most (sixteen on an int8 state, whose grid is far coarser)
  constexpr int NMAIN = EXACT ? 1 : (CS >= 16 && PH == 2 ? 4 : 2);
  constexpr int NACC = EXACT ? 1 : NMAIN + 1;
  // Slot i of the operands belongs to rank - i (modulo C), the i-th CTA to send to this one, so that the
  // slabs are consumed in the order in which they arrive.
  // CS slabs (a compile-time count: a branch between two tcgen05.mma costs more than the product, 50
  // cycles each against 12 at N = 16); slabs beyond C are zero.  Four barriers, one per CS / 4 slabs.
  constexpr int GS = CS / 4;
  constexpr uint32_t SLAB = PH * N * 64;                   // [8-row group][plane][8 rows][32 units]
  constexpr uint32_t GROUP = PH * 512;                     // bytes of an 8-row group
  // the first lo slabs that fit between the hi planes and the accumulators live in tensor memory too
  constexpr int LO_TM = PW == 2 ? ((TMEM_COLS - NACC * N - 16 * CS) / 16 < CS ? (TMEM_COLS - NACC * N - 16 * CS) / 16 : CS) : 0;
  constexpr uint32_t IDESC = umma_idesc(false, false, false, 128, N, 0u);
  constexpr int LDS = N + 1;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) unsigned long long bar_full[4], bar_empty, bar_acc;
  __shared__ uint32_t tmem_slot;
  __shared__ int dead, peer_gave_up, unhealthy;
  __shared__ float s_wscale[ROWS_A], s_inv_h[MAX_N], s_h[MAX_N];

  cg::cluster_group cluster = cg::this_cluster();
  const int warp = uniform_warp(), lane = threadIdx.x & 31, tid = threadIdx.x;
  const int C = a.C, Hb = a.Hb, H = a.H, rows8 = a.rows8;
  const int rank = blockIdx.x % C;
  const int problem = blockIdx.x / C;
  const int n = problem / a.ntiles_b;
  const int b0 = (problem - n * a.ntiles_b) * a.rows;
  const int nrows = min(a.rows, a.B - b0);
  const int u0 = rank * UNITS;
  const int T = a.T;
  volatile int* deadp = &dead;
  int* status = a.status;

  const uint32_t sent = (uint32_t)(rows8 >> 3) * GROUP;    // bytes of a slab that carry rows
  unsigned char* lo = smem;
  unsigned char* hbuf = smem + (PW == 2 ? (CS / 2) * LO_BLOCK : 0);           // LO_BLOCK is a multiple of 1024
  unsigned char* stg = hbuf + CS * SLAB;
  float* S = reinterpret_cast<float*>(stg + SLAB);
  auto slot_rank = [&](int slot) { return rank - slot < 0 ? rank - slot + C : rank - slot; };
  auto group_bytes = [&](int g) { return (uint32_t)max(0, min(GS, C - g * GS)) * sent; };

  if (tid == 0) {
    dead = peer_gave_up = 0;
    unhealthy = *reinterpret_cast<volatile int*>(status);
    for (int g = 0; g < 4; ++g) mbar_init(smem_u32(&bar_full[g]), 1);
    mbar_init(smem_u32(&bar_empty), C);
    mbar_init(smem_u32(&bar_acc), 1);
    mbar_fence_init();
    if (T > 1)
      for (int g = 0; g < 4; ++g) mbar_expect_tx(smem_u32(&bar_full[g]), group_bytes(g));
  }
  if (warp == NW) tmem_alloc(smem_u32(&tmem_slot), 512);

  // ---- weights: planes of the 96 own rows; hi rows wait in the (still unused) state buffer
  constexpr int pitch = CS * 64 + 16;
  if (warp < NW) {
    const bool vec = (a.codes == nullptr) && Hb % 4 == 0 && (reinterpret_cast<uintptr_t>(a.W) & 15u) == 0 &&
                     a.w_gate_stride % 4 == 0 && a.w_block_stride % 4 == 0;
#pragma unroll 2
    for (int i = warp; i < ROWS_A; i += NW) {
      const int g = i >> 5, j = i & 31;
      const bool own = u0 + j < Hb;
      float v[4][4];                                       // k = 128 q + 4 lane + e of the slot order
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int slot = 4 * q + (lane >> 3);
        const int k = slot < C ? slot_rank(slot) * UNITS + (lane & 7) * 4 : Hb;
#pragma unroll
        for (int e = 0; e < 4; ++e) v[q][e] = 0.f;
        if (own && k < Hb) {
          if (PW == 1) {
            const signed char* src = a.codes + ((size_t)g * H + u0 + j) * Hb + k;
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (k + e < Hb) v[q][e] = (float)src[e];
          } else {
            const float* src = a.W + (size_t)g * a.w_gate_stride + (size_t)n * a.w_block_stride + (size_t)(u0 + j) * Hb + k;
            if (vec) {
              const float4 x = __ldg(reinterpret_cast<const float4*>(src));
              v[q][0] = x.x; v[q][1] = x.y; v[q][2] = x.z; v[q][3] = x.w;
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (k + e < Hb) v[q][e] = __ldg(src + e);
            }
          }
        }
      }
      float s = 1.f, inv = 1.f;
      if (PW == 2) {
        float mx = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int e = 0; e < 4; ++e) mx = fmaxf(mx, fabsf(v[q][e]));
        pow2_row_scale(warp_max(mx), &s, &inv);
      } else {
        inv = own ? a.scales[g * H + u0 + j] : 0.f;
      }
      if (lane == 0) s_wscale[i] = (PH == 1) ? a.qin.scale * inv : inv;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int k = 128 * q + 4 * lane;
        if (k >= CS * UNITS) continue;
        __half hi[4], lw[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split2(v[q][e] * s, &hi[e], &lw[e]);
        *reinterpret_cast<uint2*>(hbuf + i * pitch + k * 2) = make_uint2(pack2(hi[0], hi[1]), pack2(hi[2], hi[3]));
        if (PW == 2)
          *reinterpret_cast<uint2*>(lo + (k >> 6) * LO_BLOCK + sw128(i, (k & 63) * 2)) =
              make_uint2(pack2(lw[0], lw[1]), pack2(lw[2], lw[3]));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  if (warp < NW) {
    const int q = warp & 3;                                // tensor-memory lanes 32 q ..
    for (int i = warp >> 2; i < CS + LO_TM; i += NW / 4) {
      const int s = i < CS ? i : i - CS;
      uint32_t v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = 0u;
      if (q < 3) {
        const int row = q * 32 + lane;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 x = i < CS ? *reinterpret_cast<const uint4*>(hbuf + row * pitch + s * 64 + j * 16)
                                : *reinterpret_cast<const uint4*>(lo + (s >> 1) * LO_BLOCK + sw128(row, (s & 1) * 64 + j * 16));
          v[4 * j] = x.x; v[4 * j + 1] = x.y; v[4 * j + 2] = x.z; v[4 * j + 3] = x.w;
        }
      }
      tmem_st16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(i * 16), v);
    }
    tmem_st_wait();
  }
  __syncthreads();

  // ---- operand form of h0, all units of the block
  if (warp < NW) {
    for (int b = warp; b < N; b += NW) {                   // all N rows and CS slabs: nothing is left undefined
      const float* src = a.h0 + (size_t)(b0 + b) * H + (size_t)n * Hb;
      const bool live = b < nrows;
      float s = 1.f, inv = 1.f;
      if (PH == 2) {
        // |h_t| never exceeds max(1, |h0|) by more than the rounding of the quantisers
        float mx = 0.f;
        if (live)
          for (int k = lane; k < Hb; k += 32) mx = fmaxf(mx, fabsf(src[k]));
        mx = fmaxf(1.f, warp_max(mx));
        if (a.qin.enabled) mx += a.qin.scale;
        if (a.qout.enabled) mx += a.qout.scale;
        pow2_row_scale(mx, &s, &inv);
        if (lane == 0) { s_h[b] = s; s_inv_h[b] = inv; }
      }
      for (int slot = 0; slot < CS; ++slot) {
        const int k = slot < C ? slot_rank(slot) * UNITS + lane : Hb;
        const float h = (live && k < Hb) ? src[k] : 0.f;
        unsigned char* dst = hbuf + (size_t)slot * SLAB + (b >> 3) * GROUP + sw64(b & 7, lane * 2);
        if (PH == 1) {
          *reinterpret_cast<__half*>(dst) = __float2half_rn(h_code(h, a.qin));
        } else {
          __half hi, lh;
          split2((a.qin.enabled ? fake_quant<true>(h, a.qin) : h) * s, &hi, &lh);
          *reinterpret_cast<__half*>(dst) = hi;
          *reinterpret_cast<__half*>(dst + 512) = lh;
        }
      }
    }
  }

  // ---- the elements this thread owns: unit u0 + lane of rows warp, warp + 16, ...
  const int u = n * Hb + u0 + lane;
  const bool unit_ok = warp < NW && u0 + lane < Hb;
  float hown[RPW], gr[RPW], gz[RPW], gn[RPW], br = 0.f, bz = 0.f, bn = 0.f;
  bool ok_row[RPW];
  if (unit_ok) { br = a.bh[u]; bz = a.bh[H + u]; bn = a.bh[2 * H + u]; }
#pragma unroll
  for (int i = 0; i < RPW; ++i) {
    const int b = warp + i * NW;
    ok_row[i] = unit_ok && b < nrows;
    hown[i] = gr[i] = gz[i] = gn[i] = 0.f;
    if (ok_row[i]) {
      hown[i] = a.h0[(size_t)(b0 + b) * H + u];
      const float* g = a.gi + (size_t)(b0 + b) * 3 * H + u;
      gr[i] = __ldcs(g); gz[i] = __ldcs(g + H); gn[i] = __ldcs(g + 2 * H);
    }
  }
  fence_async_smem();
  tc_fence_before();
  cluster.sync();                      // operands, barriers and tensor memory are ready everywhere
  tc_fence_after();

  // no step where the status word was set when rank 0 started: the cluster leaves as one
  const int steps = __any_sync(0xffffffffu, load_at_peer(map_to_rank(smem_u32(&unhealthy), 0)) != 0) ? 0 : T;
  if (warp == NW) {
    // ---- products of a step, a quarter of the slabs at a time as they arrive; one lane waits and issues
    const uint64_t dlo = umma_smem_desc(smem_u32(lo), 16, 1024);
    const uint64_t dh = desc_sw64(smem_u32(hbuf), GROUP);
    const uint32_t acc = tmem + TMEM_COLS - NACC * N;
    for (int t = 0; t < steps; ++t) {
      bool ok = true;
      if (elect_one()) {
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const uint32_t full = smem_u32(&bar_full[g]);
          if (t > 0) {
            ok = wait_cluster(full, (t - 1) & 1, deadp, status) && ok;
            if (t + 1 < T && ok) mbar_expect_tx(full, group_bytes(g));
          }
          tc_fence_after();
#pragma unroll
          for (int s = g * GS; s < (g + 1) * GS; ++s) {
            // the leading products, CS / NMAIN slabs to an accumulator
            const uint32_t a1 = acc + (uint32_t)(s * NMAIN / CS * N), a2 = acc + NMAIN * N;
            const bool more = s % (CS / NMAIN) > 0;
            const uint64_t b = dh + (s * SLAB >> 4);
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
              umma_ts(a1, tmem + (uint32_t)(s * 16 + kk * 8), b + kk * 2, IDESC, (more || kk > 0) ? 1u : 0u);
              if (PH == 2)
                umma_ts(a2, tmem + (uint32_t)(s * 16 + kk * 8), b + (512 >> 4) + kk * 2, IDESC, (s > 0 || kk > 0) ? 1u : 0u);
              if (PW == 2) {
                const uint32_t on = (PH == 2 || s > 0 || kk > 0) ? 1u : 0u;
                if (s < LO_TM) umma_ts(a2, tmem + (uint32_t)((CS + s) * 16 + kk * 8), b + kk * 2, IDESC, on);
                else umma<false>(a2, dlo + (((s >> 1) * LO_BLOCK + (s & 1) * 64) >> 4) + kk * 2, b + kk * 2, IDESC, on);
              }
            }
          }
        }
        if (ok) {
          umma_commit(smem_u32(&bar_acc));
          if (t + 1 < T) umma_commit_cluster(smem_u32(&bar_empty), (uint16_t)((1u << C) - 1));
        }
      }
      __syncwarp();
      if (t + 1 < T) {
        if (bar_all_any(!ok)) break;                       // the new slab is staged: one copy to every peer
        if (lane < C) {
          const uint32_t peer = (uint32_t)(rank + lane < C ? rank + lane : rank + lane - C);
          bulk_to_peer(map_to_rank(smem_u32(hbuf) + (uint32_t)lane * SLAB, peer), smem_u32(stg), sent,
                       map_to_rank(smem_u32(&bar_full[lane / GS]), peer));
        }
        __syncwarp();
      }
    }
  } else {
    const size_t out_step = (size_t)a.B * H, comp = (size_t)T * out_step;
    const int q = warp & 3, cg4 = warp >> 2;
    constexpr int CW = N / 4;                              // accumulator columns per warp
    const float wsc = (q < 3) ? s_wscale[q * 32 + lane] : 0.f;
    float sh[RPW];
#pragma unroll
    for (int i = 0; i < RPW; ++i) sh[i] = (PH == 2) ? s_h[warp + i * NW] : 1.f;
    for (int t = 0; t < steps; ++t) {
      float ngr[RPW], ngz[RPW], ngn[RPW];
#pragma unroll
      for (int i = 0; i < RPW; ++i) {
        ngr[i] = ngz[i] = ngn[i] = 0.f;
        if (ok_row[i] && t + 1 < T) {
          const float* g = a.gi + ((size_t)(t + 1) * a.B + b0 + warp + i * NW) * 3 * H + u;
          ngr[i] = __ldcs(g); ngz[i] = __ldcs(g + H); ngn[i] = __ldcs(g + 2 * H);
        }
      }
      bool alive = mbar_wait(smem_u32(&bar_acc), t & 1, deadp, status);
      __syncwarp();
      tc_fence_after();
      if (q < 3) {
        const uint32_t tb = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(TMEM_COLS - NACC * N + cg4 * CW);
        float x[NACC][CW / 4][4];
#pragma unroll
        for (int p = 0; p < NACC; ++p)
#pragma unroll
          for (int c = 0; c < CW / 4; ++c)
            tmem_ld4(tb + p * N + c * 4, x[p][c]);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < CW; ++c) {
          const int b = cg4 * CW + c;
          float v = x[0][c / 4][c % 4];
#pragma unroll
          for (int p = 1; p < NACC; ++p) v = v + x[p][c / 4][c % 4];
          v = v * wsc;
          if (PH == 2) v = v * s_inv_h[b];
          S[(q * 32 + lane) * LDS + b] = v;
        }
      }
      tc_fence_before();
      bar_compute();

      float r_[RPW], z_[RPW], n_[RPW], g_[RPW];
#pragma unroll
      for (int i = 0; i < RPW; ++i) {
        // rows beyond the tile run on garbage, so that the rows of a thread interleave
        const int b = warp + i * NW;
        const float ghr = S[lane * LDS + b] + br, ghz = S[(32 + lane) * LDS + b] + bz, ghn = S[(64 + lane) * LDS + b] + bn;
        const GateOut go = gru_gates(gr[i], gz[i], gn[i], ghr, ghz, ghn, hown[i]);
        hown[i] = a.qout.enabled ? fake_quant<true>(go.h_raw, a.qout) : go.h_raw;
        r_[i] = go.r; z_[i] = go.z; n_[i] = go.n; g_[i] = ghn;
      }
      if (t + 1 < T) {
        // every peer has finished reading h_{t-1} (and so has received the slab this buffer held)
        alive = wait_cluster(smem_u32(&bar_empty), t & 1, deadp, status) && alive;
        __syncwarp();
#pragma unroll
        for (int i = 0; i < RPW; ++i) {
          const int b = warp + i * NW;
          if (b < rows8) {
            unsigned char* dst = stg + (b >> 3) * GROUP + sw64(b & 7, lane * 2);
            const float h = ok_row[i] ? hown[i] : 0.f;
            if (PH == 1) {
              *reinterpret_cast<__half*>(dst) = __float2half_rn(h_code(h, a.qin));
            } else {
              __half hi, lh;
              split2((a.qin.enabled ? fake_quant<true>(h, a.qin) : h) * sh[i], &hi, &lh);
              *reinterpret_cast<__half*>(dst) = hi;
              *reinterpret_cast<__half*>(dst + 512) = lh;
            }
          }
        }
        fence_async_smem();
        if (bar_all_any(!alive)) break;
      }
#pragma unroll
      for (int i = 0; i < RPW; ++i) {
        if (ok_row[i]) {
          const size_t o = (size_t)t * out_step + (size_t)(b0 + warp + i * NW) * H + u;
          a.out[o] = hown[i];
          if (a.save != nullptr) {
            __stcs(a.save + o, r_[i]);
            __stcs(a.save + comp + o, z_[i]);
            __stcs(a.save + 2 * comp + o, n_[i]);
            __stcs(a.save + 3 * comp + o, g_[i]);
          }
        }
        gr[i] = ngr[i]; gz[i] = ngz[i]; gn[i] = ngn[i];
      }
    }
  }
  leave_together(cluster, C, deadp, &peer_gave_up);
  if (warp == NW) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------------------------------------------
// backward (serial part): dgi[t], the dh chain, dh0.  Gate activations come from `S`.
// ---------------------------------------------------------------------------------------------------
template <int N, int TILES, int PW>
__global__ void __launch_bounds__(NT, 1) tcc_bwd_kernel(const Args a) {
  constexpr int R = N / NW;                                // a compute warp owns rows warp, warp + 16, ...
  constexpr uint32_t IDESC = umma_idesc(false, false, false, 128, N, 0u);
  constexpr uint32_t LO_BLK = 128 * 64;                    // lo plane in blocks (tile, gate): 128 positions x 32 units
  constexpr int LO_TM = lo_blocks_tmem(TILES, N);          // the first of them live in tensor memory
  constexpr uint32_t PLANE = 3 * N * 64;                   // bytes of one plane of dgh: [gate][N rows][32 units]
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) unsigned long long bar_recv, bar_empty, bar_acc[4];
  __shared__ uint32_t tmem_slot;
  __shared__ int dead, peer_gave_up, unhealthy;
  __shared__ float s_fold[ROWS_A], s_scale[ROWS_A];
  __shared__ __align__(16) float s_inv[2][4 * NW];          // inverse row scales of dgh, by step parity

  cg::cluster_group cluster = cg::this_cluster();
  const int warp = uniform_warp(), lane = threadIdx.x & 31, tid = threadIdx.x;
  const int C = a.C, Hb = a.Hb, H = a.H;
  const int rank = blockIdx.x % C;
  const int problem = blockIdx.x / C;
  const int n = problem / a.ntiles_b;
  const int b0 = (problem - n * a.ntiles_b) * a.rows;
  const int nrows = min(a.rows, a.B - b0);
  const int RG = (a.rows + 3) >> 2;                        // groups of four rows that are exchanged
  const int u0 = rank * UNITS;
  const int T = a.T;
  volatile int* deadp = &dead;
  int* status = a.status;
  const uint32_t recv_bytes = (uint32_t)(C * RG * 512);

  unsigned char* lo = smem;                                // [block][128 positions][32 units]
  unsigned char* bop = smem + (PW == 2 ? (3 * TILES - LO_TM) * LO_BLK : 0);
  float* recv = reinterpret_cast<float*>(bop + 2 * PLANE); // [source][row group][unit][4 rows]
  float* stage = recv + (size_t)C * RG * 128;              // [destination][row group][unit][4 rows]

  if (tid == 0) {
    dead = peer_gave_up = 0;
    unhealthy = *reinterpret_cast<volatile int*>(status);
    mbar_init(smem_u32(&bar_recv), 1);
    mbar_init(smem_u32(&bar_empty), C);
    for (int m = 0; m < 4; ++m) mbar_init(smem_u32(&bar_acc[m]), 1);
    mbar_fence_init();
    mbar_expect_tx(smem_u32(&bar_recv), recv_bytes);
  }
  if (warp == NW) tmem_alloc(smem_u32(&tmem_slot), 512);

  // ---- scale of every own weight row: a power of two for fp32 weights (undone in dgh before it is
  // split), the code scale for int8 weights
  if (warp < NW) {
    for (int i = warp; i < ROWS_A; i += NW) {
      const int g = i >> 5, j = i & 31;
      const bool own = u0 + j < Hb;
      float s = 1.f, inv = 1.f;
      if (PW == 2) {
        // All loads in flight at once, from clamped addresses (an entry read twice does not change the maximum): under a
        // condition each waited for the one before it, and the prologue took 28 us at H = 512 instead of 17.
        const float* src = a.W + (size_t)g * a.w_gate_stride + (size_t)n * a.w_block_stride + (size_t)(own ? u0 + j : 0) * Hb;
        float mx = 0.f;
#pragma unroll
        for (int q = 0; q < TILES * 4; ++q) mx = fmaxf(mx, fabsf(__ldg(src + min(lane + 32 * q, Hb - 1))));
        pow2_row_scale(warp_max(mx), &s, &inv);
      } else {
        inv = own ? a.scales[g * H + u0 + j] : 0.f;
      }
      if (lane == 0) { s_scale[i] = s; s_fold[i] = inv; }
    }
    // rows of the operand that no thread writes stay zero
    for (int i = tid; i < (int)(2 * PLANE / 16); i += 32 * NW) reinterpret_cast<uint4*>(bop)[i] = make_uint4(0, 0, 0, 0);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t acc = tmem + (uint32_t)(TMEM_COLS - TILES * N);
  const int m_own = warp >> 2, q_own = warp & 3;           // accumulator tile and lane quarter of a compute warp
  if (warp < NW && m_own < TILES) {
    const int k = m_own * 128 + q_own * 32 + lane;         // position: row of the transposed weights
#pragma unroll 1
    for (int g = 0; g < 3; ++g) {
      uint32_t vh[16], vl[16];
      const int kc = min(k, Hb - 1);
      float w[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const int jr = min(u0 + j, Hb - 1);
        w[j] = PW == 1 ? (float)a.codes[((size_t)g * H + jr) * Hb + kc]
                       : __ldg(a.W + (size_t)g * a.w_gate_stride + (size_t)n * a.w_block_stride + (size_t)jr * Hb + kc);
      }
#pragma unroll
      for (int j2 = 0; j2 < 16; ++j2) {
        __half hi[2], lw[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int j = 2 * j2 + e;
          split2((k < Hb && u0 + j < Hb) ? w[j] * s_scale[g * 32 + j] : 0.f, &hi[e], &lw[e]);
        }
        vh[j2] = pack2(hi[0], hi[1]);
        vl[j2] = pack2(lw[0], lw[1]);
      }
      tmem_st16(tmem + ((uint32_t)(q_own * 32) << 16) + (uint32_t)(m_own * 48 + g * 16), vh);
      const int blk = m_own * 3 + g;
      if (PW == 2 && blk < LO_TM) {
        tmem_st16(tmem + ((uint32_t)(q_own * 32) << 16) + (uint32_t)(TILES * 48 + blk * 16), vl);
      } else if (PW == 2) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *reinterpret_cast<uint4*>(lo + (size_t)(blk - LO_TM) * LO_BLK + sw64((uint32_t)(k & 127), c * 16)) =
              make_uint4(vl[4 * c], vl[4 * c + 1], vl[4 * c + 2], vl[4 * c + 3]);
      }
    }
    tmem_st_wait();
  }

  const int u = n * Hb + u0 + lane;
  const bool unit_ok = warp < NW && u0 + lane < Hb;
  const size_t out_step = (size_t)a.B * H, comp = (size_t)T * out_step;
  float c_do[R], c_r[R], c_z[R], c_n[R], c_ghn[R], c_hp[R], dh_direct[R], mask_in[R];
  bool ok[R];
  const float fr = (warp < NW) ? s_fold[lane] : 0.f, fz = (warp < NW) ? s_fold[32 + lane] : 0.f, fn = (warp < NW) ? s_fold[64 + lane] : 0.f;

  const size_t row0 = (size_t)(b0 + warp) * H + u;         // first owned element; the others are NW rows apart
  auto fetch = [&](int t) {
    if (t < 0) return;
    // one base per array keeps the loop's registers down (17 warps leave 96 a thread; -Xptxas -v reports 72 to 136 bytes
    // spilled in the backward kernels, and a spill can miss the little L1 cache that is left beside shared memory)
    const size_t o = (size_t)t * out_step + row0;
    const float* pd = a.dout + o;
    const float* ps = a.S + o;
    const float* ph = (t > 0) ? a.out + (o - out_step) : a.h0 + row0;
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (ok[i]) {
        const float* q = ps + i * NW * H;
        c_do[i] = __ldcs(pd + i * NW * H);
        c_r[i] = __ldcs(q); q += comp;
        c_z[i] = __ldcs(q); q += comp;
        c_n[i] = __ldcs(q); q += comp;
        c_ghn[i] = __ldcs(q);
        c_hp[i] = ph[i * NW * H];
      }
  };
#pragma unroll
  for (int i = 0; i < R; ++i) {
    ok[i] = unit_ok && warp + NW * i < nrows;
    dh_direct[i] = 0.f; mask_in[i] = 1.f;
    c_do[i] = c_r[i] = c_z[i] = c_n[i] = c_ghn[i] = c_hp[i] = 0.f;
  }
  fetch(T - 1);
  fence_async_smem();
  tc_fence_before();
  cluster.sync();
  tc_fence_after();

  // nothing is done where the status word was set when rank 0 started: the cluster leaves as one
  const int last = __any_sync(0xffffffffu, load_at_peer(map_to_rank(smem_u32(&unhealthy), 0)) != 0) ? -1 : T;
  if (warp == NW) {
    const uint64_t db0 = desc_sw64(smem_u32(bop), 512);
    const uint64_t da0 = desc_sw64(smem_u32(lo), 512);
    for (int it = 0; it < last; ++it) {
      if (bar_all_any(false)) break;                       // dgh of this step is in place
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int m = 0; m < TILES; ++m) {
          const uint32_t d = acc + (uint32_t)(m * N);
          // one truncating accumulator: the small products first, then six of the leading ones on top of them
#pragma unroll
          for (int kk = 0; kk < 6; ++kk) {
            const uint64_t b = db0 + (((kk >> 1) * (N * 64) + (kk & 1) * 32) >> 4);
            umma_ts(d, tmem + (uint32_t)(m * 48 + kk * 8), b + (PLANE >> 4), IDESC, kk > 0 ? 1u : 0u);
            const int blk = m * 3 + (kk >> 1);
            if (PW == 2 && blk < LO_TM)
              umma_ts(d, tmem + (uint32_t)(TILES * 48 + blk * 16 + (kk & 1) * 8), b, IDESC, 1u);
            else if (PW == 2)
              umma<false>(d, da0 + (((blk - LO_TM) * LO_BLK + (kk & 1) * 32) >> 4), b, IDESC, 1u);
          }
#pragma unroll
          for (int kk = 0; kk < 6; ++kk)
            umma_ts(d, tmem + (uint32_t)(m * 48 + kk * 8), db0 + (((kk >> 1) * (N * 64) + (kk & 1) * 32) >> 4), IDESC, 1u);
          umma_commit(smem_u32(&bar_acc[m]));
        }
      }
      __syncwarp();
    }
  } else {
    bool alive = true;                                     // every wait of this warp so far
    for (int it = 0; it <= last; ++it) {
      const int t = T - 1 - it;
      float dh[R];
#pragma unroll
      for (int i = 0; i < R; ++i) dh[i] = 0.f;
      if (it > 0) {
        alive = wait_cluster(smem_u32(&bar_recv), (it - 1) & 1, deadp, status) && alive;
        __syncwarp();
        if (tid == 0 && it < T && alive) mbar_expect_tx(smem_u32(&bar_recv), recv_bytes);
        // scalar reads of [unit][4 rows]: the rows of a unit are rotated by unit / 8, so that the 32 units of a row
        // lie in 32 banks
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const int b = warp + NW * i;
          if (b < 4 * RG) {
            const float* src = recv + (b >> 2) * 128 + lane * 4 + ((b + (lane >> 3)) & 3);
            float s = 0.f;
#pragma unroll 4
            for (int r = 0; r < C; ++r, src += RG * 128) s += *src;
            dh[i] = dh_direct[i] + s * mask_in[i];
          }
        }
      }
      if (it == T) {
#pragma unroll
        for (int i = 0; i < R; ++i)
          if (ok[i]) a.dh0[row0 + i * NW * H] = dh[i];
        break;
      }
      float gr[R], gz[R], gn[R];
      // the products of the previous step have read the operand (this rank's partial sums may be
      // complete while the last tiles are still under way)
      if (it > 0) alive = mbar_wait(smem_u32(&bar_acc[TILES - 1]), (it - 1) & 1, deadp, status) && alive;
      __syncwarp();
#pragma unroll
      for (int i = 0; i < R; ++i) {
        // entries beyond the batch run on zeros, so that the rows of a thread interleave
        float d = c_do[i] + dh[i];
        if (a.qout.enabled) {
          const float h_raw = (1.0f - c_z[i]) * c_n[i] + c_z[i] * c_hp[i];
          d = d * ste_mask<true>(h_raw, a.qout);
        }
        if (!ok[i]) d = 0.f;
        const GateGrad gg = gru_gate_grads(d, c_r[i], c_z[i], c_n[i], c_ghn[i], c_hp[i]);
        dh_direct[i] = gg.dh_direct;
        mask_in[i] = a.qin.enabled ? ste_mask<true>(c_hp[i], a.qin) : 1.0f;
        gr[i] = gg.dgr; gz[i] = gg.dgz; gn[i] = gg.dgn;
        // operand planes, scaled by a power of two of this row's largest entry
        const float vr = gr[i] * fr, vz = gz[i] * fz, vn = gg.dghn * fn;
        float s, inv;
        pow2_row_scale(warp_max(fmaxf(fabsf(vr), fmaxf(fabsf(vz), fabsf(vn)))), &s, &inv);
        const int b = warp + NW * i;
        if (lane == 0) s_inv[it & 1][b] = inv;
        unsigned char* dst = bop + sw64((uint32_t)b, lane * 2);
        __half hi, lw;
        split2(vr * s, &hi, &lw);
        *reinterpret_cast<__half*>(dst) = hi; *reinterpret_cast<__half*>(dst + PLANE) = lw;
        split2(vz * s, &hi, &lw);
        *reinterpret_cast<__half*>(dst + N * 64) = hi; *reinterpret_cast<__half*>(dst + N * 64 + PLANE) = lw;
        split2(vn * s, &hi, &lw);
        *reinterpret_cast<__half*>(dst + 2 * N * 64) = hi; *reinterpret_cast<__half*>(dst + 2 * N * 64 + PLANE) = lw;
      }
      // operands of the next step: ahead of the partial sums, behind whose stores a load would queue
      fetch(t - 1);
      fence_async_smem();
      if (bar_all_any(!alive)) break;
      // the partial sums of the previous step have been read: peers may overwrite them
      if (it > 0 && warp < C && lane == 0) arrive_at_peer(map_to_rank(smem_u32(&bar_empty), (uint32_t)warp));
      __syncwarp();
      // ---- partial sums of 32 positions to the rank that owns them
      const int dest = m_own * 4 + q_own;
      if (dest < C) {
        bool ready = mbar_wait(smem_u32(&bar_acc[m_own]), it & 1, deadp, status);
        if (it > 0) ready = wait_cluster(smem_u32(&bar_empty), (it - 1) & 1, deadp, status) && ready;
        alive = alive && ready;
        __syncwarp();
        tc_fence_after();
        const uint32_t ts = acc + ((uint32_t)(q_own * 32) << 16) + (uint32_t)(m_own * N);
        const int rot = lane >> 3;
        for (int rg = 0; rg < RG; ++rg) {
          float v[4];
          tmem_ld4(ts + rg * 4, v);
          tmem_ld_wait();
          const float4 iv = *reinterpret_cast<const float4*>(&s_inv[it & 1][rg * 4]);
          float x0 = v[0] * iv.x, x1 = v[1] * iv.y, x2 = v[2] * iv.z, x3 = v[3] * iv.w;
          if (rot & 1) { const float y = x3; x3 = x2; x2 = x1; x1 = x0; x0 = y; }
          if (rot & 2) { const float y0 = x0, y1 = x1; x0 = x2; x1 = x3; x2 = y0; x3 = y1; }
          *reinterpret_cast<float4*>(stage + (size_t)(dest * RG + rg) * 128 + lane * 4) = make_float4(x0, x1, x2, x3);
        }
        tc_fence_before();
        fence_async_smem();
        __syncwarp();
        if (lane == 0 && ready)
          bulk_to_peer(map_to_rank(smem_u32(recv) + (uint32_t)(rank * RG * 512), (uint32_t)dest),
                       smem_u32(stage + (size_t)dest * RG * 128), (uint32_t)(RG * 512),
                       map_to_rank(smem_u32(&bar_recv), (uint32_t)dest));
        __syncwarp();
      }
      // off the chain
#pragma unroll
      for (int i = 0; i < R; ++i)
        if (ok[i]) {
          float* d = a.dgi + ((size_t)t * a.B + b0 + warp) * 3 * H + u + i * NW * 3 * H;
          __stcs(d, gr[i]); __stcs(d + H, gz[i]); __stcs(d + 2 * H, gn[i]);
        }
    }
  }
  leave_together(cluster, C, deadp, &peer_gave_up);
  if (warp == NW) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------
typedef void (*Kernel)(const Args);

template <int N, int CS>
static Kernel pick_fwd(int pw, int ph) {
  if (pw == 2) return ph == 2 ? tcc_fwd_kernel<N, CS, 2, 2> : tcc_fwd_kernel<N, CS, 2, 1>;
  return tcc_fwd_kernel<N, CS, 1, 1>;
}
template <int N>
static Kernel pick_n(bool fwd, int cs, int pw, int ph) {
  switch (cs) {
    case 4: return fwd ? pick_fwd<N, 4>(pw, ph) : (pw == 2 ? tcc_bwd_kernel<N, 1, 2> : tcc_bwd_kernel<N, 1, 1>);
    case 8: return fwd ? pick_fwd<N, 8>(pw, ph) : (pw == 2 ? tcc_bwd_kernel<N, 2, 2> : tcc_bwd_kernel<N, 2, 1>);
    default: return fwd ? pick_fwd<N, 16>(pw, ph) : (pw == 2 ? tcc_bwd_kernel<N, 4, 2> : tcc_bwd_kernel<N, 4, 1>);
  }
}
static Kernel pick(bool fwd, int N, int cs, int pw, int ph) {
  switch (N) {
    case 16: return pick_n<16>(fwd, cs, pw, ph);
    case 32: return pick_n<32>(fwd, cs, pw, ph);
    default: return pick_n<48>(fwd, cs, pw, ph);
  }
}
static int slab_count(int C) { return C <= 4 ? 4 : (C <= 8 ? 8 : 16); }

// Stands in for the scan kernels in the occupancy query: all of them run one CTA per SM, so the answer
// depends on the cluster size alone, and asking about each of them would load its code.
__global__ void __launch_bounds__(NT, 1) occupancy_probe_kernel() {}

constexpr size_t STATIC_SMEM = 4096;         // more than any of the kernels declares, and what the system reserves

// Clusters of C CTAs the device holds at once (0: none can be launched), the shared memory a CTA may ask for, and
// the least that every launch asks for: half of an SM's.  A CTA takes all 512 columns of tensor memory and then waits
// for its cluster; a second one on its SM would wait for those columns, and its cluster for it, for good.  Half an
// SM's memory beside the static part keeps out a second CTA of these kernels and, since they ask for more than
// that too, one of the tcgen05 products that another stream may run.
struct Device { int active[MAX_C + 1]; size_t smem, least; };
static Device device_limits(int C) {
  static std::mutex mu;
  static std::map<int, Device> cache;
  int dev = -1;
  Device none;
  memset(&none, 0, sizeof(none));
  if (cudaGetDevice(&dev) != cudaSuccess) return none;
  std::lock_guard<std::mutex> lk(mu);
  auto it = cache.find(dev);
  if (it == cache.end()) {
    Device d = none;
    for (int c = 0; c <= MAX_C; ++c) d.active[c] = -1;
    int optin = 0, per_sm = 0;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess || optin < 65536) return none;
    if (cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess) return none;
    d.smem = (size_t)optin - STATIC_SMEM;
    d.least = (size_t)per_sm / 2;
    if (d.least > d.smem) return none;
    it = cache.emplace(dev, d).first;
  }
  Device& d = it->second;
  if (d.active[C] < 0) {
    const void* fn = (const void*)occupancy_probe_kernel;
    int n = 0;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)d.smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C); cfg.blockDim = dim3(NT); cfg.dynamicSmemBytes = d.smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, fn, &cfg);
    if (e != cudaSuccess) { cudaGetLastError(); n = 0; }
    d.active[C] = n;
  }
  return d;
}

// Once per (device, kernel): the attributes of its launch.
static bool prepare_kernel(Kernel fn, size_t smem) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, bool> done;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  if (allow_dynamic_smem((const void*)fn, smem) != B200GRU_OK) return false;
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_pair(dev, (const void*)fn);
  auto it = done.find(key);
  if (it == done.end()) {
    const bool ok = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    if (!ok) cudaGetLastError();
    it = done.emplace(key, ok).first;
  }
  return it->second;
}

bool choose(bool fwd, int T, int B, int Hb, int nb, bool w_codes, const Quant& qin, Config* out, double* cycles) {
  if (Hb > UNITS * MAX_C || Hb < 1) return false;
  const int C = cdiv(Hb, UNITS);
  // one CTA per problem leaves the backward its full fixed cost and no more FMAs to save (Hb = 32, nb = 4, B = 200:
  // 131 us against 106 of the FP32 kernel at T = 32)
  if (C == 1 && !fwd && test_kernel_choice(2) != 2) return false;
  const int cs = slab_count(C);
  const int ph = (qin.enabled && qin.qmin >= -128.f && qin.qmax <= 127.f) ? 1 : 2;
  // codes of weights and state are exact in one accumulator; an unquantised state takes the fp32 form of the weights
  const int pw = w_codes && (!fwd || ph == 1) ? 1 : 2;
  const Device dev = device_limits(C);
  const int active = dev.active[C];
  if (active <= 0) return false;
  bool found = false;
  for (int N = 16; N <= MAX_N; N += 16) {
    int rows = B < N ? B : N;
    size_t smem = 0;
    auto fits = [&](int r) {
      smem = fwd ? fwd_layout(cs, N, pw, ph).total : bwd_layout(C, cs / 4, N, r, pw).total;
      return smem <= dev.smem;
    };
    while (!fits(rows) && rows > N - 12 && rows > 4) rows -= 4;        // the backward buffers grow with the rows
    if (!fits(rows)) continue;
    // spread the batch evenly over the waves that it needs anyway
    const long long waves_max = ((long long)nb * cdiv(B, rows) + active - 1) / active;
    const int per_block = (int)(waves_max * active / nb);
    if (per_block >= 1 && cdiv(B, per_block) < rows) {
      rows = cdiv(B, per_block);
      if (!fits(rows)) continue;
    }
    const long long clusters = (long long)nb * cdiv(B, rows);
    const double waves = (double)((clusters + active - 1) / active);
    // Cycles of a step as measured over C = 1 .. 16 and 1 .. 43 rows (within 15 %): a fixed part, the gate work of
    // 16 rows, and per CTA of the cluster one bulk copy and its bytes (the backward shares the SM's outgoing
    // port with dgi and is slower).  H = 512: forward 4700 at 4 rows and 11700 at 43; backward 5400 at 5, 9000 at 19.
    // With few rows the forward is bound by issuing the products of its CS slabs: 2500 cycles at 4 slabs, 4700 at 16
    // (int8 state: 2350 and 3950; integer codes of both operands fewer still).  The backward of small clusters lies above
    // its exchange as well: with 300 rows of 64 units it takes 736 us where the FP32 kernel takes 640.
    static const double least[3][3] = {{2500.0, 2950.0, 4650.0}, {2350.0, 2750.0, 3900.0}, {2100.0, 2400.0, 3400.0}};
    const double slab = fwd ? (double)ph * ((rows + 7) / 8 * 8) * 64 : (double)((rows + 3) / 4) * 512;
    double step = fwd ? 750.0 + C * (60.0 + slab / 15.0) + 1000.0 * (N / 16) : 1300.0 + C * (50.0 + slab / 8.3) + 1000.0 * (N / 16);
    if (fwd) {
      const double low = least[pw == 1 ? 2 : 2 - ph][cs / 8] + 1000.0 * (N / 16 - 1);
      if (step < low) step = low;
    } else if (cs == 4) {
      step *= 1.3;
    }
    // set-up (weights into tensor memory), from T = 1 and T = 4 launches
    const double setup = fwd ? 12000.0 + 750.0 * C : 18500.0 + 850.0 * C;
    const double cost = waves * (step * T + setup);
    if (!found || cost < *cycles) {
      found = true;
      *cycles = cost;
      out->C = C; out->N = N; out->rows = rows; out->pw = pw; out->ph = ph; out->clusters = (int)clusters;
      out->active = active; out->smem = smem > dev.least ? smem : dev.least;
    }
  }
  return found;
}

static int* status_address() {
  static std::mutex mu;
  static std::map<int, int*> table;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lk(mu);
  int*& p = table[dev];
  if (p == nullptr) {
    void* q = nullptr;
    if (cudaGetSymbolAddress(&q, g_tcc_status) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    p = static_cast<int*>(q);
  }
  return p;
}

int launch(bool fwd, const Config& c, Args a, cudaStream_t st) {
  a.C = c.C; a.rows = c.rows; a.rows8 = (c.rows + 7) / 8 * 8; a.ntiles_b = cdiv(a.B, c.rows);
  a.status = status_address();
  if (a.status == nullptr) return B200GRU_LAUNCH_FAILURE;
  Kernel fn = pick(fwd, c.N, slab_count(c.C), c.pw, c.ph);
  if (!prepare_kernel(fn, c.smem)) return B200GRU_UNSUPPORTED;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(c.C * c.clusters)); cfg.blockDim = dim3(NT); cfg.dynamicSmemBytes = c.smem; cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = c.C; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, fn, a);
  note_launch();
  return check_launch(fwd ? "tcc_fwd_kernel" : "tcc_bwd_kernel");
}

int set_status(int value) { return cudaMemcpyToSymbol(g_tcc_status, &value, sizeof(int)) == cudaSuccess ? B200GRU_OK : B200GRU_LAUNCH_FAILURE; }

int read_status(int reset) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_tcc_status, sizeof(int)) != cudaSuccess) return -1;
  if (reset && v != 0) {
    const int z = 0;
    cudaMemcpyToSymbol(g_tcc_status, &z, sizeof(int));
  }
  return v;
}

}  // namespace tcc
}  // namespace b200gru
