// A whole layer call in one C entry per direction: weight gathering, operand planes, input projection,
// scan; and backward the scan, the weight gradients, the bias sums and the input gradient.
//
// The host path of a layer call used to be Python: four concatenations, two autograd functions, a dozen
// library calls.  For one step of one sequence that was 190 us of host work around 23 us of kernels.
// Here the caller passes the layer's parameters as they lie (one pointer per gate) and buffers of
// the sizes b200gru_layer_sizes() names; one kernel gathers the weights.
//
// Reference: src/gru_qat/gru_layer.py:234-302 (dispatch), src/gru_qat/gru_cell.py:410-435 (projection).

#include <cstring>

#include <cuda_fp16.h>

#include "tc_gemm.cuh"
#include "tc_scan.cuh"

namespace b200gru {
namespace {

using namespace tc;

constexpr int ROW_CHUNK = 32768;             // rows of x / dgi whose operand planes exist at a time

struct Layer {
  b200gru_shape shape;
  int T, B, I, H, bits_i, bits_h, flags;
  size_t rows, w_elems;                      // T * B; elements of the hidden weights (all gates)
};

bool parse(const int* dims, Layer* L) {
  memset(L, 0, sizeof(*L));
  L->shape.kind = dims[0]; L->T = dims[1]; L->B = dims[2]; L->I = dims[3]; L->H = dims[4];
  L->shape.T = L->T; L->shape.B = L->B; L->shape.H = L->H; L->shape.nblocks = dims[5]; L->shape.log2_hpad = dims[6];
  L->bits_i = dims[7]; L->bits_h = dims[8]; L->flags = dims[9];
  if (L->T <= 0 || L->B <= 0 || L->I <= 0 || L->H <= 0 || (L->I & 7) || (L->H & 7)) return false;
  if ((long long)L->T * L->B > 0x7fffffffLL / 4) return false;
  if (L->bits_i < 2 || L->bits_h < 2 || (L->bits_i > 8 && L->bits_i != 32) || (L->bits_h > 8 && L->bits_h != 32)) return false;
  if (L->bits_h <= 8 && L->shape.kind != B200GRU_DENSE) return false;
  L->rows = (size_t)L->T * L->B;
  const size_t H = L->H;
  switch (L->shape.kind) {
    case B200GRU_DENSE: L->w_elems = 3 * H * H; break;
    case B200GRU_DIAGONAL: L->w_elems = 3 * H; break;
    case B200GRU_MONARCH:
      if (dims[5] <= 0 || L->H % dims[5]) return false;
      L->w_elems = 3 * H * (H / dims[5]);
      break;
    case B200GRU_BUTTERFLY:
      if (dims[5] <= 0 || dims[6] <= 0 || dims[6] > 20 || (1 << dims[6]) < L->H) return false;
      L->w_elems = (size_t)3 * dims[5] * dims[6] * ((size_t)1 << (dims[6] - 1)) * 4;
      break;
    default: return false;
  }
  return true;
}

size_t pad(size_t n) { return align_up(n, 256); }

// What the weights become, and the backward needs again.
struct Kept {
  float* Wh;             // [w_elems] gathered hidden weights (raw)
  float* b_i;            // [3H]
  float* b_h;            // [3H]
  __half* Wi_op;         // fp16 planes [2][3H][I], or one plane of codes
  float* Wi_scale;       // [3H]: inverse power-of-two row scales, or the scales of the codes
  float* Wi;             // quantised input weights: gathered raw values [3H][I]
  signed char* Wi_codes;
  signed char* Wh_codes; // quantised hidden weights
  float* Wh_scale;
  float* Wh_q;           // codes * scales
};

size_t carve(const Layer& L, char* base, Kept* k) {
  const size_t n3 = (size_t)3 * L.H, wi = n3 * L.I;
  size_t at = 0;
  auto take = [&](size_t bytes) { char* p = base == nullptr ? nullptr : base + at; at += pad(bytes); return p; };
  memset(k, 0, sizeof(*k));
  k->Wh = (float*)take(L.w_elems * 4);
  k->b_i = (float*)take(n3 * 4);
  k->b_h = (float*)take(n3 * 4);
  k->Wi_scale = (float*)take(n3 * 4);
  k->Wi_op = (__half*)take(wi * (L.bits_i <= 8 ? 2 : 4));
  if (L.bits_i <= 8) {
    k->Wi = (float*)take(wi * 4);
    k->Wi_codes = (signed char*)take(wi);
  }
  if (L.bits_h <= 8) {
    k->Wh_codes = (signed char*)take(L.w_elems);
    k->Wh_scale = (float*)take(n3 * 4);
    k->Wh_q = (float*)take(L.w_elems * 4);
  }
  return at;
}

// ---- weight gathering ------------------------------------------------------------------------------
// Blocks [0, split_blocks) turn the input weights into two row-scaled fp16 planes (a warp per row, as
// split_rows_f16_kernel does); the others copy the per-gate tensors into one.  Bound by latency: 1.5 to 9 MB.
struct Gather {
  const float* src[3];
  float* dst;
  unsigned n;            // elements per gate
  int vec;               // float4 copies
};
struct PrepArgs {
  Gather copy[4];
  int ncopy;
  const float* Wi[3];
  __half* planes;
  float* inv;
  int H, I, split_blocks;
};

__global__ void __launch_bounds__(256) layer_prep_kernel(const PrepArgs a) {
  pdl_launch_dependents();
  if ((int)blockIdx.x < a.split_blocks) {
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= 3 * a.H) return;
    const int g = row / a.H;
    const float* s = a.Wi[g] + (size_t)(row - g * a.H) * a.I;
    float mx = 0.f;
    for (int i = lane; i < a.I; i += 32) mx = fmaxf(mx, fabsf(__ldg(s + i)));
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    float sc, inv;
    pow2_row_scale(mx, &sc, &inv);
    if (lane == 0) a.inv[row] = inv;
    __half* d = a.planes + (size_t)row * a.I;
    const size_t plane = (size_t)3 * a.H * a.I;
    for (int i = lane * 2; i < a.I; i += 64) {             // I % 8 == 0
      const float x = __ldg(s + i) * sc, y = __ldg(s + i + 1) * sc;
      const __half hx = __float2half_rn(x), hy = __float2half_rn(y);
      *reinterpret_cast<__half2*>(d + i) = __halves2half2(hx, hy);
      *reinterpret_cast<__half2*>(d + plane + i) = __halves2half2(__float2half_rn(x - __half2float(hx)), __float2half_rn(y - __half2float(hy)));
    }
    return;
  }
  const size_t t0 = (size_t)(blockIdx.x - a.split_blocks) * 256 + threadIdx.x, stride = (size_t)(gridDim.x - a.split_blocks) * 256;
  for (int c = 0; c < a.ncopy; ++c) {
    const Gather& g = a.copy[c];
    for (int q = 0; q < 3; ++q) {
      float* dst = g.dst + (size_t)q * g.n;
      if (g.src[q] == nullptr) {
        for (size_t i = t0; i < g.n; i += stride) dst[i] = 0.f;
      } else if (g.vec) {
        const float4* s4 = reinterpret_cast<const float4*>(g.src[q]);
        for (size_t i = t0; i < g.n / 4; i += stride) reinterpret_cast<float4*>(dst)[i] = __ldg(s4 + i);
      } else {
        for (size_t i = t0; i < g.n; i += stride) dst[i] = __ldg(g.src[q] + i);
      }
    }
  }
}

__global__ void __launch_bounds__(256)
codes_to_f16_kernel(const signed char* __restrict__ src, __half* __restrict__ dst, size_t n4) {
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n4) return;
  const char4 c = reinterpret_cast<const char4*>(src)[i];
  __half2* d = reinterpret_cast<__half2*>(dst) + 2 * i;
  d[0] = __halves2half2(__float2half_rn((float)c.x), __float2half_rn((float)c.y));
  d[1] = __halves2half2(__float2half_rn((float)c.z), __float2half_rn((float)c.w));
}

// x -> integer codes of a frozen quantiser, exact in fp16.  A NaN stays one: the clamp would make a code of it, and a
// broken frame would come out as ordinary numbers.
__global__ void __launch_bounds__(256)
quantize_to_f16_kernel(const float* __restrict__ x, __half* __restrict__ dst, size_t n4, Quant q) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n4) return;
  const float4 v = __ldcs(reinterpret_cast<const float4*>(x) + i);
  const float e[4] = {v.x, v.y, v.z, v.w};
  __half h[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) h[k] = __float2half_rn(e[k] == e[k] ? fminf(fmaxf(fq_code(e[k], q), q.qmin), q.qmax) : e[k]);
  __half2* d = reinterpret_cast<__half2*>(dst) + 2 * i;
  d[0] = __halves2half2(h[0], h[1]);
  d[1] = __halves2half2(h[2], h[3]);
}

bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int gather_weights(const Layer& L, const Kept& k, const float* const* Wi, const float* const* Wh, const float* const* bi,
                   const float* const* bh, cudaStream_t st) {
  PrepArgs a;
  memset(&a, 0, sizeof(a));
  auto add = [&](const float* const* src, float* dst, size_t each) {
    Gather& g = a.copy[a.ncopy++];
    g.dst = dst; g.n = (unsigned)each; g.vec = (each % 4 == 0);
    for (int q = 0; q < 3; ++q) { g.src[q] = src[q]; if (!al16(src[q])) g.vec = 0; }
  };
  add(Wh, k.Wh, L.w_elems / 3);
  add(bi, k.b_i, L.H);
  add(bh, k.b_h, L.H);
  a.H = L.H; a.I = L.I;
  if (L.bits_i <= 8) {
    add(Wi, k.Wi, (size_t)L.H * L.I);
  } else {
    for (int q = 0; q < 3; ++q) a.Wi[q] = Wi[q];
    a.planes = k.Wi_op; a.inv = k.Wi_scale;
    a.split_blocks = cdiv(3 * L.H, 8);
  }
  const size_t most = (L.w_elems + (L.bits_i <= 8 ? (size_t)3 * L.H * L.I : 0)) / 4;
  int copy_blocks = (int)((most + 1023) / 1024);           // a few float4 per thread
  if (copy_blocks > 592) copy_blocks = 592;
  if (copy_blocks < 1) copy_blocks = 1;
  layer_prep_kernel<<<a.split_blocks + copy_blocks, 256, 0, st>>>(a);
  note_launch();
  int rc = check_launch("layer_prep_kernel");
  if (rc) return rc;
  if (L.bits_i <= 8) {
    rc = launch_quantize_rows(k.Wi, 3 * L.H, L.I, L.bits_i, k.Wi_codes, k.Wi_scale, nullptr, st);
    if (rc) return rc;
    const size_t n4 = (size_t)3 * L.H * L.I / 4;
    codes_to_f16_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, st>>>(k.Wi_codes, k.Wi_op, n4);
    note_launch();
  }
  if (L.bits_h <= 8) rc = launch_quantize_rows(k.Wh, 3 * L.H, L.H, L.bits_h, k.Wh_codes, k.Wh_scale, k.Wh_q, st);
  return rc ? rc : check_launch("weight preparation");
}

// Cross products of order < most, the smallest first: the accumulator of the tensor core truncates, and what it loses
// goes with what it already holds (error of a 3072-term product of two fp16 planes each: 6.2e-7 with the leading
// product first, 3.8e-7 with it last).
int fill_pairs(TcGemm* g, int na, int nb, int most) {
  g->npairs = 0;
  for (int s = most - 1; s >= 0; --s)
    for (int i = 0; i <= s; ++i)
      if (i < na && s - i < nb) { g->pa[g->npairs] = i; g->pb[g->npairs] = s - i; ++g->npairs; }
  return g->npairs;
}

size_t chunk_rows(const Layer& L) { return L.rows < (size_t)ROW_CHUNK ? L.rows : (size_t)ROW_CHUNK; }
size_t x_planes_bytes(const Layer& L) { return pad(chunk_rows(L) * L.I * 4) + pad(chunk_rows(L) * 4); }

// gi = x . Wi^T + b_i
int project(const Layer& L, const Kept& k, const float* x, const Quant& qx, float* gi, char* scratch, cudaStream_t st) {
  __half* xp = reinterpret_cast<__half*>(scratch);
  float* inv = reinterpret_cast<float*>(scratch + pad(chunk_rows(L) * L.I * 4));
  for (size_t r0 = 0; r0 < L.rows; r0 += ROW_CHUNK) {
    const int n = (int)(L.rows - r0 < (size_t)ROW_CHUNK ? L.rows - r0 : (size_t)ROW_CHUNK);
    TcGemm g;
    memset(&g, 0, sizeof(g));
    int rc;
    if (qx.enabled) {
      const size_t n4 = (size_t)n * L.I / 4;
      if (!al16(x)) return B200GRU_INVALID_ARGUMENT;
      launch_pdl(quantize_to_f16_kernel, dim3((unsigned)((n4 + 255) / 256)), dim3(256), 0, st, x + r0 * L.I, xp, n4, qx);
      note_launch();
      rc = check_launch("quantize_to_f16_kernel");
    } else {
      rc = launch_split_rows_f16(x + r0 * L.I, xp, n, L.I, (size_t)n * L.I, inv, st);
    }
    if (rc) return rc;
    g.kind = TC_KIND_F16; g.M = n; g.N = 3 * L.H; g.K = L.I;
    g.A = xp; g.B = k.Wi_op; g.a_planes = qx.enabled ? 1 : 2; g.b_planes = L.bits_i <= 8 ? 1 : 2;
    g.lda = L.I; g.ldb = L.I; g.a_plane_stride = (long long)n * L.I; g.b_plane_stride = (long long)3 * L.H * L.I;
    fill_pairs(&g, g.a_planes, g.b_planes, 2);
    g.split_k = 1; g.alpha = qx.enabled ? qx.scale : 1.0f;
    g.row_scale = qx.enabled ? nullptr : inv; g.col_scale = k.Wi_scale; g.bias = k.b_i;
    g.C = gi + r0 * 3 * L.H; g.ldc = 3 * L.H;
    rc = launch_tc_gemm(g, st);
    if (rc) return rc;
  }
  return B200GRU_OK;
}

// ---- backward of the projection ----------------------------------------------------------------------
struct LinearPlan { int splits; size_t dyp, xp, acc, sums, total; };

TcGemm wgrad_gemm(const Layer& L) {
  TcGemm g;
  memset(&g, 0, sizeof(g));
  g.kind = TC_KIND_BF16; g.M = 3 * L.H; g.N = L.I;
  g.a_planes = 2; g.b_planes = 2; g.a_mn = 1; g.b_mn = 1;
  g.lda = 3 * L.H; g.ldb = L.I;
  fill_pairs(&g, 2, 2, 2);
  g.alpha = 1.0f; g.ldc = L.I; g.split_stride = (long long)3 * L.H * L.I;
  return g;
}

LinearPlan linear_plan(const Layer& L) {
  LinearPlan p;
  const size_t chunk = chunk_rows(L), n3 = (size_t)3 * L.H;
  // K slices: about two waves of (N/128) x (I/256) tiles over the 148 SMs when the contraction is long,
  // one wave when each slice would otherwise be only a few k-blocks
  const int tiles = cdiv(3 * L.H, 128) * cdiv(L.I, 256);
  int want = tiles >= 120 ? 1 : cdiv(chunk >= 16384 ? 280 : 140, tiles);
  if ((size_t)want > chunk / 512) want = (int)(chunk / 512);
  TcGemm g = wgrad_gemm(L);
  g.K = (int)chunk;
  p.splits = tc_gemm_splits(g, want < 1 ? 1 : want);
  p.dyp = pad(2 * chunk * n3 * 2);
  p.xp = pad(2 * chunk * L.I * 2);
  p.acc = pad((size_t)p.splits * n3 * L.I * 4);
  p.sums = pad(column_sums_scratch_bytes(p.splits, (int)(n3 * L.I)));
  p.total = p.dyp + p.xp + p.acc + p.sums;
  return p;
}

// dWi, dx from dgi (either may be NULL: not wanted)
int linear_backward(const Layer& L, const Kept& k, const float* x, const float* dgi, float* dWi, float* dx,
                    char* ws, cudaStream_t st) {
  const LinearPlan p = linear_plan(L);
  char* dyp = ws; ws += p.dyp;
  char* xp = ws; ws += p.xp;
  float* acc = reinterpret_cast<float*>(ws); ws += p.acc;
  float* sums = reinterpret_cast<float*>(ws);
  const int n3 = 3 * L.H;
  const size_t w = (size_t)n3 * L.I;
  int rc = B200GRU_OK;
  float* dWq = (p.splits > 1) ? acc : (L.bits_i <= 8 ? acc : dWi);
  bool first = true;
  for (size_t r0 = 0; r0 < L.rows; r0 += ROW_CHUNK) {
    const size_t n = L.rows - r0 < (size_t)ROW_CHUNK ? L.rows - r0 : (size_t)ROW_CHUNK;
    if (dWi != nullptr) {
      // weight gradients are held to 1e-4 of their largest entry: two planes per operand and the cross
      // products down to 2^-16 (error about 1e-5 of a term, averaged over the rows)
      rc = launch_split_planes(dgi + r0 * n3, dyp, n * n3, n * n3, 2, nullptr, 0, st);
      if (!rc) rc = launch_split_planes(x + r0 * L.I, xp, n * L.I, n * L.I, 2, nullptr, 0, st);
      if (rc) return rc;
      TcGemm g = wgrad_gemm(L);
      g.K = (int)n; g.A = dyp; g.B = xp; g.a_plane_stride = (long long)n * n3; g.b_plane_stride = (long long)n * L.I;
      g.split_k = tc_gemm_splits(g, p.splits);
      g.accumulate = first ? 0 : 1;
      if (first && g.split_k != p.splits) {
        cudaMemsetAsync(dWq, 0, (size_t)p.splits * w * 4, st);
        g.accumulate = 1;
      }
      g.C = dWq;
      rc = launch_tc_gemm(g, st);
      if (rc) return rc;
      first = false;
    }
    if (dx != nullptr) {
      // dx = (dgi * row scales of the weights) . planes of the weights, rows of the weights being the contraction index
      __half* dp = reinterpret_cast<__half*>(dyp);
      float* inv = reinterpret_cast<float*>(xp);
      rc = launch_split_rows_f16_scaled(dgi + r0 * n3, dp, (int)n, n3, n * n3, inv, k.Wi_scale, st);
      if (rc) return rc;
      TcGemm g;
      memset(&g, 0, sizeof(g));
      g.kind = TC_KIND_F16; g.M = (int)n; g.N = L.I; g.K = n3;
      g.A = dp; g.B = k.Wi_op; g.a_planes = 2; g.b_planes = L.bits_i <= 8 ? 1 : 2; g.b_mn = 1;
      g.lda = n3; g.ldb = L.I; g.a_plane_stride = (long long)n * n3; g.b_plane_stride = (long long)w;
      fill_pairs(&g, g.a_planes, g.b_planes, 2);
      g.split_k = 1; g.alpha = 1.0f; g.row_scale = inv; g.C = dx + r0 * L.I; g.ldc = L.I;
      g.chunk_kb = L.bits_i <= 8 ? TC_GRADIENT_CODES_CHUNK : 0;
      rc = launch_tc_gemm(g, st);
      if (rc) return rc;
    }
  }
  if (dWi != nullptr) {
    float* full = L.bits_i <= 8 ? acc : dWi;                 // slice 0 is overwritten by the sum when it has to be
    if (p.splits > 1) rc = launch_column_sums(acc, p.splits, (int)w, full, sums, st);
    if (!rc && L.bits_i <= 8) rc = launch_quantize_rows_backward(k.Wi, full, n3, L.I, L.bits_i, dWi, st);
    if (rc) return rc;
  }
  return rc;
}

size_t scan_ws(const Layer& L, int backward) { return pad(b200gru_workspace_bytes(&L.shape, backward)); }
bool keeps_gi(const Layer& L) { return L.shape.kind == B200GRU_DIAGONAL; }     // recomputes its gates instead of saving them

b200gru_quant quant_of(const float* q) {
  b200gru_quant r;
  r.scale = q[0]; r.qmin = (int)q[1]; r.qmax = (int)q[2]; r.enabled = q[3] != 0.f ? 1 : 0;
  return r;
}

}  // namespace
}  // namespace b200gru

using namespace b200gru;

extern "C" {

int b200gru_layer_sizes(const int* dims, size_t* sizes) {
  Layer L;
  Kept k;
  if (!parse(dims, &L)) return B200GRU_INVALID_ARGUMENT;
  if (b200gru_workspace_bytes(&L.shape, 0) == (size_t)-1) return B200GRU_UNSUPPORTED;
  const int mode = keeps_gi(L) ? 1 : 2;
  sizes[0] = carve(L, nullptr, &k);
  const size_t fwd_scan = scan_ws(L, 0), proj = x_planes_bytes(L);
  sizes[1] = fwd_scan > proj ? fwd_scan : proj;
  const size_t bwd_scan = scan_ws(L, mode), lin = linear_plan(L).total;
  sizes[2] = (bwd_scan > lin ? bwd_scan : lin) + (L.bits_h <= 8 ? pad(L.w_elems * 4) : 0);
  return B200GRU_OK;
}

int b200gru_layer_forward(const int* dims, const float* quants, const void* const* ptrs, void* stream) {
  Layer L;
  Kept k;
  if (!parse(dims, &L)) return B200GRU_INVALID_ARGUMENT;
  const float* x = static_cast<const float*>(ptrs[0]);
  const float* h0 = static_cast<const float*>(ptrs[1]);
  const float* const* p = reinterpret_cast<const float* const*>(ptrs) + 2;      // Wi, Wh, bi, bh: three gates each
  float* out = static_cast<float*>(const_cast<void*>(ptrs[14]));
  float* save = static_cast<float*>(const_cast<void*>(ptrs[15]));
  char* kept = static_cast<char*>(const_cast<void*>(ptrs[16]));
  char* ws = static_cast<char*>(const_cast<void*>(ptrs[17]));
  float* gi = static_cast<float*>(const_cast<void*>(ptrs[18]));
  if (!x || !h0 || !out || !kept || !ws || !gi) return B200GRU_INVALID_ARGUMENT;
  for (int i = 0; i < 6; ++i) if (p[i] == nullptr) return B200GRU_INVALID_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  carve(L, kept, &k);
  const b200gru_quant qx = quant_of(quants), qi = quant_of(quants + 4), qo = quant_of(quants + 8);
  if ((qx.enabled && !(qx.scale > 0.f)) || (qi.enabled && !(qi.scale > 0.f)) || (qo.enabled && !(qo.scale > 0.f)))
    return B200GRU_INVALID_ARGUMENT;
  int rc = gather_weights(L, k, p, p + 3, p + 6, p + 9, st);
  if (rc) return rc;
  rc = project(L, k, x, make_quant(&qx), gi, ws, st);
  if (rc) return rc;
  const size_t n = scan_ws(L, 0);
  float* S = keeps_gi(L) ? nullptr : save;
  if (L.bits_h <= 8)
    return b200gru_dense_q8_forward(gi, h0, k.Wh_q, k.Wh_codes, k.Wh_scale, k.b_h, L.T, L.B, L.H, &qi, &qo, out, S, ws, n, stream);
  return b200gru_scan_forward(&L.shape, gi, h0, k.Wh, k.b_h, &qi, &qo, out, S, ws, n, stream);
}

int b200gru_layer_backward(const int* dims, const float* quants, const void* const* ptrs, void* stream) {
  Layer L;
  Kept k;
  if (!parse(dims, &L)) return B200GRU_INVALID_ARGUMENT;
  const bool scan = L.flags != B200GRU_LAYER_PROJECTION, projection = L.flags != B200GRU_LAYER_SCAN;
  const float* x = static_cast<const float*>(ptrs[0]);
  const float* h0 = static_cast<const float*>(ptrs[1]);
  const float* out = static_cast<const float*>(ptrs[2]);
  const float* dout = static_cast<const float*>(ptrs[3]);
  const float* save = static_cast<const float*>(ptrs[4]);
  char* kept = static_cast<char*>(const_cast<void*>(ptrs[5]));
  char* scratch = static_cast<char*>(const_cast<void*>(ptrs[6]));
  float* const* o = reinterpret_cast<float* const*>(const_cast<void* const*>(ptrs)) + 7;   // dx, dh0, dWi, dWh, dbi, dbh, dgi
  if (!kept || !scratch || !o[6]) return B200GRU_INVALID_ARGUMENT;
  if (scan && (!h0 || !out || !dout || !save || !o[1] || !o[3] || !o[5])) return B200GRU_INVALID_ARGUMENT;
  if (projection && !x) return B200GRU_INVALID_ARGUMENT;
  carve(L, kept, &k);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const b200gru_quant qi = quant_of(quants + 4), qo = quant_of(quants + 8);
  float* dgi = o[6];
  float* dWq = nullptr;
  if (L.bits_h <= 8) { dWq = reinterpret_cast<float*>(scratch); scratch += pad(L.w_elems * 4); }
  if (scan) {                           // gi is read only where the gates were not saved; dgi stands in for it
    const bool q8 = L.bits_h <= 8, gi_in = keeps_gi(L);
    int rc = layer_scan_backward(&L.shape, gi_in ? save : dgi, h0, q8 ? k.Wh_q : k.Wh, k.Wh_codes, q8 ? k.Wh_scale : nullptr, k.b_h, out,
                                 dout, gi_in ? nullptr : save, &qi, &qo, dgi, o[1], q8 ? dWq : o[3], o[5], o[4], scratch,
                                 scan_ws(L, gi_in ? 1 : 2), stream);
    if (!rc && q8) rc = launch_quantize_rows_backward(k.Wh, dWq, 3 * L.H, L.H, L.bits_h, o[3], st);
    if (rc) return rc;
  }
  return projection ? linear_backward(L, k, x, dgi, o[2], o[0], scratch, st) : B200GRU_OK;
}

}  // extern "C"
