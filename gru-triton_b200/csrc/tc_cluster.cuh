// Interface of the tensor-core cluster scan (tc_cluster.cu): all T steps of dense / block-diagonal
// problems with blocks of at most 512 units in one launch, weights resident in tensor and shared memory.
#pragma once

#include "common.cuh"

namespace b200gru {
namespace tcc {

constexpr int UNITS = 32;              // hidden units per CTA
constexpr int MAX_C = 16;              // CTAs of a cluster

struct Args {
  const float* gi;           // [T][B][3H]
  const float* h0;           // [B][H]
  const float* W;            // fp32 weights (gate / block strides below)
  const signed char* codes;  // or int8 codes [3H][H] with one scale per row (dense only)
  const float* scales;
  const float* bh;           // [3H]
  float* out;                // [T][B][H]: forward written, backward read
  float* save;               // forward: [4][T][B][H] or NULL
  const float* S;            // backward: the four saved activations
  const float* dout;
  float* dgi;
  float* dh0;
  int* status;
  int T, B, H, nb, Hb;
  long long w_gate_stride, w_block_stride;
  Quant qin, qout;
  // filled by launch()
  int C, rows, rows8, ntiles_b;
};

struct Config {
  int C, N, rows, pw, ph, clusters, active;
  size_t smem;
};

// False when no configuration applies; *cycles is the estimated time of the scan in SM cycles, comparable with
// the estimate of choose_block_config().
bool choose(bool fwd, int T, int B, int Hb, int nb, bool w_codes, const Quant& qin, Config* out, double* cycles);
int launch(bool fwd, const Config& c, Args a, cudaStream_t st);
int read_status(int reset);
int set_status(int value);              // tests only

}  // namespace tcc
}  // namespace b200gru
