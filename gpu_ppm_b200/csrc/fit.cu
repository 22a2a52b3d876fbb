// Fit statistics of model counts against observed counts (ppm_batch_fit,
// ppm_profile_fit): the reduced-chi2 helper cal_chi2 of p_devarshi24st.py:43-49
// and the Poisson log-likelihood, evaluated on the device right after the fold
// so that a sampler's likelihood loop reads back a few scalars per proposal
// instead of the [n_ch][n_bins] count arrays.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "../../include/ppm.h"
#include "engine.h"

namespace ppm {

namespace {

#define FIT_CUDA(call)                                                                           \
  do {                                                                                           \
    cudaError_t e_ = (call);                                                                     \
    if (e_ != cudaSuccess) throw Error(PPM_E_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

constexpr int kFitThreads = 256;
constexpr int kFitPerBlock = 1024, kFitMaxBlocks = 32;

// What one block sums of a profile's entries.
struct FitPart {
  double M, S, L;
  long long nz;
  int bad;
};

// Blocks of a profile: by its number of entries alone, so that its statistics do not depend on what it is batched with.
int fit_blocks(int n_el) { return std::max(1, std::min(kFitMaxBlocks, (n_el + kFitPerBlock - 1) / kFitPerBlock)); }

// grid (blocks, profiles).  Per-thread partial sums over a fixed stride, a
// fixed-order warp and block reduction; the block that finishes a profile's last
// part adds the parts in their order: the result does not depend on timing.
// Bound by the latency of the FP64 logarithm: 300 x 64 entries took 53 us on one
// block, 15 on five, 11 on the 19 that 1024 entries a block give.  done: zero before, zero after.
__global__ void __launch_bounds__(kFitThreads) fit_kernel(const long long* counts_off, const double* counts,
                                                          const double* obs, int n_el, double lgamma_sum,
                                                          FitPart* parts, int* done, ppm_fit* out) {
  __shared__ double s_red[3][kFitThreads / 32];
  __shared__ long long s_nz[kFitThreads / 32];
  __shared__ int s_bad[kFitThreads / 32];
  const double* m = counts + counts_off[blockIdx.y];
  double M = 0.0, S = 0.0, L = 0.0;
  long long nz = 0;
  int bad = 0;
  for (int i = blockIdx.x * kFitThreads + threadIdx.x; i < n_el; i += gridDim.x * kFitThreads) {
    const double mi = m[i], di = obs[i];
    M += mi;
    if (mi > 0.0) {
      const double r = di - mi;
      S += r * r / mi;
      L += di * log(mi) - mi;
    } else {
      ++nz;
      if (di != 0.0) bad = 1;
      L -= mi;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    M += __shfl_down_sync(0xffffffffu, M, o);
    S += __shfl_down_sync(0xffffffffu, S, o);
    L += __shfl_down_sync(0xffffffffu, L, o);
    nz += __shfl_down_sync(0xffffffffu, nz, o);
    bad |= __shfl_down_sync(0xffffffffu, bad, o);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    s_red[0][warp] = M;
    s_red[1][warp] = S;
    s_red[2][warp] = L;
    s_nz[warp] = nz;
    s_bad[warp] = bad;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    FitPart t{0.0, 0.0, 0.0, 0, 0};
    for (int w = 0; w < kFitThreads / 32; ++w) {
      t.M += s_red[0][w];
      t.S += s_red[1][w];
      t.L += s_red[2][w];
      t.nz += s_nz[w];
      t.bad |= s_bad[w];
    }
    FitPart* mine = parts + (size_t)blockIdx.y * gridDim.x;
    mine[blockIdx.x] = t;
    __threadfence();
    if (atomicAdd(&done[blockIdx.y], 1) != (int)gridDim.x - 1) return;
    __threadfence();
    done[blockIdx.y] = 0;
    t = FitPart{0.0, 0.0, 0.0, 0, 0};
    for (int k = 0; k < (int)gridDim.x; ++k) {
      const volatile FitPart* p = mine + k;
      t.M += p->M;
      t.S += p->S;
      t.L += p->L;
      t.nz += p->nz;
      t.bad |= p->bad;
    }
    ppm_fit f;
    f.chi2 = t.M > 0.0 ? t.S * (1e6 / t.M) : (double)NAN;
    f.loglike = t.bad ? -(double)INFINITY : t.L - lgamma_sum;
    f.model_total = t.M;
    f.n_zero_model = t.nz;
    out[blockIdx.y] = f;
  }
}

}  // namespace

int Engine::add_observed(int resp, int n_bins, const double* counts) {
  std::lock_guard<std::mutex> lk(mu);
  FIT_CUDA(cudaSetDevice(cfg.device));
  if (resp < 0 || resp >= (int)resps.size()) throw Error(PPM_E_INVALID, "no such response");
  if (n_bins <= 0) throw Error(PPM_E_INVALID, "n_bins must be positive");
  if (!counts) throw Error(PPM_E_INVALID, "null observed counts");
  Observed o;
  o.resp = resp;
  o.n_bins = n_bins;
  o.n_ch = resps[resp].n_ch;
  const size_t n = (size_t)o.n_ch * n_bins;
  for (size_t i = 0; i < n; ++i) {
    if (!(counts[i] >= 0.0) || !std::isfinite(counts[i]))
      throw Error(PPM_E_INVALID, "observed counts must be finite and non-negative");
    o.lgamma_sum += std::lgamma(counts[i] + 1.0);
  }
  FIT_CUDA(cudaMalloc(&o.d_counts, sizeof(double) * n));
  track(o.d_counts);
  FIT_CUDA(cudaMemcpy(o.d_counts, counts, sizeof(double) * n, cudaMemcpyHostToDevice));
  observed.push_back(o);
  return (int)observed.size() - 1;
}

void Engine::batch_fit(BatchImpl& B, int obs, ppm_fit* out, cudaStream_t st) {
  FIT_CUDA(cudaSetDevice(cfg.device));
  if (obs < 0 || obs >= (int)observed.size()) throw Error(PPM_E_INVALID, "no such observed data");
  if (!out) throw Error(PPM_E_INVALID, "null output");
  const Observed& o = observed[obs];
  for (int i = 0; i < B.n; ++i)
    if (B.params[i].response != o.resp || B.params[i].n_bins != o.n_bins)
      throw Error(PPM_E_INVALID, "profile " + std::to_string(i) +
                                     " does not use the observed data's response and bin count");
  if (!st) st = B.last_stream ? B.last_stream : stream;
  const int n_el = o.n_ch * o.n_bins;  // the same for every set of observed data this batch takes
  const int blocks = fit_blocks(n_el);
  std::lock_guard<std::mutex> lk(B.fit_mu);
  if (!B.d_fit) {
    // one block, and the batch has it only when it is complete: a call that runs out of memory here leaves nothing
    // half made to the next one
    const size_t n = (size_t)B.n;
    static_assert(sizeof(FitPart) % 8 == 0 && sizeof(ppm_fit) % 8 == 0, "the parts of the block are 8-byte aligned");
    unsigned char* const mem = (unsigned char*)B.mem.alloc(
        (sizeof(long long) + sizeof(ppm_fit) + sizeof(FitPart) * blocks + sizeof(int)) * n);
    long long* const off = (long long*)mem;
    ppm_fit* const fit = (ppm_fit*)(off + n);
    FitPart* const parts = (FitPart*)(fit + n);
    int* const done = (int*)(parts + (size_t)blocks * n);
    FIT_CUDA(cudaMemcpyAsync(off, B.counts_off.data(), sizeof(long long) * n, cudaMemcpyHostToDevice, st));
    FIT_CUDA(cudaMemsetAsync(done, 0, sizeof(int) * n, st));
    B.d_fit_off = off;
    B.d_fit_parts = parts;
    B.d_fit_done = done;
    B.d_fit = fit;
  }
  if (B.n > 0) {
    // (at most 65535 profiles a launch: grid y)
    for (int k = 0; k < B.n; k += 65535)
      fit_kernel<<<dim3(blocks, std::min(65535, B.n - k)), kFitThreads, 0, st>>>(
          B.d_fit_off + k, B.d_counts, o.d_counts, n_el, o.lgamma_sum, (FitPart*)B.d_fit_parts + (size_t)k * blocks,
          B.d_fit_done + k, B.d_fit + k);
    FIT_CUDA(cudaGetLastError());
    FIT_CUDA(cudaMemcpyAsync(out, B.d_fit, sizeof(ppm_fit) * (size_t)B.n, cudaMemcpyDeviceToHost, st));
  }
  FIT_CUDA(cudaStreamSynchronize(st));
}

void Engine::profile_fit(const ppm_params& p, int obs, ppm_fit* out, ppm_result_info* info) {
  std::lock_guard<std::mutex> lk(mu);
  BatchImpl B;
  pin_uploads(B);
  batch_build(B, 1, &p, stream);
  batch_enqueue(B, stream, nullptr);
  batch_fit(B, obs, out, stream);
  batch_collect(B, nullptr, nullptr, info, stream, true);
}

}  // namespace ppm
