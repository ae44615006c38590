// pipeline.cu — pipelined launches (pipeline_kernel.cuh): their layout, the kernels
// of the SUBLEQ languages, mutation masks, and the entry points on caller-owned
// buffers.
#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "pipeline_kernel.cuh"

namespace cubff {
namespace {

constexpr uint64_t kDefaultWaitLimitNs = 10ull * 1000 * 1000 * 1000;
std::atomic<uint64_t> g_wait_limit_ns{kDefaultWaitLimitNs};

// Mutation masks of MutateAndRunPrograms (common_language.h:172-180) for
// epochs [e0, e0 + E): bit i of mask[e][k] is set iff draw i of pair k, with key
// (n * seed(e0 + e) + k) * 128 + i, mutates byte i.  Bound by the draws' integer
// arithmetic; a thread takes a pair, so that the epoch's seed costs little.
__global__ void __launch_bounds__(256)
    mutation_mask_kernel(uint64_t s0, uint64_t e0, uint32_t n_epochs, uint64_t npairs, uint64_t n,
                         uint32_t prob, uint4 *out) {
  const uint64_t k = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= npairs) return;
  for (uint32_t e = blockIdx.y; e < n_epochs; e += gridDim.y) {
    const uint64_t key0 = (n * seed_from(s0, e0 + e) + k) * kPair;
    uint32_t m[4];
#pragma unroll 1
    for (int q = 0; q < 4; q++) m[q] = mutation_word(key0 + 32 * q, prob);
    out[e * npairs + k] = make_uint4(m[0], m[1], m[2], m[3]);
  }
}

}  // namespace

uint64_t pipeline_wait_limit_ns() { return g_wait_limit_ns.load(); }

namespace {
uint32_t env_u32(const char *name, uint32_t dflt, uint32_t lo, uint32_t hi) {
  const char *v = std::getenv(name);
  if (!v || !*v) return dflt;
  const long x = std::strtol(v, nullptr, 10);
  return x < long(lo) ? lo : x > long(hi) ? hi : static_cast<uint32_t>(x);
}
}  // namespace

// Default launch shape: half an epoch of pairs in flight, and for SUBLEQ 64 steps
// per visit and claims by warps whose lanes are all idle (8 epochs of 8720 subleq
// programs 205 us; with 10 of 16 idle 225; of 2^17 programs the same time).
cubff_tuning default_shape() {
  static const cubff_tuning t = {env_u32("CUBFF_LANES_PER_PAIR64", 32, 1, 64),
                                 env_u32("CUBFF_STEPS_PER_VISIT", 64, 1, 4096),
                                 env_u32("CUBFF_CLAIM_MIN", 32, 1, 32),
                                 env_u32("CUBFF_LONG_VISITS", 1, 0, 1u << 20),
                                 env_u32("CUBFF_FIRST_VISIT_STEPS", 64, 1, 4096)};
  return t;
}

bool valid_shape(const cubff_tuning &t) {
  return t.lanes_per_pair64 >= 1 && t.lanes_per_pair64 <= 64 && t.steps_per_visit >= 1 &&
         t.steps_per_visit <= 4096 && t.claim_min >= 1 && t.claim_min <= 32 &&
         t.first_visit_steps >= 1 && t.first_visit_steps <= 4096;
}

PipeTuning pipe_tuning(const cubff_tuning &t) {
  return PipeTuning{t.steps_per_visit, t.claim_min,
                    t.long_visits ? t.long_visits : 0xffffffffu, t.first_visit_steps};
}

namespace {

PipeKernels kernels_of(int lang) {
  if (lang <= kBffSelfmove) return bff_pipe_kernels(lang);
  if (lang <= kForthtrivialReset) return forth_pipe_kernels(lang);
  return lang == kSubleq ? pipe_kernels<kSubleq>() : pipe_kernels<kRsubleq4>();
}

// Blocks of a kernel that are resident on an SM at once, with the descriptors of
// n_soups soups; its shared memory limit is raised on a device's first launch.
int blocks_per_sm(const PipeKernel &k, int lang, int which, int n_soups, int device, int *out) {
  static std::atomic<uint64_t> raised[kNumLangs][kPipeWidths];  // by device (zero-initialised)
  const uint64_t bit = 1ull << (device & 63);
  if (!(raised[lang][which].load() & bit)) {
    CUBFF_CUDA_TRY(cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(k.smem_bytes(kMaxPipeSoups))));
    raised[lang][which].fetch_or(bit);
  }
  CUBFF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, k.fn, kThreads,
                                                               k.smem_bytes(n_soups)));
  return CUBFF_OK;
}

}  // namespace

int plan_pipeline(int lang, int n_soups, uint64_t total_pairs, uint32_t lanes_per_pair64,
                  int device, PipePlan *out) {
  static std::atomic<int> sms_of[64];  // by device (zero-initialised)
  int sms = sms_of[device & 63].load();
  if (sms == 0) {
    CUBFF_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    sms_of[device & 63].store(sms);
  }
  const PipeKernels k = kernels_of(lang);
  int per_sm = 0;
  const PipeWidths widths = pipe_widths(lang);
  CUBFF_TRY(blocks_per_sm(k.kernel[0], lang, 0, n_soups, device, &per_sm));
  const uint64_t lanes = lanes_wanted(total_pairs, lanes_per_pair64, sms);
  const int w = choose_width(widths, lanes, sms, per_sm);
  if (w != 0) CUBFF_TRY(blocks_per_sm(k.kernel[w], lang, w, n_soups, device, &per_sm));
  *out = PipePlan{w, grid_of(widths.width[w], lanes, sms, per_sm)};
  return CUBFF_OK;
}

int launch_pipeline(const PipeBatch &b, uint64_t total_pairs, uint32_t lanes_per_pair64,
                    int device, cudaStream_t stream) {
  if (b.n_soups <= 0 || total_pairs == 0) return CUBFF_OK;
  if (b.n_soups > kMaxPipeSoups)
    return set_error(CUBFF_EINVAL, "pipeline: %d soups over the limit of %d", b.n_soups,
                     kMaxPipeSoups);
  if (b.queue.lang < 0 || b.queue.lang >= kNumLangs)
    return set_error(CUBFF_ENOTFOUND, "unknown language id %d", b.queue.lang);
  PipePlan plan;
  CUBFF_TRY(plan_pipeline(b.queue.lang, b.n_soups, total_pairs, lanes_per_pair64, device, &plan));
  const PipeKernel k = kernels_of(b.queue.lang).kernel[plan.which];
  void *args[] = {const_cast<PipeBatch *>(&b)};
  CUBFF_CUDA_TRY(cudaLaunchKernel(k.fn, dim3(plan.grid), dim3(kThreads), args,
                                  k.smem_bytes(b.n_soups), stream));
  return CUBFF_OK;
}

int launch_mutation_masks(uint64_t s0, uint64_t e0, uint32_t n_epochs, uint64_t n, uint32_t prob,
                          uint4 *out, cudaStream_t stream) {
  const uint64_t npairs = n / 2;
  if (npairs == 0 || n_epochs == 0) return CUBFF_OK;
  const dim3 grid(static_cast<unsigned>((npairs + 255) / 256), std::min(n_epochs, 65535u));
  mutation_mask_kernel<<<grid, 256, 0, stream>>>(s0, e0, n_epochs, npairs, n, prob, out);
  CUBFF_CUDA_TRY(cudaGetLastError());
  return CUBFF_OK;
}

}  // namespace cubff

// ---------------------------------------------------------------------------
// Kernel-level pipelined run on caller-owned buffers (cubff_run_epochs).

namespace cubff {
namespace {

struct RunWs {
  uint4 *mutmask;
  uint32_t *inv, *readycnt, *queue, *ctl;
  unsigned long long *counters;
};

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

RunWs run_ws(void *base, uint64_t n, uint32_t E) {
  const uint64_t P = n / 2;
  uint8_t *p = static_cast<uint8_t *>(base);
  RunWs w;
  w.mutmask = reinterpret_cast<uint4 *>(p);
  p += align256(size_t(E) * P * sizeof(uint4));
  w.inv = reinterpret_cast<uint32_t *>(p);
  p += align256(size_t(E) * n * sizeof(uint32_t));
  w.readycnt = reinterpret_cast<uint32_t *>(p);
  p += align256(size_t(E) * P * sizeof(uint32_t));
  w.queue = reinterpret_cast<uint32_t *>(p);
  p += align256(size_t(E) * P * sizeof(uint32_t));
  w.counters = reinterpret_cast<unsigned long long *>(p);
  p += align256(size_t(E) * kPipeCountSlots * 2 * sizeof(unsigned long long));
  w.ctl = reinterpret_cast<uint32_t *>(p);
  return w;
}

// d_counts[e] += the per-slot counters of epoch e.
__global__ void reduce_counts_kernel(const unsigned long long *slots, uint32_t E,
                                     unsigned long long *out) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  unsigned long long o = 0, r = 0;
  for (int s = 0; s < kPipeCountSlots; s++) {
    o += slots[(uint64_t(e) * kPipeCountSlots + s) * 2];
    r += slots[(uint64_t(e) * kPipeCountSlots + s) * 2 + 1];
  }
  out[2 * e] += o;
  out[2 * e + 1] += r;
}

}  // namespace
}  // namespace cubff

extern "C" size_t cubff_run_epochs_workspace_bytes(uint64_t num_programs, uint32_t n_epochs) {
  using namespace cubff;
  const uint64_t P = num_programs / 2;
  return align256(size_t(n_epochs) * P * sizeof(uint4)) +
         align256(size_t(n_epochs) * num_programs * sizeof(uint32_t)) +
         2 * align256(size_t(n_epochs) * P * sizeof(uint32_t)) +
         align256(size_t(n_epochs) * kPipeCountSlots * 2 * sizeof(unsigned long long)) + 256;
}

extern "C" int cubff_run_epochs(int lang, uint8_t *d_programs, const uint32_t *d_shuf_idx,
                                const uint64_t *d_num_indices, uint64_t params_seed,
                                uint64_t first_epoch, uint32_t n_epochs, uint32_t mutation_prob,
                                uint64_t num_programs, unsigned long long *d_counts,
                                void *d_workspace, size_t workspace_bytes, void *stream) {
  return cubff_run_epochs_tuned(lang, d_programs, d_shuf_idx, d_num_indices, params_seed,
                                first_epoch, n_epochs, mutation_prob, num_programs, d_counts,
                                d_workspace, workspace_bytes, nullptr, stream);
}

extern "C" void cubff_default_tuning(cubff_tuning *out) {
  if (out) *out = cubff::default_shape();
}

extern "C" int cubff_run_epochs_tuned(int lang, uint8_t *d_programs, const uint32_t *d_shuf_idx,
                                      const uint64_t *d_num_indices, uint64_t params_seed,
                                      uint64_t first_epoch, uint32_t n_epochs,
                                      uint32_t mutation_prob, uint64_t num_programs,
                                      unsigned long long *d_counts, void *d_workspace,
                                      size_t workspace_bytes, const cubff_tuning *tuning,
                                      void *stream) {
  using namespace cubff;
  const cubff_tuning shape = tuning ? *tuning : default_shape();
  if (!valid_shape(shape)) return set_error(CUBFF_EINVAL, "run_epochs: launch shape out of range");
  if (lang < 0 || lang >= kNumLangs) return set_error(CUBFF_ENOTFOUND, "unknown language %d", lang);
  if (!d_programs || !d_shuf_idx || !d_counts || !d_workspace || num_programs < 2 ||
      num_programs % 2 != 0 || num_programs > (1ull << 31))
    return set_error(CUBFF_EINVAL, "run_epochs: bad arguments");
  if ((reinterpret_cast<uintptr_t>(d_programs) & 15) || (reinterpret_cast<uintptr_t>(d_shuf_idx) & 7) ||
      (reinterpret_cast<uintptr_t>(d_workspace) & 255))
    return set_error(CUBFF_EINVAL, "run_epochs: misaligned buffer (programs 16, indices 8, "
                                   "workspace 256 bytes)");
  if (workspace_bytes < cubff_run_epochs_workspace_bytes(num_programs, n_epochs))
    return set_error(CUBFF_EINVAL, "run_epochs: workspace too small (%zu < %zu)", workspace_bytes,
                     cubff_run_epochs_workspace_bytes(num_programs, n_epochs));
  if (n_epochs == 0) return CUBFF_OK;
  if ((num_programs / 2) * uint64_t(n_epochs) >= (1ull << 31))
    return set_error(CUBFF_EINVAL, "run_epochs: num_programs/2 * n_epochs must be < 2^31");
  int dev = 0;
  CUBFF_CUDA_TRY(cudaGetDevice(&dev));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const uint64_t n = num_programs, P = n / 2, s0 = splitmix64(params_seed);
  RunWs w = run_ws(d_workspace, n, n_epochs);
  CUBFF_CUDA_TRY(cudaMemsetAsync(w.readycnt, 0, size_t(n_epochs) * P * sizeof(uint32_t), st));
  CUBFF_CUDA_TRY(cudaMemsetAsync(w.queue, 0, size_t(n_epochs) * P * sizeof(uint32_t), st));
  CUBFF_CUDA_TRY(cudaMemsetAsync(w.counters, 0,
                                 size_t(n_epochs) * kPipeCountSlots * 2 * sizeof(unsigned long long), st));
  CUBFF_CUDA_TRY(cudaMemsetAsync(w.ctl, 0, 4 * sizeof(uint32_t), st));
  CUBFF_TRY(launch_mutation_masks(s0, first_epoch, n_epochs, n, mutation_prob, w.mutmask, st));
  CUBFF_TRY(launch_inverse(d_shuf_idx, n_epochs, n, w.inv, st));
  PipeBatch b;
  PipeSoup &sp = b.soups[0];
  sp.soup = d_programs;
  sp.perm = d_shuf_idx;
  sp.inv = w.inv;
  sp.mutmask = w.mutmask;
  sp.readycnt = w.readycnt;
  sp.num_indices = d_num_indices;
  sp.ops = w.counters;
  sp.n = n;
  sp.s0 = s0;
  sp.e0 = first_epoch;
  sp.npairs = static_cast<uint32_t>(P);
  sp.mutation_prob = mutation_prob;
  sp.task_base = 0;
  sp.init_base = 0;
  sp.lang = lang;
  sp.n_epochs = n_epochs;
  PipeQueue &q = b.queue;
  q.queue = w.queue;
  q.ctl = w.ctl;
  q.total = static_cast<uint32_t>(P * n_epochs);
  q.initial = static_cast<uint32_t>(P);
  q.first_soup = 0;
  q.n_soups = 1;
  q.lang = lang;
  b.n_soups = 1;
  b.error = reinterpret_cast<int *>(w.ctl + 2);
  b.wait_limit_ns = pipeline_wait_limit_ns();
  b.tune = pipe_tuning(shape);
  CUBFF_TRY(launch_pipeline(b, P, shape.lanes_per_pair64, dev, st));
  reduce_counts_kernel<<<(n_epochs + 127) / 128, 128, 0, st>>>(w.counters, n_epochs, d_counts);
  CUBFF_CUDA_TRY(cudaGetLastError());
  return CUBFF_OK;
}

extern "C" int cubff_run_epochs_status(const void *d_workspace, uint64_t num_programs,
                                       uint32_t n_epochs, void *stream) {
  using namespace cubff;
  if (!d_workspace) return set_error(CUBFF_EINVAL, "run_epochs_status: null workspace");
  RunWs w = run_ws(const_cast<void *>(d_workspace), num_programs, n_epochs);
  int err = 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  CUBFF_CUDA_TRY(cudaMemcpyAsync(&err, w.ctl + 2, sizeof(int), cudaMemcpyDeviceToHost, st));
  CUBFF_CUDA_TRY(cudaStreamSynchronize(st));
  if (err == 2) return set_error(CUBFF_EDEVICE, "run_epochs: a ready-queue entry was out of range");
  if (err) return set_error(CUBFF_ETIMEDOUT, "run_epochs: a pipelined wait timed out");
  return CUBFF_OK;
}

extern "C" int cubff_set_wait_limit_ns(uint64_t ns, uint64_t *previous) {
  using namespace cubff;
  if (ns == 0) return set_error(CUBFF_EINVAL, "set_wait_limit_ns: the limit must be > 0");
  const uint64_t old = g_wait_limit_ns.exchange(ns);
  if (previous) *previous = old;
  return CUBFF_OK;
}
