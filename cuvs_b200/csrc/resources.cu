#include "common.hpp"

#include <nvtx3/nvToolsExt.h>

#include <atomic>
#include <mutex>

namespace cuvs_b200 {

namespace {
nvtxDomainHandle_t nvtx_domain()
{
  static nvtxDomainHandle_t d = nvtxDomainCreateA("cuvs");
  return d;
}
}  // namespace

nvtx_range::nvtx_range(const char* fmt, ...)
{
  nvtxDomainHandle_t d = nvtx_domain();
  if (d == nullptr) { return; }  // no tool attached: the domain handle is null and nothing is recorded
  char buf[256];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  nvtxEventAttributes_t attr{};
  attr.version       = NVTX_VERSION;
  attr.size          = NVTX_EVENT_ATTRIB_STRUCT_SIZE;
  attr.messageType   = NVTX_MESSAGE_TYPE_ASCII;
  attr.message.ascii = buf;
  nvtxDomainRangePushEx(d, &attr);
  pushed_ = true;
}

nvtx_range::~nvtx_range()
{
  if (pushed_) { nvtxDomainRangePop(nvtx_domain()); }
}

void ensure_dynamic_smem(const void* kernel, size_t bytes)
{
  static std::mutex lock;
  static std::map<std::pair<const void*, int>, size_t> done;
  int dev = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> guard(lock);
  size_t& have = done[{kernel, dev}];
  if (bytes > have) {
    CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
    have = bytes;
  }
}

resources::resources()
{
  CUDA_TRY(cudaGetDevice(&device));
  cudaDeviceProp prop{};
  CUDA_TRY(cudaGetDeviceProperties(&prop, device));
  sm_count   = prop.multiProcessorCount;
  smem_optin = static_cast<int>(prop.sharedMemPerBlockOptin);
  cc_major   = prop.major;
  CUDA_TRY(cudaMallocHost(&pinned, 64));
  pinned[12] = 0;
  pinned[13] = 0;
  CUDA_TRY(cudaMalloc(&redo_counts, N_REDO_COUNTS * sizeof(*redo_counts)));
  CUDA_TRY(cudaMemset(redo_counts, 0, N_REDO_COUNTS * sizeof(*redo_counts)));
}

resources::~resources()
{
  for (auto& ev : pending) {
    for (auto& e : ev.e) { cudaEventDestroy(e); }
  }
  if (d_stats) { cudaFree(d_stats); }
  if (redo_counts) { cudaFree(redo_counts); }
  if (pinned) {
    cudaDeviceSynchronize();  // a kernel may still write its verdict or count a time-out there
    cudaFreeHost(pinned);
  }
}

void resources::adopt_tc_verdict()
{
  if (!tc_redo_pending || *static_cast<volatile uint32_t*>(pinned + 12) != tc_redo_seq) { return; }
  std::atomic_thread_fence(std::memory_order_acquire);
  tc_redo_pending = false;
  if (tc_redo_n_lists != 0u) {
    // (a time-out, which the kernels count, says nothing about the bounds)
    if (pinned[8] == 0u && tc_redo_adapts) {
      probe_level& lv = probe_levels[{tc_redo_n_lists, tc_redo_n_probes}];
      if (uint64_t(pinned[9]) * 16 > tc_redo_queries) {
        lv.rest      = lv.next_rest;
        lv.next_rest = std::min(2 * lv.next_rest, 1024u);
      } else {
        lv.next_rest = 16;
      }
    }
  } else if (pinned[8] != 0u) {
    // the coarse GEMM of that batch gave up on a bounded wait; its probes were all recomputed exactly
    tc_timeouts++;
  } else if (tc_redo_adapts) {
    tc_level& lv = tc_levels[tc_redo_n_probes];
    if (uint64_t(pinned[9]) * 256 > tc_redo_queries && lv.products < 3) {
      // more than 1/256 of the batch failed the exactness guard: one more product of the TF32 split,
      // and never fewer again on this handle for this n_probes
      lv.products++;
      lv.floor = lv.products;
    } else if (lv.products > lv.floor && uint64_t(pinned[11]) * 1024 <= tc_redo_queries) {
      // (almost) every query of the batch would have passed the guard with one product less
      lv.products--;
    }
  }
}

bool resources::probes_by_passes(uint32_t n_lists, uint32_t n_probes)
{
  adopt_tc_verdict();
  if (probe_levels.size() > 4096) { probe_levels.clear(); }
  const auto at = probe_levels.find({n_lists, n_probes});
  if (at == probe_levels.end() || at->second.rest == 0u) { return true; }
  at->second.rest--;
  return false;
}

uint32_t* resources::tc_redo_record(uint32_t n_queries, uint32_t n_probes, uint32_t n_lists, bool adapts)
{
  if (tc_redo_pending) { return nullptr; }
  tc_redo_queries  = n_queries;
  tc_redo_n_probes = n_probes;
  tc_redo_n_lists  = n_lists;
  tc_redo_adapts   = adapts;
  tc_redo_pending  = true;
  tc_redo_seq++;
  return pinned + 8;
}

void resources::sync()
{
  CUDA_TRY(cudaStreamSynchronize(stream));
  adopt_tc_verdict();
}

void resources::stats_enable(bool on)
{
  if (on && !d_stats) {
    CUDA_TRY(cudaMalloc(&d_stats, 16));
    CUDA_TRY(cudaMemset(d_stats, 0, 16));
  }
  stats_enabled = on;
}

void resources::stats_mark(stage_events& ev, int i)
{
  if (i == 0) {
    for (auto& e : ev.e) { CUDA_TRY(cudaEventCreate(&e)); }
  }
  CUDA_TRY(cudaEventRecord(ev.e[i], stream));
}

void resources::stats_resolve()
{
  CUDA_TRY(cudaStreamSynchronize(stream));
  for (auto& ev : pending) {
    for (int i = 0; i < 5; i++) {
      float ms = 0.0f;
      CUDA_TRY(cudaEventElapsedTime(&ms, ev.e[i], ev.e[i + 1]));
      stage_ms[i] += ms;
    }
    for (auto& e : ev.e) { cudaEventDestroy(e); }
    stat_batches++;
  }
  pending.clear();
}

}  // namespace cuvs_b200
