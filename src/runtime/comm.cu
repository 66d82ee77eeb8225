// Communicator runtime: symmetric heap, peer mapping, program cache and the
// launcher of the fused executor.
//
// The reference's counterpart is the scratch-buffer manager inside its
// ncclCommInitRank hook (src/piccl.c:175-199: three process-global buffers,
// 16 GiB per process, no error checks).  Here every communicator owns one heap
// of a few hundred MiB that peers map through CUDA IPC; the handles travel by
// whatever the caller has (real NCCL in the preload shim, torch.distributed
// in the Python package, a pipe in the benchmark).
#include "comm.h"
#include "../include/piccl_slice.h"
#include "nvls.h"
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>
#include <algorithm>
#include <chrono>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <thread>
#include <unistd.h>

namespace piccl {

thread_local std::string g_last_error;
int fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap; va_start(ap, fmt); vsnprintf(buf, sizeof buf, fmt, ap); va_end(ap);
  g_last_error = buf;
  log_msg(1, "error: %s", buf);
  return code;
}

#define CUDA_TRY(expr)                                                                              \
  do {                                                                                              \
    cudaError_t e_ = (expr);                                                                        \
    if (e_ != cudaSuccess) return fail(PICCL_CUDA_ERROR, "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e_), __FILE__, __LINE__); \
  } while (0)

static unsigned long long host_hash() {
  char h[256] = {0}; gethostname(h, sizeof h - 1);
  unsigned long long x = 1469598103934665603ull;
  for (char* p = h; *p; p++) { x ^= (unsigned char)*p; x *= 1099511628211ull; }
  // CUDA IPC needs one PID namespace as well as one host: the boot id tells hosts apart,
  // the host name tells containers apart
  if (FILE* f = fopen("/proc/sys/kernel/random/boot_id", "r")) { int c; while ((c = fgetc(f)) != EOF) { x ^= (unsigned char)c; x *= 1099511628211ull; } fclose(f); }
  return x;
}

static long long round_up(long long v, long long a) { return (v + a - 1) / a * a; }

struct DevGuard {
  int prev = -1; bool changed = false;
  explicit DevGuard(int dev) { if (cudaGetDevice(&prev) == cudaSuccess && prev != dev) { cudaSetDevice(dev); changed = true; } }
  ~DevGuard() { if (changed) cudaSetDevice(prev); }
};

}  // namespace piccl

using namespace piccl;

extern "C" {

const char* piccl_last_error(void) { return g_last_error.c_str(); }

int piccl_comm_create(int rank, int nranks, int device, const piccl_config_t* user_cfg, piccl_comm_t** out) {
  if (!out || nranks < 1 || nranks > kMaxRanks || rank < 0 || rank >= nranks) return fail(PICCL_INVALID_ARGUMENT, "bad rank/nranks %d/%d", rank, nranks);
  const Env& e = env();
  piccl_config_t cfg; memset(&cfg, 0, sizeof cfg);
  if (user_cfg) cfg = *user_cfg;
  if (cfg.max_cta <= 0) cfg.max_cta = e.max_cta;
  if (cfg.nslot <= 0) cfg.nslot = e.nslot;
  if (cfg.nslot < 2) cfg.nslot = 2;                        // fused receive+forward needs two entries in flight
  if (cfg.slot_bytes <= 0) cfg.slot_bytes = (long long)e.slot_kb * 1024;
  cfg.slot_bytes = round_up(cfg.slot_bytes, 16);
  if (cfg.scratch_bytes <= 0) cfg.scratch_bytes = (long long)e.scratch_mb << 20;
  if (cfg.block_size <= 0) cfg.block_size = e.block_size_set ? e.block_size : 512;
  if (cfg.block_size > kMaxBlock) cfg.block_size = kMaxBlock;
  if (cfg.block_size < 64) cfg.block_size = 64;
  cfg.block_size = cfg.block_size / 32 * 32;
  if (cfg.timeout_ms <= 0) cfg.timeout_ms = e.timeout_ms;
  if (cfg.max_cta > 128) cfg.max_cta = 128;
  if (cfg.nvls_cta <= 0) cfg.nvls_cta = e.nvls_cta;

  DevGuard g(device);
  piccl_comm* c = new piccl_comm();
  c->rank = rank; c->nranks = nranks; c->device = device; c->cfg = cfg;
  c->host_id = host_hash();
  RankCtx& x = c->h_ctx; memset(&x, 0, sizeof x);
  x.rank = rank; x.nranks = nranks; x.max_cta = cfg.max_cta; x.nslot = cfg.nslot; x.slot_bytes = cfg.slot_bytes;
  long long flags = round_up((long long)nranks * cfg.max_cta * kFlagStride, 4096);
  // low-latency slots: [parity][step][source rank], each 2 x the largest payload (line = 8 B data + 8 B flags)
  long long ll_payload = (long long)e.ll_kb * 1024;
  x.ll_slot_bytes = round_up(2 * ll_payload, 4096);
  long long ll_bytes = ll_payload > 0 ? 2LL * kLLMaxSteps * nranks * x.ll_slot_bytes : 0;
  if (cfg.tp_bytes <= 0) cfg.tp_bytes = (long long)e.tp_mb << 20;
  c->cfg.tp_bytes = cfg.tp_bytes;
  const long long tp_flags = cfg.tp_bytes > 0 ? (1 << 20) : 0;
  x.tail_off = 0; x.head_off = flags; x.ll_off = 2 * flags; x.tp_flag_off = x.ll_off + ll_bytes;
  // low-latency FIFO of the executor (all collectives, small messages): head counters, then the lines
  x.llf_head_off = x.tp_flag_off + tp_flags;
  x.llf_off = x.llf_head_off + round_up((long long)nranks * kLLFifoCta * kFlagStride, 4096);
  x.scratch_off = x.llf_off + (long long)nranks * kLLFifoCta * kLLFifoSlots * kLLFifoSlotBytes; x.scratch_bytes = round_up(cfg.scratch_bytes, 4096);
  c->llf_max_bytes = (long long)e.llf_kb * 1024;
  c->ll_max_bytes = ll_payload;
  x.fifo_off = x.scratch_off + x.scratch_bytes;
  x.tp_data_off = round_up(x.fifo_off + (long long)nranks * cfg.max_cta * cfg.nslot * cfg.slot_bytes, 4096);
  x.tp_bytes = round_up(cfg.tp_bytes, 4096);
  x.heap_bytes = x.tp_data_off + x.tp_bytes;
  c->heap_bytes = x.heap_bytes;

  cudaError_t err;
#define CREATE_TRY(expr) if ((err = (expr)) != cudaSuccess) { int rc = fail(PICCL_CUDA_ERROR, "%s failed: %s", #expr, cudaGetErrorString(err)); piccl_comm_destroy(c); return rc; }
  CREATE_TRY(cudaMalloc(&c->heap, c->heap_bytes));
  CREATE_TRY(cudaMemset(c->heap, 0, x.scratch_off));          // counters start at zero; payload needs no clearing
  size_t cnt_bytes = (size_t)nranks * cfg.max_cta * sizeof(unsigned long long);
  CREATE_TRY(cudaMalloc(&c->d_sent, cnt_bytes)); CREATE_TRY(cudaMemset(c->d_sent, 0, cnt_bytes));
  CREATE_TRY(cudaMalloc(&c->d_rcvd, cnt_bytes)); CREATE_TRY(cudaMemset(c->d_rcvd, 0, cnt_bytes));
  size_t cnt_ll = (size_t)nranks * kLLFifoCta * sizeof(unsigned long long);
  CREATE_TRY(cudaMalloc(&c->d_sent_ll, cnt_ll)); CREATE_TRY(cudaMemset(c->d_sent_ll, 0, cnt_ll));
  CREATE_TRY(cudaMalloc(&c->d_rcvd_ll, cnt_ll)); CREATE_TRY(cudaMemset(c->d_rcvd_ll, 0, cnt_ll));
  CREATE_TRY(cudaMalloc(&c->d_abort, sizeof(int))); CREATE_TRY(cudaMemset(c->d_abort, 0, sizeof(int)));
  CREATE_TRY(cudaHostAlloc(&c->h_status, sizeof(piccl_status_t), cudaHostAllocMapped));
  memset(c->h_status, 0, sizeof(piccl_status_t));
  CREATE_TRY(cudaHostGetDevicePointer((void**)&c->d_status, c->h_status, 0));
  CREATE_TRY(cudaMalloc(&c->d_ctx, sizeof(RankCtx)));
  CREATE_TRY(cudaDeviceSynchronize());
#undef CREATE_TRY
  x.sent = c->d_sent; x.rcvd = c->d_rcvd; x.sent_ll = c->d_sent_ll; x.rcvd_ll = c->d_rcvd_ll; x.abort_flag = c->d_abort; x.status = c->d_status;
  int sms = 0; cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device); c->sm_count = sms > 0 ? sms : 148;
  log_msg(2, "comm %p: rank %d/%d dev %d heap %.1f MiB (max_cta %d nslot %d slot %lld KiB scratch %lld MiB)", (void*)c, rank, nranks, device,
          c->heap_bytes / 1048576.0, cfg.max_cta, cfg.nslot, cfg.slot_bytes >> 10, x.scratch_bytes >> 20);
  *out = c;
  return PICCL_OK;
}

int piccl_comm_local_handle(piccl_comm_t* c, piccl_handle_t* out) {
  if (!c || !out) return fail(PICCL_INVALID_ARGUMENT, "null argument");
  DevGuard g(c->device);
  HandleBlob b; memset(&b, 0, sizeof b);
  b.magic = kHandleMagic; b.rank = c->rank; b.nranks = c->nranks; b.pid = (int)getpid(); b.device = c->device;
  b.host_id = c->host_id; b.heap_bytes = (unsigned long long)c->heap_bytes; b.raw_ptr = (unsigned long long)(uintptr_t)c->heap;
  b.max_cta = c->cfg.max_cta; b.nslot = c->cfg.nslot; b.slot_bytes = (unsigned long long)c->cfg.slot_bytes;
  cudaError_t e = cudaIpcGetMemHandle(&b.ipc, c->heap);
  b.ipc_ok = (e == cudaSuccess) ? 1 : 0;
  if (env().nvls && nvls_device_capable(c->device)) b.ipc_ok |= 2;
  b.ipc_ok |= (c->cfg.nvls_cta & 0xff) << 8;                 // the window geometry must agree on all ranks
  if (e != cudaSuccess) { cudaGetLastError(); log_msg(1, "cudaIpcGetMemHandle: %s (peers in other processes cannot map this rank)", cudaGetErrorString(e)); }
  static_assert(sizeof(HandleBlob) <= sizeof(piccl_handle_t), "handle blob too large");
  memset(out, 0, sizeof *out); memcpy(out->bytes, &b, sizeof b);
  return PICCL_OK;
}

int piccl_comm_connect(piccl_comm_t* c, const piccl_handle_t* all) {
  if (!c || !all) return fail(PICCL_INVALID_ARGUMENT, "null argument");
  if (c->connected) return fail(PICCL_INVALID_USAGE, "communicator already connected");
  DevGuard g(c->device);
  for (int p = 0; p < c->nranks; p++) {
    HandleBlob b; memcpy(&b, all[p].bytes, sizeof b);
    if (b.magic != kHandleMagic || b.rank != p || b.nranks != c->nranks) return fail(PICCL_INVALID_ARGUMENT, "handle %d is not a handle of rank %d of this communicator", p, p);
    if (b.max_cta != c->cfg.max_cta || b.nslot != c->cfg.nslot || (long long)b.slot_bytes != c->cfg.slot_bytes || (long long)b.heap_bytes != c->heap_bytes)
      return fail(PICCL_INVALID_USAGE, "rank %d uses a different heap layout (PICCL_MAX_CTA/NSLOT/SLOT_KB/SCRATCH_MB must agree)", p);
    if (((b.ipc_ok >> 8) & 0xff) != (c->cfg.nvls_cta & 0xff)) return fail(PICCL_INVALID_USAGE, "rank %d uses a different number of in-switch CTAs (nvls_cta / PICCL_NVLS_CTA must agree)", p);
    if (p == c->rank) { c->h_ctx.heap[p] = c->heap; continue; }
    if (b.host_id != c->host_id) return fail(PICCL_UNSUPPORTED, "rank %d is on another host: peer memory is not reachable", p);
    if (b.pid == (int)getpid()) {
      // same process: the pointer itself is valid; another device needs peer access
      if (b.device != c->device) {
        int can = 0; cudaDeviceCanAccessPeer(&can, c->device, b.device);
        if (!can) return fail(PICCL_UNSUPPORTED, "no peer access from device %d to %d", c->device, b.device);
        cudaError_t e = cudaDeviceEnablePeerAccess(b.device, 0);
        if (e != cudaSuccess && e != cudaErrorPeerAccessAlreadyEnabled) return fail(PICCL_CUDA_ERROR, "cudaDeviceEnablePeerAccess: %s", cudaGetErrorString(e));
        cudaGetLastError();
      }
      c->h_ctx.heap[p] = (char*)(uintptr_t)b.raw_ptr;
    } else {
      if (!(b.ipc_ok & 1)) return fail(PICCL_UNSUPPORTED, "rank %d could not export its heap", p);
      void* ptr = nullptr;
      cudaError_t e = cudaIpcOpenMemHandle(&ptr, b.ipc, cudaIpcMemLazyEnablePeerAccess);
      if (e != cudaSuccess) { cudaGetLastError(); return fail(PICCL_UNSUPPORTED, "cudaIpcOpenMemHandle(rank %d): %s", p, cudaGetErrorString(e)); }
      c->h_ctx.heap[p] = (char*)ptr; c->ipc_opened[p] = true;
    }
  }
  CUDA_TRY(cudaMemcpy(c->d_ctx, &c->h_ctx, sizeof(RankCtx), cudaMemcpyHostToDevice));
  c->connected = true;
  if (c->nranks >= 2) {
    // In-switch collectives: a multicast window if every rank asked for it and can do it, and no two ranks share a process
    // (each rank binds its own device to the multicast object, and the set-up blocks until all ranks take part).
    // All ranks inside this process on this device (virtual ranks): a plain window each, the kernels emulate the switch.
    bool want = true, one_process = true; int root_pid = 0; unsigned long long root_id = 0;
    for (int p = 0; p < c->nranks; p++) {
      HandleBlob b; memcpy(&b, all[p].bytes, sizeof b);
      want &= (b.ipc_ok & 2) != 0;
      one_process &= b.pid == (int)getpid() && b.device == c->device;
      if (p == 0) { root_pid = b.pid; root_id = b.raw_ptr; }
      for (int q = 0; q < p; q++) { HandleBlob o; memcpy(&o, all[q].bytes, sizeof o); if (o.pid == b.pid) want = false; }
    }
    if (one_process) { if (env().nvls && c->nranks <= kMaxVRanks) nvls_setup_emulated(c); }
    else if (want) nvls_setup(c, root_pid, root_id);
  }
  return PICCL_OK;
}

// A consumer's kernel acknowledges the last entries this rank sent by writing head counters into THIS rank's heap, and that
// can happen after this rank's own kernels have ended.  Before the heap is freed: wait on the host, with a limit, until every
// entry sent has been acknowledged.  (Everything peers sent to this rank was consumed by kernels that have ended.)
static void quiesce_fifos(piccl_comm* c) {
  if (!c->connected || !c->heap || c->nranks < 2 || c->broken || (c->h_status && c->h_status->aborted)) return;
  const RankCtx& x = c->h_ctx;
  const int n = c->nranks, mc = c->cfg.max_cta;
  std::vector<unsigned long long> sent((size_t)n * mc), sent_ll((size_t)n * kLLFifoCta);
  const size_t head_bytes = (size_t)n * mc * kFlagStride, llh_bytes = (size_t)n * kLLFifoCta * kFlagStride;
  std::vector<char> head(head_bytes), llh(llh_bytes);
  if (cudaMemcpy(sent.data(), c->d_sent, sent.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess ||
      cudaMemcpy(sent_ll.data(), c->d_sent_ll, sent_ll.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess) { cudaGetLastError(); return; }
  for (int tries = 0; tries < 200; tries++) {
    if (cudaMemcpy(head.data(), c->heap + x.head_off, head_bytes, cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(llh.data(), c->heap + x.llf_head_off, llh_bytes, cudaMemcpyDeviceToHost) != cudaSuccess) { cudaGetLastError(); return; }
    bool done = true;
    for (int p = 0; p < n && done; p++) {
      if (p == c->rank) continue;
      for (int b = 0; b < mc && done; b++) { unsigned long long h; memcpy(&h, &head[(size_t)(p * mc + b) * kFlagStride], 8); if (h < sent[(size_t)p * mc + b]) done = false; }
      for (int b = 0; b < kLLFifoCta && done; b++) { unsigned long long h; memcpy(&h, &llh[(size_t)(p * kLLFifoCta + b) * kFlagStride], 8); if (h < sent_ll[(size_t)p * kLLFifoCta + b]) done = false; }
    }
    if (done) return;
    usleep(5000);
  }
  log_msg(1, "rank %d: peers did not acknowledge everything this rank sent within 1 s", c->rank);
}

int piccl_comm_destroy(piccl_comm_t* c) {
  if (!c) return PICCL_OK;
  DevGuard g(c->device);
  cudaDeviceSynchronize();
  quiesce_fifos(c);
  persist_destroy(c);
  nvls_destroy(c);
  if (!env().trace_file.empty()) trace_dump(c);
  if (env().log_level >= 1) {
    const piccl_stats_t& s = c->stats;
    log_msg(1, "comm rank %d: calls ag %llu ar %llu bc %llu rd %llu rs %llu, launches %llu, cache hit/miss %llu/%llu, fallbacks %llu, timeouts %llu", c->rank,
            s.calls[0], s.calls[1], s.calls[2], s.calls[3], s.calls[4], s.launches, s.program_cache_hits, s.program_cache_misses, s.fallbacks, s.timeouts);
  }
  for (int p = 0; p < c->nranks; p++) if (c->ipc_opened[p]) cudaIpcCloseMemHandle(c->h_ctx.heap[p]);
  for (auto* chunks : {&c->chunks, &c->flow_chunks}) for (auto& ch : *chunks) { cudaFree(ch.dev); cudaFreeHost(ch.host); }
  for (auto& kv : c->cache) if (kv.second.ready) cudaEventDestroy(kv.second.ready);
  for (auto& t : c->trace) { if (t.start) cudaEventDestroy(t.start); if (t.stop) cudaEventDestroy(t.stop); }
  if (c->d_tp_status) cudaFree(c->d_tp_status);
  cudaFree(c->d_sent_ll); cudaFree(c->d_rcvd_ll);
  cudaFree(c->heap); cudaFree(c->d_sent); cudaFree(c->d_rcvd); cudaFree(c->d_abort); cudaFree(c->d_ctx);
  if (c->h_status) cudaFreeHost(c->h_status);
  cudaGetLastError();
  delete c;
  return PICCL_OK;
}

int piccl_comm_abort(piccl_comm_t* c) {
  if (!c) return PICCL_OK;
  DevGuard g(c->device);
  int one = 1;
  // a blocking copy on the legacy stream would wait for the very kernel we want to stop
  cudaStream_t s; if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) return fail(PICCL_CUDA_ERROR, "stream create failed");
  cudaMemcpyAsync(c->d_abort, &one, sizeof one, cudaMemcpyHostToDevice, s);
  cudaStreamSynchronize(s); cudaStreamDestroy(s);
  if (!c->h_status->aborted) { c->h_status->code = 3; c->h_status->rank = c->rank; c->h_status->aborted = 1; }
  c->broken = true;
  return PICCL_OK;
}

int piccl_comm_status(piccl_comm_t* c, piccl_status_t* out) {
  if (!c || !out) return fail(PICCL_INVALID_ARGUMENT, "null argument");
  memcpy(out, (const void*)c->h_status, sizeof *out);
  return PICCL_OK;
}
int piccl_get_stats(piccl_comm_t* c, piccl_stats_t* out) {
  if (!c || !out) return fail(PICCL_INVALID_ARGUMENT, "null argument");
  std::lock_guard<std::mutex> l(c->mu); *out = c->stats; out->timeouts += c->h_status->aborted && c->h_status->code != 3 ? 1 : 0; return PICCL_OK;
}
int piccl_comm_rank(piccl_comm_t* c) { return c ? c->rank : -1; }
int piccl_comm_nranks(piccl_comm_t* c) { return c ? c->nranks : -1; }

}  // extern "C"

// ------------------------------------------------------------------ program cache
namespace piccl {

struct CallDesc { Coll coll; const void* send; void* recv; size_t count; int dtype, op, root; Algo algo; int k; };

// What is uploaded is kept for the life of the communicator (kernels in flight may read it): programs and data flows may take this much each.
constexpr size_t kKeptBytes = (size_t)256 << 20;
static size_t held(const std::vector<ProgChunk>& chunks) {
  size_t n = 0;
  for (const auto& ch : chunks) n += ch.cap;
  return n;
}
// `bytes` of `data` on the device; they stay as long as the communicator.
static int upload(std::vector<ProgChunk>& chunks, const void* data, size_t data_bytes, size_t bytes, cudaStream_t stream, ProgEntry& e, const void** dev) {
  bytes = (bytes + 255) / 256 * 256;
  if (chunks.empty() || chunks.back().used + bytes > chunks.back().cap) {
    ProgChunk ch; ch.cap = std::max<size_t>(1 << 20, bytes); ch.used = 0;
    CUDA_TRY(cudaMalloc(&ch.dev, ch.cap));
    cudaError_t er = cudaHostAlloc(&ch.host, ch.cap, cudaHostAllocDefault);
    if (er != cudaSuccess) { cudaFree(ch.dev); return fail(PICCL_CUDA_ERROR, "cudaHostAlloc: %s", cudaGetErrorString(er)); }
    chunks.push_back(ch);
  }
  ProgChunk& ch = chunks.back();
  memcpy(ch.host + ch.used, data, data_bytes);
  *dev = ch.dev + ch.used; e.origin = stream; e.synced = false;
  if (data_bytes) CUDA_TRY(cudaMemcpyAsync(ch.dev + ch.used, ch.host + ch.used, data_bytes, cudaMemcpyHostToDevice, stream));
  CUDA_TRY(cudaEventCreateWithFlags(&e.ready, cudaEventDisableTiming));
  CUDA_TRY(cudaEventRecord(e.ready, stream));
  ch.used += bytes;
  return PICCL_OK;
}
static int upload_program(piccl_comm* c, const Program& p, cudaStream_t stream, ProgEntry& e) {
  const void* dev = nullptr;
  const int rc = upload(c->chunks, p.actions.data(), p.actions.size() * sizeof(Action), std::max<size_t>(p.actions.size(), 1) * sizeof(Action), stream, e, &dev);
  e.dev = static_cast<const Action*>(dev); e.n_actions = (int)p.actions.size(); e.scratch_elems = p.scratch_elems;
  return rc;
}
// The entry's upload is done, or `stream` waits for it.
static int after_upload(ProgEntry& e, cudaStream_t stream) {
  if (e.synced) return PICCL_OK;
  // Asked first, and in the relaxed mode: a stream in capture cannot wait for an upload outside it, and a question in the global mode would end the capture.
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (cudaEventQuery(e.ready) == cudaSuccess) e.synced = true; else cudaGetLastError();
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (!e.synced && e.origin != stream) CUDA_TRY(cudaStreamWaitEvent(stream, e.ready, 0));
  return PICCL_OK;
}

// PICCL_DEBUG=1: every action of a freshly compiled program is checked against the extents of the
// buffers of the call before it is ever given to the device (ranges, peers, scratch capacity); a data flow's operations likewise (flow.cc: check_flow).
static const char* check_program(const Program& p, const CollArgs& a, long long scratch_cap_elems) {
  const long long st = a.block_stride ? a.block_stride : a.count;
  long long in_elems = a.count, out_elems = a.count;
  if (a.coll == COLL_ALLGATHER) out_elems = (a.nranks - 1) * st + a.count;
  if (a.coll == COLL_REDUCE_SCATTER) in_elems = (a.nranks - 1) * st + a.count;
  for (const Action& ac : p.actions) {
    if (ac.count <= 0 || ac.n_recv > kMaxActionPeers || ac.n_send > kMaxActionPeers) return "bad operand count";
    for (int i = 0; i < ac.n_recv; i++) if (ac.recv_peer[i] >= a.nranks || ac.recv_peer[i] == p.rank) return "bad receive peer";
    for (int i = 0; i < ac.n_send; i++) if (ac.send_peer[i] >= a.nranks || ac.send_peer[i] == p.rank) return "bad send peer";
    const long long slim = ac.src_buf == BUF_IN ? in_elems : ac.src_buf == BUF_OUT ? out_elems : scratch_cap_elems;
    if (ac.src_buf != BUF_NONE && (ac.src_off < 0 || ac.src_off + ac.count > slim)) return "source range outside its buffer";
    const long long dlim = ac.dst_buf == BUF_OUT ? out_elems : scratch_cap_elems;
    if (ac.dst_buf == BUF_IN) return "write to the send buffer";
    if (ac.dst_buf != BUF_NONE && (ac.dst_off < 0 || ac.dst_off + ac.count > dlim)) return "destination range outside its buffer";
  }
  return nullptr;
}

static int get_program(piccl_comm* c, const CollArgs& a, cudaStream_t stream, const ProgEntry** out) {
  ProgKey k{(int)a.coll, (int)a.algo, a.k, a.root, a.elem_size, a.in_place ? 1 : 0, a.count, a.block_stride};
  auto it = c->cache.find(k);
  if (it == c->cache.end()) {
    // A new program needs device and pinned memory and an upload on the caller's stream: not inside a stream capture (an
    // allocation ends a capture in the global mode, and the upload's event would belong to the graph).  The caller runs
    // the call once before capturing, or, in the preload library, the call goes to NCCL.
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone) {
      c->stats.fallbacks++;
      return fail(PICCL_UNSUPPORTED, "%s %s of %lld elements was never run outside a stream capture: its program cannot be built while capturing", coll_name(a.coll), algo_name(a.algo), a.count);
    }
    cudaGetLastError();
    if (held(c->chunks) > kKeptBytes) {
      c->stats.fallbacks++;
      return fail(PICCL_UNSUPPORTED, "program cache full (%zu MiB for %zu distinct calls)", held(c->chunks) >> 20, c->cache.size());
    }
    c->stats.program_cache_misses++;
    Program p = compile(a, c->rank);
    if (env().debug) {
      if (const char* why = check_program(p, a, c->h_ctx.scratch_bytes / std::max(1, a.elem_size)))
        return fail(PICCL_INTERNAL_ERROR, "program check failed (%s %s, rank %d): %s", coll_name(a.coll), algo_name(a.algo), c->rank, why);
    }
    ProgEntry e;
    for (const Action& ac : p.actions) e.offsets_aligned &= (ac.src_off * a.elem_size) % 16 == 0 && (ac.dst_off * a.elem_size) % 16 == 0;
    int rc = upload_program(c, p, stream, e); if (rc) return rc;
    it = c->cache.emplace(k, e).first;
  } else {
    c->stats.program_cache_hits++;
    if (int rc = after_upload(it->second, stream)) return rc;
  }
  *out = &it->second;
  return PICCL_OK;
}

// May this launch run the call's data flow (flow.cc) in place of the ranks' programs?  All ranks in one launch on one GPU; no receive buffer may overlap another rank's buffers, or,
// but for an all-gather or broadcast in place, which never write what others read, its own send buffer: an operation could overwrite what another is still to read.
static bool may_flow(piccl_comm** comms, int n, const CallDesc* calls, long long bytes) {
  const CallDesc& d0 = calls[0];
  if (n != comms[0]->nranks || n < 2) return false;
  struct Span { const char *lo, *hi; } in[kMaxVRanks], out[kMaxVRanks];
  auto meet = [](const Span& a, const Span& b) { return a.lo < b.hi && b.lo < a.hi; };
  const long long blocks_in = d0.coll == COLL_REDUCE_SCATTER ? n : 1, blocks_out = d0.coll == COLL_ALLGATHER ? n : 1;
  const bool moves = d0.coll == COLL_ALLGATHER || d0.coll == COLL_BROADCAST;
  int in_place = 0;
  for (int i = 0; i < n; i++) {
    if (comms[i]->rank != i || comms[i]->slots_only) return false;
    const char *s = (const char*)calls[i].send, *r = (const char*)calls[i].recv;
    const bool reads = d0.coll != COLL_BROADCAST || i == d0.root, writes = d0.coll != COLL_REDUCE || i == d0.root;
    in[i] = {s, s + (reads ? blocks_in * bytes : 0)}; out[i] = {r, r + (writes ? blocks_out * bytes : 0)};
    in_place += moves && s == r + (d0.coll == COLL_ALLGATHER ? i * bytes : 0);
  }
  if (in_place != 0 && in_place != n) return false;
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      if (i < j && meet(out[i], out[j])) return false;
      if (meet(out[i], in[j]) && !(i == j && in_place)) return false;
    }
  return true;
}

// CTAs for one collective: enough to fill NVLink for large messages, one for tiny ones.
// All ranks compute the same number from the same arguments.  The reference's grid formula
// grid = clamp(count / block, MIN, MAX) (src/kernels/permutation_kernel.cu:76-77) is kept when
// PICCL_MIN/MAX_GRID_SIZE are set; the result is capped by the FIFO channel count.
static int choose_cta(const piccl_comm* c, const CollArgs& a, int n_vrank) {
  long long bytes = a.count * a.elem_size;
  if (a.coll == COLL_ALLREDUCE && (a.algo == ALGO_RING || a.algo == ALGO_K_RING)) bytes /= std::max(1, a.nranks);
  if (a.algo == ALGO_DIRECT && a.coll != COLL_ALLGATHER && a.coll != COLL_REDUCE_SCATTER) bytes /= std::max(1, a.coll == COLL_ALLREDUCE ? a.nranks : a.nranks - 1);
  const Env& e = env();
  // (all ranks in one launch, whose steps cost less than a way over NVLink: 280 KB among eight ranks 42 us at 32 KiB a CTA, 35 at 16.  Part of the ranks
  // in one launch: the others may be in launches of other sizes and have to come to the same number)
  const long long per = n_vrank > 1 && n_vrank == c->nranks ? 16384 : 32768;
  long long n = (bytes + per - 1) / per;
  if (e.min_grid_set || e.max_grid_set) {
    long long g = a.count / std::max(1, c->cfg.block_size);
    n = std::max<long long>(e.min_grid_set ? e.min_grid : 1, std::min<long long>(e.max_grid_set ? e.max_grid : g, g));
  }
  n = std::max<long long>(1, std::min<long long>(n, c->cfg.max_cta));
  if (n_vrank > 1) n = std::min<long long>(n, std::max(1, c->sm_count / n_vrank));
  return (int)n;
}

// threads of an executor CTA: the configured block moves data, two more warps wait and publish
static int exec_block(const piccl_comm* c) { return c->cfg.block_size + kCtlThreads; }

// Do the caller's buffers of a launch of n ranks, read and written, crowd what is on its way between ranks out of L2 (126 MB)?  Then the executor asks L2 to let go of
// the caller's lines first, each with its last use (exec_impl.cuh: stream): of operands (1) and of results (2).
// Operands, us without and with: all-reduce on the ring 8 x 16 MiB 109.7 / 108.1, 8 x 32 209 / 200.6, 8 x 64 407 / 392, recursive doubling 4 x 17 93.1 / 89.2; reduce-scatter
// 2 x 16 MiB 33.2 / 31.5, 8 x 8 216 / 202.5, 8 x 16 418 / 392; reduce 4 x 16 49.5 / 47.9; below their lines no gain or a loss (all-reduce 8 x 4 MiB 75 / 80, reduce-scatter 2 x 8 19.9 / 21.1).
// (Of an all-reduce more stays in L2 from one call to the next: its line lies higher.)  A reader of the operands after the call loses nothing (reduce-scatter 2 x 16 47.8 / 46.7).
// Results are read by whoever called, and those that L2 could keep are worth more there.  Call, and call with a kernel that scales the results in place, without and with:
// reduce-scatter 2 x 32 MiB (64 MiB of results) 56.3 / 55.1, but 72.5 / 77.7; broadcast 4 x 16 (64) 50 / 50, 68.4 / 72.6; all-gather 4 x 4 (64) 35.5 / 34.3, 51.9 / 54.0, 2 x 26 (104)
// 48.5 / 45.3, 76.5 / 80.5; all-reduce 2 x 40 (80) 59.4 / 54.9, 81.9 / 84.3, 8 x 12 (96) 97.2 / 97.3, 126 / 128.  So results leave first only where they do not fit in any case: all-gather 4 x 8 (128)
// 61.2 / 55.7, 99.6 / 96.6, 4 x 16 (256) 115 / 102, 195 / 186; reduce-scatter 2 x 64 (128) 102.8 / 99.3, 141.5 / 141.6; broadcast 8 x 32 (256) 157.8 / 153.2, 239.6 / 235.8; all-reduce
// 8 x 32 (256) 200.6 / 193, 281 / 274.6, 8 x 64 392 / 369.5, 551 / 529.  An all-reduce passes over them again for each step, and gains from 100 MiB on: recursive doubling 4 x 25 131 / 128.5, 162.9 / 161.
// All of this is of launches that carry every rank on one GPU: elsewhere the slots are filled by other GPUs, and nothing leaves first.
static int leave_first(const CollArgs& a, int n, bool one_gpu) {
  if (!one_gpu) return 0;
  const long long one = (long long)a.count * a.elem_size, MiB = 1 << 20;
  long long bytes = 0, line = 72 * MiB, results = n * one, results_line = 120 * MiB;
  switch (a.coll) {
    case COLL_ALLREDUCE: bytes = 2 * n * one; line = 128 * MiB; results_line = 98 * MiB; break;
    case COLL_ALLGATHER: bytes = n * (1 + a.nranks) * one; results = n * a.nranks * one; break;
    case COLL_REDUCE_SCATTER: bytes = n * (1 + a.nranks) * one; break;
    case COLL_REDUCE: bytes = (n + 1) * one; results = one; break;
    default: bytes = (n + 1) * one; break;
  }
  return bytes <= line ? 0 : results > results_line ? 3 : 1;
}

// Segments of the executor.  Two are walked together where there are slots for it (the protocol needs two slots per segment of a window): the way from a
// peer's stores to my loads then hides behind the other one.  One launch for all ranks: segments of at most 128 KiB, a quarter of the default
// slot, so that what is on its way between ranks stays in L2 (512 KiB slots of 144 CTAs are 300 MB).  Measured with 512 threads, 8 x 64 MiB all-reduce on the
// ring: 408 us with 128 KiB, 463 with 64 or 256 KiB, 446 with the slots as they are; at least 32 KiB, a round of four packs a thread, and
// a message is cut into two where it can be.  Ranks in launches of their own keep the communicator's slots: they may be a call apart.
static void cut_fifo(const piccl_comm* c, int n_vrank, int n_cta, const CollArgs& a, KernelArgs* ka) {
  const RankCtx& x = c->h_ctx;
  ka->seg_bytes = x.slot_bytes; ka->nslot = x.nslot; ka->window = window_of(x.nslot);
  if (n_vrank != c->nranks || n_vrank < 2) return;
  const long long chan = x.nslot * x.slot_bytes, round = (long long)c->cfg.block_size * 64;
  long long slice = a.count * a.elem_size;
  if (a.coll == COLL_ALLREDUCE && (a.algo == ALGO_RING || a.algo == ALGO_K_RING)) slice /= c->nranks;
  slice = (slice + n_cta - 1) / n_cta;
  const long long seg = std::min<long long>(round_up((slice + 1) / 2, round), std::max<long long>(round, 131072 / round * round));
  ka->nslot = 4; ka->window = window_of(4);
  ka->seg_bytes = std::max<long long>(16, std::min<long long>(seg, chan / 4 / 16 * 16));
}

static bool fault_now(piccl_comm* c) {
  const Env& e = env();
  if (e.fault_rank != c->rank) return false;
  unsigned long long call = c->call_index;
  if ((long long)call != e.fault_call) return false;
  if (e.fault_delay_ms > 0) { log_msg(1, "fault injection: delaying call %llu by %d ms", call, e.fault_delay_ms); std::this_thread::sleep_for(std::chrono::milliseconds(e.fault_delay_ms)); return false; }
  if (e.fault_skip) { log_msg(1, "fault injection: skipping call %llu", call); return true; }
  return false;
}

// CTAs of a low-latency kernel: one line per thread as far as the SMs go (a thread takes its lines one after the other, each with its
// own round trip: 32 KiB among eight ranks 12.3 us with four lines a thread, 6.3 us with one), never fewer than the kernel's most lines per thread need.
static int ll_ctas(long long nlines, int most_lines, int sms) {
  const long long spread = std::min<long long>((nlines + kLLBlock - 1) / kLLBlock, std::max(1, sms));
  return (int)std::max(spread, (nlines + most_lines - 1) / most_lines);
}

// Fills `out` with the call-independent part of a low-latency all-reduce; false: the schedule is not one of exchanges among all ranks.
static bool ll_plan(piccl_comm** comms, int n, Algo algo, int k, LLArgs* out) {
  piccl_comm* c0 = comms[0];
  std::lock_guard<std::mutex> l(c0->mu);
  for (const LLPlan& p : c0->ll_plans) {
    if (p.n != n || p.algo != (int)algo || p.k != k) continue;
    bool same = true;
    for (int i = 0; i < n; i++) same &= p.ranks[i] == comms[i]->rank;
    if (same) { if (p.usable) *out = p.args; return p.usable; }
  }
  LLPlan p; memset(&p, 0, sizeof p);
  p.n = n; p.algo = (int)algo; p.k = k;
  for (int i = 0; i < n; i++) p.ranks[i] = comms[i]->rank;
  const Resolved rs = resolve(COLL_ALLREDUCE, algo, k, c0->nranks);
  p.usable = rs.core == c0->nranks && !rs.radices.empty() && (int)rs.radices.size() <= kLLMaxSteps && rs.algo == algo;
  if (p.usable) {
    const bool permuted = algo == ALGO_PRD || algo == ALGO_PRM;
    p.args.n_vrank = n; p.args.nsteps = (int)rs.radices.size();
    for (int i = 0; i < n; i++)
      for (int s = 0; s < p.args.nsteps; s++) {
        std::vector<int> pe = step_peers(comms[i]->rank, s, rs.radices, c0->nranks, permuted);
        std::sort(pe.begin(), pe.end());
        p.args.npeers[s] = (uint8_t)pe.size();
        int below = 0;
        for (size_t j = 0; j < pe.size(); j++) { p.args.peers[i][s][j] = (uint8_t)pe[j]; if (pe[j] < comms[i]->rank) below++; }
        p.args.self_pos[i][s] = (uint8_t)below;
      }
  }
  if (c0->ll_plans.size() >= 64) c0->ll_plans.clear();      // a program uses a handful of algorithms
  c0->ll_plans.push_back(p);
  if (p.usable) *out = p.args;
  return p.usable;
}

// Is this a small exchange-type all-reduce, which the low-latency kernel takes (flags travel inside the data lines)?  Its call-independent arguments then.
static bool ll_takes(piccl_comm** comms, int n, const CallDesc& d, int esz, LLArgs* la) {
  piccl_comm* c0 = comms[0];
  if (d.coll != COLL_ALLREDUCE || c0->ll_max_bytes <= 0 || (long long)d.count * esz > c0->ll_max_bytes) return false;
  if (d.algo != ALGO_RD && d.algo != ALGO_RM && d.algo != ALGO_PRD && d.algo != ALGO_PRM) return false;
  if (!ll_plan(comms, n, d.algo, d.k, la)) return false;
  const int E = 8 / esz;
  const long long nlines = ((long long)d.count + E - 1) / E;
  // (the persistent server is one CTA: what fits one goes to it)
  la->n_cta = env().launch_persistent && nlines <= ll_lines_per_cta() ? 1 : ll_ctas(nlines, ll_lines_per_cta(), c0->sm_count / n);
  return n * la->n_cta <= c0->sm_count;
}
// A small all-gather / reduce-scatter whose schedule is one exchange with every rank (DIRECT, or RM / PRM with a radix of at least the rank count): the low-latency exchange kernel.
static bool llx_takes(piccl_comm** comms, int n, const CallDesc& d, int esz, LLXArgs* xa) {
  piccl_comm* c0 = comms[0];
  if ((d.coll != COLL_ALLGATHER && d.coll != COLL_REDUCE_SCATTER) || c0->ll_max_bytes <= 0 || c0->nranks < 2 ||
      (long long)d.count * esz > std::min<long long>(c0->ll_max_bytes, (long long)env().llx_kb * 1024)) return false;
  if (d.algo != ALGO_DIRECT && !((d.algo == ALGO_RM || d.algo == ALGO_PRM) && d.k >= c0->nranks)) return false;
  memset(xa, 0, sizeof *xa);
  xa->count = d.coll == COLL_ALLGATHER ? (long long)d.count * esz : (long long)d.count;
  const long long nlines = d.coll == COLL_ALLGATHER ? (xa->count + 7) / 8 : ((long long)d.count + (8 / esz) - 1) / (8 / esz);
  xa->n_cta = ll_ctas(nlines, llx_lines_per_cta(), c0->sm_count / n);
  return n * xa->n_cta <= c0->sm_count;
}

// Slices to an operation: blocks of 4 KiB, one 16-byte pack a thread, while there are SMs for more of them, and no larger than 64 KiB, so that the last wave is short (figures in flow.cc).
static int flow_slices(const piccl_comm* c, long long bytes, long long ops, long long* slice_bytes) {
  const long long even = (ops * bytes / (12LL * c->sm_count) + 4095) / 4096 * 4096;
  *slice_bytes = std::max<long long>(4096, std::min<long long>(65536, even));
  return (int)std::max<long long>(1, (bytes + *slice_bytes - 1) / *slice_bytes);
}

// The call's data flow, all ranks in this launch; ll: of a call that a low-latency kernel would take, whose averages it gives; *fresh: it was not known before.  PICCL_UNSUPPORTED: nothing was done, the ranks' programs are to run.
static int run_flow(piccl_comm** comms, int n, const CallDesc* calls, long long count, int esz, int op, bool avg, bool ll, bool capturing, bool* fresh, cudaStream_t stream) {
  piccl_comm* c0 = comms[0];
  const CallDesc& d0 = calls[0];
  *fresh = false;
  const bool reducing = d0.coll == COLL_ALLREDUCE || d0.coll == COLL_REDUCE || d0.coll == COLL_REDUCE_SCATTER;
  CollArgs a; a.coll = d0.coll; a.algo = d0.algo; a.k = d0.k; a.nranks = n; a.root = d0.root; a.count = count; a.elem_size = esz;
  a.in_place = !reducing && d0.send == d0.recv;              // (an all-gather's rank 0: its block is the buffer's first; may_flow: all ranks or none)
  ProgKey k{(int)a.coll, (int)a.algo, a.k, a.root, a.elem_size, a.in_place ? 1 : 0, a.count, 0};
  const bool floats = !reducing || d0.dtype == DT_F16 || d0.dtype == DT_F32 || d0.dtype == DT_F64 || d0.dtype == DT_BF16;
  const FlowKind kind = !floats ? FLOW_INTEGERS : !avg || esz != 2 ? FLOW_FLOATS : ll ? FLOW_ALL_SHARES : d0.dtype == DT_F16 ? FLOW_SMALL_SHARES : FLOW_FLOATS;
  k.flow = kind;
  ProgEntry* e = nullptr;
  {
    std::lock_guard<std::mutex> l(c0->mu);
    auto it = c0->cache.find(k);
    if (it == c0->cache.end()) {
      if (capturing || held(c0->flow_chunks) > kKeptBytes) return PICCL_UNSUPPORTED;      // (the programs, which take a fraction of the room, or what their path says)
      std::vector<Program> progs;
      for (int r = 0; r < n; r++) progs.push_back(compile(a, r));
      std::vector<FlowOp> ops;
      ProgEntry x;
      if (data_flow(progs, ops, kind)) {
        if (env().debug) if (const char* why = check_flow(ops, a)) return fail(PICCL_INTERNAL_ERROR, "data flow check failed (%s %s): %s", coll_name(a.coll), algo_name(a.algo), why);
        for (const FlowOp& o : ops) {
          x.most = std::max<long long>(x.most, o.count); x.leaves = std::max<int>(x.leaves, o.n_leaf);
          for (int i = 0; i < o.n_leaf; i++) x.offsets_aligned &= o.leaf_off[i] * esz % 16 == 0;
          for (int i = 0; i < o.n_dst; i++) x.offsets_aligned &= o.dst_off[i] * esz % 16 == 0;
        }
        x.n_ops = (int)ops.size();
      }
      const void* dev = nullptr;
      if (int rc = upload(c0->flow_chunks, ops.data(), ops.size() * sizeof(FlowOp), std::max<size_t>(1, ops.size()) * sizeof(FlowOp), stream, x, &dev)) return rc;
      x.ops = static_cast<const FlowOp*>(dev);
      it = c0->cache.emplace(k, x).first;
      *fresh = true;
      for (int i = 0; i < n; i++) comms[i]->stats.program_cache_misses++;
    } else {
      if (int rc = after_upload(it->second, stream)) return rc;
      for (int i = 0; i < n; i++) comms[i]->stats.program_cache_hits++;
    }
    e = &it->second;
  }
  if (e->n_ops == 0) return PICCL_UNSUPPORTED;
  FlowArgs fa; memset(&fa, 0, sizeof fa);
  fa.n_ops = e->n_ops; fa.avg = avg ? 1 : 0; fa.scale = avg ? 1.0f / (float)n : 1.0f; fa.ops = e->ops;
  fa.leave_first = leave_first(a, n, true);
  fa.n_slices = flow_slices(c0, e->most * esz, e->n_ops, &fa.slice_bytes);
  bool aligned = e->offsets_aligned, skip = false;
  for (int i = 0; i < n; i++) {
    fa.in[i] = calls[i].send; fa.out[i] = calls[i].recv;
    aligned &= ((reinterpret_cast<uintptr_t>(calls[i].send) | reinterpret_cast<uintptr_t>(calls[i].recv)) & 15) == 0;
  }
  // Small sums at odd addresses, whose code takes longer to fetch than their data: those that the low-latency kernels make in one launch too stay with them.  us there and as a data flow: all-reduce of
  // 20 KB of fp16 among four ranks 6.6 / 8.1, among eight 7.5 / 13.8, of 80 KB 12.3 / 13.9 (160 KB 26.7 / 13.9, four ranks 9.2 / 8.2); reduce of 300 bytes of bf16 among eight in two rings 8.2 / 10.4, of 14 KB 8.9 / 11.2
  // (40 KB in fours 12.4 / 8.5; up to four ranks 7.4 / 5.0).  (A captured call has nothing else that could run.)
  if (!aligned && !capturing && ((ll && e->leaves >= 4 && count * esz <= 98304) || (d0.coll == COLL_REDUCE && e->leaves > 4 && count * esz <= 16384))) return PICCL_UNSUPPORTED;
  for (int i = 0; i < n; i++) {
    std::lock_guard<std::mutex> l(comms[i]->mu);
    comms[i]->stats.launches++;
    skip |= fault_now(comms[i]); comms[i]->call_index++;
  }
  if (skip) return PICCL_OK;
  TraceRec* tr = trace_begin(c0, d0.coll, d0.algo, d0.k, count * esz, fa.n_slices, stream);
  nvtxRangePushA(coll_name(d0.coll));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((long long)fa.n_ops * fa.n_slices)); cfg.blockDim = dim3(kFlowBlock); cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  void* args[] = {&fa};
  const cudaError_t err = cudaLaunchKernelExC(&cfg, (const void*)(reducing ? exec_flow_kernel_for(d0.dtype, op, !aligned) : exec_flow_copy_kernel(!aligned)), args);
  nvtxRangePop();
  trace_end(c0, tr, stream);
  if (err != cudaSuccess) return fail(PICCL_CUDA_ERROR, "launch of a data flow failed: %s", cudaGetErrorString(err));
  for (int i = 0; i < n; i++) { comms[i]->flow_calls++; comms[i]->stats.calls[d0.coll]++; comms[i]->stats.bytes[d0.coll] += (unsigned long long)count * esz; }
  return PICCL_OK;
}

// Runs one collective over `n` communicators of this process (n == 1: the normal case).
static int run(piccl_comm** comms, int n, const CallDesc* calls, cudaStream_t stream) {
  piccl_comm* c0 = comms[0];
  const CallDesc& d0 = calls[0];
  if (n > kMaxVRanks) return fail(PICCL_INVALID_ARGUMENT, "at most %d communicators per group launch", kMaxVRanks);
  for (int i = 0; i < n; i++) {
    if (!comms[i]->connected) return fail(PICCL_INVALID_USAGE, "communicator is not connected");
    if (comms[i]->broken || comms[i]->h_status->aborted) { comms[i]->broken = true; return fail(PICCL_REMOTE_ERROR, "communicator aborted earlier (code %d, peer %d)", comms[i]->h_status->code, comms[i]->h_status->peer); }
    if (comms[i]->device != c0->device) return fail(PICCL_INVALID_ARGUMENT, "group launch needs one device");
  }
  const int esz_real = dtype_size(d0.dtype);
  if (!esz_real) { c0->stats.fallbacks++; return fail(PICCL_UNSUPPORTED, "unsupported data type %d", d0.dtype); }
  const bool reducing = d0.coll == COLL_ALLREDUCE || d0.coll == COLL_REDUCE || d0.coll == COLL_REDUCE_SCATTER;
  int op = d0.op; bool avg = false;
  if (reducing) {
    if (op == 4) { avg = true; op = 0; if (!(d0.dtype == DT_F32 || d0.dtype == DT_F16 || d0.dtype == DT_BF16 || d0.dtype == DT_F64)) { c0->stats.fallbacks++; return fail(PICCL_UNSUPPORTED, "avg on integer types"); } }
    if (op < 0 || op > 3) { c0->stats.fallbacks++; return fail(PICCL_UNSUPPORTED, "unsupported reduction op %d", d0.op); }
  }
  if (d0.root < 0 || d0.root >= c0->nranks) return fail(PICCL_INVALID_ARGUMENT, "root %d out of range", d0.root);
  if (d0.count == 0) return PICCL_OK;
  DevGuard g(c0->device);

  // data-moving collectives run the byte-wise instantiation
  const int esz = reducing ? esz_real : 1;
  const long long count = reducing ? (long long)d0.count : (long long)d0.count * esz_real;
  // small messages of every collective run the low-latency variant of the executor (flags inside the data lines)
  const bool use_llf = c0->llf_max_bytes > 0 && (long long)d0.count * esz_real <= c0->llf_max_bytes;
  ExecKernelFn fn = use_llf ? (reducing ? exec_ll_kernel_for(d0.dtype, op) : exec_ll_copy_kernel())
                   : (reducing ? exec_kernel_for(d0.dtype, op) : exec_copy_kernel());
  if (!fn) return fail(PICCL_INTERNAL_ERROR, "no kernel for dtype %d op %d", d0.dtype, op);

  // All ranks in this launch: the call's data flow, where neither a way between the ranks (PICCL_PROTO, the persistent server, the switch) nor a size of the grid (PICCL_MIN_GRID_SIZE,
  // PICCL_MAX_GRID_SIZE) is asked for by name.  Among eight ranks the low-latency kernels, which are cooperative launches, take 8.2 us for an all-reduce of 64 KiB and for an all-gather of 4 KiB
  // blocks, the data flow 4.9.  An exchange of up to 16 KiB would gain as much (1 KiB 5.9 and 5.1, 4 KiB one after the other 8.2 and 4.9): there the kernel that one rank per GPU runs at these sizes
  // has been kept, so that programs and tests of one GPU run it too.
  constexpr long long kOwnKernelBytes = 16384;
  const Env& ev = env();
  const bool flows = ev.proto == 0 && !ev.launch_persistent && !ev.min_grid_set && !ev.max_grid_set && d0.algo != ALGO_NVLS && may_flow(comms, n, calls, (long long)d0.count * esz_real);
  // (the low-latency kernels not while the stream is being captured: the call epoch is a launch argument, a replay would reuse it)
  cudaStreamCaptureStatus cap_state = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &cap_state) != cudaSuccess) { cudaGetLastError(); cap_state = cudaStreamCaptureStatusNone; }
  const bool capturing = cap_state != cudaStreamCaptureStatusNone;
  LLArgs la;
  LLXArgs xa;
  const bool ll = ll_takes(comms, n, d0, esz_real, &la), llx = llx_takes(comms, n, d0, esz_real, &xa);
  if (flows && !capturing && (ll ? (long long)d0.count * esz_real > kOwnKernelBytes : llx)) {
    bool fresh;
    const int rc = run_flow(comms, n, calls, count, esz, op, avg, true, false, &fresh, stream);
    if (rc != PICCL_UNSUPPORTED) return rc;
  }
  if (ll && !capturing) {
    if (LLKernelFn lf = ll_kernel_for(d0.dtype, op)) {
      la.avg = avg ? 1 : 0; la.scale = avg ? 1.0f / (float)c0->nranks : 1.0f;
      la.count = (long long)d0.count; la.timeout_ns = (unsigned long long)c0->cfg.timeout_ms * 1000000ull;
      bool skip = false;
      for (int i = 0; i < n; i++) {
        piccl_comm* c = comms[i];
        std::lock_guard<std::mutex> l(c->mu);
        la.r[i].ctx = c->d_ctx; la.r[i].in = calls[i].send; la.r[i].out = calls[i].recv;
        la.epoch = ++c->ll_epoch;
        c->stats.launches++; c->stats.calls[COLL_ALLREDUCE]++; c->stats.bytes[COLL_ALLREDUCE] += (unsigned long long)d0.count * esz_real;
        skip |= fault_now(c); c->call_index++;
      }
      if (skip) return PICCL_OK;
      if (env().launch_persistent) {
        const void* ins[kMaxVRanks]; void* outs[kMaxVRanks];
        for (int i = 0; i < n; i++) { ins[i] = calls[i].send; outs[i] = calls[i].recv; }
        if (persist_allreduce(comms, n, la, ins, outs, (long long)d0.count, d0.dtype, op, avg ? 1 : 0, (int)d0.algo, d0.k, stream) == PICCL_OK) { c0->stats.persistent_calls++; return PICCL_OK; }
      }
      nvtxRangePushA("allreduce_ll");
      void* args[] = {&la};
      cudaError_t e;
      if (n > 1) e = cudaLaunchCooperativeKernel((const void*)lf, dim3(n * la.n_cta), dim3(kLLBlock), args, 0, stream);
      else e = cudaLaunchKernel((const void*)lf, dim3(la.n_cta), dim3(kLLBlock), args, 0, stream);
      nvtxRangePop();
      if (e != cudaSuccess) return fail(PICCL_CUDA_ERROR, "low-latency launch failed: %s", cudaGetErrorString(e));
      return PICCL_OK;
    }
  }

  if (llx && !capturing) {
    LLXKernelFn xf = d0.coll == COLL_ALLGATHER ? llx_allgather_kernel() : llx_reduce_scatter_kernel_for(d0.dtype, op);
    xa.n_vrank = n; xa.avg = avg ? 1 : 0; xa.scale = avg ? 1.0f / (float)c0->nranks : 1.0f;
    xa.timeout_ns = (unsigned long long)c0->cfg.timeout_ms * 1000000ull;
    if (xf) {
      bool skip = false;
      for (int i = 0; i < n; i++) {
        piccl_comm* c = comms[i];
        std::lock_guard<std::mutex> l(c->mu);
        xa.r[i].ctx = c->d_ctx; xa.r[i].in = calls[i].send; xa.r[i].out = calls[i].recv;
        xa.epoch = ++c->ll_epoch;
        c->stats.launches++; c->stats.calls[d0.coll]++; c->stats.bytes[d0.coll] += (unsigned long long)d0.count * esz_real;
        skip |= fault_now(c); c->call_index++;
      }
      if (skip) return PICCL_OK;
      nvtxRangePushA("exchange_ll");
      void* args[] = {&xa};
      cudaError_t e;
      if (n > 1) e = cudaLaunchCooperativeKernel((const void*)xf, dim3(n * xa.n_cta), dim3(kLLBlock), args, 0, stream);
      else e = cudaLaunchKernel((const void*)xf, dim3(xa.n_cta), dim3(kLLBlock), args, 0, stream);
      nvtxRangePop();
      if (e != cudaSuccess) return fail(PICCL_CUDA_ERROR, "low-latency exchange launch failed: %s", cudaGetErrorString(e));
      return PICCL_OK;
    }
  }

  // through the switch: all ranks of the communicator in this launch (one real rank, or every virtual rank of an emulated group)
  if (d0.algo == ALGO_NVLS || env().proto == 3) {
    bool can = (op == 0 || op == 2 || op == 3 || !reducing) && (n == 1 ? !nvls_emulated(c0) : nvls_emulated(c0) && n == c0->nranks);
    for (int i = 0; i < n && can; i++) can = nvls_eligible(comms[i], d0.coll, d0.dtype, op, d0.count);
    if (can) {
      bool skip = false;
      for (int i = 0; i < n; i++) { std::lock_guard<std::mutex> l(comms[i]->mu); skip |= fault_now(comms[i]); comms[i]->call_index++; }
      if (skip) return PICCL_OK;
      const void* ins[kMaxVRanks]; void* outs[kMaxVRanks];
      for (int i = 0; i < n; i++) { ins[i] = calls[i].send; outs[i] = calls[i].recv; }
      TraceRec* tr = trace_begin(c0, d0.coll, ALGO_NVLS, 0, (long long)d0.count * esz_real, 0, stream);
      nvtxRangePushA("in_switch");
      int rc = nvls_collective(comms, n, d0.coll, ins, outs, d0.count, d0.dtype, op, avg, d0.root, stream);
      nvtxRangePop();
      trace_end(c0, tr, stream);
      if (rc == PICCL_OK) {
        for (int i = 0; i < n; i++) { piccl_comm* c = comms[i]; c->stats.launches++; c->stats.nvls_calls++; c->stats.calls[d0.coll]++; c->stats.bytes[d0.coll] += (unsigned long long)d0.count * esz_real; }
        return rc;
      }
      if (rc != PICCL_UNSUPPORTED) return rc;
    }
  }
  if (d0.algo == ALGO_NVLS) {
    // no window, or a type / operator / size the switch path does not take: what AUTO picks without a window
    CallDesc alt[kMaxVRanks];
    int k2 = d0.k;
    const Algo a2 = select_algo_p2p(c0, d0.coll, d0.count * (size_t)esz_real, &k2);
    for (int i = 0; i < n; i++) { alt[i] = calls[i]; alt[i].algo = a2; alt[i].k = k2; }
    return run(comms, n, alt, stream);
  }

  // slabs: bound the local scratch of the recursive reduce-scatters
  long long slab = count, stride = 0;
  if (d0.coll == COLL_REDUCE_SCATTER) {
    const ProgKey pk{(int)d0.coll, (int)d0.algo, d0.k, 0, esz, 0, count, 0};
    long long scratch_elems = -1;
    { std::lock_guard<std::mutex> l(c0->mu); auto it = c0->scratch_need.find(pk); if (it != c0->scratch_need.end()) scratch_elems = it->second; }
    if (scratch_elems < 0) {
      CollArgs probe; probe.coll = d0.coll; probe.algo = d0.algo; probe.k = d0.k; probe.nranks = c0->nranks; probe.count = count; probe.elem_size = esz;
      scratch_elems = compile(probe, 0).scratch_elems;
      std::lock_guard<std::mutex> l(c0->mu);
      if (c0->scratch_need.size() >= 65536) c0->scratch_need.clear();
      c0->scratch_need.emplace(pk, scratch_elems);
    }
    if (scratch_elems * esz > c0->h_ctx.scratch_bytes) {
      long long blocks = (scratch_elems + count - 1) / count + 1;
      slab = c0->h_ctx.scratch_bytes / esz / blocks / 64 * 64;
      if (slab <= 0) return fail(PICCL_UNSUPPORTED, "scratch too small");
      stride = count;
    }
  }

  // the call of rank i on `cur` elements from `done` on
  auto part_of = [&](int i, long long done, long long cur, const char** s, char** r) {
    const piccl_comm* c = comms[i]; const CallDesc& d = calls[i];
    CollArgs a; a.coll = d.coll; a.algo = d.algo; a.k = d.k; a.nranks = c->nranks; a.root = d.root; a.count = cur; a.block_stride = stride; a.elem_size = esz;
    *s = (const char*)d.send; *r = (char*)d.recv;
    switch (d.coll) {
      case COLL_ALLGATHER: a.in_place = (*s == *r + (long long)c->rank * count); *s += done; *r += done; if (stride == 0 && slab != count) a.block_stride = count; break;
      case COLL_REDUCE_SCATTER: a.in_place = (*r == *s + (long long)c->rank * count * esz); *s += done * esz; *r += done * esz; break;
      default: a.in_place = (*s == *r); break;
    }
    if (d.coll == COLL_REDUCE && c->rank != d.root) a.in_place = false;
    return a;
  };

  if (flows) {
    bool fresh;
    const int flow = run_flow(comms, n, calls, count, esz, op, avg, ll || llx, capturing, &fresh, stream);
    if (flow == PICCL_OK && fresh && !capturing) {
      // The ranks' programs too: the same call may come again inside a stream capture with buffers that overlap, when nothing can be built any more.  (What cannot be kept is refused there.)
      int rc = PICCL_OK;
      for (long long done = 0; done < count && rc == PICCL_OK; done += slab)
        for (int i = 0; i < n && rc == PICCL_OK; i++) {
          std::lock_guard<std::mutex> l(comms[i]->mu);
          const char* s; char* r;
          const ProgEntry* pe = nullptr;
          rc = get_program(comms[i], part_of(i, done, std::min(slab, count - done), &s, &r), stream, &pe);
        }
    }
    if (flow != PICCL_UNSUPPORTED) return flow;
  }

  nvtxRangePushA(coll_name(d0.coll));
  int rc = PICCL_OK;
  for (long long done = 0; done < count && rc == PICCL_OK; done += slab) {
    long long cur = std::min(slab, count - done);
    KernelArgs ka; memset(&ka, 0, sizeof ka);
    ka.n_vrank = n; ka.elem_size = esz; ka.avg = avg ? 1 : 0; ka.scale = avg ? 1.0f / (float)c0->nranks : 1.0f;
    int n_cta = 0;
    bool aligned = true;
    CollArgs priorities_of;
    for (int i = 0; i < n && rc == PICCL_OK; i++) {
      piccl_comm* c = comms[i];
      std::lock_guard<std::mutex> l(c->mu);
      const char* s; char* r;
      const CollArgs a = part_of(i, done, cur, &s, &r);
      const ProgEntry* pe = nullptr;
      rc = get_program(c, a, stream, &pe); if (rc) break;
      if (i == 0) {
        n_cta = choose_cta(c, a, n);
        if (use_llf) {   // a line (8 bytes) per thread and action while there are CTAs, then several; a segment holds 4 KiB
          long long ab = a.count * a.elem_size;
          if (a.coll == COLL_ALLREDUCE && (a.algo == ALGO_RING || a.algo == ALGO_K_RING)) ab /= std::max(1, a.nranks);
          if (a.algo == ALGO_DIRECT && a.coll != COLL_ALLGATHER && a.coll != COLL_REDUCE_SCATTER) ab /= std::max(1, a.coll == COLL_ALLREDUCE ? a.nranks : a.nranks - 1);
          n_cta = (int)std::max<long long>(1, std::min<long long>((ab + kLLBlock * 8 - 1) / (kLLBlock * 8), kLLFifoCta));
          if (n > 1) n_cta = std::min(n_cta, std::max(1, c->sm_count / n));
        }
        ka.n_cta = n_cta; if (!use_llf) cut_fifo(c, n, n_cta, a, &ka);
        priorities_of = a;
        ka.one_gpu = n == c->nranks;
        ka.timeout_ns = (unsigned long long)c->cfg.timeout_ms * 1000000ull;
      }
      ka.one_gpu &= c->device == c0->device;
      ka.r[i].ctx = c->d_ctx; ka.r[i].actions = pe->dev; ka.r[i].n_actions = pe->n_actions; ka.r[i].in = s; ka.r[i].out = r;
      aligned &= pe->offsets_aligned && ((reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(r)) & 15) == 0;
      c->stats.launches++;
    }
    if (rc) break;
    ka.leave_first = leave_first(priorities_of, n, ka.one_gpu);
    bool skip = false;
    for (int i = 0; i < n; i++) skip |= fault_now(comms[i]);
    for (int i = 0; i < n; i++) comms[i]->call_index++;
    if (skip) continue;
    TraceRec* tr = trace_begin(c0, d0.coll, d0.algo, d0.k, cur * esz, n_cta, stream);
    void* args[] = {&ka};
    cudaError_t e;
    const int block = use_llf ? kLLBlock : exec_block(c0);
    // which kernel a rank runs is its own business: both speak the same protocol
    const ExecKernelFn f = (aligned || use_llf) ? fn : reducing ? exec_shift_kernel_for(d0.dtype, op) : exec_shift_copy_kernel();
    if (n > 1) e = cudaLaunchCooperativeKernel((const void*)f, dim3(n * n_cta), dim3(block), args, 0, stream);
    else e = cudaLaunchKernel((const void*)f, dim3(n_cta), dim3(block), args, 0, stream);
    if (e != cudaSuccess) rc = fail(PICCL_CUDA_ERROR, "executor launch failed: %s", cudaGetErrorString(e));
    trace_end(c0, tr, stream);
  }
  nvtxRangePop();
  if (rc == PICCL_OK) for (int i = 0; i < n; i++) { comms[i]->stats.calls[d0.coll]++; comms[i]->stats.bytes[d0.coll] += (unsigned long long)d0.count * esz_real; }
  return rc;
}

}  // namespace piccl

extern "C" {

static int one(piccl_comm_t* c, CallDesc d, void* stream) {
  if (!c) return fail(PICCL_INVALID_ARGUMENT, "null communicator");
  if (d.algo == ALGO_DEFAULT_NCCL || d.algo == ALGO_AUTO) d.algo = select_algo(c, d.coll, d.count * (size_t)dtype_size(d.dtype), &d.k);
  piccl_comm* cs[1] = {c};
  return run(cs, 1, &d, (cudaStream_t)stream);
}

int piccl_allreduce(piccl_comm_t* c, const void* send, void* recv, size_t count, int dtype, int op, int algo, int k, void* stream) {
  return one(c, CallDesc{COLL_ALLREDUCE, send, recv, count, dtype, op, 0, (Algo)algo, k}, stream);
}
int piccl_allgather(piccl_comm_t* c, const void* send, void* recv, size_t sendcount, int dtype, int algo, int k, void* stream) {
  return one(c, CallDesc{COLL_ALLGATHER, send, recv, sendcount, dtype, 0, 0, (Algo)algo, k}, stream);
}
int piccl_reduce_scatter(piccl_comm_t* c, const void* send, void* recv, size_t recvcount, int dtype, int op, int algo, int k, void* stream) {
  return one(c, CallDesc{COLL_REDUCE_SCATTER, send, recv, recvcount, dtype, op, 0, (Algo)algo, k}, stream);
}
int piccl_reduce(piccl_comm_t* c, const void* send, void* recv, size_t count, int dtype, int op, int root, int algo, int k, void* stream) {
  return one(c, CallDesc{COLL_REDUCE, send, recv, count, dtype, op, root, (Algo)algo, k}, stream);
}
int piccl_broadcast(piccl_comm_t* c, const void* send, void* recv, size_t count, int dtype, int root, int algo, int k, void* stream) {
  return one(c, CallDesc{COLL_BROADCAST, send, recv, count, dtype, 0, root, (Algo)algo, k}, stream);
}

int piccl_group_collective(piccl_comm_t** comms, int ncomms, int coll, const void* const* send, void* const* recv,
                           size_t count, int dtype, int op, int root, int algo, int k, void* stream) {
  if (!comms || ncomms < 1 || ncomms > kMaxVRanks) return fail(PICCL_INVALID_ARGUMENT, "bad group size %d", ncomms);
  CallDesc d[kMaxVRanks];
  Algo al = (Algo)algo;
  if (al == ALGO_DEFAULT_NCCL || al == ALGO_AUTO) al = select_algo(comms[0], (Coll)coll, count * (size_t)dtype_size(dtype), &k);
  for (int i = 0; i < ncomms; i++) d[i] = CallDesc{(Coll)coll, send[i], recv[i], count, dtype, op, root, al, k};
  return run(comms, ncomms, d, (cudaStream_t)stream);
}

// Which of the caller's lines the executor asks L2 to let go of first (1 operands, 2 results), for blocks of `bytes` in a launch of `in_launch` of `nranks` ranks.
int piccl_test_leave_first(int coll, int nranks, int in_launch, int one_device, long long bytes) {
  CollArgs a; a.coll = (Coll)coll; a.nranks = nranks; a.count = bytes; a.elem_size = 1;
  return leave_first(a, in_launch, one_device && in_launch == nranks);
}
// on != 0: everything that crosses goes through the slots as it does between GPUs, also where one launch carries all ranks.
int piccl_test_slots_only(piccl_comm_t* c, int on) {
  if (!c) return fail(PICCL_INVALID_ARGUMENT, "null communicator");
  c->slots_only = on != 0;
  return PICCL_OK;
}
long long piccl_test_flow_calls(const piccl_comm_t* c) { return c ? (long long)c->flow_calls : -1; }
int piccl_test_unmatched_wait(piccl_comm_t* c, int timeout_ms, void* stream) {
  if (!c || !c->connected) return fail(PICCL_INVALID_USAGE, "communicator is not connected");
  DevGuard g(c->device);
  // one action: receive 16 bytes from the next rank (or from myself), which never sends
  Program p; p.rank = c->rank; p.nranks = c->nranks;
  Action a; a.n_recv = 1; a.recv_peer[0] = (uint8_t)((c->rank + 1) % c->nranks); a.dst_buf = BUF_SCRATCH; a.dst_off = 0; a.count = 16;
  p.actions.push_back(a);
  ProgEntry e;
  int rc = upload_program(c, p, (cudaStream_t)stream, e); if (rc) return rc;
  c->cache.emplace(ProgKey{-1, 0, 0, 0, 1, 0, (long long)c->cache.size(), 0}, e);
  KernelArgs ka; memset(&ka, 0, sizeof ka);
  ka.n_vrank = 1; ka.n_cta = 1; ka.elem_size = 1; ka.seg_bytes = c->h_ctx.slot_bytes; ka.nslot = c->h_ctx.nslot; ka.window = 1; ka.scale = 1.f; ka.timeout_ns = (unsigned long long)timeout_ms * 1000000ull;
  ka.r[0].ctx = c->d_ctx; ka.r[0].actions = e.dev; ka.r[0].n_actions = 1;
  void* args[] = {&ka};
  CUDA_TRY(cudaLaunchKernel((const void*)exec_copy_kernel(), dim3(1), dim3(exec_block(c)), args, 0, (cudaStream_t)stream));
  return PICCL_OK;
}

}  // extern "C"
