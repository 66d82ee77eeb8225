// Forward and backward pass of the GPT-2 training step as one native call (piccl_b200/models/gpt2.py keeps the parameters).
//
// Why native: the step is a few dozen launches per layer, and issued from Python each cost about 15 us of host time: two layers of
// 256 columns took 1.4 ms for 0.3 ms of kernels, eight layers of 768 columns 4.5 ms for 2.7 ms.  Here a launch of this framework's
// own kernels is a plain call (2 to 3 us); attention goes through ATen's fused kernels without autograd, but for heads of 64 columns the way back, and
// the forward pass of an evaluation, are this framework's where those are the faster kernels (piccl_ops_attn_pays).
//
// A step of the same shape on the same input buffers is captured into a CUDA graph by the caller (models/gpt2.py).  Its weight gradients and
// column sums, which nothing in the backward pass waits for, can then go to a second stream: small ones fill the SMs that the chain of
// input gradients leaves idle, and in a graph the events between the streams cost no host time.
//
// The gradient buffer is laid out in the order in which the backward pass finishes it; `ready(end)` tells the caller that elements
// [0, end) are final, which is where bucketed all-reduces start (the overlap that the reference gets from torch DDP).
// Bias, gamma and beta gradients are column sums of tensors that some kernel holds in registers: each leaves partial rows in fp32,
// one launch per layer folds the partial rows of all eight vectors.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>
#include <c10/core/GradMode.h>
#include <torch/csrc/autograd/autograd.h>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>
#include "../ops/piccl_ops.h"

namespace {

thread_local std::string g_error;

enum { W_QKV, W_O, W_FC, W_PROJ, LN1_G, LN1_B, B_QKV, B_O, LN2_G, LN2_B, B_FC, B_PROJ, PER_LAYER };
enum { NT = 0, NN = 1, TN = 2 };
enum { EPI_BIAS = 0, EPI_GELU = 1, EPI_GELU_GRAD = 3 };
typedef uint16_t b16;       // storage of a bf16 value
typedef void (*ReadyFn)(long long end);

struct Desc {               // mirrored in piccl_b200/models/gpt2.py
  int L, C, H, V, Vp, seq_len;
  float eps;
  int pad;
  b16 *p, *g;               // flat parameters and gradients
  const long long* off;     // element offsets: lnf_g, lnf_b, wpe, wte, then PER_LAYER per layer
};

struct Saved { at::Tensor q, k, v, out, lse, cq, ck, seed, offset; c10::SymInt mq = 0, mk = 0; bool direct = false; };

constexpr size_t kSplitBytes = (size_t)40 << 20;

// The streams that steps are captured on.  They are nobody else's, unlike those of PyTorch's pool: cuBLAS's workspace, which belongs to a
// stream, is written by every replay.  Streams of a model that is gone serve the next one, and so does that workspace.
struct Streams { cudaStream_t main = nullptr, side = nullptr; int device = -1; };
std::mutex g_streams_mutex;
std::vector<Streams> g_streams;

bool take_streams(Streams& st) {
  const int device = at::cuda::current_device();
  std::lock_guard<std::mutex> lock(g_streams_mutex);
  for (auto it = g_streams.begin(); it != g_streams.end(); ++it)
    if (it->device == device) { st = *it; g_streams.erase(it); return true; }
  int low, high;
  if (cudaDeviceGetStreamPriorityRange(&low, &high) != cudaSuccess || cudaStreamCreateWithPriority(&st.main, cudaStreamNonBlocking, std::max(high, low - 1)) != cudaSuccess) return false;
  if (cudaStreamCreateWithPriority(&st.side, cudaStreamNonBlocking, low) != cudaSuccess) { cudaStreamDestroy(st.main); st.main = nullptr; return false; }
  st.device = device;
  return true;
}
void give_back(const Streams& st) {
  std::lock_guard<std::mutex> lock(g_streams_mutex);
  g_streams.push_back(st);
}


struct Model {
  Desc d;
  std::vector<long long> off;
  at::Tensor arena;         // activations and workspace, grown to the largest shape so far
  bool in_callers_graph = false;       // the caller captured launches that use this arena into a graph of its own
  std::vector<at::Tensor> kept;        // such arenas, outgrown since: that graph may be replayed as long as the model lives
  at::Tensor stage, owner;  // fp32 table of embedding gradients (all zero between calls), one row of the batch per token id
  at::Tensor split;         // workspace of the products that split K
  bool split_zero = false, stage_zero = false;      // their zeros have been written, not only captured
  void* ws[2] = {nullptr, nullptr};      // of the main and the second stream
  Streams streams;
  cudaEvent_t ev_fork = nullptr, ev_layer[2] = {nullptr, nullptr};
  std::vector<Saved> saved;
  long long launches = 0, cublas = 0, tcgen05 = 0;
  bool captured = false;
  int backend = 0;          // 0: by size, 1: this framework's GEMM, 2: cuBLAS

  ~Model() {
    for (cudaEvent_t e : {ev_fork, ev_layer[0], ev_layer[1]}) if (e) cudaEventDestroy(e);
    if (streams.side) give_back(streams);
  }

  b16* p(int l, int which) const { return d.p + off[4 + l * PER_LAYER + which]; }
  b16* g(int l, int which) const { return d.g + off[4 + l * PER_LAYER + which]; }
};

#define TRY(expr)                                                                             \
  do {                                                                                        \
    const int rc_ = (expr);                                                                   \
    if (rc_ != 0) { g_error = std::string(#expr) + " failed (code " + std::to_string(rc_) + ")"; return rc_; } \
    m.launches++;                                                                             \
  } while (0)

// hands out 256-byte aligned pieces of the arena; with base = null it only adds up
struct Carve {
  char* base; size_t used = 0;
  template <typename T> T* get(size_t n) {
    T* r = reinterpret_cast<T*>(base + used);
    used += (n * sizeof(T) + 255) / 256 * 256;
    return base ? r : nullptr;
  }
};

struct Layer { b16 *ln1, *qkv, *att, *x2, *ln2, *h, *gl, *x3; float *mean1, *rstd1, *mean2, *rstd2; };
struct Buffers {
  b16 *x0, *a, *pr, *logits, *dln, *dln2, *datt, *dln1;
  b16 *dxa[3], *dxb[2], *dg[2], *dqkv[2];      // taken in turn by the layers: weight gradients may still read those of the layer above
  float *loss_rows, *parts[2], *row_sums;
  std::vector<Layer> layer;         // L + 1: the last one holds the input of the head
};

// row_floats: scratch of the attention kernels, 0 where attention is ATen's
void carve(Carve& c, const Desc& d, size_t T, bool train, size_t part_floats, size_t row_floats, Buffers& b) {
  const size_t C = d.C;
  b.x0 = c.get<b16>(T * C); b.a = c.get<b16>(T * C); b.pr = c.get<b16>(T * C);
  b.layer.resize(d.L + 1);
  for (int l = 0; l <= d.L; l++) {
    Layer& y = b.layer[l];
    if (!train && l >= 2) { y = b.layer[l - 2]; continue; }      // nothing is kept for a backward pass: two sets take turns
    y.ln1 = c.get<b16>(T * C); y.mean1 = c.get<float>(T); y.rstd1 = c.get<float>(T);
    if (train && l == d.L) continue;
    y.qkv = c.get<b16>(T * 3 * C); y.x2 = c.get<b16>(T * C); y.ln2 = c.get<b16>(T * C); y.mean2 = c.get<float>(T); y.rstd2 = c.get<float>(T);
    y.att = row_floats && !train ? c.get<b16>(T * C) : nullptr;
    y.h = train ? c.get<b16>(T * 4 * C) : nullptr; y.gl = c.get<b16>(T * 4 * C); y.x3 = c.get<b16>(T * C);
  }
  b.logits = c.get<b16>(T * d.Vp); b.loss_rows = c.get<float>(T);
  if (!train) return;
  for (b16*& x : b.dxa) x = c.get<b16>(T * C);
  for (int q = 0; q < 2; q++) { b.dxb[q] = c.get<b16>(T * C); b.dg[q] = c.get<b16>(T * 4 * C); b.dqkv[q] = c.get<b16>(T * 3 * C); }
  b.row_sums = c.get<float>(row_floats);
  b.dln = c.get<b16>(T * C); b.dln2 = c.get<b16>(T * C); b.datt = c.get<b16>(T * C); b.dln1 = c.get<b16>(T * C); for (float*& x : b.parts) x = c.get<float>(part_floats);
}

at::Tensor view(b16* p, at::IntArrayRef sizes, at::IntArrayRef strides = {}) {
  static thread_local int dev = -1;
  dev = at::cuda::current_device();
  const auto opt = at::TensorOptions().dtype(at::kBFloat16).device(at::kCUDA, dev);
  return strides.empty() ? at::from_blob(p, sizes, opt) : at::from_blob(p, sizes, strides, [](void*) {}, opt);
}

// C[M, N] = A op B, bf16 row-major: layout NT A [M,K] B [N,K], NN A [M,K] B [K,N], TN A [K,M] B [K,N]
// Plain products of more than some GFLOP go to cuBLAS unless the "tcgen05" backend is asked for: it has more tile shapes to fit ragged sizes
// to the chip (GPT-2 medium step 23.5 ms with it, 24.7 without; 8 layers of 768 columns on 3 x 777 tokens 2.97 / 3.10 ms).  Below, the launch counts: issued call by call this framework's kernel costs a third of
// the host time (2 layers of 256 columns 342 us, 500 with cuBLAS); replayed from a graph it does not, and the line lies lower (the same
// step 236 us at 2 GFLOP, 217 at 0.1; 12 layers of 512 columns on 4 x 512 tokens 1985 us, 1857).  So a product between the two lines runs on one back end issued and on the other replayed: the sums are the same up to
// their order.
constexpr double kOwnProductFlops = 2e9, kOwnProductFlopsReplayed = 1e8;
int product(Model& m, int layout, b16* A, b16* B, b16* C, const b16* bias, int M, int N, int K, void* s, int which_ws = 0) {
  if (m.backend == 2 || (m.backend == 0 && 2.0 * M * N * K > (m.captured ? kOwnProductFlopsReplayed : kOwnProductFlops))) {
    at::Tensor out = view(C, {M, N});
    at::Tensor a = layout == TN ? view(A, {K, M}).t() : view(A, {M, K}), b = layout == NT ? view(B, {N, K}).t() : view(B, {K, N});
    if (bias) at::addmm_out(out, view(const_cast<b16*>(bias), {N}), a, b); else at::mm_out(out, a, b);
    m.cublas++;
    return 0;
  }
  TRY(piccl_ops_gemm(layout, EPI_BIAS, A, B, C, nullptr, bias, nullptr, nullptr, m.ws[which_ws], kSplitBytes, M, N, K, s));
  m.tcgen05++;
  return 0;
}
#define DO(expr) do { const int rc_ = (expr); if (rc_ != 0) return rc_; } while (0)

// What scaled_dot_product_attention would pick for q, k, v within packed rows.
int64_t sdp_choice(b16* qkv, int B, int S, int H, int D) {
  const int64_t C = (int64_t)H * D, sizes[4] = {B, H, S, D}, strides[4] = {(int64_t)S * 3 * C, D, 3 * C, 1};
  return at::_fused_sdp_choice(view(qkv, sizes, strides), view(qkv + C, sizes, strides), view(qkv + 2 * C, sizes, strides), {}, 0.0, true);
}
constexpr int64_t kCudnnAttention = 3;       // sdp::SDPBackend::cudnn_attention

// Causal attention of qkv [B * S, 3 C]; the [B, S, H, D] output is contiguous.
at::Tensor attention(Saved& sv, b16* qkv, int B, int S, int H, int D, bool train) {
  const int64_t C = (int64_t)H * D, sizes[4] = {B, H, S, D}, strides[4] = {(int64_t)S * 3 * C, D, 3 * C, 1};
  sv.q = view(qkv, sizes, strides); sv.k = view(qkv + C, sizes, strides); sv.v = view(qkv + 2 * C, sizes, strides);
  // the kernel that scaled_dot_product_attention would pick: cuDNN's is called without autograd, any other through it
  sv.direct = at::_fused_sdp_choice(sv.q, sv.k, sv.v, {}, 0.0, true) == kCudnnAttention;
  if (sv.direct) {
    auto r = at::_scaled_dot_product_cudnn_attention(sv.q, sv.k, sv.v, {}, train, 0.0, true, false);
    sv.out = std::get<0>(r); sv.lse = std::get<1>(r); sv.cq = std::get<2>(r); sv.ck = std::get<3>(r); sv.mq = std::get<4>(r); sv.mk = std::get<5>(r);
    sv.seed = std::get<6>(r); sv.offset = std::get<7>(r);
    return sv.out.transpose(1, 2).contiguous();
  }
  c10::AutoGradMode grad(train);
  if (train) { sv.q.requires_grad_(true); sv.k.requires_grad_(true); sv.v.requires_grad_(true); }
  sv.out = at::scaled_dot_product_attention(sv.q, sv.k, sv.v, {}, 0.0, true);
  return sv.out.detach().transpose(1, 2).contiguous();
}

void attention_grad(const Saved& sv, b16* dout, int B, int S, int H, int D, at::Tensor (&d)[3]) {
  const at::Tensor go = view(dout, {B, S, H, D}).transpose(1, 2);
  if (sv.direct) {
    auto r = at::_scaled_dot_product_cudnn_attention_backward_symint(go, sv.q, sv.k, sv.v, sv.out, sv.lse, sv.seed, sv.offset, at::Tensor(), sv.cq, sv.ck, sv.mq, sv.mk, 0.0, true);
    d[0] = std::get<0>(r); d[1] = std::get<1>(r); d[2] = std::get<2>(r);
  } else {
    auto r = torch::autograd::grad({sv.out}, {sv.q, sv.k, sv.v}, {go});
    for (int i = 0; i < 3; i++) d[i] = r[i];
  }
  for (auto& t : d) if (t.stride(3) != 1) t = t.contiguous();
}

bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(s, &st) == cudaSuccess && st != cudaStreamCaptureStatusNone;
}

int run(Model& m, const long long* idx, const long long* tgt, int B, int S, float* loss, bool train, ReadyFn ready) {
  const Desc& d = m.d;
  const int T = B * S, C = d.C, L = d.L, H = d.H, D = C / H;
  const cudaStream_t main_stream = at::cuda::getCurrentCUDAStream().stream();
  void* s = main_stream;
  c10::NoGradGuard no_grad;
  const auto opt = at::TensorOptions().device(at::kCUDA, at::cuda::current_device());

  // partial rows of the column sums: dgamma, dbeta and bias gradient of both LayerNorms, the MLP's and the attention's bias gradients
  const int n_ln = piccl_ops_ln_bwd_parts(T, C), n_qkv = piccl_ops_col_parts(T, 3 * C), n_fc_own = (T + 31) / 32, n_fc_sep = piccl_ops_col_parts(T, 4 * C);
  // Heads of 64 columns: this framework's kernels, where they are the faster ones and PyTorch would take cuDNN's (a program that asks for another back end gets that one; any
  // address will do for the question).  A training step keeps cuDNN's forward kernel, whose sums of exponentials the way back takes as they are: the two forward kernels are equally
  // exact and fast (2.0e-3 off fp64; 8 x 1024 tokens 40 us, own 41), but another order of its sums rolls the rounding of every activation above it anew, and gradients
  // of one step then differ by 0.95 % from those that this model has had, with the own way back alone by 0.48 % (8 layers of 768 columns).
  const bool own_attention = D == 64 && piccl_ops_attn_pays(train, B, S, H, at::cuda::getCurrentDeviceProperties()->multiProcessorCount) && sdp_choice(d.p, B, S, H, D) == kCudnnAttention;
  const int n_att = own_attention ? piccl_ops_attn_parts(B, S) : 0;
  const size_t row = (size_t)n_ln * C, fc_floats = (size_t)std::max(n_fc_own, n_fc_sep) * 4 * C, part_floats = 6 * row + fc_floats + (size_t)std::max(n_qkv, n_att) * 3 * C;
  const size_t row_floats = own_attention ? (size_t)2 * B * H * piccl_ops_attn_rows(S) : 0;
  Buffers b;
  Carve count{nullptr};
  carve(count, d, T, train, part_floats, row_floats, b);
  if (!m.arena.defined() || (size_t)m.arena.numel() < count.used) {
    if (m.in_callers_graph) m.kept.push_back(m.arena);
    m.in_callers_graph = false;
    m.arena = at::Tensor(); m.arena = at::empty({(int64_t)count.used}, opt.dtype(at::kByte));
  }
  // (captures of the model's own steps come with m.captured; models/gpt2.py drops those graphs when the arena moves)
  const bool in_capture = capturing(main_stream);
  m.in_callers_graph |= !m.captured && in_capture;
  Carve c{static_cast<char*>(m.arena.data_ptr())};
  carve(c, d, T, train, part_floats, row_floats, b);
  b16 *const lnf_g = d.p + m.off[0], *const lnf_b = d.p + m.off[1], *const wpe = d.p + m.off[2], *const wte = d.p + m.off[3];
  if (!m.split.defined()) {
    m.split = at::empty({2, (int64_t)kSplitBytes}, opt.dtype(at::kByte));
    for (int q = 0; q < 2; q++) m.ws[q] = m.split.select(0, q).data_ptr();
    if (!take_streams(m.streams)) { g_error = "cudaStreamCreate failed"; return -1001; }
    for (cudaEvent_t* e : {&m.ev_fork, &m.ev_layer[0], &m.ev_layer[1]}) if (cudaEventCreateWithFlags(e, cudaEventDisableTiming) != cudaSuccess) { g_error = "cudaEventCreate failed"; return -1001; }
  }
  if (!m.split_zero) {                // in a capture the zeros come with every replay, and the next call writes them again
    m.split.narrow(1, 0, 64 << 10).zero_();
    m.split_zero = !in_capture;
  }
  if ((int)m.saved.size() < L) m.saved.resize(L);

  // ---------------- forward
  TRY(piccl_ops_embed_fwd(idx, wte, wpe, b.x0, T, S, C, s));
  TRY(piccl_ops_ln_fwd(b.x0, nullptr, m.p(0, LN1_G), m.p(0, LN1_B), nullptr, b.layer[0].ln1, b.layer[0].mean1, b.layer[0].rstd1, T, C, d.eps, s));
  const b16* xin = b.x0;
  std::vector<at::Tensor> att(L);
  for (int l = 0; l < L; l++) {
    Layer& y = b.layer[l]; Layer& z = b.layer[l + 1];
    DO(product(m, NT, y.ln1, m.p(l, W_QKV), y.qkv, m.p(l, B_QKV), T, 3 * C, C, s));
    if (own_attention && !train) TRY(piccl_ops_attn_fwd(y.qkv, y.att, nullptr, B, S, H, s));
    else { att[l] = attention(m.saved[l], y.qkv, B, S, H, D, train); y.att = static_cast<b16*>(att[l].data_ptr()); }
    DO(product(m, NT, y.att, m.p(l, W_O), b.a, m.p(l, B_O), T, C, C, s));
    if (!train) { m.saved[l] = Saved(); att[l] = at::Tensor(); }
    TRY(piccl_ops_ln_fwd(b.a, xin, m.p(l, LN2_G), m.p(l, LN2_B), y.x2, y.ln2, y.mean2, y.rstd2, T, C, d.eps, s));
    if (m.backend == 2) {
      b16* h = y.h ? y.h : y.gl;
      DO(product(m, NT, y.ln2, m.p(l, W_FC), h, nullptr, T, 4 * C, C, s));
      TRY(piccl_ops_bias_gelu_fwd(h, m.p(l, B_FC), y.h, y.gl, T, 4 * C, s));
    } else {
      TRY(piccl_ops_gemm(NT, EPI_GELU, y.ln2, m.p(l, W_FC), y.gl, y.h, m.p(l, B_FC), nullptr, nullptr, nullptr, 0, T, 4 * C, C, s));
      m.tcgen05++;
    }
    DO(product(m, NT, y.gl, m.p(l, W_PROJ), b.pr, m.p(l, B_PROJ), T, C, 4 * C, s));
    const bool last = l + 1 == L;
    TRY(piccl_ops_ln_fwd(b.pr, y.x2, last ? lnf_g : m.p(l + 1, LN1_G), last ? lnf_b : m.p(l + 1, LN1_B), y.x3, z.ln1, z.mean1, z.rstd1, T, C, d.eps, s));
    xin = y.x3;
  }
  Layer& f = b.layer[L];
  DO(product(m, NT, f.ln1, wte, b.logits, nullptr, T, d.Vp, C, s));
  TRY(piccl_ops_ce(b.logits, tgt, b.loss_rows, T, d.V, d.Vp, 1.0f / (float)T, train, s));
  // The loss comes last, since it also tells whether a kernel of the pass gave up on a wait: its products or gradients are left over from another layer or step then.
  if (!train) { TRY(piccl_ops_pass_loss(b.loss_rows, loss, T, s)); return 0; }

  // ---------------- backward (logits now hold d loss / d logits)
  b16 *const g_lnf_g = d.g + m.off[0], *const g_lnf_b = d.g + m.off[1], *const g_wpe = d.g + m.off[2], *const g_wte = d.g + m.off[3];
  // Captured, the weight gradients and column sums of small models run beside the chain of input gradients.  Above 4 Mi elements of the
  // residual stream a product fills the chip by itself, and a block of another kernel on one SM costs it a wave (8192 x 1024: 22.5 ms with
  // weight gradients on the second stream, 23.3 with the column sums there as well, 22.4 with neither; 4096 x 768: 5.13 ms and 5.26).
  const bool fork = m.captured && (long)T * C <= (4 << 20);
  auto to_side = [&] {                // what comes next on the second stream sees all that the main one has done
    cudaEventRecord(m.ev_fork, main_stream);
    cudaStreamWaitEvent(m.streams.side, m.ev_fork, 0);
  };
  auto finish = [&](const piccl_finish_job* jobs, int n, int q) -> int {
    if (!fork) { TRY(piccl_ops_finish_parts(jobs, n, s)); return 0; }
    to_side();
    TRY(piccl_ops_finish_parts(jobs, n, m.streams.side));
    cudaEventRecord(m.ev_layer[q], m.streams.side);
    return 0;
  };
  auto done = [&](const b16* last_of, size_t n) { if (ready) ready((long long)(last_of - d.g) + (long long)n); };
  // G[M, N] = A[T, M]^T B[T, N], on the second stream once the main one has come this far
  auto weight_grad = [&](b16* A, b16* B, b16* G, int M, int N) -> int {
    if (!fork) return product(m, TN, A, B, G, nullptr, M, N, T, s);
    to_side();
    c10::cuda::CUDAStreamGuard guard(c10::cuda::getStreamFromExternal(m.streams.side, m.streams.device));
    return product(m, TN, A, B, G, nullptr, M, N, T, m.streams.side, 1);
  };
  DO(weight_grad(b.logits, f.ln1, g_wte, d.Vp, C));
  DO(product(m, NN, b.logits, wte, b.dln, nullptr, T, C, d.Vp, s));
  b16* dx = b.dxa[L % 3];             // gradient of the residual stream above the layer at hand
  {
    float* const ws1 = b.parts[L & 1] + 3 * row;
    TRY(piccl_ops_ln_bwd(b.dln, xin, lnf_g, f.mean1, f.rstd1, nullptr, dx, ws1, 1, T, C, s));
    const piccl_finish_job jobs[3] = {{ws1, g_lnf_g, n_ln, C, 0, 0}, {ws1 + row, g_lnf_b, n_ln, C, 0, 0}, {ws1 + 2 * row, m.g(L - 1, B_PROJ), n_ln, C, 0, 0}};
    DO(finish(jobs, 3, L & 1));
  }
  done(g_lnf_b, C);
  for (int l = L - 1; l >= 0; l--) {
    Layer& y = b.layer[l];
    const int q = l & 1;
    b16 *const dg = b.dg[q], *const dxb = b.dxb[q], *const dqkv = b.dqkv[q], *const dx_below = b.dxa[l % 3];
    float *const ws2 = b.parts[q], *const ws1 = ws2 + 3 * row, *const ws_fc = ws1 + 3 * row, *const ws_qkv = ws_fc + fc_floats;
    if (fork && l + 2 <= L) cudaStreamWaitEvent(main_stream, m.ev_layer[q], 0);      // layer l + 2 is done with the buffers that this one writes
    // x3 = x2 + gelu(ln2 Wfc + bfc) Wproj + bproj
    DO(weight_grad(dx, y.gl, m.g(l, W_PROJ), C, 4 * C));
    int n_fc = n_fc_own;
    if (m.backend == 2) {
      n_fc = n_fc_sep;
      DO(product(m, NN, dx, m.p(l, W_PROJ), dg, nullptr, T, 4 * C, C, s));
      TRY(piccl_ops_gelu_bwd(dg, y.h, dg, ws_fc, T, 4 * C, s));
    } else {
      TRY(piccl_ops_gemm(NN, EPI_GELU_GRAD, dx, m.p(l, W_PROJ), dg, nullptr, nullptr, y.h, ws_fc, nullptr, 0, T, 4 * C, C, s));
      m.tcgen05++;
    }
    DO(weight_grad(dg, y.ln2, m.g(l, W_FC), 4 * C, C));
    DO(product(m, NN, dg, m.p(l, W_FC), b.dln2, nullptr, T, C, 4 * C, s));
    TRY(piccl_ops_ln_bwd(b.dln2, y.x2, m.p(l, LN2_G), y.mean2, y.rstd2, dx, dxb, ws2, 1, T, C, s));
    // x2 = xin + attention Wo + bo
    DO(weight_grad(dxb, y.att, m.g(l, W_O), C, C));
    DO(product(m, NN, dxb, m.p(l, W_O), b.datt, nullptr, T, C, C, s));
    int n_q = n_qkv;
    if (own_attention && m.saved[l].direct) {
      n_q = n_att;
      const at::Tensor lse = m.saved[l].lse.contiguous();      // [B, H, S]
      TRY(piccl_ops_attn_bwd(y.qkv, y.att, b.datt, lse.data_ptr<float>(), b.row_sums, dqkv, ws_qkv, B, S, H, s));
      m.launches++;                   // two kernels
    } else {
      at::Tensor dq[3];
      attention_grad(m.saved[l], b.datt, B, S, H, D, dq);
      const void* ptr[3]; long long st[9];
      for (int i = 0; i < 3; i++) { ptr[i] = dq[i].data_ptr(); for (int j = 0; j < 3; j++) st[3 * i + j] = dq[i].stride(j); }
      bool words = D % 8 == 0;          // rows of a head are whole 16-byte words
      for (int i = 0; i < 3; i++) words &= (reinterpret_cast<uintptr_t>(ptr[i]) % 16 | (st[3 * i] | st[3 * i + 1] | st[3 * i + 2]) % 8) == 0;
      if (words) TRY(piccl_ops_qkv_grad(ptr, st, dqkv, ws_qkv, B, S, H, D, s));
      else {                            // heads of 4 columns, say: packed by ATen, the column sums from the packed rows
        const at::Tensor packed = view(dqkv, {B, S, 3, H, D});
        for (int i = 0; i < 3; i++) packed.select(2, i).copy_(dq[i].transpose(1, 2));
        const int per = (T + n_qkv - 1) / n_qkv;
        n_q = (T + per - 1) / per;
        TRY(piccl_ops_colsum(dqkv, nullptr, ws_qkv, T, 3 * C, per, 0, s));
      }
    }
    DO(weight_grad(dqkv, y.ln1, m.g(l, W_QKV), 3 * C, C));
    DO(product(m, NN, dqkv, m.p(l, W_QKV), b.dln1, nullptr, T, C, 3 * C, s));
    TRY(piccl_ops_ln_bwd(b.dln1, l ? b.layer[l - 1].x3 : b.x0, m.p(l, LN1_G), y.mean1, y.rstd1, dxb, dx_below, ws1, l > 0, T, C, s));
    const piccl_finish_job jobs[8] = {{ws2, m.g(l, LN2_G), n_ln, C, 0, 0}, {ws2 + row, m.g(l, LN2_B), n_ln, C, 0, 0}, {ws2 + 2 * row, m.g(l, B_O), n_ln, C, 0, 0},
                                      {ws_fc, m.g(l, B_FC), n_fc, 4 * C, 0, 0}, {ws_qkv, m.g(l, B_QKV), n_q, 3 * C, 0, 0}, {ws1, m.g(l, LN1_G), n_ln, C, 0, 0},
                                      {ws1 + row, m.g(l, LN1_B), n_ln, C, 0, 0}, {ws1 + 2 * row, l ? m.g(l - 1, B_PROJ) : nullptr, n_ln, C, 0, 0}};
    DO(finish(jobs, l ? 8 : 7, q));
    dx = dx_below;
    done(m.g(l, B_PROJ), C);
    m.saved[l] = Saved();
    if (!fork) att[l] = at::Tensor();  // the second stream may still read it
  }
  TRY(piccl_ops_wpe_bwd(dx, g_wpe, B, S, d.seq_len, C, 0, s));
  done(g_wpe, (size_t)d.seq_len * C);
  if (!m.stage.defined()) { m.stage = at::empty({d.Vp, C}, opt.dtype(at::kFloat)); m.owner = at::empty({d.Vp}, opt.dtype(at::kInt)); }
  if (!m.stage_zero) {
    m.stage.zero_();
    m.stage_zero = !in_capture;
  }
  if (fork) {
    cudaEventRecord(m.ev_fork, m.streams.side);
    cudaStreamWaitEvent(main_stream, m.ev_fork, 0);
  }
  TRY(piccl_ops_wte_bwd_rows(idx, dx, m.stage.data_ptr<float>(), m.owner.data_ptr<int>(), g_wte, T, C, s));
  m.launches++;                       // two kernels
  done(g_wte, (size_t)d.Vp * C);
  TRY(piccl_ops_pass_loss(b.loss_rows, loss, T, s));
  return 0;
}

}  // namespace

extern "C" {

void* piccl_gpt2_create(const void* desc) {
  Model* m = new Model();
  memcpy(&m->d, desc, sizeof(Desc));
  m->off.assign(m->d.off, m->d.off + 4 + m->d.L * PER_LAYER);
  return m;
}
void piccl_gpt2_destroy(void* h) { delete static_cast<Model*>(h); }

// idx / tgt: int64 [B * S] on the device; loss: one float on the device; captured: the call is captured into a graph.  counts[4] (optional): launches of this framework's kernels,
// products on tcgen05, products on cuBLAS since the last call.  0, or an error code whose text piccl_gpt2_error() holds.
int piccl_gpt2_run(void* h, const long long* idx, const long long* tgt, int B, int S, float* loss, int train, int backend, int captured, ReadyFn ready, long long* counts) {
  Model& m = *static_cast<Model*>(h);
  m.launches = m.cublas = m.tcgen05 = 0;
  m.backend = backend;
  m.captured = captured != 0;
  int rc;
  try { rc = run(m, idx, tgt, B, S, loss, train != 0, ready); }
  catch (const std::exception& e) { g_error = e.what(); rc = -1000; }
  if (counts) { counts[0] = m.launches; counts[1] = m.tcgen05; counts[2] = m.cublas; }
  return rc;
}
// The stream on which a step is captured (nullptr before the first step).
void* piccl_gpt2_capture_stream(void* h) { return static_cast<Model*>(h)->streams.main; }
// Where the activations are: a graph captured earlier is of no use once this has changed.
const void* piccl_gpt2_arena(void* h) { const Model& m = *static_cast<Model*>(h); return m.arena.defined() ? m.arena.data_ptr() : nullptr; }
const char* piccl_gpt2_error(void) { return g_error.c_str(); }

}  // extern "C"
