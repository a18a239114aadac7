// extern "C" surface of libflashoptim_b200.so: argument checking, building the kernel
// parameter tables, launching.  No allocation, no synchronisation, caller's stream only.
#include <cstdarg>
#include <cstdio>
#include <cstring>

#include "fo_step.cuh"

namespace fo {

static thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

// the kernel with the asked features: one of its own for one feature, else the one that carries them all
static Launcher find_launcher(int opt, int pdt, int ecc_bits, int state, bool generic, int mode, int group_size, int gdt) {
#define FO_PICK(stem)                                                    \
  switch (mode) {                                                        \
    case kPlain: return stem##_plain(pdt, ecc_bits, gdt);                     \
    case kClip: return stem##_clip(pdt, ecc_bits, gdt);                       \
    case kOut: return stem##_out(pdt, ecc_bits, gdt);                         \
    case kPeer: return stem##_peer(pdt, ecc_bits, gdt);                       \
    default: return stem##_all(pdt, ecc_bits, gdt);                           \
  }
  if (opt == FO_OPT_ADAM) {
    if (generic) return lookup_adam_generic(pdt, ecc_bits, gdt);
    if (mode == kGroup) return group_size < 16 ? lookup_adam_quant_group8(pdt, ecc_bits, gdt) : lookup_adam_quant_group(pdt, ecc_bits, gdt);
    if (mode == kDelta) return state == FO_STATE_QUANT ? lookup_adam_quant_delta(pdt, ecc_bits, gdt) : lookup_adam_full_delta(pdt, ecc_bits, gdt);
    if (state == FO_STATE_QUANT) { FO_PICK(lookup_adam_quant) }
    if (state == FO_STATE_FULL) { FO_PICK(lookup_adam_full) }
  } else if (opt == FO_OPT_LION) {
    if (generic) return lookup_lion_generic(pdt, ecc_bits, gdt);
    if (mode == kGroup) return group_size < 16 ? lookup_lion_quant_group8(pdt, ecc_bits, gdt) : lookup_lion_quant_group(pdt, ecc_bits, gdt);
    if (state == FO_STATE_QUANT) { FO_PICK(lookup_lion_quant) }
    if (state == FO_STATE_FULL) { FO_PICK(lookup_lion_full) }
  } else if (opt == FO_OPT_SGD) {
    if (generic) return lookup_sgd_generic(pdt, ecc_bits, gdt);
    if (mode == kGroup) return group_size < 16 ? lookup_sgd_quant_group8(pdt, ecc_bits, gdt) : lookup_sgd_quant_group(pdt, ecc_bits, gdt);
    if (state == FO_STATE_QUANT) { FO_PICK(lookup_sgd_quant) }
    if (state == FO_STATE_FULL) { FO_PICK(lookup_sgd_full) }
    if (state == FO_STATE_NONE) { FO_PICK(lookup_sgd_none) }
  }
#undef FO_PICK
  return Launcher{nullptr, 0u, 0, false};
}
static PieceFn find_pieces(int opt, int pdt, int ecc_bits, int state) {
  if (opt == FO_OPT_ADAM) return state == FO_STATE_QUANT ? lookup_adam_quant_piece(pdt, ecc_bits) : lookup_adam_full_piece(pdt, ecc_bits);
  if (opt == FO_OPT_LION) return state == FO_STATE_QUANT ? lookup_lion_quant_piece(pdt, ecc_bits) : lookup_lion_full_piece(pdt, ecc_bits);
  if (state == FO_STATE_NONE) return lookup_sgd_none_piece(pdt, ecc_bits);
  return state == FO_STATE_QUANT ? lookup_sgd_quant_piece(pdt, ecc_bits) : lookup_sgd_full_piece(pdt, ecc_bits);
}

// Up to this many elements in whole chunks a call goes through piece_kernel alone: its blocks of 1024
// elements spread a small problem over all SMs in one launch, where step_kernel has one block of 4096 to 6144
// elements on few of them and leaves the ragged ends to a second launch.
#ifndef FO_SMALL_ELEMS
#define FO_SMALL_ELEMS (148ull * 8192ull)
#endif
// The same where tile_kernel takes over, whose warps spread tiles of 512 elements.  In us with pieces and with tiles, whole steps in a graph, at 606720
// elements: AdamW 24-bit masters 7.4 / 6.2, 32-bit 7.5 / 6.1, fp32 7.2 / 5.7, groups of 128 7.6 / 6.1, Lion 24-bit 5.1 / 4.8, fp32 5.1 / 4.5, SGDW 24-bit 5.1 / 4.7, fp32
// 5.1 / 4.3, groups of 256 5.2 / 4.8; with a ragged end (620100) AdamW 8.0 / 7.0, Lion 5.4 / 5.5, SGDW 5.4 / 5.5.  At 2^19 pieces lead under AdamW (4.5 / 4.7,
// the kernels alone).
constexpr unsigned long long kSmallElemsTiles = 148ull * 4096ull;

static DevHyper make_dev_hyper(const FoHyper& h, int opt) {
  DevHyper d;
  memset(&d, 0, sizeof(d));
  d.lr = h.lr; d.wd = h.wd; d.b1 = h.b1; d.b2 = h.b2;
  d.omb1 = h.one_minus_b1; d.omb2 = h.one_minus_b2;
  d.eps = h.eps; d.bc1 = h.bc1; d.bc2 = h.bc2;
  // single IEEE fp32 operations, as the reference forms them (adamw.py:103-105)
  volatile float prod = h.lr * h.wd;
  d.decay = 1.0f - prod;
  d.flags = h.flags & (FO_FLAG_DECOUPLED_WD | FO_FLAG_NESTEROV | FO_FLAG_LION_LERP | FO_FLAG_LP_DELTA | FO_FLAG_SCALE_FLOOR);
  if (opt == FO_OPT_ADAM) {
    d.lr_bc1 = h.lr / h.bc1;
    d.sqrt_bc2 = sqrtf(h.bc2);
    d.rcp_sqrt_bc2 = 1.0f / d.sqrt_bc2;
    if (adam_is_tame(h.eps, d.sqrt_bc2)) d.flags |= kFlagTameAdam;
    d.least = adam_least_new(h.eps);
  }
  d.dyn = h.dev_scalars;
  return d;
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// SM count of the device that is current on the calling thread (cached per device ordinal; atomics,
// so that concurrent first calls from several threads are well defined: they store the same number)
static int sm_count_of_current_device() {
  static std::atomic<int> cache[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -1;
  if (dev >= 0 && dev < 64) {
    const int known = cache[dev].load(std::memory_order_acquire);
    if (known > 0) return known;
  }
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
  if (dev >= 0 && dev < 64) cache[dev].store(sms, std::memory_order_release);
  return sms;
}

}  // namespace fo

using namespace fo;

extern "C" int fo_step(const FoStepDesc* d, void* cuda_stream) { return fo_step_ex(d, nullptr, cuda_stream); }

extern "C" int fo_step_ex(const FoStepDesc* d, const FoStepMore* more, void* cuda_stream) {
  if (d == nullptr) return fail(FO_ERR_INVALID_ARG, "fo_step: null descriptor");
  if (d->struct_size != sizeof(FoStepDesc))
    return fail(FO_ERR_INVALID_ARG, "fo_step: struct_size %u != %zu (ABI mismatch)", d->struct_size, sizeof(FoStepDesc));
  if (more != nullptr && more->struct_size != sizeof(FoStepMore))
    return fail(FO_ERR_INVALID_ARG, "fo_step_ex: struct_size %u != %zu (ABI mismatch)", more->struct_size, sizeof(FoStepMore));
  const FoLeafOut* const outs = more != nullptr ? more->outs : nullptr;
  if (d->opt < FO_OPT_ADAM || d->opt > FO_OPT_SGD) return fail(FO_ERR_INVALID_ARG, "fo_step: bad opt %d", d->opt);
  if (d->param_dtype < FO_F32 || d->param_dtype > FO_F16) return fail(FO_ERR_INVALID_ARG, "fo_step: bad param_dtype %d", d->param_dtype);
  if (d->grad_dtype < FO_F32 || d->grad_dtype > FO_F16) return fail(FO_ERR_INVALID_ARG, "fo_step: bad grad_dtype %d", d->grad_dtype);
  if (d->ecc_bits != 0 && d->ecc_bits != 8 && d->ecc_bits != 16) return fail(FO_ERR_INVALID_ARG, "fo_step: ecc_bits must be 0, 8 or 16, got %d", d->ecc_bits);
  if (d->param_dtype == FO_F32 && d->ecc_bits != 0) return fail(FO_ERR_INVALID_ARG, "fo_step: fp32 params carry no ECC");
  if (d->state < FO_STATE_QUANT || d->state > FO_STATE_NONE) return fail(FO_ERR_INVALID_ARG, "fo_step: bad state %d", d->state);
  if (d->state == FO_STATE_NONE && d->opt != FO_OPT_SGD) return fail(FO_ERR_INVALID_ARG, "fo_step: only SGD can run without a momentum buffer");
  if (d->n_leaves == 0) return FO_OK;
  if (d->leaves == nullptr || d->hypers == nullptr) return fail(FO_ERR_INVALID_ARG, "fo_step: null table");
  if (d->n_hypers == 0) return fail(FO_ERR_INVALID_ARG, "fo_step: no hyper-parameter set");
  if (d->n_hypers > FO_MAX_HYPERS) return fail(FO_ERR_TOO_LARGE, "fo_step: %u hyper sets, at most %d per call", d->n_hypers, FO_MAX_HYPERS);
  bool generic = false;
  int group_shift = 5;
  if (d->state == FO_STATE_QUANT) {
    if (d->group_size < 1) return fail(FO_ERR_INVALID_ARG, "fo_step: group_size %d", d->group_size);
    if (d->group_size > kGenericTile) return fail(FO_ERR_UNSUPPORTED, "fo_step: group_size %d > %d", d->group_size, kGenericTile);
    // a group is 1 to 32 lanes of 8 elements for 8, 16, ..., 256; other sizes run a kernel of their own
    generic = d->group_size < 8 || d->group_size > 256 || (d->group_size & (d->group_size - 1)) != 0;
    for (group_shift = 0; (2 << group_shift) <= d->group_size; ++group_shift) {}
  }
  if (d->n_peers > (uint32_t)kMaxPeers) return fail(FO_ERR_TOO_LARGE, "fo_step: %u peers, at most %d", d->n_peers, kMaxPeers);
  if (d->n_peers > 0 && d->peer_param_offsets == nullptr && d->peer_grad_offsets == nullptr)
    return fail(FO_ERR_INVALID_ARG, "fo_step: n_peers without peer_param_offsets or peer_grad_offsets");
  if (d->n_peers > 0 && d->state == FO_STATE_QUANT && d->group_size != 32) return fail(FO_ERR_UNSUPPORTED, "fo_step: peer replicas need group_size 32");
  if (find_launcher(d->opt, d->param_dtype, d->ecc_bits, d->state, generic, kPlain, 32, d->grad_dtype).launch == nullptr)
    return fail(FO_ERR_UNSUPPORTED, "fo_step: no kernel for this combination");

  const bool need_mu = d->state != FO_STATE_NONE;
  const bool need_nu = need_mu && d->opt == FO_OPT_ADAM;
  const bool need_scales = d->state == FO_STATE_QUANT;
  for (uint32_t i = 0; i < d->n_leaves; ++i) {
    const FoLeaf& L = d->leaves[i];
    if (L.n == 0) continue;
    if (L.grad == nullptr || L.param == nullptr) return fail(FO_ERR_INVALID_ARG, "fo_step: leaf %u: null grad/param", i);
    if (d->ecc_bits != 0 && L.ecc == nullptr) return fail(FO_ERR_INVALID_ARG, "fo_step: leaf %u: null ecc", i);
    if (need_mu && L.mu == nullptr) return fail(FO_ERR_INVALID_ARG, "fo_step: leaf %u: null mu", i);
    if (need_nu && L.nu == nullptr) return fail(FO_ERR_INVALID_ARG, "fo_step: leaf %u: null nu", i);
    if (need_scales && L.mu_scales == nullptr) return fail(FO_ERR_INVALID_ARG, "fo_step: leaf %u: null mu_scales", i);
    if (need_scales && need_nu && L.nu_scales == nullptr) return fail(FO_ERR_INVALID_ARG, "fo_step: leaf %u: null nu_scales", i);
    if (outs != nullptr) {
      const FoLeafOut& O = outs[i];
      if (O.param == nullptr || (d->ecc_bits != 0 && O.ecc == nullptr) || (need_mu && O.mu == nullptr) || (need_nu && O.nu == nullptr) ||
          (need_scales && O.mu_scales == nullptr) || (need_scales && need_nu && O.nu_scales == nullptr))
        return fail(FO_ERR_INVALID_ARG, "fo_step: leaf %u: null output", i);
    }
    if (L.hyper >= d->n_hypers) return fail(FO_ERR_INVALID_ARG, "fo_step: leaf %u: hyper index %u out of range", i, L.hyper);
  }

  if (outs != nullptr && d->n_peers > 0) return fail(FO_ERR_UNSUPPORTED, "fo_step: peers and separate outputs");

  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  DevHyper hyper[FO_MAX_HYPERS];
  bool lp_delta = false, coupled = false;
  for (uint32_t h = 0; h < d->n_hypers; ++h) {
    hyper[h] = make_dev_hyper(d->hypers[h], d->opt);
    lp_delta = lp_delta || (hyper[h].flags & FO_FLAG_LP_DELTA) != 0;
    coupled = coupled || (d->opt != FO_OPT_LION && (hyper[h].flags & FO_FLAG_DECOUPLED_WD) == 0 && hyper[h].wd != 0.0f);
  }
  Peers peers;
  memset(&peers, 0, sizeof(peers));
  if (d->peer_param_offsets != nullptr) {
    peers.n = (int)d->n_peers;
    for (uint32_t r = 0; r < d->n_peers; ++r) peers.delta[r] = (long long)d->peer_param_offsets[r];
  }
  if (d->peer_grad_offsets != nullptr && d->n_peers > 0) {
    const uint32_t ranks = d->n_peers + 1;
    peers.ng = (int)d->n_peers;
    for (uint32_t r = 0; r < d->n_peers; ++r) peers.gdelta[r] = (long long)d->peer_grad_offsets[r];
    peers.neg_ranks = -(float)ranks;
    peers.rcp_ranks = 1.0f / (float)ranks;  // correctly rounded (IEEE division on the host)
    peers.ranks_pow2 = (ranks & (ranks - 1)) == 0;
  }
  if (d->mc_param_offset != 0) {
    if (d->peer_param_offsets == nullptr || d->n_peers == 0) return fail(FO_ERR_INVALID_ARG, "fo_step: mc_param_offset without peer_param_offsets");
    peers.mc_pdelta = (long long)d->mc_param_offset;
  }
  if (d->mc_grad_offset != 0) {
    if (d->peer_grad_offsets == nullptr || d->n_peers == 0) return fail(FO_ERR_INVALID_ARG, "fo_step: mc_grad_offset without peer_grad_offsets");
    peers.mc_gdelta = (long long)d->mc_grad_offset;
  }
  const bool with_peers = peers.n > 0 || peers.ng > 0;
  const int features = (d->grad_sq_norm != nullptr ? kClip : 0) | (outs != nullptr ? kOut : 0) |
                       (d->state == FO_STATE_QUANT && d->group_size != 32 ? kGroup : 0) | (lp_delta ? kDelta : 0);
  const int mode = with_peers ? kPeer : features;
  const Launcher launcher = find_launcher(d->opt, d->param_dtype, d->ecc_bits, d->state, generic, mode, d->group_size, d->grad_dtype);
  const PieceFn pieces = generic ? nullptr : find_pieces(d->opt, d->param_dtype, d->ecc_bits, d->state);
  if (launcher.launch == nullptr || (!generic && pieces == nullptr)) return fail(FO_ERR_UNSUPPORTED, "fo_step: no kernel for this combination");

  HostLeaf table[kMaxLeaves];
  HostStep hs;
  hs.leaf = table; hs.n_leaves = 0;
  hs.hyper = hyper; hs.n_hypers = (int)d->n_hypers;
  hs.grad_dtype = d->grad_dtype; hs.group_shift = group_shift; hs.group_size = d->state == FO_STATE_QUANT ? d->group_size : 32;
  hs.sm_count = sm_count_of_current_device();
  if (hs.sm_count <= 0) return fail(FO_ERR_CUDA, "fo_step: cannot query the current device");
  hs.sq_norm = d->grad_sq_norm; hs.max_norm = d->max_grad_norm;
  hs.peers = &peers;
  hs.outs = outs != nullptr;
  hs.coupled = coupled;
  // Launches that touch peers' memory start in stream order, behind the exchange in front of them.
  const bool same_step = more != nullptr && (more->launch_flags & FO_LAUNCH_CHAINED) != 0;
  bool chained = same_step || !with_peers;
  hs.wait = !same_step && !with_peers;
  const int most_leaves = outs != nullptr ? kMaxLeavesFlex : launcher.most_leaves;
  const unsigned long long unit = generic ? generic_tile_elems(d->group_size) : kPieceElems;
  const unsigned long long kMaxBlocks = 0x7FFFFFFFull;
  unsigned long long blocks = 0, whole = 0;
  auto flush = [&]() -> int {
    if (hs.n_leaves == 0) return FO_OK;
    cudaError_t e = cudaSuccess;
    if (generic) {
      e = launcher.launch(hs, chained, stream);
    } else {
      // with peers the whole chunks always take the kernel that knows them (the pieces' path is scalar there)
      const unsigned long long small = launcher.tiles ? kSmallElemsTiles : FO_SMALL_ELEMS;
      const unsigned int main_chunk = (with_peers ? whole > 0 : whole > small) ? launcher.chunk : 0u;
      if (main_chunk != 0) e = launcher.launch(hs, chained, stream);
      if (e == cudaSuccess) e = pieces(hs, main_chunk, chained, stream);
    }
    hs.n_leaves = 0;
    blocks = whole = 0;
    if (e != cudaSuccess) return fail(FO_ERR_CUDA, "fo_step: launch failed: %s", cudaGetErrorString(e));
    return FO_OK;
  };
  // The 32-group kernels address elements with 32-bit offsets: a longer leaf goes in as several
  // leaves of 2^31 elements (a multiple of the pieces of 1024 and of the group, so every piece keeps
  // its alignment and its own whole groups; what the chunks leave over goes to piece_kernel).
  const unsigned long long kMaxLeafElems = generic ? ~0ull : (1ull << 31);
  const size_t grad_size = d->grad_dtype == FO_F32 ? 4 : 2, param_size = d->param_dtype == FO_F32 ? 4 : 2;
  const size_t ecc_size = (size_t)d->ecc_bits / 8, moment_size = d->state == FO_STATE_FULL ? 4 : 1;
  auto advance = [](const void* base, unsigned long long elems, size_t size) -> void* {
    return base == nullptr ? nullptr : (void*)((const char*)base + elems * size);
  };
  auto distance = [](const void* to, const void* from) -> long long { return from == nullptr ? 0ll : (long long)((const char*)to - (const char*)from); };
  for (uint32_t i = 0; i < d->n_leaves; ++i) {
    const FoLeaf& L = d->leaves[i];
    DevOut out = {};
    bool aligned = aligned16(L.grad) && aligned16(L.param) && aligned16(L.ecc) && aligned16(L.mu) && aligned16(L.nu);
    if (outs != nullptr && L.n != 0) {
      const FoLeafOut& O = outs[i];
      out.param = distance(O.param, L.param);
      out.ecc = distance(O.ecc, L.ecc);
      out.mu = distance(O.mu, L.mu);
      out.mu_scales = distance(O.mu_scales, L.mu_scales);
      out.nu = distance(O.nu, L.nu);
      out.nu_scales = distance(O.nu_scales, L.nu_scales);
      aligned = aligned && ((out.param | out.ecc | out.mu | out.nu) & 15) == 0;
    }
    for (unsigned long long done = 0; done < L.n; done += kMaxLeafElems) {
      const unsigned long long n = L.n - done < kMaxLeafElems ? L.n - done : kMaxLeafElems;
      const unsigned long long nb = (n + unit - 1) / unit;
      if (nb > kMaxBlocks) return fail(FO_ERR_TOO_LARGE, "fo_step: leaf %u with %llu elements exceeds one launch", i, (unsigned long long)L.n);
      if (hs.n_leaves == most_leaves || blocks + nb > kMaxBlocks) {
        int rc = flush();
        if (rc != FO_OK) return rc;
      }
      HostLeaf& H = table[hs.n_leaves];
      DevLeaf& D = H.src;
      D.grad = advance(L.grad, done, grad_size);
      D.param = advance(L.param, done, param_size);
      D.ecc = advance(L.ecc, done, ecc_size);
      D.mu = advance(L.mu, done, moment_size);
      D.nu = advance(L.nu, done, moment_size);
      D.mu_scales = advance(L.mu_scales, done >> group_shift, 2);
      D.nu_scales = advance(L.nu_scales, done >> group_shift, 2);
      D.n = n;
      H.out = out;  // (zeros without outs: the kernel that carries all features adds them)
      H.hyper = (uint8_t)L.hyper;
      const DevHyper& dh = hyper[L.hyper];
      bool hot = aligned && !(mode == kPeer && (dh.flags & FO_FLAG_LP_DELTA) != 0);
      if (d->opt == FO_OPT_ADAM && dh.dyn == nullptr) hot = hot && (dh.flags & kFlagTameAdam) != 0;
      // Lion's first pass on quantized moments takes the sign of a NaN for 1.  Moments and gradients that bring one show in the group's maximum; factors
      // that do (finite ones only where both products overflow) are found here.  (Asked in the kernel, before the loop, that made Lion on fp16 parameters
      // 2 to 5 % slower: 16.8 M elements 30.0 -> 30.6 us by a bound of the maxima, 31.6 by factors that make such moments NaN.)
      if (d->opt == FO_OPT_LION && d->state == FO_STATE_QUANT) hot = hot && fabsf(dh.b1) <= 1.0e30f && fabsf(dh.omb1) <= 3.4e38f;
#ifdef FO_NAIVE_MATH
      hot = false;
#endif
      H.hot = hot ? 1 : 0;
      if (hot && !generic) whole += n / launcher.chunk * launcher.chunk;
      blocks += nb;
      ++hs.n_leaves;
    }
  }
  return flush();
}

extern "C" int fo_version(void) { return FO_ABI_VERSION; }

extern "C" const char* fo_status_string(int status) {
  switch (status) {
    case FO_OK: return "ok";
    case FO_ERR_INVALID_ARG: return "invalid argument";
    case FO_ERR_UNSUPPORTED: return "unsupported configuration";
    case FO_ERR_CUDA: return "CUDA error";
    case FO_ERR_TOO_LARGE: return "size beyond a stated maximum";
    default: return "unknown status";
  }
}

extern "C" const char* fo_last_error(void) { return fo::g_err; }
