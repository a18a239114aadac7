// The step on quantized moments, in tiles of 512 elements per warp: what step_kernel (fo_step.cuh) is for the other kinds of state.
//
// Bound: a sweep over 10 to 19 bytes per element whose arithmetic takes about as long as its memory traffic, under the chip's
// power cap.  A warp works for itself: it copies its next tile into a slot of shared memory of its own (cp.async, 16 bytes per
// lane, no block barrier), and a lane owns 16 consecutive elements of it.  Against 8 elements per lane that halves
// everything that is per lane and not per element (group maxima and their shuffles, reciprocals, range checks, votes, address
// steps; a 32-element group is two lanes), makes every copy 16 bytes wide, also of the one-byte streams, and lets a lane store whole
// 32-byte sectors.
//
//   * Dequantization tables: row b holds 32 copies of the momentum value of code b, one per lane and bank, and 32
//     copies of b / 255 for the second moment.  A row is 256 bytes, so one byte permutation of (codes, lane * 4) is the address, and no
//     look-up has a bank conflict.  64 KB of the SM's 227.
//   * Slots: 16-byte units are stored at positions permuted inside 128 bytes (see Units), so that both the coalesced copies and
//     the reads of a lane's 32 or 64 consecutive bytes fall on all banks.
//   * All range checks are known once the group maxima are: one vote, then the stores of parameter and ECC, then the codes.  For bf16 parameters
//     with codes most of them are one look at the new parameters (tile_run).
//   * Two slots per warp and a loop body that is not unrolled: three slots and an unrolled body measured the same.
//
// Measured (one bf16 leaf of 2^28 elements, AdamW, 32-bit master weights): 712 us with step_kernel, 588 here when it was written; with the power cap reached
// 798 and 675 (691 -> 682 on another box when the checks moved).  51 instructions per element instead of 63; a packed one keeps the FMA pipe for two cycles (60 % busy, 64 % of
// the issue slots).  Warps of a block, and blocks, end up to 10 % of a launch of 9 to 25 M elements apart.  Dealing the last tiles while the kernel runs
// (clusterlaunchcontrol, a unit of one to four tiles for a warp that has nothing left) made 2^28 elements 3 to 8 % faster until the cap is reached, 1 to 2 %
// slower then, and 9 M 24 -> 29 us: an answer takes a microsecond, and the device gives two per nanosecond.
#pragma once

namespace fo {

inline namespace FO_SHAPE_NS {

constexpr int kTileElems = 512;   // of a warp
constexpr int kEnd = 256;         // elements of the warp's pieces that a leaf's ragged end is taken in
constexpr int kWarps = kThreads / 32;
constexpr int kTableBytes = 256 * 256;
constexpr int kAnyGrad = -1;      // gradient dtype known at run time only

template <int MODE>
struct TileParams : StepParams<MODE> {
  uint16_t first_end[((MODE & kOut) != 0 ? kMaxLeavesFlex : kMaxLeaves) + 1];  // first piece of each leaf's ragged end
};
static_assert(sizeof(TileParams<kOut>) <= 32764 && sizeof(TileParams<kPlain>) <= 32764, "kernel parameters");

template <int OPT, int PDT, int ECC_BITS, int GDT>
struct TileSlot {
  static constexpr int kParamUnits = PDT == FO_F32 ? 4 : 2;  // 16-byte units per lane
  static constexpr int kEccUnits = ECC_BITS / 8;
  static constexpr int kGradUnits = (GDT == FO_F32 || GDT == kAnyGrad) ? 4 : 2;
  static constexpr int kEcc = kParamUnits * 512;  // byte offsets
  static constexpr int kMu = kEcc + kEccUnits * 512;
  static constexpr int kNu = kMu + 512;
  static constexpr int kGrad = kNu + (OPT == FO_OPT_ADAM ? 512 : 0);
  static constexpr int kScales = kGrad + kGradUnits * 512;  // up to 32 of the first moment, then as many of the second
  static constexpr int kBytes = kScales + 128;
};
constexpr int kTileStages = 2;
constexpr int kSmemPerBlock = 227 * 1024 - 64;  // (the clipping constants are static)
template <int OPT, int PDT, int ECC_BITS, int GDT>
__host__ __device__ constexpr int tile_smem() {
  return kTableBytes + kTileStages * kWarps * TileSlot<OPT, PDT, ECC_BITS, GDT>::kBytes;
}

// Streams of U 16-byte units per lane (U x 512 bytes per tile).  Unit u goes to position u ^ (u >> 3 & (U - 1)): lane l copies units
// l + 32 i, which stay eight to a row of 128 bytes, and the eight lanes of a quarter warp that read their j-th units U l + j
// find them in eight different places of a row.
template <int U>
struct Units {
  static FO_DEVI uint32_t copy_to(uint32_t lane) { return (lane ^ ((lane >> 3) & (U - 1))) * 16u; }
  static FO_DEVI uint32_t read_at(uint32_t lane) { return (lane * U + (((lane * U) >> 3) & (U - 1))) * 16u; }  // unit j: ^ (j * 16)
  static FO_DEVI uint32_t unit_at(uint32_t u) { return (u ^ ((u >> 3) & (U - 1))) * 16u; }
};
template <int U>
FO_DEVI void copy_units(const uint32_t at, const char* src) {
#pragma unroll
  for (int i = 0; i < U; ++i) copy_async16(at + 512u * i, src + 512 * i);
}
FO_DEVI void copy_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
FO_DEVI float lds_half(uint32_t a) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
  return __half2float(__ushort_as_half(v));
}

// 32 bytes of a lane.  An array that starts on a 16-byte boundary only takes two stores.
FO_DEVI void store32(void* p, const uint4& a, const uint4& b, const bool wide) {
  if (wide) {
    asm volatile("st.global.cs.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x),
                 "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
  } else {
    __stcs((uint4*)p, a);
    __stcs((uint4*)p + 1, b);
  }
}
FO_DEVI uint4 bits_of(const float2& a, const float2& b) {
  return make_uint4(__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(b.x), __float_as_uint(b.y));
}

// The tables: thread t makes the values of one code and stores eight copies at a time, rotated by its lane, so that the lanes of
// a store fall on different banks.
template <int OPT>
FO_DEVI void build_tables(char* table) {
  for (int i = threadIdx.x; i < (OPT == FO_OPT_ADAM ? 512 : 256); i += kThreads) {
    const int code = i & 255;
    const float x = i < 256 ? kDeqM.v[code] : fdiv((float)code, 255.0f);
    float4* row = reinterpret_cast<float4*>(table + code * 256 + (i < 256 ? 0 : 128));
#pragma unroll
    for (int k = 0; k < 8; ++k) row[(k + threadIdx.x) & 7] = make_float4(x, x, x, x);
  }
  __syncthreads();
}
// the values of the codes in bytes b and b + 1 of w; lane4: four times the lane
FO_DEVI float2 table_pair(const char* table, const uint32_t w, const int b, const uint32_t lane4) {
  return make_float2(*reinterpret_cast<const float*>(table + __byte_perm(w, lane4, 0x5504u | (uint32_t)(b << 4))),
                     *reinterpret_cast<const float*>(table + __byte_perm(w, lane4, 0x5504u | (uint32_t)((b + 1) << 4))));
}

// Where a lane's copies of a tile come from, and the copies.
template <int OPT, int PDT, int ECC_BITS, int GDT>
struct TileSource {
  using S = TileSlot<OPT, PDT, ECC_BITS, GDT>;
  static constexpr bool kAdam = OPT == FO_OPT_ADAM;
  static constexpr int kPsz = PDT == FO_F32 ? 4 : 2, kEsz = ECC_BITS / 8;
  const char* grad;
  char* param;
  char* ecc;
  char* mu;
  char* nu;
  // The group scales travel with the tile in words of four bytes, the first moment's by lanes 0 to 15, the second's by the others.  (Loaded
  // into registers one tile ahead, they shared a scoreboard with the loads from shared memory, which then waited for DRAM: 615 to
  // 750 us per 2^28 elements, as the compiler happened to assign it.)  Arrays that begin in the middle of a word still do that.
  const char* sc;
  bool sc_words, sc_mine;
  static FO_DEVI bool in_words(const DevLeaf& L) {
    return ((reinterpret_cast<uintptr_t>(L.mu_scales) | (kAdam ? reinterpret_cast<uintptr_t>(L.nu_scales) : 0)) & 3u) == 0;
  }
  FO_DEVI TileSource(const DevLeaf& L, const uint32_t t, const int gsz, const int gshift, const uint32_t lane) {
    const size_t e0 = (size_t)t * kTileElems;
    grad = (const char*)L.grad + e0 * (size_t)gsz + lane * 16u;
    param = (char*)L.param + e0 * kPsz + lane * 16u;
    ecc = (char*)L.ecc + e0 * kEsz + lane * 16u;
    mu = (char*)L.mu + e0 + lane * 16u;
    nu = (char*)L.nu + e0 + lane * 16u;
    sc = (const char*)(kAdam && lane >= 16u ? L.nu_scales : L.mu_scales) + (e0 >> gshift) * 2u + (lane & 15u) * 4u;
    sc_words = in_words(L);
    sc_mine = sc_words && (lane & 15u) < (256u >> gshift) && (kAdam || lane < 16u);
  }
  // the lane's units of the tile `ahead` steps on
  FO_DEVI void fill(const uint32_t slot, const int ahead, const int gdt, const int gshift, const uint32_t lane) const {
    constexpr int kStep = kWarps * kTileElems;
    copy_units<S::kParamUnits>(slot + Units<S::kParamUnits>::copy_to(lane), param + ahead * (kStep * kPsz));
    if constexpr (ECC_BITS != 0) copy_units<S::kEccUnits>(slot + S::kEcc + Units<S::kEccUnits>::copy_to(lane), ecc + ahead * (kStep * kEsz));
    copy_units<1>(slot + S::kMu + lane * 16u, mu + ahead * kStep);
    if constexpr (kAdam) copy_units<1>(slot + S::kNu + lane * 16u, nu + ahead * kStep);
    if (gdt == FO_F32) copy_units<4>(slot + S::kGrad + Units<4>::copy_to(lane), grad + ahead * (kStep * 4));
    else copy_units<2>(slot + S::kGrad + Units<2>::copy_to(lane), grad + ahead * (kStep * 2));
    if (sc_mine) copy_async4(slot + S::kScales + lane * 4u, sc + ahead * ((kStep >> gshift) * 2));
  }
};

// What a lane owns of a tile's half in pieces of eight elements, from the warp's slot (the group scales of a leaf whose scales do not travel in words from
// memory).
template <int OPT, int PDT, int ECC_BITS, int GDT>
FO_DEVI void slot_read(const DevLeaf& L, const uint32_t slot, const uint32_t half, const int gdt, const int gshift, const uint32_t i0, const bool sc_words,
                       Raw<OPT, PDT, ECC_BITS, FO_STATE_QUANT>& r) {
  using S = TileSlot<OPT, PDT, ECC_BITS, GDT>;
  const uint32_t piece = half * 32u + (threadIdx.x & 31u);
  if constexpr (PDT == FO_F32) {
    r.p0 = lds128(slot + Units<4>::unit_at(2u * piece));
    r.p1 = lds128(slot + Units<4>::unit_at(2u * piece + 1u));
  } else {
    r.p0 = lds128(slot + Units<2>::unit_at(piece));
  }
  if constexpr (ECC_BITS == 16) r.e = lds128(slot + S::kEcc + Units<2>::unit_at(piece));
  if constexpr (ECC_BITS == 8) {
    const uint2 e = lds64(slot + S::kEcc + piece * 8u);
    r.e.x = e.x; r.e.y = e.y;
  }
  r.mq = lds64(slot + S::kMu + piece * 8u);
  if constexpr (OPT == FO_OPT_ADAM) r.vq = lds64(slot + S::kNu + piece * 8u);
  if (sc_words) {
    const uint32_t at = slot + S::kScales + ((piece * 8u >> gshift) << 1);
    r.msc = __float2half(lds_half(at));
    if constexpr (OPT == FO_OPT_ADAM) r.vsc = __float2half(lds_half(at + 64u));
  } else {
    r.msc = ((const __half*)L.mu_scales)[i0 >> gshift];
    if constexpr (OPT == FO_OPT_ADAM) r.vsc = ((const __half*)L.nu_scales)[i0 >> gshift];
  }
  if (gdt == FO_F32) {
    r.g0 = lds128(slot + S::kGrad + Units<4>::unit_at(2u * piece));
    r.g1 = lds128(slot + S::kGrad + Units<4>::unit_at(2u * piece + 1u));
  } else {
    r.g0 = lds128(slot + S::kGrad + Units<2>::unit_at(piece));
  }
}

// The magnitudes of new bf16 parameters that tile_run accepts, from `least` (rounded up) to 2^126: x = 2 w + range.x, in each half of a word of two parameters,
// counts from twice the smallest and is below range.y for them only (a carry out of the lower half can make it one or two more).
constexpr uint32_t kMostBits = 0x7E80u;  // 2^126
FO_DEVI uint2 range_from(const float least) {
  const uint32_t low = min((__float_as_uint(least) >> 16) + 2u, kMostBits);
  return make_uint2((0x8000u - low) * 0x00020002u, 2u * (kMostBits - low));
}

// Half of a tile that holds a value outside the shortcuts' ranges, 256 elements (sixteen lanes' worth): once more, by the repairing pass, from the warp's slot,
// which still holds it.  It works out for itself what only it needs, rows at rest among it: asked in the loop that cost ordinary tiles
// up to 5 %.  (Storing a half that holds no such value from the first pass made the loop slower, AdamW with 8-bit codes 588 -> 623 us per 2^28
// elements; under SGD and Lion it made such tiles themselves slower, 8192 x 8192 with 0.1 % zeros under SGD 233 -> 262.)
template <int OPT, int PDT, int ECC_BITS, int GDT, int MODE>
__device__ __noinline__ void redo_half(const StepCommon& c, const DevLeaf& L, const DevOut* out, const DevHyper& dh, const uint32_t e0, const uint32_t slot, const uint32_t half) {
  const int gdt = GDT == kAnyGrad ? c.grad_dtype : GDT, gshift = (MODE & kGroup) != 0 ? c.group_shift : 5;
  const uint32_t i0 = e0 + half * 256u + (threadIdx.x & 31u) * 8u;
  Raw<OPT, PDT, ECC_BITS, FO_STATE_QUANT> raw;
  slot_read<OPT, PDT, ECC_BITS, GDT>(L, slot, half, gdt, gshift, i0, TileSource<OPT, PDT, ECC_BITS, GDT>::in_words(L), raw);
  warm_finish<OPT, PDT, ECC_BITS, FO_STATE_QUANT, MODE & ~kCoupled>(c, L, out, dh, i0, nullptr, raw);
}

// 256 elements from i0 - 8 * lane on of a leaf's ragged end: the code of piece_kernel.
template <int OPT, int PDT, int ECC_BITS, bool OUT>
__device__ __noinline__ void end_piece(const StepCommon& c, const DevLeaf& L, const DevOut* out, const DevHyper& dh, const uint32_t i0) {
  const Hyp h = load_hyper<OPT>(dh);
  if (OPT != FO_OPT_ADAM || (h.flags & kFlagTameAdam) != 0) {
    const Clip clip = load_clip(c.sq_norm, c.max_norm, c.grad_dtype);
    ragged_piece<OPT, PDT, ECC_BITS, FO_STATE_QUANT, OUT>(c, L, out, dh, h, clip, i0, (uint32_t)L.n);
  } else {
    cold_piece<OPT, PDT, ECC_BITS, FO_STATE_QUANT>(L, out, dh, c.grad_dtype, c.group_shift, i0, nullptr, c.sq_norm, c.max_norm);
  }
}

// One warp's tiles t, t + kWarps, ... below t1 of a leaf.  `primed`: the first one's copies are under way, in the first slot.
//
// bf16 parameters with codes (kLate; not under a decay added to the gradient): what the shortcuts ask of the old parameter and of the first moment follows
// from the new parameter, so that one look at it takes the place of four range checks of every element.  Let it be |p| >= L, L >= 2^-68, and |decay| <= 2.
//   * An old parameter below 2^-100, which the packed reconstruction may get wrong (it stays below 2^-99), has left nothing in p: decayed it is below 2^-98, and
//     a quarter of a unit in the last place of the update that it was added to, which is above L / 2, is 2^-27 L at least.  (Lion and SGD ask for no more.)
//   * A numerator below 2^-102, for which neg_div2 is not exact, makes an update below 2^-102 / eps, exact or not.  With L >= 2^-76 / eps that is less than half a
//     unit in the last place of anything that rounds to p: it adds nothing.  Above, up to 2^60 (am_most), neg_div2 is exact or its quotient as small.
//   * Clipping a bf16 gradient below 2^-100, whose quotient may be off, makes a gradient below 2^-100 G, where G is 2 or, under a limit below zero, up to 2^16
//     (Clip::div_ok) times as large as the norm, |limit| / norm.  The second moment is that of the element's past, or below the 1e-30 that is checked.  The
//     first moment is that of the past too, or (|b1| >= 2^-20 or 0, |omb1| <= 2) below 2^-99 G: its code is 0 and its update, below 2^-99 G lr / bc1 / eps, less
//     than half a unit of p with L >= 2^-73 G lr / bc1 / eps.
// (Hyp::least.  With eps = 1e-8 and lr / bc1 up to 1/16 it is 2^-49.  A range that began at 2^-28 sent most tiles of a matrix that started at zero to the repairs:
// AdamW with 8-bit codes, 4096 x 4096, the first 20 steps of a warm-up 954 -> 1572 us, Lion 698 -> 979.)
// The look is taken at the packed words (range_from): an addition per word and a maximum per two.  (A test of single bits that passes 2^-31 to 2 with half
// of that, and a comparison behind it for the rest, made leaves with larger parameters 5 % slower.)
// AdamW with 8-bit codes, 2^28 elements 580 -> 560 us, with the power cap reached 662 -> 648, 4 M elements in the L2 12.3 -> 11.7; clipping 649 -> 597, 717 ->
// 674, 14.4 -> 13.6; 16-bit codes 691 -> 682 at the cap; Lion 472 -> 441 and 9.1 -> 8.5, half of it by its sign in two instructions; SGDW 461 -> 454.
template <int OPT, int PDT, int ECC_BITS, int GDT, int MODE, typename OUT>
FO_DEVI void tile_run(const bool primed, const StepCommon& c, const DevLeaf& L, const DevOut* out, const DevHyper& dh, const Hyp& h, const SharedClip& clip, uint32_t t,
                      const uint32_t t1, const uint32_t slots, const char* table, const OUT& distance) {
  using namespace fast2;
  using S = TileSlot<OPT, PDT, ECC_BITS, GDT>;
  constexpr bool kAdam = OPT == FO_OPT_ADAM;
  constexpr int kStep = kWarps * kTileElems;  // elements from one of the warp's tiles to the next
  constexpr int kPsz = PDT == FO_F32 ? 4 : 2, kEsz = ECC_BITS / 8;
  constexpr bool kLate = PDT == FO_BF16 && ECC_BITS != 0 && (MODE & kCoupled) == 0;
  // Where the look stands makes 2 to 12 % by what the compiler makes of the loop around it (repeats differ by 0.3 %).  8.4 M elements in the L2, us behind the
  // maxima / in front of them / with each half: AdamW 8-bit codes 21.6 / 20.3 / 22.2, handing back 22.2 / 21.5 / 22.7, results elsewhere 21.8 / 23.2 / 21.7,
  // clipping 23.1 / 23.4 / 23.6, under fp32 gradients 24.4 / 24.3 / 24.9, groups of 128 22.3 / 22.9 / 22.2; 16-bit codes 21.7 / 21.9 / 22.8, handing back 22.1 / 22.3 / 22.5,
  // clipping 24.0 / 24.1 / 23.9, under gradients of any dtype 25.4 / 25.0 / 25.3, groups 22.6 / 22.4 / 21.9; Lion 14.6 / 14.6 / 14.3, clipping 18.7 / 18.6 / 18.0, 16-bit codes
  // 15.9 / 15.6 / 15.5, results elsewhere 15.3 / - / 17.2, groups 16.0 / 15.8 / 17.2; SGDW 14.8 / 15.0 / 14.9, 16-bit codes 14.6 / 15.0 / 14.9, groups of 256 15.4 / 16.3 / 15.9, under fp32 gradients
  // 16.0 / 16.8 / 15.8.
  enum { kNowhere, kBehind, kInFront, kWithEachHalf };
  constexpr bool kEachHalf = OPT == FO_OPT_LION ? (MODE & (kOut | kGroup)) == 0 : (MODE & kGroup) != 0 && (kAdam || (ECC_BITS == 8 && GDT == FO_F32));
  constexpr bool kFront = kAdam && (MODE & kOut) == 0 && ((MODE & kClip) != 0 ? GDT != FO_BF16 : ECC_BITS == 8);
  constexpr int kLook = !kLate ? kNowhere : kEachHalf ? kWithEachHalf : kFront ? kInFront : kBehind;
  const int gdt = GDT == kAnyGrad ? c.grad_dtype : GDT;
  const int gsz = gdt == FO_F32 ? 4 : 2;
  const int gshift = (MODE & kGroup) != 0 ? c.group_shift : 5;  // 4 to 8 here
  uint32_t tid;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));  // read once: otherwise re-read at every use
  const uint32_t lane = tid & 31u, lane4 = lane * 4u, lane16 = lane * 16u;
  const size_t e0 = (size_t)t * kTileElems;
  TileSource<OPT, PDT, ECC_BITS, GDT> s(L, t, gsz, gshift, lane);
  char* s_msc = (char*)L.mu_scales + ((e0 + lane16) >> gshift) * 2u;  // the scale of the lane's group
  char* s_vsc = (char*)L.nu_scales + ((e0 + lane16) >> gshift) * 2u;
  const int sc_step = (kStep >> gshift) * 2;
  bool wide = ((reinterpret_cast<uintptr_t>(L.param) | (ECC_BITS == 16 ? reinterpret_cast<uintptr_t>(L.ecc) : 0)) & 31u) == 0;
  if constexpr ((MODE & kOut) != 0) wide = wide && ((distance(&DevOut::param) | (ECC_BITS == 16 ? distance(&DevOut::ecc) : 0)) & 31) == 0;
  // Lion and SGD have the range in the code, and a leaf under another decay fails by its scales.
  float least = kAdam ? h.least : kLeastNew;
  if constexpr (kLate && kAdam && (MODE & kClip) != 0) {
    if (clip.active) {
      const Clip k = clip.get();
      least *= fmaxf(1.0f, 0.5f * fabsf(k.m_g) * k.rcp_n);
    }
  }
  const uint2 range = range_from(least);
  float am_most = kAdam ? fminf(1.0e30f, h.m_hi) : 1.0e30f;  // of a group scale: the reciprocal's range, the update's numerator
  if constexpr (kLate && !kAdam) am_most = fabsf(h.decay) <= 2.0f ? am_most : -1.0f;
  uint32_t slot = slots;
  if (!primed) {
    __syncwarp();
    s.fill(slot, 0, gdt, gshift, lane);
    copy_commit();
  }
  __half msc = __float2half(0.0f), vsc = msc;
  if (!s.sc_words) {
    msc = *(const __half*)s_msc;
    if constexpr (kAdam) vsc = *(const __half*)s_vsc;
  }
  while (true) {
    const bool more = t + kWarps < t1;
    __syncwarp();
    if (more) s.fill(2u * slots + S::kBytes - slot, 1, gdt, gshift, lane);
    copy_commit();
    copy_wait<1>();
    __syncwarp();
    float2 msc2, vsc2 = sp(0.0f);
    if (s.sc_words) {
      const uint32_t sc_at = slot + S::kScales + ((lane16 >> gshift) << 1);
      msc2 = sp(lds_half(sc_at));
      if constexpr (kAdam) vsc2 = sp(lds_half(sc_at + 64u));
    } else {
      msc2 = sp(__half2float(msc));
      if constexpr (kAdam) vsc2 = sp(__half2float(vsc));
      if (more) {
        msc = *(const __half*)(s_msc + sc_step);
        if constexpr (kAdam) vsc = *(const __half*)(s_vsc + sc_step);
      }
    }
    const uint4 mq = lds128(slot + S::kMu + lane16);
    uint4 vq = make_uint4(0, 0, 0, 0), eq = vq;
    if constexpr (kAdam) vq = lds128(slot + S::kNu + lane16);
    if constexpr (ECC_BITS == 8) eq = lds128(slot + S::kEcc + lane16);
    bool rare = false;
    float2 m[2][4], nroot[2][4], theta[2][4];
    uint32_t nw[2][4];
    uint4 ecc_out[2];
    float am = 0.0f, av = 0.0f;
    [[maybe_unused]] uint32_t most = 0u;  // of the new parameters, as range_from counts
    auto look_at = [&](int k) {
#pragma unroll
      for (int j = 0; j < 4; j += 2) most = __vimax3_u16x2(most, 2u * nw[k][j] + range.x, 2u * nw[k][j + 1] + range.x);
    };
    auto answer = [&]() { rare = rare || (most & 0xFFFFu) >= range.y || (most >> 16) >= range.y; };
    const uint32_t p_at = slot + Units<S::kParamUnits>::read_at(lane);
#pragma unroll
    for (int k = 0; k < 2; ++k) {  // the lane's first and second eight elements
      Unpacked u;
      if (gdt == FO_F32) {
        const uint32_t g_at = slot + S::kGrad + Units<4>::read_at(lane);
        pairs_of(lds128(g_at ^ (32u * k)), lds128(g_at ^ (32u * k + 16u)), u.g);
      } else {
        const uint4 w = lds128((slot + S::kGrad + Units<2>::read_at(lane)) ^ (16u * k));
        if (gdt == FO_BF16) pairs_of16<FO_BF16>(w, u.g);
        else pairs_of16<FO_F16>(w, u.g);
      }
      uint4 p0, p1 = make_uint4(0, 0, 0, 0), e = p1;
      if constexpr (PDT == FO_F32) { p0 = lds128(p_at ^ (32u * k)); p1 = lds128(p_at ^ (32u * k + 16u)); }
      else p0 = lds128(p_at ^ (16u * k));
      if constexpr (ECC_BITS == 16) e = lds128((slot + S::kEcc + Units<2>::read_at(lane)) ^ (16u * k));
      if constexpr (ECC_BITS == 8) { e.x = k ? eq.z : eq.x; e.y = k ? eq.w : eq.y; }
      bool odd = unpack_master<false, PDT, ECC_BITS, !kLate>(p0, p1, e, u.theta);
      const uint32_t mw[2] = {k ? mq.z : mq.x, k ? mq.w : mq.y}, vw[2] = {k ? vq.z : vq.x, k ? vq.w : vq.y};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        u.m[j] = mul2(table_pair(table, mw[j >> 1], 2 * (j & 1), lane4), msc2);  // quantization.py:52-55
        if constexpr (kAdam) {                                                   // quantization.py:74-77
          const float2 s = mul2(table_pair(table + 128, vw[j >> 1], 2 * (j & 1), lane4), vsc2);
          u.v[j] = mul2(s, s);
        }
      }
      if constexpr ((MODE & kClip) != 0) {
        if (clip.active) odd = clip_grads<false, !(kLate && kAdam)>(u.g, gdt, clip) || odd;
      }
      float am_lane, av_lane;
      odd = update_pairs<false, OPT, FO_STATE_QUANT, (MODE & kCoupled) != 0, !kLate>(h, c.one, u, nroot[k], am_lane, av_lane) || odd;
      // (Infinite parameters and NaNs take part in a weight decay of zero that is added to the gradient, which this pass leaves out.  Where there
      // is an error-correction code stored_form sees them.)
      if constexpr (ECC_BITS == 0 && OPT != FO_OPT_LION && (MODE & kCoupled) == 0) odd = odd || !(maxabs8(u.theta) <= 3.4e38f);
      odd = stored_form<false, PDT, ECC_BITS, !kLate>(u.theta, nw[k], ecc_out[k]) || odd;
      if constexpr (kLook == kWithEachHalf) look_at(k);
      rare = rare || odd;
      am = k ? max2<true>(am, am_lane) : am_lane;
      av = k ? max2<true>(av, av_lane) : av_lane;
#pragma unroll
      for (int j = 0; j < 4; ++j) { m[k][j] = u.m[j]; theta[k][j] = u.theta[j]; }
    }
    if constexpr (kLook == kInFront) {
      look_at(0);
      look_at(1);
      answer();
    }
    // ---- group maxima, and one decision per warp ------------------------------------------------------------
    if constexpr ((MODE & kGroup) != 0) {
      for (int o = 1; o < (1 << (gshift - 4)); o <<= 1) {
        am = max2<true>(am, __shfl_xor_sync(0xFFFFFFFFu, am, o));
        if constexpr (kAdam) av = max2<true>(av, __shfl_xor_sync(0xFFFFFFFFu, av, o));
      }
    } else {
      am = max2<true>(am, __shfl_xor_sync(0xFFFFFFFFu, am, 1));
      if constexpr (kAdam) av = max2<true>(av, __shfl_xor_sync(0xFFFFFFFFu, av, 1));
    }
    rare = rare || !(am >= 1.0e-12f && am <= am_most);                           // an all-zero group, or beyond
    if constexpr (kAdam) rare = rare || !(av >= 1.0e-12f && av <= 1.0737418e9f);  // 2^30: also the limit of the packed division
    if constexpr (kLook == kBehind) {
      look_at(0);
      look_at(1);
    }
    if constexpr (kLook == kBehind || kLook == kWithEachHalf) answer();
    if (__any_sync(0xFFFFFFFFu, rare)) {
      // (A loop under Adam, two calls under Lion and SGD: which of them leaves the loop around it fewer instructions differs, AdamW 9 M elements in
      // the L2 22.2 and 24.6 us, Lion 17.4 and 17.0, SGDW 15.1 and 14.9; through one call for both halves 24.1, 17.5 and 14.9.)
#pragma unroll (kAdam ? 1 : 2)
      for (uint32_t half = 0; half < 2u; ++half) redo_half<OPT, PDT, ECC_BITS, GDT, MODE>(c, L, out, dh, t * (uint32_t)kTileElems, slot, half);
    } else {
      // ---- stores: parameter and ECC, scales, codes -------------------------------------------------------------
      auto to = [&](char* base, long long DevOut::*d) {
        if constexpr ((MODE & kOut) != 0) return base + distance(d);
        else return base;
      };
      if constexpr ((MODE & kDelta) != 0) {
        if (h.flags & FO_FLAG_LP_DELTA) {  // (the old parameter is still in the slot)
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            if constexpr (PDT == FO_F32) hand_back_delta<PDT>(lds128(p_at ^ (32u * k)), lds128(p_at ^ (32u * k + 16u)), nw[k], theta[k]);
            else hand_back_delta<PDT>(lds128(p_at ^ (16u * k)), make_uint4(0, 0, 0, 0), nw[k], theta[k]);
          }
        }
      }
      char* const o_param = to(s.param, &DevOut::param) + lane16 * (S::kParamUnits - 1);
      if constexpr (PDT == FO_F32) {
        store32(o_param, bits_of(theta[0][0], theta[0][1]), bits_of(theta[0][2], theta[0][3]), wide);
        store32(o_param + 32, bits_of(theta[1][0], theta[1][1]), bits_of(theta[1][2], theta[1][3]), wide);
      } else {
        store32(o_param, make_uint4(nw[0][0], nw[0][1], nw[0][2], nw[0][3]), make_uint4(nw[1][0], nw[1][1], nw[1][2], nw[1][3]), wide);
      }
      if constexpr (ECC_BITS == 16) store32(to(s.ecc, &DevOut::ecc) + lane16, ecc_out[0], ecc_out[1], wide);
      if constexpr (ECC_BITS == 8) __stcs((uint4*)to(s.ecc, &DevOut::ecc), make_uint4(ecc_out[0].x, ecc_out[0].y, ecc_out[1].x, ecc_out[1].y));
      // all lanes of a group store its scale: same value to the same address, one unpredicated instruction
      *(__half*)to(s_msc, &DevOut::mu_scales) = __float2half_rn(am);
      if constexpr (kAdam) *(__half*)to(s_vsc, &DevOut::nu_scales) = __float2half_rn(av);
      uint32_t q[2][8];
      {
        const float2 nam = sp(-am), rm2 = sp(fast::rcp_rn(am));
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int j = 0; j < 4; ++j) softsign_code_bits2(div_by_rcp2(m[k][j], nam, rm2), q[k][2 * j], q[k][2 * j + 1]);
        __stcs((uint4*)to(s.mu, &DevOut::mu), make_uint4(pack_bytes(q[0][0], q[0][1], q[0][2], q[0][3]), pack_bytes(q[0][4], q[0][5], q[0][6], q[0][7]),
                                                         pack_bytes(q[1][0], q[1][1], q[1][2], q[1][3]), pack_bytes(q[1][4], q[1][5], q[1][6], q[1][7])));
      }
      if constexpr (kAdam) {
        const float2 av2 = sp(av), nrv2 = sp(-fast::rcp_rn(av));
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int j = 0; j < 4; ++j) quant_v_bits2(nroot[k][j], av2, nrv2, q[k][2 * j], q[k][2 * j + 1]);
        __stcs((uint4*)to(s.nu, &DevOut::nu), make_uint4(pack_bytes(q[0][0], q[0][1], q[0][2], q[0][3]), pack_bytes(q[0][4], q[0][5], q[0][6], q[0][7]),
                                                         pack_bytes(q[1][0], q[1][1], q[1][2], q[1][3]), pack_bytes(q[1][4], q[1][5], q[1][6], q[1][7])));
      }
    }
    if (!more) return;
    t += kWarps;
    slot = 2u * slots + S::kBytes - slot;
    s.grad += kStep * gsz;
    s.param += kStep * kPsz;
    if constexpr (ECC_BITS != 0) s.ecc += kStep * kEsz;
    s.mu += kStep;
    s.sc += sc_step;
    s_msc += sc_step;
    if constexpr (kAdam) { s.nu += kStep; s_vsc += sc_step; }
  }
}

// Persistent grid, one block per SM.  The tiles of all leaves form one sequence, cut into runs of p.run_chunks tiles; block b takes
// runs b, b + grid, ..., and tile i of a run belongs to warp i modulo the number of warps.  One run per block is even to a tile; of several the remainders add up on
// a block's first warps (49810 tiles in runs of 85: 32 tiles for the first of twelve, 28 for the others), and above 1536 * 4 tiles per block some blocks have a run more
// than others (3.76 M tiles: 26112 against a mean of 25379).
template <int OPT, int PDT, int ECC_BITS, int GDT, int MODE>
__global__ void __launch_bounds__(kThreads, 1) tile_kernel(const __grid_constant__ TileParams<MODE> p) {
  extern __shared__ __align__(128) unsigned char tile_mem[];  // the tables, then every warp's slots
  char* const table = reinterpret_cast<char*>(tile_mem);
  using S = TileSlot<OPT, PDT, ECC_BITS, GDT>;
  const uint32_t warp = threadIdx.x / 32u;
  const uint32_t slots = (uint32_t)__cvta_generic_to_shared(tile_mem) + (uint32_t)kTableBytes + warp * (uint32_t)(kTileStages * S::kBytes);
  const uint32_t total = p.t.first_block[p.n_leaves];
  // The block's first run, and its first leaf, are known before the wait: a warp that has a tile there asks for it right behind.
  // (The hyper-parameters, clipping constants and ends then pass under the latency of the copies.  AdamW, 24-bit masters, cold arrays of 2^21,
  // 2^22, 2^24 elements: 8.4, 14.5, 43.7 us without, 7.5, 13.5, 41.6 so; Lion on 5.3 M 12.7, 12.4.  Asking for the first tile
  // of every later run or leaf ahead as well gave nothing more.)
  const int l0 = leaf_of(p.t.first_block, p.n_leaves, blockIdx.x * p.run_chunks);
  const uint32_t t0 = blockIdx.x * p.run_chunks - p.t.first_block[l0] + warp;
  const bool primed0 = blockIdx.x * p.run_chunks < total &&
                       t0 < min(p.t.first_block[l0 + 1], min(total, (blockIdx.x + 1u) * p.run_chunks)) - p.t.first_block[l0];
  const int gdt0 = GDT == kAnyGrad ? p.grad_dtype : GDT, gshift0 = (MODE & kGroup) != 0 ? p.group_shift : 5;
  const TileSource<OPT, PDT, ECC_BITS, GDT> source0(p.t.leaf[l0], t0, gdt0 == FO_F32 ? 4 : 2, gshift0, threadIdx.x & 31u);
  build_tables<OPT>(table);
  if (p.wait) chain_wait();
  chain_release();
  if (primed0) source0.fill(slots, 0, gdt0, gshift0, threadIdx.x & 31u);
  copy_commit();
  SharedClip clip{false, 0u};
  if constexpr ((MODE & kClip) != 0) {
    __shared__ float4 clip_constants;
    const Clip k = load_clip(p.sq_norm, p.max_norm, p.grad_dtype);
    if (threadIdx.x == 0) clip_constants = make_float4(k.n_g, k.rcp_n, k.m_g, __uint_as_float(k.div_ok ? 1u : 0u));
    __syncthreads();
    clip.active = k.active;
    clip.at = (uint32_t)__cvta_generic_to_shared(&clip_constants);
  }
  // Ragged ends first, one piece to a block at a time, beginning with the last blocks and warps, which have the fewest tiles: their
  // latency then passes behind the other warps' work.  (As a launch of piece_kernel they came behind the last tile, and
  // cost the host a launch: Lion on 2999 x 1777 and its bias 13.2 us, now 12.2.)
  for (uint32_t q = (kWarps - 1u - warp) * gridDim.x + (gridDim.x - 1u - blockIdx.x); q < p.first_end[p.n_leaves]; q += kWarps * gridDim.x) {
    const int l = leaf_of(p.first_end, p.n_leaves, (uint16_t)q);
    const DevLeaf& L = p.t.leaf[l];
    const DevOut* out = nullptr;
    if constexpr ((MODE & kOut) != 0) out = &p.out[l];
    const uint32_t i0 = (uint32_t)(L.n / kTileElems) * kTileElems + (q - p.first_end[l]) * kEnd + (threadIdx.x & 31u) * kPiece;
    end_piece<OPT, PDT, ECC_BITS, (MODE & kOut) != 0>(p, L, out, p.hyper[p.t.hyper_of[l]], i0);
  }
  bool primed = primed0;
  for (uint32_t run0 = blockIdx.x * p.run_chunks; run0 < total; run0 += gridDim.x * p.run_chunks) {
    uint32_t at = run0;  // this block's next position in the sequence
    const uint32_t run1 = min(total, run0 + p.run_chunks);
    for (int l = leaf_of(p.t.first_block, p.n_leaves, at); l < p.n_leaves; ++l) {
      if (at >= run1) break;
      const uint32_t first = p.t.first_block[l];
      const uint32_t next = min(p.t.first_block[l + 1], run1);
      if (at >= next) continue;
      uint32_t t = at - first + (warp + kWarps - (at - run0) % kWarps) % kWarps;  // the warp's first tile of the leaf in this run
      const uint32_t t1 = next - first;
      at = next;
      if (t >= t1) continue;
      const DevLeaf& L = p.t.leaf[l];
      const DevHyper& dh = p.hyper[p.t.hyper_of[l]];
      const DevOut* out = nullptr;
      if constexpr ((MODE & kOut) != 0) out = &p.out[l];
      const Hyp h = load_hyper<OPT>(dh);
      if constexpr (OPT == FO_OPT_ADAM) {
        // device-resident scalars can leave the range the reciprocal shortcut in the denominator is proven for
        if ((h.flags & kFlagTameAdam) == 0) {
          copy_wait<0>();
          primed = false;
          for (; t < t1; t += kWarps)
            for (uint32_t half = 0; half < 2u; ++half)
              cold_piece<OPT, PDT, ECC_BITS, FO_STATE_QUANT>(L, out, dh, p.grad_dtype, (MODE & kGroup) != 0 ? p.group_shift : 5,
                                                             (unsigned long long)t * kTileElems + half * 256u + (threadIdx.x & 31u) * 8u, nullptr,
                                                             (MODE & kClip) != 0 ? p.sq_norm : nullptr, p.max_norm);
          continue;
        }
      }
      if constexpr ((MODE & kOut) != 0)
        tile_run<OPT, PDT, ECC_BITS, GDT, MODE>(primed, p, L, out, dh, h, clip, t, t1, slots, table, OutOf{p, l});
      else
        tile_run<OPT, PDT, ECC_BITS, GDT, MODE>(primed, p, L, out, dh, h, clip, t, t1, slots, table, OutAt{nullptr});
      primed = false;
    }
  }
  chain_end();
}

template <int OPT, int PDT, int ECC_BITS, int GDT, int MODE>
cudaError_t launch_tiles(HostStep& hs, bool& chained, cudaStream_t s) {
  if constexpr (OPT != FO_OPT_LION && (MODE & kCoupled) == 0) {
    if (hs.coupled) return launch_tiles<OPT, PDT, ECC_BITS, GDT, MODE | kCoupled>(hs, chained, s);
  }
  auto kernel = tile_kernel<OPT, PDT, ECC_BITS, GDT, MODE>;
  constexpr int smem = tile_smem<OPT, PDT, ECC_BITS, GDT>();
  static_assert(smem <= kSmemPerBlock, "the slots fit a block");
  // whether a device's copy of the function has been opted in above 48 KB (per instantiation; concurrent first calls may both set it)
  static std::atomic<bool> opted_in[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64 || !opted_in[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) opted_in[dev].store(true, std::memory_order_release);
  }
  TileParams<MODE> p;  // filled as far as it is used
  fill_common(p, hs);
  uint32_t total = 0, ends = 0;
  int n = 0;
  for (int i = 0; i < hs.n_leaves; ++i) {
    const HostLeaf& l = hs.leaf[i];
    if (!l.hot || l.src.n == 0) continue;
    p.t.leaf[n] = l.src;
    p.t.hyper_of[n] = l.hyper;
    p.t.first_block[n] = total;
    p.first_end[n] = (uint16_t)ends;
    if constexpr ((MODE & kOut) != 0) p.out[n] = l.out;
    total += (uint32_t)(l.src.n / kTileElems);
    ends += (uint32_t)((l.src.n % kTileElems + kEnd - 1) / kEnd);
    ++n;
  }
  if (n == 0) return cudaSuccess;
  p.n_leaves = n;
  p.t.first_block[n] = total;
  p.first_end[n] = (uint16_t)ends;
  const unsigned int grid = (unsigned int)hs.sm_count;
  // Run length: a launch of at most 256 tiles per block (it lasts tens of microseconds) goes out as one run per block, to within a
  // tile; a larger one in runs of a quarter of a block's share, at most 1536 tiles, so that regions that cost more (rows at rest, values
  // outside the shortcuts' ranges) are spread over all blocks.
  const unsigned int share = (total + grid - 1u) / grid;
  unsigned int run = share;
  if (share > 256u) run = (total + grid * 4u - 1u) / (grid * 4u);
  else if (share <= 64u && ends <= 4u && total >= (unsigned int)kWarps) {
    // A ragged end is cold code for one warp and lasts about as long as one and a half tiles of each warp.  A few ends get blocks with that much less to do:
    // the others take a tile more where the last ones would be full.  (AdamW, 24-bit masters, 909412, 1137000, 1212000 elements 10.4, 9.4, 10.2 us
    // with full last blocks, 7.2, 7.2, 7.7 so; Lion 1137000 5.8 and 5.3, SGDW 6.6 and 5.4.)
    const unsigned int room = share > 5u * kWarps / 2u ? share - 3u * kWarps / 2u : (unsigned int)kWarps - 1u;
    const unsigned int spare = (total - room + grid - ends - 1u) / (grid - ends);
    if (spare > run) run = spare;
  }
  p.run_chunks = run < 1u ? 1u : (run > 1536u ? 1536u : run);
  return launched(hs, launch_chained(kernel, grid, kThreads, smem, chained, s, p));
}

}  // namespace FO_SHAPE_NS

}  // namespace fo
