// Stand-alone codecs over fp32 arrays: the pieces of the step that the reference also
// exposes on their own (quantize_* / dequantize_* of flashoptim_jax/quantization.py,
// split_leaf / reconstruct_leaf of flashoptim_jax/compression.py).  Used for state
// initialisation from existing moments, checkpoint export/import and tests; same device
// arithmetic as the step kernels.
//
// All are bound by memory: a thread owns eight consecutive elements (32-byte fp32 accesses, 8 or 16 bytes on the other
// streams), a group's maximum is a few xor-shuffles, and a pytree's leaves go into one launch.  On 16.8 M elements,
// against one element per thread and group maxima through shared-memory atomics: quantize 114 -> 20 us, dequantize
// 43 -> 17 us; split of a 33.5 M element leaf 46 -> 44 us, but a launch per call instead of one per leaf.
#include "fo_step.cuh"

namespace fo {
int fail(int code, const char* fmt, ...);
constexpr int kCodecThreads = 256;
constexpr unsigned long long kCodecTile = (unsigned long long)kCodecThreads * kPiece;  // elements a block takes at a time

// eight fp32 values as one 32-byte access
FO_DEVI void load8(const float* p, float (&v)[8]) {
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p));
}
// the same, giving way in the L2
FO_DEVI void load8_once(const float* p, float (&v)[8]) {
  asm volatile("ld.global.L1::no_allocate.L2::evict_first.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p));
}
FO_DEVI void store8(float* p, const float (&v)[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]),
               "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}

// Moments that are quantized are not read again, the codes are.  Up to about the size of the L2 the moments therefore give way in it, and what
// dequantizes the codes, or the other moment, finds more of it there.  Both moments quantized and dequantized, 4.2 / 16.8 / 67 M elements: 20.5 / 62.8 / 222 us,
// 19.8 / 59.6 / 223 with loads that give way; 25 / 29 / 33.6 M 90.2 / 105.3 / 116.9 and 87.0 / 102.9 / 114.4.  A single quantization has 21.0 / 25.8 / 27.8 there and 20.0 /
// 25.4 / 27.7, but at 42 / 50 / 67 M 34.0 / 40.1 / 52.5 and 35.0 / 41.6 / 54.6, where the four together still gain 1 % or nothing: the line lies between.  (Blocks that stay and load a tile ahead 21.1 / 67.7 / 254, one
// tile per block 20.4 / 64.8 / 227, blocks of 128 threads 22.0 / 73.3 / 275; the split of fp32 weights 306 and 318 with such loads.)
constexpr unsigned long long kOnce = 1ull << 25;

// Groups of 8 to 256 elements: 1 to 32 lanes.  (The maximum is taken over magnitude bits, so that a NaN survives.)
template <bool VARIANCE>
__global__ void __launch_bounds__(kCodecThreads) quantize_kernel(const float* x, void* values, __half* scales,
                                                                 unsigned long long n, int gshift, int floor_mode, int aligned) {
  using namespace fast2;
  chain_wait();
  chain_release();
  const unsigned long long tiles = (n + kCodecTile - 1) / kCodecTile;
  const int lanes = 1 << (gshift - 3);
  for (unsigned long long t = blockIdx.x; t < tiles; t += gridDim.x) {
    const unsigned long long i0 = t * kCodecTile + threadIdx.x * kPiece;
    const bool whole = i0 + kPiece <= n;
    float v[8];
    if (whole && aligned) {
      if (n <= kOnce) load8_once(x + i0, v);
      else load8(x + i0, v);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = i0 + j < n ? x[i0 + j] : 0.0f;
    }
    if constexpr (VARIANCE) {
      float lo = v[0];
#pragma unroll
      for (int j = 1; j < 8; ++j) lo = fminf(lo, v[j]);
      bool finite = true;
#pragma unroll
      for (int j = 0; j < 8; ++j) finite = finite && v[j] <= 3.0e38f;
      if (lo >= 1.0e-30f && finite) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const f2 r = neg_sqrt_core2(mk(-v[2 * k], -v[2 * k + 1]));
          v[2 * k] = -r.x; v[2 * k + 1] = -r.y;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = fsqrt(v[j]);
      }
    }
    uint32_t top = 0u;
#pragma unroll
    for (int j = 0; j < 8; ++j) top = max(top, __float_as_uint(v[j]) & 0x7FFFFFFFu);
    for (int o = 1; o < lanes; o <<= 1) top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
    const float a = __uint_as_float(top);
    uint32_t q[8];
    if (a >= 1.0e-12f && a <= 1.0e30f) {
      const float y = fast::rcp_rn(a);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const f2 e = mk(v[2 * k], v[2 * k + 1]);
        if constexpr (VARIANCE) quant_v_bits2(mk(-e.x, -e.y), sp(a), sp(-y), q[2 * k], q[2 * k + 1]);
        else softsign_code_bits2(div_by_rcp2(e, sp(-a), sp(y)), q[2 * k], q[2 * k + 1]);
      }
    } else {
      const float safe = ieee::safe_scale(a, floor_mode != 0);
#pragma unroll
      for (int j = 0; j < 8; ++j) q[j] = VARIANCE ? repair_code_v(v[j], safe) : repair_code_m(v[j], safe);
    }
    const uint2 w = make_uint2(pack_bytes(q[0], q[1], q[2], q[3]), pack_bytes(q[4], q[5], q[6], q[7]));
    if (whole && aligned) {
      *(uint2*)((unsigned char*)values + i0) = w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (i0 + j < n) ((unsigned char*)values)[i0 + j] = (unsigned char)((j < 4 ? w.x : w.y) >> (8 * (j & 3)));
    }
    if ((threadIdx.x & (lanes - 1)) == 0 && i0 < n) scales[i0 >> gshift] = __float2half_rn(a);
  }
}

// Any other group size 1..1024: one block per tile of whole groups, group maxima through
// shared-memory atomics on non-negative float bit patterns.
template <bool VARIANCE>
__global__ void __launch_bounds__(256) quantize_any_kernel(const float* x, void* values, __half* scales, unsigned long long n, int G, int floor_mode) {
  chain_wait();
  chain_release();
  __shared__ unsigned int smax[kGenericTile];
  const int groups_per_tile = max(1, kGenericTile / G);
  const int tile = groups_per_tile * G;
  const unsigned long long base = (unsigned long long)blockIdx.x * tile;
  for (int i = threadIdx.x; i < groups_per_tile; i += kCodecThreads) smax[i] = 0u;
  __syncthreads();
  constexpr int kPer = kGenericTile / kCodecThreads;
  float val[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int li = threadIdx.x + k * kCodecThreads;
    const unsigned long long i = base + li;
    val[k] = 0.0f;
    if (li < tile && i < n) {
      float v = x[i];
      val[k] = VARIANCE ? fast::sqrt_rn(v) : v;
      atomicMax(&smax[li / G], __float_as_uint(fabsf(val[k])));
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int li = threadIdx.x + k * kCodecThreads;
    const unsigned long long i = base + li;
    if (li < tile && i < n) {
      const float a = __uint_as_float(smax[li / G]);
      const fast::GroupScale gs = fast::group_scale(a, floor_mode != 0);
      if (VARIANCE) ((unsigned char*)values)[i] = (unsigned char)fast::quant_v(val[k], gs);
      else ((signed char*)values)[i] = (signed char)fast::quant_m(val[k], gs);
      if (li % G == 0) scales[i / G] = __float2half_rn(a);
    }
  }
}

template <bool VARIANCE>
FO_DEVI float dequantize_one(unsigned int b, float sc) {
  if (VARIANCE) {
    const float s = fmul(ieee::deq_v_norm((int)b), sc);
    return fmul(s, s);
  }
  return fmul(__ldg(&kDeqM.v[b]), sc);
}

// Groups of 2^gshift = 8 to 256 elements, aligned arrays: whole pieces lie in one group.
template <bool VARIANCE>
__global__ void __launch_bounds__(kCodecThreads) dequantize_kernel(const void* values, const __half* scales, float* out, unsigned long long n, int gshift) {
  using namespace fast2;
  chain_wait();
  chain_release();
  const unsigned long long tiles = (n + kCodecTile - 1) / kCodecTile;
  for (unsigned long long t = blockIdx.x; t < tiles; t += gridDim.x) {
    const unsigned long long i0 = t * kCodecTile + threadIdx.x * kPiece;
    if (i0 + kPiece <= n) {
      const uint2 w = *(const uint2*)((const unsigned char*)values + i0);
      const uint32_t word[2] = {w.x, w.y};
      const f2 sc = sp(__half2float(scales[i0 >> gshift]));
      float v[8];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        f2 e;
        if constexpr (VARIANCE) {
          e = mul2(codes_over_255(word[k >> 1], 2 * (k & 1)), sc);
          e = mul2(e, e);
        } else {
          e = mul2(LutGlobal{}.pair(word[k >> 1], 2 * (k & 1)), sc);
        }
        v[2 * k] = e.x; v[2 * k + 1] = e.y;
      }
      store8(out + i0, v);
    } else {
      for (int j = 0; j < 8; ++j)
        if (i0 + j < n) out[i0 + j] = dequantize_one<VARIANCE>(((const unsigned char*)values)[i0 + j], __half2float(scales[(i0 + j) >> gshift]));
    }
  }
}

// Any other group size, and arrays that are not aligned: one element per thread at a time, neighbours side by side; a shift for
// powers of two (gshift >= 0), else one wide division per tile and a narrow one per element.  A kernel of its own, so that the one above keeps its registers.  (Eight elements in a row per thread took twice
// as long: 16.8 M elements in groups of 48 69 us, this 36; unaligned in groups of 32 69 and 21.)
template <bool VARIANCE>
__global__ void __launch_bounds__(kCodecThreads) dequantize_any_kernel(const void* values, const __half* scales, float* out, unsigned long long n, unsigned int G, int gshift) {
  chain_wait();
  chain_release();
  const unsigned long long tiles = (n + kCodecTile - 1) / kCodecTile;
  for (unsigned long long t = blockIdx.x; t < tiles; t += gridDim.x) {
    const unsigned long long base = t * kCodecTile, group = gshift >= 0 ? base >> gshift : base / G;
    const uint32_t rest = (uint32_t)(base - group * G) + threadIdx.x;  // below 2^31 + 2^8: the group size is an int
    unsigned int code[8];
    float sc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const unsigned long long i = base + j * kCodecThreads + threadIdx.x;
      if (i < n) {
        code[j] = ((const unsigned char*)values)[i];
        const uint32_t r = rest + j * kCodecThreads;
        sc[j] = __half2float(scales[group + (gshift >= 0 ? r >> gshift : r / G)]);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const unsigned long long i = base + j * kCodecThreads + threadIdx.x;
      if (i < n) out[i] = dequantize_one<VARIANCE>(code[j], sc[j]);
    }
  }
}

// ---- fp32 <-> (16-bit parameter, ECC), a table of leaves per launch --------------------------------------------
// Two table sizes: a launch copies its whole parameter block (9.5 KB of the large one), which shows on a call for a leaf or two:
// 100 000 elements 5.9 us with the large table, 4.2 with the small one.
constexpr int kSplitLeavesSmall = 8, kSplitLeaves = 256;
template <int N>
struct SplitParams {
  FoSplitLeaf leaf[N];
  uint32_t first_tile[N + 1];
  int32_t n_leaves;
};

template <int PDT, int ECC_BITS>
FO_DEVI void split_one(const FoSplitLeaf& L, const unsigned long long i, const float theta) {
  uint32_t nb;
  int e = 0;
  if constexpr (ECC_BITS != 0) fast::split<PDT, ECC_BITS>(theta, nb, e);
  else nb = Lp<PDT>::from_f32(theta);
  ((unsigned short*)L.lp)[i] = (unsigned short)nb;
  if constexpr (ECC_BITS == 16) ((short*)L.ecc)[i] = (short)e;
  if constexpr (ECC_BITS == 8) ((signed char*)L.ecc)[i] = (signed char)e;
}
template <int PDT, int ECC_BITS>
FO_DEVI float reconstruct_one(const uint32_t bits, const int e) {
  if constexpr (ECC_BITS != 0) return fast::reconstruct<PDT, ECC_BITS>(bits, e);
  else return Lp<PDT>::to_f32(bits);
}
template <int ECC_BITS>
FO_DEVI int code_at(const void* ecc, const unsigned long long i) {
  if constexpr (ECC_BITS == 16) return ((const short*)ecc)[i];
  if constexpr (ECC_BITS == 8) return ((const signed char*)ecc)[i];
  return 0;
}

// A leaf that is not aligned: one element per thread at a time, neighbours side by side, eight loads in flight.  A launch per
// leaf, in kernels of their own, so that those below keep their registers.  (Eight elements in a row per thread took twice as
// long: 16.8 M elements with 16-bit codes 87 us split and 71 reconstructed, this 25 and 26.)
template <int PDT, int ECC_BITS>
__global__ void __launch_bounds__(kCodecThreads) split_unaligned_kernel(const FoSplitLeaf L) {
  chain_wait();
  chain_release();
  for (unsigned long long base = blockIdx.x * kCodecTile + threadIdx.x; base < L.n; base += gridDim.x * kCodecTile) {
    float theta[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (base + j * kCodecThreads < L.n) theta[j] = L.theta[base + j * kCodecThreads];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (base + j * kCodecThreads < L.n) split_one<PDT, ECC_BITS>(L, base + j * kCodecThreads, theta[j]);
  }
}
template <int PDT, int ECC_BITS>
__global__ void __launch_bounds__(kCodecThreads) reconstruct_unaligned_kernel(const FoSplitLeaf L) {
  chain_wait();
  chain_release();
  for (unsigned long long base = blockIdx.x * kCodecTile + threadIdx.x; base < L.n; base += gridDim.x * kCodecTile) {
    uint32_t bits[8];
    int e[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const unsigned long long i = base + j * kCodecThreads;
      if (i < L.n) {
        bits[j] = ((const unsigned short*)L.lp)[i];
        e[j] = code_at<ECC_BITS>(L.ecc, i);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (base + j * kCodecThreads < L.n) L.theta[base + j * kCodecThreads] = reconstruct_one<PDT, ECC_BITS>(bits[j], e[j]);
  }
}

template <int PDT, int ECC_BITS, int N>
__global__ void __launch_bounds__(kCodecThreads) split_kernel(const __grid_constant__ SplitParams<N> p) {
  chain_wait();
  chain_release();
  const uint32_t total = p.first_tile[p.n_leaves];
  for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {
    const int l = leaf_of(p.first_tile, p.n_leaves, t);
    const FoSplitLeaf& L = p.leaf[l];
    const unsigned long long i0 = (unsigned long long)(t - p.first_tile[l]) * kCodecTile + threadIdx.x * kPiece;
    if (i0 + kPiece <= L.n) {
      float v[8];
      load8(L.theta + i0, v);
      uint32_t nw[4];
      uint4 e;
      float2 theta[4];
      uint32_t hi = 0u;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        theta[k] = make_float2(v[2 * k], v[2 * k + 1]);
        hi = max(hi, max(__float_as_uint(v[2 * k]) & 0x7FFFFFFFu, __float_as_uint(v[2 * k + 1]) & 0x7FFFFFFFu));
      }
      stored_form<true, PDT, ECC_BITS>(theta, nw, e);
      if (ECC_BITS != 0 && hi > 0x7E967699u) {  // above 1e38, or not finite: beyond the packed shortcut's range
        uint32_t ew[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) ew[j] = (uint32_t)repair_ecc<PDT, ECC_BITS>(v[j]);
        if constexpr (ECC_BITS == 16) e = make_uint4(pack_halves(ew[0], ew[1]), pack_halves(ew[2], ew[3]), pack_halves(ew[4], ew[5]), pack_halves(ew[6], ew[7]));
        else e = make_uint4(pack_bytes(ew[0], ew[1], ew[2], ew[3]), pack_bytes(ew[4], ew[5], ew[6], ew[7]), 0u, 0u);
      }
      *(uint4*)((unsigned short*)L.lp + i0) = make_uint4(nw[0], nw[1], nw[2], nw[3]);
      if constexpr (ECC_BITS == 16) *(uint4*)((short*)L.ecc + i0) = e;
      if constexpr (ECC_BITS == 8) *(uint2*)((signed char*)L.ecc + i0) = make_uint2(e.x, e.y);
    } else {
      for (unsigned long long i = i0; i < L.n && i < i0 + kPiece; ++i) split_one<PDT, ECC_BITS>(L, i, L.theta[i]);
    }
  }
}

template <int PDT, int ECC_BITS, int N>
__global__ void __launch_bounds__(kCodecThreads) reconstruct_kernel(const __grid_constant__ SplitParams<N> p) {
  chain_wait();
  chain_release();
  const uint32_t total = p.first_tile[p.n_leaves];
  for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {
    const int l = leaf_of(p.first_tile, p.n_leaves, t);
    const FoSplitLeaf& L = p.leaf[l];
    const unsigned long long i0 = (unsigned long long)(t - p.first_tile[l]) * kCodecTile + threadIdx.x * kPiece;
    if (i0 + kPiece <= L.n) {
      const uint4 w = *(const uint4*)((const unsigned short*)L.lp + i0);
      uint4 e = make_uint4(0u, 0u, 0u, 0u);
      if constexpr (ECC_BITS == 16) e = *(const uint4*)((const short*)L.ecc + i0);
      if constexpr (ECC_BITS == 8) {
        const uint2 x = *(const uint2*)((const signed char*)L.ecc + i0);
        e.x = x.x; e.y = x.y;
      }
      float2 theta[4];
      unpack_master<true, PDT, ECC_BITS>(w, make_uint4(0u, 0u, 0u, 0u), e, theta);
      float v[8];
#pragma unroll
      for (int k = 0; k < 4; ++k) { v[2 * k] = theta[k].x; v[2 * k + 1] = theta[k].y; }
      store8((float*)L.theta + i0, v);
    } else {
      for (unsigned long long i = i0; i < L.n && i < i0 + kPiece; ++i)
        L.theta[i] = reconstruct_one<PDT, ECC_BITS>(((const unsigned short*)L.lp)[i], code_at<ECC_BITS>(L.ecc, i));
    }
  }
}

// enough blocks to fill the device several times over, each a few tiles
static unsigned int tile_grid(unsigned long long tiles) {
  const unsigned long long cap = 148ull * 8ull * 4ull;
  return (unsigned int)(tiles < cap ? (tiles ? tiles : 1) : cap);
}
// The same for the kernels that write half of what they read or more (splitting, reconstructing, dequantizing): above two tiles per block, 9472 tiles, blocks of two.  In
// us, with the grid above and so: split without codes 71 M elements 64.6 and 62.2, 160 M 144 and 138, back 67.5 and 64.9, 151 and 143;
// split into 8- / 16-bit codes 71 M elements 77.0 / 88.2 and 75.7 / 84.2, 160 M 174 / 201 and 167 / 187; reconstructed from them 79.1 / 86.7 and 77.1 / 83.7, 177 / 195
// and 171 / 187; moments dequantized 71 M 60.2 / 59.6 and 56.7 / 55.4.  25 M elements differ by 1 %, 16.8 M (1.7 tiles per block) have 18.6 / 20.3 and with blocks
// of two 19.1 / 21.0.  Blocks of three and four tiles are no better.  Quantizing, which writes a quarter, is slower so: 71 M 55.9 / 59.8 and 56.9 / 61.1, 160 M 126 / 138 and 134 / 146.
static unsigned int write_grid(unsigned long long tiles) {
  const unsigned int grid = tile_grid(tiles);
  return tiles > 2ull * grid ? (unsigned int)((tiles < 0x7FFFFFFFull ? tiles + 1ull : 0x7FFFFFFFull) / 2ull) : grid;
}
static bool aligned_to(const void* p, unsigned long long a) { return ((uintptr_t)p & (a - 1)) == 0; }
// log2 of a group size of 8, 16, ..., 256; else 0
static int small_group_shift(int G) {
  for (int s = 3; s <= 8; ++s)
    if (G == 1 << s) return s;
  return 0;
}

// The kernels of this file begin with chain_wait().  (Their pointers are not __restrict__: loads through the read-only
// path may be moved in front of it.)
template <typename... P, typename... A>
static int launch_codec(const char* what, void (*kernel)(P...), unsigned int grid, void* stream, const A&... args) {
  bool chained = true;
  const cudaError_t e = launch_chained<P...>(kernel, grid, (unsigned int)kCodecThreads, 0, chained, (cudaStream_t)stream, static_cast<const P&>(args)...);
  if (e != cudaSuccess) return fail(FO_ERR_CUDA, "%s: launch failed: %s", what, cudaGetErrorString(e));
  return FO_OK;
}

template <bool VARIANCE>
static int quantize_entry(const float* x, void* values, void* scales, uint64_t n, int32_t G, int32_t floor_mode, void* stream,
                          const char* what) {
  if (n == 0) return FO_OK;
  if (x == nullptr || values == nullptr || scales == nullptr) return fail(FO_ERR_INVALID_ARG, "%s: null pointer", what);
  if (G < 1) return fail(FO_ERR_INVALID_ARG, "%s: group_size %d", what, G);
  if (G > kGenericTile) return fail(FO_ERR_UNSUPPORTED, "%s: group_size %d > %d", what, G, kGenericTile);
  if (const int gshift = small_group_shift(G)) {
    const int aligned = aligned_to(x, 32) && aligned_to(values, 8);
    return launch_codec(what, quantize_kernel<VARIANCE>, tile_grid((n + kCodecTile - 1) / kCodecTile), stream, x, values, (__half*)scales, n, gshift, floor_mode, aligned);
  }
  const unsigned long long tile = (unsigned long long)(kGenericTile / G) * G;
  const unsigned long long blocks = (n + tile - 1) / tile;
  if (blocks > 0x7FFFFFFFull) return fail(FO_ERR_TOO_LARGE, "%s: %llu elements exceed one launch", what, (unsigned long long)n);
  return launch_codec(what, quantize_any_kernel<VARIANCE>, (unsigned int)blocks, stream, x, values, (__half*)scales, n, G, floor_mode);
}

template <bool VARIANCE>
static int dequantize_entry(const void* values, const void* scales, float* out, uint64_t n, int32_t G, void* stream,
                            const char* what) {
  if (n == 0) return FO_OK;
  if (values == nullptr || scales == nullptr || out == nullptr) return fail(FO_ERR_INVALID_ARG, "%s: null pointer", what);
  if (G < 1) return fail(FO_ERR_INVALID_ARG, "%s: group_size %d", what, G);
  const unsigned long long tiles = (n + kCodecTile - 1) / kCodecTile;
  const unsigned int grid = tile_grid(tiles);
  const int gshift = small_group_shift(G);
  if (gshift != 0 && aligned_to(out, 32) && aligned_to(values, 8))
    return launch_codec(what, dequantize_kernel<VARIANCE>, write_grid(tiles), stream, values, (const __half*)scales, out, n, gshift);
  int power = 30;
  while (power >= 0 && G != 1 << power) --power;
  return launch_codec(what, dequantize_any_kernel<VARIANCE>, grid, stream, values, (const __half*)scales, out, n, (unsigned int)G, power);
}

template <int N>
static int split_table(const FoSplitLeaf* leaves, uint32_t n_leaves, int32_t pdt, int32_t ecc_bits, void* stream, bool split, const char* what) {
  void (*kernel)(const SplitParams<N>) = nullptr;
  void (*unaligned)(const FoSplitLeaf) = nullptr;
#define X(P, E)                                                                            \
  if (pdt == P && ecc_bits == E) {                                                         \
    kernel = split ? split_kernel<P, E, N> : reconstruct_kernel<P, E, N>;                  \
    unaligned = split ? split_unaligned_kernel<P, E> : reconstruct_unaligned_kernel<P, E>; \
  }
  X(FO_BF16, 0) X(FO_BF16, 8) X(FO_BF16, 16) X(FO_F16, 0) X(FO_F16, 8) X(FO_F16, 16)
#undef X
  if (kernel == nullptr) return fail(FO_ERR_INVALID_ARG, "%s: param_dtype %d with ecc_bits %d", what, pdt, ecc_bits);
  SplitParams<N> p;  // filled as far as it is used
  p.n_leaves = 0;
  unsigned long long tiles = 0;
  for (uint32_t i = 0; i <= n_leaves; ++i) {
    const unsigned long long more = i < n_leaves ? (leaves[i].n + kCodecTile - 1) / kCodecTile : 0ull;
    if (more > 0x7FFFFFFFull) return fail(FO_ERR_TOO_LARGE, "%s: leaf %u with %llu elements exceeds one launch", what, i, (unsigned long long)leaves[i].n);
    if (p.n_leaves > 0 && (i == n_leaves || p.n_leaves == N || tiles + more > 0x7FFFFFFFull)) {
      p.first_tile[p.n_leaves] = (uint32_t)tiles;
      if (int rc = launch_codec(what, kernel, write_grid(tiles), stream, p)) return rc;
      p.n_leaves = 0;
      tiles = 0;
    }
    if (i == n_leaves || leaves[i].n == 0) continue;
    const FoSplitLeaf& L = leaves[i];
    if (L.theta == nullptr || L.lp == nullptr || (ecc_bits != 0 && L.ecc == nullptr)) return fail(FO_ERR_INVALID_ARG, "%s: null pointer", what);
    if (!(aligned_to(L.theta, 32) && aligned_to(L.lp, 16) && aligned_to(L.ecc, 16))) {
      if (int rc = launch_codec(what, unaligned, tile_grid(more), stream, L)) return rc;
      continue;
    }
    p.leaf[p.n_leaves] = L;
    p.first_tile[p.n_leaves] = (uint32_t)tiles;
    tiles += more;
    ++p.n_leaves;
  }
  return FO_OK;
}
static int split_entry(const FoSplitLeaf* leaves, uint32_t n_leaves, int32_t pdt, int32_t ecc_bits, void* stream, bool split, const char* what) {
  if (n_leaves > 0 && leaves == nullptr) return fail(FO_ERR_INVALID_ARG, "%s: null table", what);
  return n_leaves <= kSplitLeavesSmall ? split_table<kSplitLeavesSmall>(leaves, n_leaves, pdt, ecc_bits, stream, split, what)
                                       : split_table<kSplitLeaves>(leaves, n_leaves, pdt, ecc_bits, stream, split, what);
}

}  // namespace fo

using namespace fo;

extern "C" int fo_quantize_momentum(const float* x, int8_t* values, void* scales, uint64_t n, int32_t G, int32_t floor_mode,
                                    void* stream) {
  return quantize_entry<false>(x, values, scales, n, G, floor_mode, stream, "fo_quantize_momentum");
}
extern "C" int fo_quantize_variance(const float* x, uint8_t* values, void* scales, uint64_t n, int32_t G, int32_t floor_mode,
                                    void* stream) {
  return quantize_entry<true>(x, values, scales, n, G, floor_mode, stream, "fo_quantize_variance");
}
extern "C" int fo_dequantize_momentum(const int8_t* values, const void* scales, float* out, uint64_t n, int32_t G, void* stream) {
  return dequantize_entry<false>(values, scales, out, n, G, stream, "fo_dequantize_momentum");
}
extern "C" int fo_dequantize_variance(const uint8_t* values, const void* scales, float* out, uint64_t n, int32_t G, void* stream) {
  return dequantize_entry<true>(values, scales, out, n, G, stream, "fo_dequantize_variance");
}

extern "C" int fo_split(const float* theta, void* lp, void* ecc, int32_t pdt, int32_t ecc_bits, uint64_t n, void* stream) {
  if (n == 0) return FO_OK;
  const FoSplitLeaf leaf = {const_cast<float*>(theta), lp, ecc, n};
  return split_entry(&leaf, 1, pdt, ecc_bits, stream, true, "fo_split");
}
extern "C" int fo_reconstruct(const void* lp, const void* ecc, float* theta, int32_t pdt, int32_t ecc_bits, uint64_t n,
                              void* stream) {
  if (n == 0) return FO_OK;
  const FoSplitLeaf leaf = {theta, const_cast<void*>(lp), const_cast<void*>(ecc), n};
  return split_entry(&leaf, 1, pdt, ecc_bits, stream, false, "fo_reconstruct");
}
extern "C" int fo_split_many(const FoSplitLeaf* leaves, uint32_t n_leaves, int32_t pdt, int32_t ecc_bits, void* stream) {
  return split_entry(leaves, n_leaves, pdt, ecc_bits, stream, true, "fo_split_many");
}
extern "C" int fo_reconstruct_many(const FoSplitLeaf* leaves, uint32_t n_leaves, int32_t pdt, int32_t ecc_bits, void* stream) {
  return split_entry(leaves, n_leaves, pdt, ecc_bits, stream, false, "fo_reconstruct_many");
}
