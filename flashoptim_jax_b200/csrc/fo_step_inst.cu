// Instantiates one slice of the step-kernel family.  Compiled once per (optimizer, state kind,
// kernel) with -DFO_INST_OPT=<FO_OPT_*> -DFO_INST_KIND=<0 quantized | 1 full | 2 none | 3 any group size>
// -DFO_INST_MODE=<the kernel's features, fo_step.cuh; -1 pieces> -DFO_INST_NAME=<lookup function name>, and -DFO_INST_TILES for
// tile_kernel in place of step_kernel, so the slices build in parallel and each can have its own block size (-DFO_THREADS, -DFO_MIN_BLOCKS_*, and a namespace
// -DFO_SHAPE_NS of its own for what depends on it).
#include "fo_step.cuh"

#if !defined(FO_INST_OPT) || !defined(FO_INST_KIND) || !defined(FO_INST_NAME) || !defined(FO_INST_MODE)
#error "FO_INST_OPT, FO_INST_KIND, FO_INST_MODE and FO_INST_NAME must be defined"
#endif

namespace fo {

#define FO_COMBOS(X) \
  X(FO_BF16, 0) X(FO_BF16, 8) X(FO_BF16, 16) X(FO_F16, 0) X(FO_F16, 8) X(FO_F16, 16) X(FO_F32, 0)

#if FO_INST_MODE == -1
PieceFn FO_INST_NAME(int pdt, int ecc_bits) {
#define X(P, E) \
  if (pdt == P && ecc_bits == E) return &launch_pieces<FO_INST_OPT, P, E, FO_INST_KIND>;
  FO_COMBOS(X)
#undef X
  return nullptr;
}
#else
Launcher FO_INST_NAME(int pdt, int ecc_bits, int gdt) {
  constexpr int most_leaves = (FO_INST_MODE & kOut) != 0 ? kMaxLeavesFlex : kMaxLeaves;
  (void)gdt;
#if FO_INST_KIND == 3
#define X(P, E) \
  if (pdt == P && ecc_bits == E) return Launcher{&launch_generic<FO_INST_OPT, P, E>, 0u, kMaxLeaves, false};
#elif defined(FO_INST_TILES)
  // gradients of the parameter's dtype or fp32, which is what steps have, by kernels of their own
#define X(P, E)                                                                                                       \
  if (pdt == P && ecc_bits == E) {                                                                                    \
    if (gdt == P) return Launcher{&launch_tiles<FO_INST_OPT, P, E, P, FO_INST_MODE>, 1u, most_leaves, true};              \
    if (gdt == FO_F32) return Launcher{&launch_tiles<FO_INST_OPT, P, E, FO_F32, FO_INST_MODE>, 1u, most_leaves, true};    \
    return Launcher{&launch_tiles<FO_INST_OPT, P, E, kAnyGrad, FO_INST_MODE>, 1u, most_leaves, true};                     \
  }
#else
#define X(P, E) \
  if (pdt == P && ecc_bits == E) return Launcher{&launch_main<FO_INST_OPT, P, E, FO_INST_KIND, FO_INST_MODE>, (unsigned int)kChunk, most_leaves, false};
#endif
  FO_COMBOS(X)
#undef X
  return Launcher{nullptr, 0u, 0, false};
}
#endif

}  // namespace fo
