// Template instantiation and dispatch of the all-pairs kernel.  Compiled once
// per precision (LMG_REAL = float | double) so the two halves build in
// parallel.
#include "launch_count.hpp"
#include "mdot_launch.cuh"

#ifndef LMG_REAL
#define LMG_REAL float
#endif

namespace lmg {

namespace {
constexpr int kThreads = 128;

// CTAs that share a target tile.  An SM runs FP64 at the rate of two lanes, so
// a tile's 128 x 128 pairs keep one SM for hundreds of microseconds while a
// small system has fewer tiles than the GPU has SMs: in FP64 each warp of a
// tile is a CTA of its own (the sums of a target are the same, bit for bit).
template <class R> constexpr int kSub = sizeof(R) == 8 ? 4 : 1;

// Packed wall pairs (FP32): up to this many sources a batch, close pairs are
// dealt out over the warp before the sums (kDenseForm); beyond, they are rare and
// are evaluated where they are met, with fewer registers.  Above a wall at one
// particle per unit area, dealt out and in place: N = 300 with torques 52 and
// 64 us, 2048 41 and 45 us, 16384 1475 and 1397 us.
constexpr int kDenseSpan = 4096;

// Outside a solve FP32 batches smaller than a tile take a form of their own (the
// sums of a solve keep their bits, and the compiler contracts other products in
// it): 1 000 000 batches of one above a wall with torques 206 us, 279 in the plain
// form, 125 000 of 8 379 and 474 (forces 243 and 301).
template <class R, int GEOM, bool HF, bool HT, bool ANG, int TPT>
void *kernel_ptr(int form) {
  constexpr int S = TPT == 1 ? kSub<R> : 1;
  if constexpr (sizeof(R) == 4 && HF && HT == ANG) {
    if constexpr (GEOM == kWall && TPT == 1) {
      if (form == kDenseForm)
        return (void *)mdot_kernel<R, GEOM, HF, HT, ANG, TPT, kThreads, S, kDenseForm>;
    }
    if (form == kTinyForm)
      return (void *)mdot_kernel<R, GEOM, HF, HT, ANG, TPT, kThreads, S, kTinyForm>;
  }
  return (void *)mdot_kernel<R, GEOM, HF, HT, ANG, TPT, kThreads, S, kPlainForm>;
}

// kernel pointer for a shape; TPT in {1, 2}
template <class R>
void *select_kernel(const MdotShape &s, int tpt, int form) {
#define LMG_SEL(G, HF, HT, A)                                              \
  if (s.geom == G && s.has_f == HF && s.has_t == HT && s.ang == A)         \
    return tpt == 2 ? kernel_ptr<R, G, HF, HT, A, 2>(form) : kernel_ptr<R, G, HF, HT, A, 1>(form);
  LMG_SEL(kOpen, true, false, false)
  LMG_SEL(kOpen, true, false, true)
  LMG_SEL(kOpen, false, true, true)
  LMG_SEL(kOpen, true, true, true)
  LMG_SEL(kWall, true, false, false)
  LMG_SEL(kWall, true, false, true)
  LMG_SEL(kWall, false, true, true)
  LMG_SEL(kWall, true, true, true)
#undef LMG_SEL
  return nullptr;
}
}  // namespace

template <class R>
cudaError_t mdot_plan(const MdotShape &s, int N, int max_src_span, int num_sms, int force_tpt,
                      int force_split, MdotPlan &plan) {
  plan = MdotPlan{};
  plan.threads = kThreads;
  // FP32: two targets per thread once there are enough targets to keep every
  // SM busy; FP64 stays at one (register pressure, the FP64 pipe is the limit)
  int tpt = 1;
  if (sizeof(R) == 4 && N >= 2 * kThreads * num_sms) tpt = 2;
  if (force_tpt == 1 || force_tpt == 2) tpt = force_tpt;
  plan.tpt = tpt;
  plan.sub = tpt == 1 ? kSub<R> : 1;
  const int bt = kThreads * tpt;
  plan.tiles = (N + bt - 1) / bt;
  // (the splits are planned for the kernel without it, whichever runs)
  void *k = select_kernel<R>(s, tpt, kPlainForm);
  if (!k) return cudaErrorInvalidValue;
  int per_sm = 0;
  cudaError_t e =
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kThreads / plan.sub, 0);
  if (e != cudaSuccess) return e;
  per_sm = std::max(per_sm / plan.sub, 1);
  // two waves of CTAs, and at least 32 CTAs per SM: kernels with few
  // resident CTAs (the wall kernel holds 5 per SM) otherwise lose a large
  // share of the last wave; measured on wall N = 16384 / 65536, 32 splits
  // beat 12 by 7 % and 3 by 10 %
  const long want = std::max(2L * num_sms * per_sm, 32L * num_sms);
  int nsplit = (int)std::max(1L, (want + plan.tiles - 1) / plan.tiles);
  // at least one full source tile per split
  const int max_split = std::max(1, max_src_span / kThreads);
  nsplit = std::min(nsplit, max_split);
  if (force_split > 0) nsplit = force_split;
  nsplit = std::min(nsplit, 65535);
  int chunk = (max_src_span + nsplit - 1) / nsplit;
  chunk = (chunk + kThreads - 1) / kThreads * kThreads;
  if (chunk <= 0) chunk = kThreads;
  nsplit = (max_src_span + chunk - 1) / chunk;
  if (nsplit < 1) nsplit = 1;
  // With few CTAs, a split of several source tiles is cut into one split per
  // tile, and the reduction sums those of a former split first: the same sums
  // bit for bit, on more SMs (a span of 2000 gave 8 splits of 256 sources, one
  // of 2048 gave 16 of 128: N = 2000 wall with torques 54 us, N = 2048 47).
  const long warps = (long)plan.tiles * nsplit * (kThreads / 32);
  if (force_split <= 0 && chunk > kThreads && warps < 8L * num_sms) {
    plan.group = chunk / kThreads;
    chunk = kThreads;
    nsplit = (max_src_span + chunk - 1) / chunk;
  }
  plan.nsplit = nsplit;
  plan.chunk = chunk;
  plan.dense = max_src_span <= kDenseSpan;
  const int nc = s.ang ? 6 : 3;
  plan.part_elems = nsplit > 1 ? (size_t)plan.tiles * nsplit * 2 * nc * bt : 0;
  plan.tickets = nsplit > 1 ? (size_t)plan.tiles * plan.sub : 0;
  return cudaSuccess;
}

template <class R>
cudaError_t mdot_launch(const MdotShape &s, const MdotArgs<R> &args, const MdotPlan &plan,
                        cudaStream_t stream, bool early, bool tiny) {
  const int form = tiny ? kTinyForm : plan.dense ? kDenseForm : kPlainForm;
  void *k = select_kernel<R>(s, plan.tpt, form);
  if (!k) return cudaErrorInvalidValue;
  MdotArgs<R> a = args;
  a.chunk = plan.chunk;
  a.group = plan.group;
  a.part_cap = plan.part_elems;
  a.ticket_cap = plan.tickets;
  dim3 grid(plan.tiles * plan.sub, plan.nsplit);
  void *params[] = {(void *)&a};
  count_launch();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(plan.threads / plan.sub);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelExC(&cfg, k, params);
}

// this translation unit's bounds status (the checked build; 0 otherwise)
#define LMG_STATUS_FN(tag) bounds_status_mdot_##tag
#define LMG_STATUS_NAME(tag) LMG_STATUS_FN(tag)
unsigned long long LMG_STATUS_NAME(LMG_REAL)(bool reset) { return bounds_status_here(reset); }

template cudaError_t mdot_plan<LMG_REAL>(const MdotShape &, int, int, int, int, int, MdotPlan &);
template cudaError_t mdot_launch<LMG_REAL>(const MdotShape &, const MdotArgs<LMG_REAL> &,
                                           const MdotPlan &, cudaStream_t, bool, bool);

}  // namespace lmg
