// fp32 convolutions on the tensor cores without threads in the operand path: y = act(conv(x, W) + b + residual) with every
// product formed as three TF32 MMAs (x = x_hi + x_lo, W = W_hi + W_lo: hi.hi, hi.lo and lo.hi; the hi.hi sums taken over into
// registers every 32 k with IEEE additions, the cross sums scaled by 2^10), both operands read from shared memory where the
// TMA puts them.
//
// Replaces, for layers of 128 products and more, the reference's cuDNN lowerings fortis_conv2d / fortis_conv3d
// (runtime/fortis_rt.c:108-156) and the further kernels for bias, residual and activation (compiler/FortisFuse.cpp:626-655).
//
// Activations lie in HBM as a SPLIT VOLUME: channels last, every value already split, [plane hi | lo][row][channels], one row per
// position of a grid that holds the zero padding:
//     row = ((n * Dq + d) * Hq + h) * Wq + w,      output (od, oh, ow) under tap (kd, kh, kw) reads row(out) + shift(tap)
// For stride 1 a line's right padding is the next line's left padding (Wq = W + pad; the same for planes and volumes); for other
// strides there is one such volume per residue of the position modulo the stride ("phase"), so that a tap is a shift again.  So an
// operand tile is 128 consecutive rows, whatever the tap: no im2col, no masks, no bounds tests; rows that are padding are computed
// too and written as zeros (the next layer's padding) or not at all.
//
//   * pairs of CTAs (cta_group::2), 128 rows each; a pair's leader issues the MMAs.  A stage of the activation ring holds the rows
//     that all taps of one kd (or of one line, or one tap) read, 32 channels, hi and lo: taps read it through descriptors whose start
//     address moves by whole rows (the 128-byte swizzle is a function of the address).
//   * kernels three wide (LINE): one step multiplies the unshifted rows by the three taps of a line (N = 3 x 32 or 3 x 64 columns), and
//     the epilogue adds the sums of neighbouring rows: an activation is read once for three taps, and lines need no padding.
//     Others: one tap a step, x_hi . [W_hi | W_lo] as one MMA of twice the columns.
//   * eight epilogue warps (thread = row, half of the features) hold the sums in registers and put finished rows into a stash in
//     shared memory; four more warps add bias and residual, activate, split and store whole lines.
// Bound: with 64 features the tensor core, 1152 clk a step of 3 taps x 32 channels, plus some 3000 clk at a tile's end, when the next
// tile's second step waits for the epilogue (a step was measured at 1160); with few features and channels the tile's end.
// Measured against the kernel before, whose threads loaded the taps and split them once per tap (a step of one tap 1240 clk): see
// conv_layer in fortis_conv3d.cu.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <string>
#include <type_traits>

#include "fortis_device.cuh"
#include "fortis_kernels.h"
#include "fortis_model.h"
#include "fortis_tc.cuh"

namespace fortis {

namespace {

using namespace tc;

constexpr int kM = 128, kKt = 32;
// The tensor core takes subnormal operands as zero: x_lo is stored times 2^10 (exact), so that it is normal wherever x is, and the
// cross sums are multiplied by 2^-10.  Without it x_lo is lost from |x| < 2^-102 on (2^-118: error 2.2e-6).  (x_lo is below 2^-10 of
// the largest value, so the product stays finite.)
constexpr float kLoScale = 1024.f;
// The tensor core truncates as it accumulates, so the sums are taken over after every step of 32 k (14-layer network: error against 64 bits
// 1.02e-6, every 64 k 1.66e-6; FFMA 2.5e-6).
// warps: 0 activations, 1 weights (TMA), 2 and 3 MMA issuers, then the epilogue and the storers
constexpr int kEWarps = 8, kWarpE0 = 4, kWarpS0 = kWarpE0 + kEWarps, kThreads = (kWarpS0 + 4) * 32;
constexpr int kMaxStages = 8;
// A turn barrier is used again a weight ring later, which the first issuer cannot reach before the second has issued the step and let go
// of its weights.  Where the weights stay it is kTurns steps, and the first can be ahead by the tile's steps and the next tile's first two
// (two accumulators, and the epilogue ends a tile with the second issuer's sums).
constexpr int kTurns = 8, kMaxResident = kTurns - 2;
constexpr int kBarBytes = 512;
constexpr int kSmemMax = 227 * 1024;
enum { VST_A_FULL = 21, VST_A_EMPTY = 22, VST_ACC_FULL = 23, VST_ACC_EMPTY = 24, VST_ALIGN = 25, VST_W_FULL = 26, VST_W_EMPTY = 27, VST_STASH_FULL = 28,
       VST_STASH_EMPTY = 29 };                 // as the other fp32 kernel numbers its waits

struct VolParams {
  CUtensorMap amap;                            // [plane 2][row][channel], box 2 x box_rows x 32
  CUtensorMap wmap;                            // [step][channel block][tile of features][CTA][row] rows of 32
  VolGeom g;
  int nchb, ntn;
  int ng, tpg, sub_w;                          // stages per channel block, steps per stage, steps of one line among them
  int box_rows, a_stages, w_stages;
  // the rows in pieces (the whole volume, or the images of a batch) of `rows` output rows up to the last one that is a real output,
  // piece_stride apart, each in pairs of tiles of its own
  int pieces, pairs_piece; long long rows, piece_stride;
  const float* bias; int act; float slope; int F;
  // output: a split volume of the same grid (pitch: channels of a row) ...
  float* out; long long out_plane; int out_pitch; long long out_shift;
  int remap; VolMap next;                      // ... or one of another grid, the next layer's, whose padding is zero already
  const float* skip;                           // the residual, a split volume like `out`
  // ... or a plain array, with a plain residual
  float* y; long long ys_n, ys_d, ys_h, ys_w, ys_c;
  const float* res; long long rs_n, rs_d, rs_h, rs_w, rs_c;
  int* status;
  unsigned int wait_limit; int test_skip_stage;
};

__host__ __device__ constexpr uint32_t idesc_tf32_pair(int n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)((2 * kM) >> 4) << 24);
}
// Low words of K-major 128-byte-swizzled shared-memory descriptors; the high word is the same for all of them
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return (saddr >> 4) & 0x3FFFu; }
// D[tmem of both CTAs] (+)= A . B^T over a step of 32 k (FULL), or its first nk8 < 4 parts of 8 k (32 bytes of a row each), one
// elected lane of the leader issues
template <uint32_t IDESC, bool FULL>
__device__ __forceinline__ void mma_step32(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t accumulate, int nk8) {
  if constexpr (FULL)
    asm volatile(
        "{\n\t.reg .pred e, q;\n\t.reg .b64 a0, a1, a2, a3, b0, b1, b2, b3;\n\t"
        "mov.b64 a0, {%1, %4};\n\tmov.b64 b0, {%2, %4};\n\t"
        "add.s64 a1, a0, 2;\n\tadd.s64 b1, b0, 2;\n\tadd.s64 a2, a0, 4;\n\tadd.s64 b2, b0, 4;\n\tadd.s64 a3, a0, 6;\n\tadd.s64 b3, b0, 6;\n\t"
        "setp.ne.b32 q, %5, 0;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.mma.cta_group::2.kind::tf32 [%0], a0, b0, %3, q;\n\t"
        "@e tcgen05.mma.cta_group::2.kind::tf32 [%0], a1, b1, %3, 1;\n\t"
        "@e tcgen05.mma.cta_group::2.kind::tf32 [%0], a2, b2, %3, 1;\n\t"
        "@e tcgen05.mma.cta_group::2.kind::tf32 [%0], a3, b3, %3, 1;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "n"(IDESC), "n"(kDescHi), "r"(accumulate) : "memory");
  else
    for (int j = 0; j < nk8; j++)
      asm volatile(
          "{\n\t.reg .pred e, q;\n\t.reg .b64 a0, b0;\n\tmov.b64 a0, {%1, %4};\n\tmov.b64 b0, {%2, %4};\n\t"
          "setp.ne.b32 q, %5, 0;\n\telect.sync _|e, 0xffffffff;\n\t"
          "@e tcgen05.mma.cta_group::2.kind::tf32 [%0], a0, b0, %3, q;\n\t}"
          ::"r"(d_tmem), "r"(a_lo + 2 * j), "r"(b_lo + 2 * j), "n"(IDESC), "n"(kDescHi), "r"(accumulate | (uint32_t)j) : "memory");
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {     // two IEEE additions
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
  return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)),
      "l"(*reinterpret_cast<unsigned long long*>(&c)));
  return *reinterpret_cast<float2*>(&d);
}
// A bounded wait without a function call, which would empty the uniform registers and fix one register budget for all warps.  Every
// lane of a warp goes on or gives up together; a CTA in which a wait has given up polls no more.
__device__ __forceinline__ bool wait_polling(uint32_t bar, uint32_t parity, uint32_t limit, volatile int* abort_flag, int* status, int code) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .u32 i;\n\tmov.u32 i, 0;\n"
      "WAIT_LOOP_%=:\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "@p bra WAIT_DONE_%=;\n\t"
      "add.u32 i, i, 1;\n\t"
      "setp.lt.u32 q, i, %3;\n\t"
      "@q bra WAIT_LOOP_%=;\n"
      "WAIT_DONE_%=:\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity), "r"(*abort_flag ? 1u : limit) : "memory");
  if (__all_sync(0xffffffffu, ok)) return true;
  if ((threadIdx.x & 31) == 0) {
    *abort_flag = 1;
    atomicCAS(status, 0, code);
  }
  return false;
}
__device__ __forceinline__ float4 ld_plain4(const float* p) {   // not read-only: the grid in front may have written it
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_plain(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ void drain_wait(uint32_t bar, uint32_t parity, uint32_t limit) {
  for (uint32_t i = 0; i < limit; i++)
    if (mbar_try_wait(bar, parity)) return;
}

// LINE: a step is the three taps of a line, and a tile has 126 output rows (the first and last computed ones only feed their
// neighbours).  Otherwise a step is one tap.
template <int NT, bool LINE> struct Form {
  static constexpr int kTaps = LINE ? 3 : 1;
  static constexpr int kRowsOut = LINE ? kM - 2 : kM, kHalo = LINE ? 1 : 0;
  static constexpr int kWRows = LINE ? 3 * NT : NT;            // weight rows of a step held by one CTA, W_hi then W_lo
  static constexpr int kWBytes = kWRows * kKt * 4;
  // tensor memory: two accumulators of kAcc columns, then the cross sums.  The accumulators take alternate steps, or where there is
  // no room for two (kHalves) 32 features each.
  static constexpr bool kHalves = LINE && NT == 64;
  static constexpr int kAcc = LINE ? 96 : 2 * NT, kCross = LINE ? 3 * NT : NT;
  static constexpr uint32_t kColCross = 2 * kAcc;
  static_assert(2 * kAcc + kCross <= 512, "tensor memory");
  // LINE: a half's 96 rows (3 taps x 32 features) lie 48 in each CTA; the columns of the cross sums follow
  static __device__ __forceinline__ int cross_col(int half, int n) { return kHalves ? (n < 48 ? half * 48 + n : half * 48 + n + 48) : n; }
  static constexpr int kXchBytes = LINE ? 2 * 4 * NT * 4 : 0;          // rows exchanged between epilogue warps: [up | down][quadrant][feature]
};

// first row of stage g_ relative to the output row
template <bool LINE>
__device__ __forceinline__ long long stage_shift(const VolParams& P, int g_) {
  const VolGeom& g = P.g;
  const int nw = LINE ? 1 : g.KW, per_kd = P.tpg == g.KH * nw ? 1 : P.tpg == nw ? g.KH : g.KH * nw;      // stages of one kd
  const int kd = g_ / per_kd, r = g_ - kd * per_kd, kh = per_kd == 1 ? 0 : P.tpg == nw ? r : r / nw, kw = P.tpg == 1 ? r % nw : 0;
  const int phase = ((kd % g.sd) * g.fh + kh % g.sh) * g.fw + kw % g.sw;
  return phase * g.P + ((long long)(g.od0 + kd / g.sd) * g.Hq + g.oh0 + kh / g.sh) * g.Wq + g.ow0 + (LINE ? 1 : kw / g.sw);
}

// RESIDENT: the weight ring holds all steps of a tile and is loaded once
template <int NT, bool LINE, bool RESIDENT>
__global__ void __launch_bounds__(kThreads, 1) __cluster_dims__(2, 1, 1) conv_vol_kernel(const __grid_constant__ VolParams P) {
  using FM = Form<NT, LINE>;
  constexpr int kWBytes = FM::kWBytes;
  constexpr int NH = NT / 2;                                   // features per epilogue thread
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t base = smem_u32(smem);
  if (base & 1023u) {                                          // the same in both CTAs of a pair
    if (threadIdx.x == 0) atomicCAS(P.status, 0, VST_ALIGN);
    return;
  }
  const uint32_t a_plane = (uint32_t)P.box_rows * kKt * 4, a_bytes = 2 * a_plane;
  const uint32_t w_ring = base + P.a_stages * a_bytes, bars = w_ring + P.w_stages * kWBytes;
  uint8_t* tail = smem + (bars - base);
  // a_full [8] | a_empty [8] | w_full [8] | w_empty [8] | acc_full [2] | acc_empty [2] | cross_full | cross_empty | drained [2];
  // at 320 the tensor-memory base, at 324 the abort flag, at 328 turn [8] | stash_full | stash_empty
  const uint32_t a_full = bars, a_empty = bars + 64, w_full = bars + 128, w_empty = bars + 192, acc_full = bars + 256, acc_empty = bars + 272,
                 cross_full = bars + 288, cross_empty = bars + 296, drained = bars + 304, turn = bars + 328, stash_full = bars + 392, stash_empty = bars + 400;
  uint32_t* tmem_slot = (uint32_t*)(tail + 320);
  volatile int* abort_flag = (volatile int*)(tail + 324);
  // through a shuffle, so that the compiler knows the roles' branches, loops and addresses to be the same in a whole warp
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank();
  const long long ntiles = (long long)P.pieces * P.pairs_piece * P.ntn;
  // a tile's piece and its first computed row there
  auto piece_of = [&](long long t) { return (uint32_t)(t / P.ntn) / (uint32_t)P.pairs_piece; };
  auto first_row = [&](long long t, uint32_t piece) {
    return (2 * ((long long)(uint32_t)(t / P.ntn) - (long long)piece * P.pairs_piece) + crank) * FM::kRowsOut - FM::kHalo;
  };
  const long long t0 = blockIdx.x >> 1, t_step = gridDim.x >> 1;
  const int nkt = P.ng * P.tpg * P.nchb;       // steps of a tile

  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxStages; s++) {
      mbar_init(a_full + 8 * s, 1); mbar_init(a_empty + 8 * s, 2);
      mbar_init(w_full + 8 * s, 1); mbar_init(w_empty + 8 * s, 2); mbar_init(turn + 8 * s, 1);
    }
    for (int s = 0; s < 2; s++) { mbar_init(acc_full + 8 * s, 1); mbar_init(acc_empty + 8 * s, FM::kHalves ? kEWarps : 2 * kEWarps); mbar_init(drained + 8 * s, 1); }
    mbar_init(cross_full, 1); mbar_init(cross_empty, 2 * kEWarps); mbar_init(stash_full, kEWarps); mbar_init(stash_empty, 4);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0 && lane < 2)
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(lane ? &P.wmap : &P.amap)) : "memory");
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                          // both CTAs' barriers exist before either signals the other's
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  // Programmatic dependent launch: the next layer's CTAs set up and load weights while this grid drains.  Not before both CTAs have
  // their tensor memory.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  auto wait = [&](uint32_t bar, uint32_t parity, int code) { return wait_polling(bar, parity, P.wait_limit, abort_flag, P.status, code); };
  // The epilogue warps of the widest form hold 96 sums a thread and up to 96 loaded values.  56 x 256 + 200 x 256 = 128 x 512
  // registers: what the block is launched with (checked before the launch).
  if (warp < kWarpE0) {
    if constexpr (FM::kHalves) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA: activations, this CTA's rows
      asm volatile("griddepcontrol.wait;" ::: "memory");        // what the kernel in front wrote is complete and visible
      const uint32_t full0 = map_to_cta(a_full, 0);
      uint32_t s = 0, ph = 0;
      bool stop = false;
      for (long long t = t0; t < ntiles && !stop; t += t_step) {
        const uint32_t piece = piece_of(t);
        const long long m0 = piece * P.piece_stride + first_row(t, piece);
        for (int g = 0; g < P.ng && !stop; g++) {
          const int y0 = (int)(m0 + stage_shift<LINE>(P, g));
          for (int cb = 0; cb < P.nchb; cb++) {
            if (!wait(a_empty + 8 * s, ph ^ 1, VST_A_EMPTY)) { stop = true; break; }
            const bool skip = P.test_skip_stage && blockIdx.x == 0 && t == t0 && g == 0 && cb == 0;    // test only: the stage never completes
            if (crank == 0) mbar_expect_tx(a_full + 8 * s, 2 * a_bytes);
            if (!skip) tma_load_3d_pair(base + s * a_bytes, &P.amap, cb * kKt, y0, 0, full0 + 8 * s);
            if (++s == (uint32_t)P.a_stages) { s = 0; ph ^= 1; }
          }
        }
      }
      if (crank == 0)
        for (uint32_t q = 0; q < (uint32_t)P.a_stages; q++) drain_wait(a_full + 8 * q, q < s ? ph : ph ^ 1, P.wait_limit);
    } else if (warp == 1) {
      // ---------------------------------------------------------------- TMA: weights, this CTA's half of the features
      const uint32_t full0 = map_to_cta(w_full, 0);
      uint32_t s = 0, ph = 0;
      bool stop = false;
      for (long long t = t0; t < ntiles && !stop; t += t_step) {
        const int nt = (int)(t % P.ntn);
        for (int g = 0; g < P.ng && !stop; g++)
          for (int cb = 0; cb < P.nchb && !stop; cb++)
            for (int tp = 0; tp < P.tpg; tp++) {
              if (!wait(w_empty + 8 * s, ph ^ 1, VST_W_EMPTY)) { stop = true; break; }
              if (crank == 0) mbar_expect_tx(w_full + 8 * s, 2 * kWBytes);
              tma_load_2d_pair(w_ring + s * kWBytes, &P.wmap, 0, ((((g * P.tpg + tp) * P.nchb + cb) * P.ntn + nt) * 2 + (int)crank) * FM::kWRows, full0 + 8 * s);
              if (++s == (uint32_t)P.w_stages) { s = 0; ph ^= 1; }
            }
        if constexpr (RESIDENT) break;
      }
      if (crank == 0)
        for (uint32_t q = 0; q < (uint32_t)P.w_stages; q++) drain_wait(w_full + 8 * q, q < s ? ph : ph ^ 1, P.wait_limit);
    } else if (crank == 0) {
      // ---------------------------------------------------------------- MMA issuers (the leader's, for both CTAs).  A warp needs several
      // hundred clocks for the waits, commits and counting of a step, in which it issues nothing, so two share a step: the first takes
      // x_hi . [W_hi | W_lo], or with LINE x_hi . W_hi, into accumulators that the epilogue takes over step by step, the second the
      // other cross products, each step when the first has issued its part: the cross products of a step then run while the epilogue
      // takes over the sums (one warp: 1220 clk a step of 432 clk of MMAs; with LINE and no order the first waits for the epilogue
      // behind the second's queued MMAs).
      const uint32_t cross = tmem + FM::kColCross, line = (uint32_t)(P.g.Wq - P.sub_w + 1) * 8;
      auto issue = [&](auto first_) {
        constexpr bool kFirst = decltype(first_)::value;
        uint32_t as = 0, aph = 0, ws = 0, wph = 0, chunk_it = 0, tile_it = 0;
        for (long long t = t0; t < ntiles; t += t_step, tile_it++) {
          int kt = 0, cb = 0;
          for (int st = P.ng * P.nchb; st > 0; st--) {
            if (kFirst && !wait(a_full + 8 * as, aph, VST_A_FULL)) return;
            const int left = P.g.C - cb * kKt, nk8 = left >= kKt ? 4 : (left + 7) >> 3;   // behind the last channel both operands are zero
            if (++cb == P.nchb) cb = 0;
            int dw = 0;
            uint32_t row_ = desc_lo(base + as * a_bytes);        // the stage's row of the tile's first row under the present step
            for (int tp = P.tpg; tp > 0; tp--, kt++) {
              // the second follows the first: what the first has waited for is there
              const uint32_t turn_bar = turn + 8 * (RESIDENT ? chunk_it % kTurns : ws);
              if (!wait(kFirst ? w_full + 8 * ws : turn_bar, !RESIDENT ? wph : kFirst ? 0 : chunk_it / kTurns & 1, VST_W_FULL)) return;
              // through shuffles: an MMA whose operands the compiler does not know to be the same in all lanes costs 18 clk and more
              // to issue (7 otherwise)
              const uint32_t row = __shfl_sync(0xffffffffu, row_, 0), wd = __shfl_sync(0xffffffffu, desc_lo(w_ring + ws * kWBytes), 0);
              const uint32_t b = chunk_it & 1;
              auto groups = [&](auto full_) {
                constexpr bool kFull = decltype(full_)::value;
                if constexpr (kFirst && FM::kHalves) {
#pragma unroll
                  for (int h = 0; h < 2; h++) {
                    if (!wait(acc_empty + 8 * h, b ^ 1, VST_ACC_EMPTY)) return false;
                    tc_fence_after();
                    mma_step32<idesc_tf32_pair(FM::kAcc), kFull>(tmem + h * FM::kAcc, row, wd + h * (48 * 128 >> 4), 0u, nk8);
                    tc_commit_pair(acc_full + 8 * h);
                  }
                } else if constexpr (kFirst) {
                  if (!wait(acc_empty + 8 * b, ((chunk_it >> 1) & 1) ^ 1, VST_ACC_EMPTY)) return false;
                  tc_fence_after();
                  mma_step32<idesc_tf32_pair(FM::kAcc), kFull>(tmem + b * FM::kAcc, row, wd, 0u, nk8);
                  tc_commit_pair(acc_full + 8 * b);
                } else {
                  if (kt == 0 && !wait(cross_empty, (tile_it & 1) ^ 1, VST_ACC_EMPTY)) return false;   // the previous tile's cross sums have been read
                  tc_fence_after();
                  if constexpr (LINE) mma_step32<idesc_tf32_pair(FM::kCross), kFull>(cross, row, wd + ((uint32_t)(FM::kWBytes / 2) >> 4), (uint32_t)kt, nk8);
                  mma_step32<idesc_tf32_pair(FM::kCross), kFull>(cross, row + (a_plane >> 4), wd, LINE ? 1u : (uint32_t)kt, nk8);
                }
                if constexpr (kFirst) {
                  __syncwarp();
                  if (lane == 0) mbar_arrive(turn_bar);
                }
                return true;
              };
              if (!(nk8 == 4 ? groups(std::true_type{}) : groups(std::false_type{}))) return;
              chunk_it++;
              if constexpr (!RESIDENT) tc_commit_pair(w_empty + 8 * ws);
              if (++ws == (uint32_t)P.w_stages) { ws = 0; wph ^= 1; }
              if (++dw == P.sub_w) { dw = 0; row_ += line; } else row_ += 8;
            }
            tc_commit_pair(a_empty + 8 * as);
            if (++as == (uint32_t)P.a_stages) { as = 0; aph ^= 1; }
          }
          if constexpr (!kFirst) tc_commit_pair(cross_full);
        }
      };
      if (warp == 2) issue(std::true_type{}); else issue(std::false_type{});
      tc_commit_pair(drained + 8 * (warp - 2));                  // nothing may still read shared or tensor memory when the CTAs end
      drain_wait(drained + 8 * (warp - 2), 0, P.wait_limit);
    }
  } else if (warp >= kWarpS0) {
    if constexpr (FM::kHalves) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    // ------------------------------------------------------------------ storers: bias, residual, activation, and the tile's rows to
    // global memory, from the stash, while the epilogue warps take over the next tile's sums
    const VolGeom& G = P.g;
    constexpr int LPR = NT / 4, RPI = 32 / LPR;                  // lanes per row, rows per access
    const int quad = warp & 3;
    const float* stash = (const float*)(tail + kBarBytes + FM::kXchBytes) + quad * 32 * NT;
    auto activate = [&](float (&v)[4]) {
      if (P.act == ACT_RELU) {
#pragma unroll
        for (int e = 0; e < 4; e++) v[e] = max_nan(v[e], 0.f);
      } else if (P.act == ACT_LEAKY) {
#pragma unroll
        for (int e = 0; e < 4; e++) v[e] = v[e] > 0.f ? v[e] : v[e] * P.slope;
      }
    };
    asm volatile("griddepcontrol.wait;" ::: "memory");           // before the first read of the residual and the first store
    uint32_t tile_it = 0;
    for (long long t = t0; t < ntiles; t += t_step, tile_it++) {
      const int r = quad * 32 + lane, n0 = (int)(t % P.ntn) * NT;
      const uint32_t piece = piece_of(t);
      const long long local = first_row(t, piece) + r, p = piece * P.piece_stride + local;
      const bool in_rows = local < P.rows && (!LINE || (r >= 1 && r <= FM::kRowsOut));
      const uint32_t q0 = (uint32_t)(in_rows ? p : 0), q1 = q0 / (uint32_t)G.Wq, q2 = q1 / (uint32_t)G.Hq, q3 = q2 / (uint32_t)G.Dq;
      const int ow = (int)(q0 - q1 * G.Wq), oh = (int)(q1 - q2 * G.Hq), od = (int)(q2 - q3 * G.Dq), on = (int)q3;
      const bool live = in_rows && ow < G.Wo && oh < G.Ho && od < G.Do;
      const uint32_t live_mask = __ballot_sync(0xffffffffu, live);
      if (!wait(stash_full, tile_it & 1, VST_STASH_FULL)) break;
      if (P.out) {
        // this lane's row in the output volume (fewer than 2^30), or -1
        const int row_out = P.remap ? (live ? (int)vol_row(P.next, on, od, oh, ow) : -1) : in_rows ? (int)(p + P.out_shift) : -1;
        // lanes along a row: whole lines of the split volume
        const int c = lane % LPR, f = n0 + 4 * c;
        const bool inside = f < P.out_pitch;
        float b[4];
#pragma unroll
        for (int e = 0; e < 4; e++) b[e] = P.bias && f + e < P.F ? __ldg(P.bias + f + e) : 0.f;
#pragma unroll 2
        for (int i = 0; i < 32; i += RPI) {
          const int rr = i + lane / LPR;
          const int row = __shfl_sync(0xffffffffu, row_out, rr);
          const bool mine = inside && row >= 0, lv = (live_mask >> rr) & 1u;
          const long long o = (long long)row * P.out_pitch + f;
          float4 sh = make_float4(0.f, 0.f, 0.f, 0.f), sl = sh;
          if (P.skip && lv && inside) { sh = ld_plain4(P.skip + o); sl = ld_plain4(P.skip + P.out_plane + o); }
          const float4 q = *reinterpret_cast<const float4*>(stash + rr * NT + ((c ^ (rr & 7)) << 2));
          float v[4] = {q.x + b[0], q.y + b[1], q.z + b[2], q.w + b[3]}, h[4], l[4];
          if (P.skip) {
            v[0] += fmaf(sl.x, 1.f / kLoScale, sh.x); v[1] += fmaf(sl.y, 1.f / kLoScale, sh.y); v[2] += fmaf(sl.z, 1.f / kLoScale, sh.z); v[3] += fmaf(sl.w, 1.f / kLoScale, sh.w);
          }
          activate(v);
#pragma unroll
          for (int e = 0; e < 4; e++) vol_split(lv && f + e < P.F ? v[e] : 0.f, h[e], l[e]);   // the next layer's padding, and channels, are zero
          if (mine) {
            *reinterpret_cast<float4*>(P.out + o) = make_float4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<float4*>(P.out + P.out_plane + o) = make_float4(l[0], l[1], l[2], l[3]);
          }
        }
      } else {
        // lane = row: whole lines of a channel-major array
        float* dst = P.y + ((long long)on * P.ys_n + (long long)od * P.ys_d + (long long)oh * P.ys_h + (long long)ow * P.ys_w + (long long)n0 * P.ys_c);
        const float* src = P.res ? P.res + ((long long)on * P.rs_n + (long long)od * P.rs_d + (long long)oh * P.rs_h + (long long)ow * P.rs_w + (long long)n0 * P.rs_c) : nullptr;
        float b[NT / 32];                                            // of feature n0 + 32 i + lane
#pragma unroll
        for (int i = 0; i < NT / 32; i++) b[i] = P.bias && n0 + 32 * i + lane < P.F ? __ldg(P.bias + n0 + 32 * i + lane) : 0.f;
#pragma unroll
        for (int c = 0; c < LPR; c++) {
          if (n0 + 4 * c >= P.F) break;
          const float4 q = *reinterpret_cast<const float4*>(stash + lane * NT + ((c ^ (lane & 7)) << 2));
          float v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int e = 0; e < 4; e++) {
            v[e] += __shfl_sync(0xffffffffu, b[c / 8], (4 * c + e) & 31);
            if (src && live && n0 + 4 * c + e < P.F) v[e] += ld_plain(src + (4 * c + e) * P.rs_c);
          }
          activate(v);
#pragma unroll
          for (int e = 0; e < 4; e++) {
            if (live && n0 + 4 * c + e < P.F) *dst = v[e];
            dst += P.ys_c;
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(stash_empty);
    }
  } else {
    if constexpr (FM::kHalves) asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
    // ------------------------------------------------------------------ epilogue: thread = row, half of the features.  A wait that gives
    // up ends no warp here: the others would wait for it at the row exchange.  The waits behind it return at once.
    const VolGeom& G = P.g;
    const int quad = warp & 3, half = (warp - kWarpE0) >> 2;
    const uint32_t lane_addr = tmem + ((uint32_t)(quad * 32) << 16);
    float* xch = (float*)(tail + kBarBytes);
    float* stash = (float*)(tail + kBarBytes + FM::kXchBytes);
    const uint32_t arr_acc = map_to_cta(acc_empty, 0), arr_cross = map_to_cta(cross_empty, 0);   // the leader's
    uint32_t chunk_it = 0, tile_it = 0;
    for (long long t = t0; t < ntiles; t += t_step, tile_it++) {
      const int r = quad * 32 + lane;
      // the row's position in its line, for its neighbours
      const long long local = LINE ? first_row(t, piece_of(t)) + r : 0;      // pieces start at a line's start
      const int ow = LINE ? (int)((uint32_t)(local > 0 && local < P.rows ? local : 0) % (uint32_t)G.Wq) : 0;
      float sum[FM::kTaps][NH], vx[LINE ? 1 : NH];
#pragma unroll
      for (int k = 0; k < FM::kTaps; k++)
#pragma unroll
        for (int j = 0; j < NH; j++) sum[k][j] = -0.f;           // -0 + x is x, also where x is -0
      if constexpr (!LINE) {
#pragma unroll
        for (int j = 0; j < NH; j++) vx[j] = 0.f;
      }
      for (int kt = 0; kt < nkt; kt++, chunk_it++) {
        const uint32_t b = FM::kHalves ? half : chunk_it & 1;
        wait(acc_full + 8 * b, (FM::kHalves ? chunk_it : chunk_it >> 1) & 1, VST_ACC_FULL);
        tc_fence_after();
        if constexpr (LINE) {
          uint32_t a[3][NH];
#pragma unroll
          for (int k = 0; k < 3; k++) tmem_ldn(lane_addr + b * FM::kAcc + k * 32 + (FM::kHalves ? 0 : half * NH), a[k]);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster_relaxed(arr_acc + 8 * b);
#pragma unroll
          for (int k = 0; k < 3; k++)
#pragma unroll
            for (int j = 0; j < NH; j += 2) {
              const float2 v = add2(make_float2(sum[k][j], sum[k][j + 1]), make_float2(__uint_as_float(a[k][j]), __uint_as_float(a[k][j + 1])));
              sum[k][j] = v.x; sum[k][j + 1] = v.y;
            }
        } else {
          uint32_t a[NH];
          tmem_ldn(lane_addr + b * FM::kAcc + half * NT, a);     // a half's W_hi columns, then its W_lo columns
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < NH; j++) sum[0][j] = __fadd_rn(sum[0][j], __uint_as_float(a[j]));
          tmem_ldn(lane_addr + b * FM::kAcc + half * NT + NH, a);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster_relaxed(arr_acc + 8 * b);
#pragma unroll
          for (int j = 0; j < NH; j++) vx[j] = __fadd_rn(vx[j], __uint_as_float(a[j]));
        }
      }
      wait(cross_full, tile_it & 1, VST_ACC_FULL);
      tc_fence_after();
      // What follows runs once a tile, so it is fetched instruction by instruction while the next tile's second step waits for these
      // warps: as few instructions as possible (packed arithmetic, whole rows to and from shared memory, no branch per feature).
      {
        uint32_t a[FM::kTaps][NH / 16][16];
#pragma unroll
        for (int k = 0; k < FM::kTaps; k++)
#pragma unroll
          for (int c = 0; c < NH / 16; c++)
            tmem_ldn(lane_addr + FM::kColCross + (LINE ? FM::cross_col(half, k * 32 + (FM::kHalves ? 0 : half * NH) + 16 * c) : half * NH + 16 * c), a[k][c]);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster_relaxed(arr_cross);
#pragma unroll
        for (int k = 0; k < FM::kTaps; k++)
#pragma unroll
          for (int j = 0; j < NH; j += 2) {
            float2 x = make_float2(__uint_as_float(a[k][j / 16][j % 16]), __uint_as_float(a[k][j / 16][j % 16 + 1]));
            if constexpr (!LINE) x = add2(make_float2(vx[j], vx[j + 1]), x);
            const float2 v = fma2(x, make_float2(1.f / kLoScale, 1.f / kLoScale), make_float2(sum[k][j], sum[k][j + 1]));
            sum[k][j] = v.x; sum[k][j + 1] = v.y;
          }
      }
      float vh[NH];
      if constexpr (LINE) {
        // out[row] = sum0[row - 1] + sum1[row] + sum2[row + 1], where the neighbour is a position of the same line; rows on either side
        // of a warp boundary go through shared memory
        float* xu = xch + half * NH;                                 // tap 0's sums of each quadrant's last row
        float* xd = xu + 4 * NT;                                     // tap 2's sums of each quadrant's first row
        if (half == 0) asm volatile("bar.sync 1, 128;" ::: "memory"); else asm volatile("bar.sync 2, 128;" ::: "memory");   // the last tile's rows have been read
        if (lane == 31) {
#pragma unroll
          for (int j = 0; j < NH; j += 4) *reinterpret_cast<float4*>(xu + quad * NT + j) = make_float4(sum[0][j], sum[0][j + 1], sum[0][j + 2], sum[0][j + 3]);
        }
        if (lane == 0) {
#pragma unroll
          for (int j = 0; j < NH; j += 4) *reinterpret_cast<float4*>(xd + quad * NT + j) = make_float4(sum[2][j], sum[2][j + 1], sum[2][j + 2], sum[2][j + 3]);
        }
        if (half == 0) asm volatile("bar.sync 1, 128;" ::: "memory"); else asm volatile("bar.sync 2, 128;" ::: "memory");
        const bool has_up = ow + G.ow0 >= 0, has_dn = ow + G.ow0 + 2 < G.Wq;
        const float* eu = xu + (quad > 0 ? quad - 1 : 0) * NT;       // what lanes 0 and 31 take instead (tile rows 0 and 127 are not outputs)
        const float* ed = xd + (quad < 3 ? quad + 1 : 3) * NT;
#pragma unroll
        for (int j = 0; j < NH; j += 4) {
          const float4 u4 = *reinterpret_cast<const float4*>(eu + j), d4 = *reinterpret_cast<const float4*>(ed + j);
          const float u[4] = {u4.x, u4.y, u4.z, u4.w}, d[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const float su = __shfl_up_sync(0xffffffffu, sum[0][j + e], 1), sd = __shfl_down_sync(0xffffffffu, sum[2][j + e], 1);
            const float up = lane == 0 ? u[e] : su, dn = lane == 31 ? d[e] : sd;
            vh[j + e] = sum[1][j + e] + (has_up ? up : 0.f) + (has_dn ? dn : 0.f);
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < NH; j++) vh[j] = sum[0][j];
      }
      // 16-byte pieces at piece ^ (row % 8): no bank conflicts, whichever way the storers read
      wait(stash_empty, (tile_it & 1) ^ 1, VST_STASH_EMPTY);
#pragma unroll
      for (int j = 0; j < NH; j += 4)
        *reinterpret_cast<float4*>(stash + r * NT + ((((half * NH + j) >> 2) ^ (r & 7)) << 2)) = make_float4(vh[j], vh[j + 1], vh[j + 2], vh[j + 3]);
      __syncwarp();
      if (lane == 0) mbar_arrive(stash_full);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0)
    for (int i = 0; i < 2000; i++) __nanosleep(1000);          // let the partner's copies in flight land before the memory is given back
  __syncthreads();
  cluster_sync_all();                          // neither CTA leaves while its partner can still signal its barriers
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// A strided fp32 array -> split volume: 128 rows x 32 channels per block, turned in shared memory; padding is written as zeros.  The
// array is pooled or repeated on the way where the source says so (2-D networks), so that such a layer's output is never stored.
// Latency of the reads bounds it: a row's position (five divisions) is worked out once per block, not by each of its warps, and a thread
// has 16 loads in flight (8 with 64 rows per block; the source's kind is a template argument, so that no branch lies between the loads).
// A layer of 32 -> 64 channels at 40^3: 55.0 -> 50.3 us; a 2-D operator network at 4 x 180^2 (pooling, upsampling): 229 -> 215 us.
template <int OP>
__global__ void __launch_bounds__(256) pack_volume_kernel(const float* __restrict__ x, float* __restrict__ out, long long plane, int pitch, VolGeom g,
                                                          VolSource src) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the layer may set up and load weights while this kernel runs
  __shared__ float tile[128][33];
  __shared__ long long pos[128];                               // element of channel 0, or -1 for padding
  const uint32_t P32 = (uint32_t)g.P, R = P32 * (uint32_t)(g.fd * g.fh * g.fw), r0 = blockIdx.x * 128u;
  const int c0 = blockIdx.y * 32, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < 128) {
    const uint32_t r = r0 + threadIdx.x;
    const uint32_t ph = r / P32, q0 = r - ph * P32, q1 = q0 / (uint32_t)g.Wq, q2 = q1 / (uint32_t)g.Hq, q3 = q2 / (uint32_t)g.Dq;
    const int w = (int)(q0 - q1 * g.Wq) * g.sw + (int)(ph % (uint32_t)g.fw) - g.pw;
    const int h = (int)(q1 - q2 * g.Hq) * g.sh + (int)((ph / (uint32_t)g.fw) % (uint32_t)g.fh) - g.ph;
    const int d = (int)(q2 - q3 * g.Dq) * g.sd + (int)(ph / (uint32_t)(g.fw * g.fh)) - g.pd;
    long long o = -1;
    if (r < R && w >= 0 && w < g.W && h >= 0 && h < g.H && d >= 0 && d < g.D) {
      const uint32_t hs = OP == VolSource::UPSAMPLE ? (uint32_t)h / (uint32_t)src.kh : OP == VolSource::MAXPOOL ? (uint32_t)(h * src.sh) : (uint32_t)h;
      const uint32_t ws = OP == VolSource::UPSAMPLE ? (uint32_t)w / (uint32_t)src.kw : OP == VolSource::MAXPOOL ? (uint32_t)(w * src.sw) : (uint32_t)w;
      o = (long long)q3 * src.xs_n + (long long)d * src.xs_d + (long long)hs * src.xs_h + (long long)ws * src.xs_w;
    }
    pos[threadIdx.x] = o;
  }
  __syncthreads();
  long long o[4];
#pragma unroll
  for (int i = 0; i < 4; i++) o[i] = pos[i * 32 + lane];
  float v[4][4];
  // one value of each of the thread's 16 outputs, all in flight together
  auto load = [&](long long off, float (&t)[4][4]) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int c = c0 + warp * 4 + k;
      const float* p = x + (long long)c * src.xs_c + off;
#pragma unroll
      for (int i = 0; i < 4; i++) t[k][i] = o[i] >= 0 && c < g.C ? __ldg(p + o[i]) : 0.f;
    }
  };
  load(0, v);
  if constexpr (OP == VolSource::MAXPOOL) {
    for (int a = 0; a < src.kh; a++)
      for (int b = a == 0 ? 1 : 0; b < src.kw; b++) {
        float t[4][4];
        load(a * src.xs_h + b * src.xs_w, t);
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
          for (int i = 0; i < 4; i++) v[k][i] = max_nan(v[k][i], t[k][i]);
      }
  }
#pragma unroll
  for (int k = 0; k < 4; k++)
#pragma unroll
    for (int i = 0; i < 4; i++) tile[i * 32 + lane][warp * 4 + k] = v[k][i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int rr = i * 32 + (threadIdx.x >> 3), c = (threadIdx.x & 7) * 4;
    if (r0 + rr >= R) continue;
    float h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; e++) vol_split(tile[rr][c + e], h[e], l[e]);
    float* q = out + (long long)(r0 + rr) * pitch + c0 + c;
    *reinterpret_cast<float4*>(q) = make_float4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<float4*>(q + plane) = make_float4(l[0], l[1], l[2], l[3]);
  }
}

// weights (F, C, taps) -> the steps' images [step][channel block][tile][CTA][W_hi rows | W_lo rows][32]; one tap: half of the tile's
// features in each CTA; three taps: for every 32 features 96 rows [tap][feature], half of them in each CTA
__global__ void pack_vol_weights_kernel(const float* __restrict__ W, int F, int C, int taps, int kw, int nchb, int ntn, int NT, float* __restrict__ out) {
  const int half_rows = kw * NT / 2;                           // one CTA's
  const long long n_el = (long long)(taps / kw) * nchb * ntn * 4 * half_rows * kKt;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n_el; i += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(i % kKt);
    long long rest = i / kKt;
    const int row = (int)(rest % (2 * half_rows)); rest /= 2 * half_rows;
    const int cta = (int)(rest & 1); rest >>= 1;
    const int nt = (int)(rest % ntn); rest /= ntn;
    const int cb = (int)(rest % nchb), step = (int)(rest / nchb);
    const int r = row % half_rows, n = kw == 3 ? cta * 48 + r % 48 : cta * half_rows + r;
    const int f = nt * NT + (kw == 3 ? r / 48 * 32 + n % 32 : n), tap = kw == 3 ? step * 3 + n / 32 : step, c = cb * kKt + k;
    float h = 0.f, l = 0.f;
    if (f < F && c < C) vol_split(W[((long long)f * C + c) * taps + tap], h, l);
    out[i] = row < half_rows ? h : l;
  }
}

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                             const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  if (fn) return fn;
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || !p) return nullptr;
  return fn = (EncodeFn)p;
}

int vol_nt(int F) { return F <= 32 ? 32 : 64; }

// How a stage serves steps: those of a kd, of a line, or one; the widest sharing whose rows fit a box and leave two stages.  What
// shared memory is left goes to the ring that reaches less far ahead, in steps.  Where a tile's steps are so few that all their weights
// fit, and two steps' activations beside the present one's, the weights stay (2-D network 4 x 180^2, a line's
// rows a stage: a quarter of what a step brings in; its layers 29.4 -> 28.4, 38.9 -> 37.4 and 39.5 -> 38.0 us, a call 173.6 -> 169.7).
struct Sharing { int ng, tpg, sub_w, box_rows, a_stages, w_stages; bool resident; size_t smem; };
bool pick_sharing(const VolGeom& g, int F, Sharing* o) {
  const bool line = g.line;
  const int NT = vol_nt(F), nw = line ? 1 : g.KW, w_bytes = (line ? 3 : 1) * NT * kKt * 4;
  const int fixed = kBarBytes + (line ? Form<32, true>::kXchBytes / 32 * NT : 0) + kM * NT * 4;
  for (int level = 0; level < 3; level++) {
    long long span;
    if (level == 0) {
      if (g.sh != 1 || (!line && g.sw != 1)) continue;
      span = (long long)(g.KH - 1) * g.Wq + nw - 1;
      o->ng = g.KD; o->tpg = g.KH * nw; o->sub_w = nw;
    } else if (level == 1) {
      if (!line && g.sw != 1) continue;
      span = nw - 1;
      o->ng = g.KD * g.KH; o->tpg = nw; o->sub_w = nw;
    } else {
      span = 0;
      o->ng = g.KD * g.KH * nw; o->tpg = 1; o->sub_w = 1;
    }
    if (kM + span > 256) continue;
    o->box_rows = (int)(kM + span + 7) / 8 * 8;
    const int a_bytes = 2 * o->box_rows * kKt * 4;
    int left = kSmemMax - fixed - 2 * a_bytes - 2 * w_bytes;
    if (left < 0) continue;
    const long long steps = (long long)o->ng * o->tpg * ((g.C + kKt - 1) / kKt);
    o->resident = false;
    if (F <= NT && steps <= kMaxResident) {
      const int n = (kSmemMax - fixed - (int)steps * w_bytes) / a_bytes, a_stages = n < kMaxStages ? n : kMaxStages;
      if (a_stages >= 2 && (a_stages - 1) * o->tpg >= 2) {
        o->resident = true; o->a_stages = a_stages; o->w_stages = (int)steps;
        o->smem = fixed + (size_t)a_stages * a_bytes + (size_t)steps * w_bytes;
        return true;
      }
    }
    o->a_stages = o->w_stages = 2;
    for (;;) {
      const bool a_ok = o->a_stages < kMaxStages && left >= a_bytes, w_ok = o->w_stages < kMaxStages && left >= w_bytes;
      if (w_ok && (o->w_stages <= (o->a_stages - 1) * o->tpg || !a_ok)) { o->w_stages++; left -= w_bytes; }
      else if (a_ok) { o->a_stages++; left -= a_bytes; }
      else break;
    }
    o->smem = kSmemMax - left;
    return true;
  }
  return false;
}

int sm_count() {
  static int sms = 0;
  if (sms) return sms;
  int n = 148, dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return sms = n;
}

bool vol_line(int kw, int sw, int pw) { return kw == 3 && sw == 1 && pw <= 1; }       // the taps of a line in one step

}  // namespace

// `front`: zero positions in front of every line, plane and volume of the grid, at least the layer's own padding (a network whose
// layers pad differently takes the widest for all); layers that take a line's taps in one step need none in front of lines
VolGeom vol_geom(const ConvGeom& c, int front_d, int front_h, int front_w) {
  VolGeom g;
  std::memset(&g, 0, sizeof g);
  g.N = c.N; g.D = c.D; g.H = c.H; g.W = c.W; g.C = c.C; g.Do = c.Do; g.Ho = c.Ho; g.Wo = c.Wo;
  g.KD = c.KD; g.KH = c.KH; g.KW = c.KW; g.sd = c.sd; g.sh = c.sh; g.sw = c.sw;
  g.pd = front_d; g.ph = front_h; g.pw = front_w;
  // stride 1: a line's right padding is the next one's left padding; never fewer positions than outputs (padding of K and more)
  auto axis = [](int ext, int front, int stride, int out) {
    const int n = stride == 1 ? ext + front : (ext + 2 * front + stride - 1) / stride;
    return n > out ? n : out;
  };
  g.Dq = axis(c.D, front_d, c.sd, c.Do); g.Hq = axis(c.H, front_h, c.sh, c.Ho); g.Wq = axis(c.W, front_w, c.sw, c.Wo);
  g.fd = c.KD < c.sd ? c.KD : c.sd; g.fh = c.KH < c.sh ? c.KH : c.sh; g.fw = c.KW < c.sw ? c.KW : c.sw;
  g.line = vol_line(c.KW, c.sw, c.pw);
  g.od0 = front_d - c.pd; g.oh0 = front_h - c.ph; g.ow0 = front_w - c.pw;
  g.P = (long long)g.N * g.Dq * g.Hq * g.Wq;
  return g;
}

VolMap vol_map(const VolGeom& g) { return VolMap{g.Dq, g.Hq, g.Wq, g.pd, g.ph, g.pw, g.sd, g.sh, g.sw, g.fd, g.fh, g.fw, g.P}; }

int vol_front_w(const ConvGeom& c) { return vol_line(c.KW, c.sw, c.pw) ? 0 : c.pw; }

size_t vol_bytes(const VolGeom& g, int pitch) { return (size_t)g.P * g.fd * g.fh * g.fw * pitch * 8; }

typedef void (*VolKernel)(VolParams);
const VolKernel kVolKernels[8] = {conv_vol_kernel<32, false, false>, conv_vol_kernel<64, false, false>, conv_vol_kernel<32, true, false>, conv_vol_kernel<64, true, false>,
                                  conv_vol_kernel<32, false, true>, conv_vol_kernel<64, false, true>, conv_vol_kernel<32, true, true>, conv_vol_kernel<64, true, true>};

// The widest form (the one that moves registers between its warps) needs the number the compiler gave it (128 a thread); with another
// compiler's the layers stay on the other kernels.
bool vol_available() {
  static const bool ok = [] {
    cudaFuncAttributes fa;
    for (VolKernel k : kVolKernels)
      if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax) != cudaSuccess) { cudaGetLastError(); return false; }
    for (int k : {3, 7})
      if (!(cudaFuncGetAttributes(&fa, kVolKernels[k]) == cudaSuccess && fa.numRegs == 128)) { cudaGetLastError(); return false; }
    return true;
  }();
  return ok;
}

bool vol_alloc(void** p, size_t bytes) {
  g_launches.volume_allocs++;
  if (!(g_tc_test.volume_limit && bytes > g_tc_test.volume_limit) && cudaMalloc(p, bytes) == cudaSuccess) return true;
  cudaGetLastError();
  *p = nullptr;
  return false;
}

bool vol_supported(const ConvGeom& c) {
  if (c.dd != 1 || c.dh != 1 || c.dw != 1) return false;                // transposed convolutions
  // the most products an output can have: taps that lie inside the volume, times channels
  const long long inside = (long long)(c.KD < c.D ? c.KD : c.D) * (c.KH < c.H ? c.KH : c.H) * (c.KW < c.W ? c.KW : c.W);
  if (inside * c.C < kF32TcConvMinProducts) return false;
  if ((long long)c.KD * c.KH * c.KW * ((c.C + 31) / 32) * ((c.F + 31) / 32) > (1 << 20)) return false;   // rows of the weight images in 32 bits
  // channels are padded to 32, features to 32 or 64: no more memory than that is worth (1 -> 1 channel of 33^3 taps: 294 MB of weights for
  // 144 KB; 1 channel on 512^3: 34 GB for 0.5)
  const long long taps = (long long)c.KD * c.KH * c.KW, w_bytes = taps * ((c.C + 31) / 32) * (c.F <= 32 ? 32 : (c.F + 63) / 64 * 64) * kKt * 8;
  if (w_bytes > (32LL << 20) && w_bytes > 4 * taps * c.C * c.F * 8) return false;
  const VolGeom g = vol_geom(c, c.pd, c.ph, vol_front_w(c));
  if (vol_bytes(g, (c.C + 31) / 32 * 32) > (16ULL << 30)) return false;
  Sharing s;
  // rows, and the last ones a tile may ask for, in 32 bits
  return g.P * g.fd * g.fh * g.fw < (1LL << 30) && (long long)c.KD * g.Hq * g.Wq < (1LL << 29) && pick_sharing(g, c.F, &s) && vol_available();
}

// The rows as one piece, or image by image (which leaves the padding planes between them out) where that takes fewer rounds of tiles:
// 14-layer network, 2 x 33^3: 299 pairs of tiles, 4.04 rounds, or 294, 3.97.
struct Pieces { int n, pairs; long long rows, stride; };
Pieces pick_pieces(const VolGeom& g, int ntn) {
  const long long per_pair = 2 * (g.line ? Form<64, true>::kRowsOut : Form<64, false>::kRowsOut), on_device = sm_count() / 2 > 0 ? sm_count() / 2 : 1;
  const long long stride = (long long)g.Dq * g.Hq * g.Wq, image = ((long long)(g.Do - 1) * g.Hq + g.Ho - 1) * g.Wq + g.Wo, all = (g.N - 1) * stride + image;
  const long long one = (all + per_pair - 1) / per_pair, each = (image + per_pair - 1) / per_pair;
  if ((each * g.N * ntn + on_device - 1) / on_device < (one * ntn + on_device - 1) / on_device) return Pieces{g.N, (int)each, image, stride};
  return Pieces{1, (int)one, all, 0};
}

// Estimated device time of a layer, ns: rounds of tiles, and in each the steps and the tile's end.  The constants are those of 520 timed
// layers and networks, on the high side of the fits (a line's taps 365 and 610 ns a step, a tap 330 to 380 with shared stages and 510 to
// 530 without, packing 5.4 TB/s of what it writes and 6 us), so that a call near the line stays with the general kernel.  A block of up to
// 24 channels issues its MMAs one by one: 24 -> 24 channels 5x5x5 on 2 x 40^3 450 us, on the general kernel 409, without that term taken
// for 421 and 435.
long long vol_kernel_cost(const VolGeom& g, int F) {
  const int NT = vol_nt(F), blocks = (g.C + 31) / 32, last = g.C % 32;
  Sharing s;
  if (!pick_sharing(g, F, &s)) return 1LL << 60;
  const Pieces pc = pick_pieces(g, (F + NT - 1) / NT);
  const long long pairs = sm_count() / 2 > 0 ? sm_count() / 2 : 1, tiles = (long long)pc.n * pc.pairs * ((F + NT - 1) / NT), rounds = (tiles + pairs - 1) / pairs;
  const long long taps = s.ng * s.tpg, step = g.line ? (NT == 64 ? 680 : 500) : s.tpg > 1 ? 380 : 570, end = g.line ? (NT == 64 ? 2600 : 2000) : 1500;
  return rounds * (taps * (blocks * step + (!g.line && last > 0 && last <= 24 ? 50 : 0)) + end);
}
long long vol_pack_cost(const VolGeom& g) { return 6500 + (long long)(vol_bytes(g, (g.C + 31) / 32 * 32) / 1600); }
long long vol_cost(const ConvGeom& c) {
  const VolGeom g = vol_geom(c, c.pd, c.ph, vol_front_w(c));
  return vol_pack_cost(g) + vol_kernel_cost(g, c.F);
}

struct VolW { int F = 0, C = 0, taps = 0, kw = 1, NT = 0, nchb = 0, ntn = 0; float* img = nullptr; CUtensorMap map; };     // kw: taps of a step

void vol_weights_free(VolW* w) {
  if (!w) return;
  cudaFree(w->img);
  delete w;
}

VolW* vol_weights_pack(const float* w_dev, int F, int C, int taps, bool line, cudaStream_t s, std::string* err) {
  VolW* w = new VolW();
  w->F = F; w->C = C; w->taps = taps; w->kw = line ? 3 : 1; w->NT = vol_nt(F); w->nchb = (C + kKt - 1) / kKt; w->ntn = (F + w->NT - 1) / w->NT;
  const long long rows = (long long)(taps / w->kw) * w->nchb * w->ntn * (line ? 6 : 2) * w->NT;
  if (!vol_alloc((void**)&w->img, (size_t)rows * kKt * 4)) {
    if (err) *err = "out of device memory for split conv weights";
    delete w;
    return nullptr;
  }
  const cuuint64_t dims[2] = {(cuuint64_t)kKt, (cuuint64_t)rows}, strides[1] = {kKt * 4};
  const cuuint32_t box[2] = {kKt, (cuuint32_t)((line ? 3 : 1) * w->NT)}, estr[2] = {1, 1};
  EncodeFn enc = encode_fn();
  if (!enc || enc(&w->map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, w->img, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
    if (err) *err = "cuTensorMapEncodeTiled failed for split conv weights";
    vol_weights_free(w);
    return nullptr;
  }
  const long long n = rows * kKt;
  pack_vol_weights_kernel<<<(unsigned)((n + 255) / 256 < 1184 ? (n + 255) / 256 : 1184), 256, 0, s>>>(w_dev, F, C, taps, w->kw, w->nchb, w->ntn, w->NT, w->img);
  return w;
}

void vol_pack(const float* x, float* vol, int pitch, const VolGeom& g, const VolSource& src, cudaStream_t s) {
  const long long R = g.P * g.fd * g.fh * g.fw;
  const dim3 grid((unsigned)((R + 127) / 128), (unsigned)((g.C + 31) / 32));
  if (src.op == VolSource::MAXPOOL) pack_volume_kernel<VolSource::MAXPOOL><<<grid, 256, 0, s>>>(x, vol, R * pitch, pitch, g, src);
  else if (src.op == VolSource::UPSAMPLE) pack_volume_kernel<VolSource::UPSAMPLE><<<grid, 256, 0, s>>>(x, vol, R * pitch, pitch, g, src);
  else pack_volume_kernel<VolSource::PLAIN><<<grid, 256, 0, s>>>(x, vol, R * pitch, pitch, g, src);
}

bool vol_conv(const VolW* w, const float* vol, int pitch, const VolGeom& g, const VolOut& o, const float* bias, int act, float slope, int* status,
              cudaStream_t s, bool early, std::string* err) {
  auto fail = [&](const char* why) { if (err) *err = why; return false; };
  Sharing sh;
  if (!pick_sharing(g, w->F, &sh)) return fail("convolution: no stage layout");
  VolParams P;
  std::memset(&P, 0, sizeof P);
  const long long R = g.P * g.fd * g.fh * g.fw;
  const cuuint64_t dims[3] = {(cuuint64_t)pitch, (cuuint64_t)R, 2}, strides[2] = {(cuuint64_t)pitch * 4, (cuuint64_t)R * pitch * 4};
  const cuuint32_t box[3] = {kKt, (cuuint32_t)sh.box_rows, 2}, estr[3] = {1, 1, 1};
  EncodeFn enc = encode_fn();
  if (!enc || enc(&P.amap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(vol), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return fail("cuTensorMapEncodeTiled failed for a split volume");
  P.wmap = w->map; P.g = g; P.nchb = w->nchb; P.ntn = w->ntn;
  P.ng = sh.ng; P.tpg = sh.tpg; P.sub_w = sh.sub_w; P.box_rows = sh.box_rows; P.a_stages = sh.a_stages; P.w_stages = sh.w_stages;
  const Pieces pc = pick_pieces(g, w->ntn);
  P.pieces = pc.n; P.pairs_piece = pc.pairs; P.rows = pc.rows; P.piece_stride = pc.stride;
  P.bias = bias; P.act = act; P.slope = slope; P.F = w->F;
  P.out = o.vol; P.remap = o.remap; P.next = o.next; P.out_plane = o.remap ? o.plane : g.P * o.pitch; P.out_pitch = o.pitch; P.out_shift = ((long long)g.pd * g.Hq + g.ph) * g.Wq + g.pw;
  P.skip = o.skip; P.y = o.y; P.ys_n = o.ys_n; P.ys_d = o.ys_d; P.ys_h = o.ys_h; P.ys_w = o.ys_w; P.ys_c = o.ys_c;
  P.res = o.res; P.rs_n = o.rs_n; P.rs_d = o.rs_d; P.rs_h = o.rs_h; P.rs_w = o.rs_w; P.rs_c = o.rs_c;
  P.status = status;
  P.wait_limit = g_tc_test.wait_limit ? g_tc_test.wait_limit : kWaitLimit;
  P.test_skip_stage = g_tc_test.skip_stage;
  if (!vol_available()) return fail("convolution: shared memory or register split not available");
  const long long tiles = (long long)pc.n * pc.pairs * P.ntn, pairs = sm_count() / 2 > 0 ? sm_count() / 2 : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * (tiles < pairs ? tiles : pairs))); cfg.blockDim = dim3(kThreads); cfg.dynamicSmemBytes = sh.smem; cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  static const bool pdl = std::getenv("FORTIS_NO_PDL") == nullptr;
  cfg.attrs = at; cfg.numAttrs = (pdl && early) ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kVolKernels[4 * sh.resident + 2 * g.line + (w->NT == 64)], P);
  if (e != cudaSuccess) { if (err) *err = std::string("convolution launch: ") + cudaGetErrorString(e); return false; }
  g_launches.vol_conv++;
  return true;
}

}  // namespace fortis
