// fp32 MLP layers of many rows on pairs of CTAs, both operands read from shared memory where the TMA puts them:
// C = act(A . W^T + b), every product as three TF32 MMAs on operands that are split once.
//
// The arithmetic of an MLP step is that of f32tc_kernel (fortis_mlp_f32tc.cu), sum by sum: the three products of 8 k one after another
// (hi.hi, hi.lo, lo.hi) in one accumulator that is taken over every 128 k with IEEE additions.  The results are the same bits; this
// form takes over where there are rows and features enough for its wide tiles (f32tc_pair_wanted).
//
// Replaces the same reference lowering: fortis_gemm = cuBLAS SGEMM per layer with further kernels for bias and activation
// (runtime/fortis_rt.c:45-75, compiler/FortisFuse.cpp:616-624, 687-760), fortis_gather_k in front and fortis_scatter_k behind.
//
// Activations lie between the layers as they are multiplied: [plane x_hi | x_lo][row][feature], features padded to 32.  In f32tc_kernel
// the threads that split them (once per tile of features) set the pace: 1140 to 1520 clk a step of 32 k whose MMAs take 384 to 768.
// Here they are split once, by the layer's epilogue or while the inputs are gathered (gather_split_kernel), and no thread is in the
// operand path.
//   * tiles of 256 rows (128 a CTA, cta_group::2) x NT = 256 or 128 features; a stage is 32 k of both operands, hi and lo: 64 or 48 KB a
//     CTA; one MMA of N = 256 takes 128 clk and reads 8 KB of shared memory a CTA, the copies write 43 B/clk: bound by the tensor core.
//   * one warp copies, one issues (12 MMAs a step), two accumulators of NT columns; eight epilogue warps (thread = row, half of the
//     features) hold up to 128 sums a thread, so that the next tile's first two chunks (12,288 clk) run under a tile's end.
// Measured: column network 244 -> 768 x4 -> 128, 30,011 rows, inputs that change from call to call 749 -> 680 us (the same inputs again 757 -> 592);
// a hidden layer 316,000 -> 249,700 clk, 184,300 of them MMAs (151 us at the 1.65 GHz that the part runs at under this load): what is left is
// the tiles' ends, 262 KB of split activations stored by every CTA at about the same time.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <string>

#include "fortis_device.cuh"
#include "fortis_kernels.h"
#include "fortis_model.h"
#include "fortis_mlp_pair.h"
#include "fortis_tc.cuh"

namespace fortis {

namespace {

using namespace tc;

constexpr int kM = 128, kKt = 32, kChunkSteps = 4;
constexpr int kEWarps = 8, kWarpE0 = 4, kThreads = (kWarpE0 + kEWarps) * 32;
constexpr int kBarBytes = 512, kScratch = 32 * 32 * 4;        // one warp's 32 x 32 transpose
constexpr int kTabOut = 256;
constexpr int kSmemMax = 227 * 1024;
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
enum { PST_FULL = 21, PST_EMPTY = 22, PST_ACC_FULL = 23, PST_ACC_EMPTY = 24, PST_ALIGN = 25 };      // as f32tc_kernel numbers its waits

template <int NT> struct Cfg {
  static constexpr int kStages = NT == 256 ? 3 : 4;
  static constexpr int kABytes = 2 * kM * kKt * 4, kWHalf = NT / 2 * kKt * 4, kStage = kABytes + 2 * kWHalf;
  static constexpr int kSmem = kStages * kStage + kBarBytes + kEWarps * kScratch + (NT == 128 ? kTabOut * 8 : 0);
  static_assert(kSmem <= kSmemMax, "shared memory");
};

struct StrideClassP { long long si, sj, sk; };
struct PairParams {
  CUtensorMap map_a, map_hi, map_lo;           // A [2][rows][K_pad], box 2 x 128 x 32; W_hi / W_lo [N_pad][K_pad], box NT/2 x 32
  int nkt, ntn, N_real;
  const float* bias; int act; float slope;
  const float* out_mul; const float* relu_mask;    // last layer only, optional
  long long nrows;
  float* out; long long out_plane; int out_pitch;  // split output ...
  float* Y; long long ldc;                         // ... or row-major ...
  const Access* store_by_slot; ArrayTable TS; StrideClassP cout[2]; RowGeom g;    // ... or scattered into host arrays (NT = 128)
  double* partials; double* sum; unsigned int* done;
  int* status;
  unsigned int wait_limit; int test_skip_stage;
};

__host__ __device__ constexpr uint32_t idesc_pair(int n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)((2 * kM) >> 4) << 24);
}
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return (saddr >> 4) & 0x3FFFu; }
// 8 k: x_hi . W_hi, x_hi . W_lo, x_lo . W_hi into one accumulator, one elected lane issues
template <uint32_t IDESC>
__device__ __forceinline__ void mma_products(uint32_t d_tmem, uint32_t ah, uint32_t al, uint32_t wh, uint32_t wl, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred e, q;\n\t.reg .b64 a, b, c, d;\n\t"
      "mov.b64 a, {%1, %6};\n\tmov.b64 b, {%2, %6};\n\tmov.b64 c, {%3, %6};\n\tmov.b64 d, {%4, %6};\n\t"
      "setp.ne.b32 q, %7, 0;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::tf32 [%0], a, c, %5, q;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::tf32 [%0], a, d, %5, 1;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::tf32 [%0], b, c, %5, 1;\n\t}"
      ::"r"(d_tmem), "r"(ah), "r"(al), "r"(wh), "r"(wl), "n"(IDESC), "n"(kDescHi), "r"(accumulate) : "memory");
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {     // two IEEE additions
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
  return *reinterpret_cast<float2*>(&d);
}
// x = hi + lo, lo exact in fp32 (the MMA truncates it to TF32)
__device__ __forceinline__ void split_plain(float x, float& hi, float& lo) {
  uint32_t h;
  asm("cvt.rna.satfinite.tf32.f32 %0, %1;" : "=r"(h) : "f"(x));
  hi = __uint_as_float(h);
  lo = x - hi;
}
// A bounded wait without a function call (one register budget per role).  Every lane goes on or gives up together; a CTA in which a wait
// has given up polls no more.
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
__device__ __forceinline__ void drain_wait(uint32_t bar, uint32_t parity, uint32_t limit) {
  for (uint32_t i = 0; i < limit; i++)
    if (mbar_try_wait(bar, parity)) return;
}

template <int NT>
__global__ void __launch_bounds__(kThreads, 1) __cluster_dims__(2, 1, 1) mlp_pair_kernel(const __grid_constant__ PairParams P) {
  using CF = Cfg<NT>;
  constexpr int NH = NT / 2;                                   // features per epilogue thread
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t base = smem_u32(smem);
  if (base & 1023u) {                                          // the same in both CTAs of a pair
    if (threadIdx.x == 0) atomicCAS(P.status, 0, PST_ALIGN);
    return;
  }
  uint8_t* tail = smem + CF::kStages * CF::kStage;
  const uint32_t bars = base + CF::kStages * CF::kStage;
  // full [4] | empty [4] | acc_full [2] | acc_empty [2] | drained; at 128 the tensor-memory base, at 132 the abort flag, at 192 the
  // checksum's warp sums; then a transpose per epilogue warp and the table of the scatter
  const uint32_t full = bars, empty = bars + 32, acc_full = bars + 64, acc_empty = bars + 80, drained = bars + 96;
  uint32_t* tmem_slot = (uint32_t*)(tail + 128);
  volatile int* abort_flag = (volatile int*)(tail + 132);
  unsigned long long* o_tab = (unsigned long long*)(tail + kBarBytes + kEWarps * kScratch);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank();
  const long long npairs = (P.nrows + 2 * kM - 1) / (2 * kM), ntiles = npairs * P.ntn;
  const long long t0 = blockIdx.x >> 1, t_step = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 4; s++) { mbar_init(full + 8 * s, 1); mbar_init(empty + 8 * s, 1); }
    for (int s = 0; s < 2; s++) { mbar_init(acc_full + 8 * s, 1); mbar_init(acc_empty + 8 * s, 2 * kEWarps); }
    mbar_init(drained, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if constexpr (NT == 128)
    if (P.store_by_slot)
      for (int n = threadIdx.x; n < kTabOut; n += kThreads) {
        unsigned long long e = 0;                              // 64-bit addresses (bit 0: stride class, 0: not stored)
        if (n < P.N_real && P.store_by_slot[n].array >= 0) {
          const Access a = P.store_by_slot[n];
          const bool c0 = a.si == P.cout[0].si && a.sj == P.cout[0].sj && a.sk == P.cout[0].sk;
          e = (unsigned long long)((float*)P.TS.base[a.array] + a.off0) | (c0 ? 0ull : 1ull);
        }
        o_tab[n] = e;
      }
  if (warp == 0 && lane < 3)
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(lane == 0 ? &P.map_a : lane == 1 ? &P.map_hi : &P.map_lo)) : "memory");
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                          // both CTAs' barriers exist before either signals the other's
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  // Programmatic dependent launch, not before both CTAs have their tensor memory
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  auto wait = [&](uint32_t bar, uint32_t parity, int code) { return wait_polling(bar, parity, P.wait_limit, abort_flag, P.status, code); };

  // 56 x 128 + 224 x 256 = 168 x 384 registers: what the block is launched with (checked before the launch)
  if (warp < kWarpE0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA: both operands of every step, this CTA's rows and half of the features
      asm volatile("griddepcontrol.wait;" ::: "memory");        // what the kernel in front wrote is complete and visible
      const uint32_t full0 = map_to_cta(full, 0);
      uint32_t s = 0, ph = 0;
      bool stop = false;
      for (long long t = t0; t < ntiles && !stop; t += t_step) {
        const int m0 = (int)((2 * (t / P.ntn) + crank) * kM), n0 = (int)(t % P.ntn) * NT + (int)crank * (NT / 2);
        for (int kt = 0; kt < P.nkt; kt++) {
          if (!wait(empty + 8 * s, ph ^ 1, PST_EMPTY)) { stop = true; break; }
          const bool skip = P.test_skip_stage && blockIdx.x == 0 && t == t0 && kt == 0;    // test only: the stage never completes
          if (crank == 0) mbar_expect_tx(full + 8 * s, 2 * CF::kStage);
          const uint32_t st = base + s * CF::kStage;
          if (!skip) {
            tma_load_3d_pair(st, &P.map_a, kt * kKt, m0, 0, full0 + 8 * s);
            tma_load_2d_pair(st + CF::kABytes, &P.map_hi, kt * kKt, n0, full0 + 8 * s);
            tma_load_2d_pair(st + CF::kABytes + CF::kWHalf, &P.map_lo, kt * kKt, n0, full0 + 8 * s);
          }
          if (++s == CF::kStages) { s = 0; ph ^= 1; }
        }
      }
      if (crank == 0)
        for (uint32_t q = 0; q < CF::kStages; q++) drain_wait(full + 8 * q, q < s ? ph : ph ^ 1, P.wait_limit);
    } else if (warp == 2 && crank == 0) {
      // ---------------------------------------------------------------- MMA issuer (the leader's, for both CTAs)
      auto issue = [&]() {
        uint32_t s_ = 0, ph = 0, chunk_it = 0;
        for (long long t = t0; t < ntiles; t += t_step) {
          int in_chunk = 0;
          for (int kt = 0; kt < P.nkt; kt++) {
            const uint32_t b = chunk_it & 1;
            if (in_chunk == 0 && !wait(acc_empty + 8 * b, ((chunk_it >> 1) & 1) ^ 1, PST_ACC_EMPTY)) return;
            if (!wait(full + 8 * s_, ph, PST_FULL)) return;
            tc_fence_after();
            const uint32_t ah = __shfl_sync(0xffffffffu, desc_lo(base + s_ * CF::kStage), 0);   // uniform: see fortis_conv3d_f32.cu
            const uint32_t al = ah + (CF::kABytes >> 5), wh = ah + (CF::kABytes >> 4), wl = wh + (CF::kWHalf >> 4);
            const uint32_t acc = tmem + b * NT, first = __shfl_sync(0xffffffffu, (uint32_t)in_chunk, 0);
#pragma unroll
            for (int j = 0; j < 4; j++)                         // 8 tf32 = 32 bytes: the address field moves by 2
              mma_products<idesc_pair(NT)>(acc, ah + 2 * j, al + 2 * j, wh + 2 * j, wl + 2 * j, first | (uint32_t)j);
            tc_commit_pair(empty + 8 * s_);
            if (++in_chunk == kChunkSteps || kt == P.nkt - 1) { tc_commit_pair(acc_full + 8 * b); chunk_it++; in_chunk = 0; }
            if (++s_ == CF::kStages) { s_ = 0; ph ^= 1; }
          }
        }
      };
      issue();
      tc_commit_pair(drained);                                  // nothing may still read shared or tensor memory when the CTAs end
      drain_wait(drained, 0, P.wait_limit);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    // ------------------------------------------------------------------ epilogue: thread = row, half of the features
    asm volatile("griddepcontrol.wait;" ::: "memory");           // the buffer written here may still be read by the kernel in front
    const int quad = warp & 3, half = (warp - kWarpE0) >> 2;
    const uint32_t lane_addr = tmem + ((uint32_t)(quad * 32) << 16) + half * NH;
    float* scratch = (float*)(tail + kBarBytes + (warp - kWarpE0) * kScratch);
    const uint32_t arr_acc = map_to_cta(acc_empty, 0);           // the leader's
    const int nch = (P.nkt + kChunkSteps - 1) / kChunkSteps;
    uint32_t chunk_it = 0;
    double csum = 0.0;
    bool ok = true;
    auto act4 = [&](float (&v)[4]) {
      if (P.act == ACT_RELU) {
#pragma unroll
        for (int e = 0; e < 4; e++) v[e] = max_nan(v[e], 0.f);
      } else if (P.act == ACT_LEAKY) {
#pragma unroll
        for (int e = 0; e < 4; e++) v[e] = v[e] > 0.f ? v[e] : v[e] * P.slope;
      }
    };
    for (long long t = t0; t < ntiles && ok; t += t_step) {
      const long long mw = (2 * (t / P.ntn) + crank) * kM + quad * 32, row = mw + lane;
      const int n0 = (int)(t % P.ntn) * NT + half * NH;
      float v[NH];
#pragma unroll
      for (int j = 0; j < NH; j++) v[j] = -0.f;                  // -0 + x is x, also where x is -0
      for (int ch = 0; ch < nch; ch++, chunk_it++) {
        const uint32_t b = chunk_it & 1;
        ok = wait(acc_full + 8 * b, (chunk_it >> 1) & 1, PST_ACC_FULL);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int c0 = 0; c0 < NH; c0 += 64) {
          uint32_t a0[32], a1[32];
          tmem_ld32(lane_addr + b * NT + c0, a0);
          tmem_ld32(lane_addr + b * NT + c0 + 32, a1);
          tmem_ld_wait();
          if (c0 + 64 == NH) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster_relaxed(arr_acc + 8 * b);
          }
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float2 x = add2(make_float2(v[c0 + j], v[c0 + j + 1]), make_float2(__uint_as_float(a0[j]), __uint_as_float(a0[j + 1])));
            const float2 y = add2(make_float2(v[c0 + 32 + j], v[c0 + 33 + j]), make_float2(__uint_as_float(a1[j]), __uint_as_float(a1[j + 1])));
            v[c0 + j] = x.x; v[c0 + j + 1] = x.y; v[c0 + 32 + j] = y.x; v[c0 + 33 + j] = y.y;
          }
        }
      }
      if (!ok) break;
      if (NT == 128 && P.store_by_slot) {
        // lane = row: every store writes 32 neighbouring elements of a host array
        float bl[NH / 32], ml[NH / 32], rl[NH / 32];             // of feature n0 + 32 i + lane
#pragma unroll
        for (int i = 0; i < NH / 32; i++) {
          const int n = n0 + 32 * i + lane;
          const bool real = n < P.N_real;
          bl[i] = P.bias && real ? __ldg(P.bias + n) : 0.f;
          ml[i] = P.out_mul && real ? __ldg(P.out_mul + n) : 1.f;
          rl[i] = P.relu_mask && real ? __ldg(P.relu_mask + n) : 0.f;
        }
        const bool live = row < P.nrows;
        long long ci, cj, kk;
        row_to_pos(P.g, live ? row : 0, &ci, &cj, &kk);
        const long long op0 = 4 * (ci * P.cout[0].si + cj * P.cout[0].sj + kk * P.cout[0].sk);
        const long long op1 = 4 * (ci * P.cout[1].si + cj * P.cout[1].sj + kk * P.cout[1].sk);
#pragma unroll
        for (int j = 0; j < NH; j += 4) {
          float o[4];
#pragma unroll
          for (int e = 0; e < 4; e++) o[e] = v[j + e] + __shfl_sync(0xffffffffu, bl[j / 32], (j + e) & 31);
          act4(o);
#pragma unroll
          for (int e = 0; e < 4; e++) {
            if (P.out_mul) o[e] *= __shfl_sync(0xffffffffu, ml[j / 32], (j + e) & 31);
            if (P.relu_mask && __shfl_sync(0xffffffffu, rl[j / 32], (j + e) & 31) != 0.f) o[e] = max_nan(o[e], 0.f);
            const unsigned long long a = n0 + j + e < kTabOut ? o_tab[n0 + j + e] : 0ull;
            if (live && a != 0ull) {
              *reinterpret_cast<float*>((a & ~1ull) + (unsigned long long)((a & 1ull) ? op1 : op0)) = o[e];
              csum += (double)o[e];
            }
          }
        }
        continue;
      }
      // blocks of 32 rows x 32 features turned in shared memory: whole lines of a row, eight lanes each.  One compact loop, the sums moved
      // down after each block: straight code for all blocks took longer to fetch (26,000 clk a tile) than two chunks to multiply.
      const int c = lane & 7;
      float b[NH / 32][4];
#pragma unroll
      for (int k = 0; k < NH / 32; k++)
#pragma unroll
        for (int e = 0; e < 4; e++) b[k][e] = P.bias && n0 + 32 * k + 4 * c + e < P.N_real ? __ldg(P.bias + n0 + 32 * k + 4 * c + e) : 0.f;
#pragma unroll 1
      for (int c0 = 0; c0 < NH; c0 += 32) {
#pragma unroll
        for (int i = 0; i < 8; i++)
          *reinterpret_cast<float4*>(scratch + lane * 32 + ((i ^ (lane & 7)) << 2)) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        __syncwarp();
        const int n = n0 + c0 + 4 * c;
#pragma unroll 2
        for (int i = 0; i < 8; i++) {
          const int rr = 4 * i + (lane >> 3);
          const float4 q = *reinterpret_cast<const float4*>(scratch + rr * 32 + ((c ^ (rr & 7)) << 2));
          float o[4] = {q.x + b[0][0], q.y + b[0][1], q.z + b[0][2], q.w + b[0][3]};
          act4(o);
          if (P.out) {
            float h[4], l[4];
#pragma unroll
            for (int e = 0; e < 4; e++) split_plain(n + e < P.N_real ? o[e] : 0.f, h[e], l[e]);
            if (mw + rr < P.nrows && n < P.out_pitch) {
              float* dst = P.out + (mw + rr) * P.out_pitch + n;
              *reinterpret_cast<float4*>(dst) = make_float4(h[0], h[1], h[2], h[3]);
              *reinterpret_cast<float4*>(dst + P.out_plane) = make_float4(l[0], l[1], l[2], l[3]);
            }
          } else if (mw + rr < P.nrows) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
              if (n + e >= P.N_real) continue;
              if (P.out_mul) o[e] *= __ldg(P.out_mul + n + e);
              if (P.relu_mask && __ldg(P.relu_mask + n + e) != 0.f) o[e] = max_nan(o[e], 0.f);
              P.Y[(mw + rr) * P.ldc + n + e] = o[e];
            }
          }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j + 32 < NH; j++) v[j] = v[j + 32];
#pragma unroll
        for (int k = 0; k + 1 < NH / 32; k++)
#pragma unroll
          for (int e = 0; e < 4; e++) b[k][e] = b[k + 1][e];
      }
    }
    if (P.partials) {
      // per-CTA checksum partial in a fixed order; the last CTA to finish folds all partials into the step checksum
      double* wsum = (double*)(tail + 192);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) csum += __shfl_down_sync(0xffffffffu, csum, o);
      if (lane == 0) wsum[warp - kWarpE0] = csum;
      asm volatile("bar.sync 1, %0;" ::"n"(kEWarps * 32) : "memory");
      if (warp == kWarpE0 && lane == 0) {
        double part = 0.0;
        for (int w = 0; w < kEWarps; w++) part += wsum[w];
        P.partials[blockIdx.x] = part;
        if (P.sum) {
          __threadfence();
          if (atomicAdd(P.done, 1u) == gridDim.x - 1) {
            __threadfence();
            double total = *P.sum;
            for (unsigned i = 0; i < gridDim.x; i++) total += __ldcg(P.partials + i);
            *P.sum = total;
            *P.done = 0u;
          }
        }
      }
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

// Model inputs -> split rows: 128 rows x 32 inputs per block, turned in shared memory.  From host arrays through the slot table (lane =
// row: a load reads 32 neighbouring elements; a thread has 16 in flight) ...
__global__ void __launch_bounds__(256) gather_split_kernel(const Access* __restrict__ slots, ArrayTable T, RowGeom g, int n_in, const float* __restrict__ in_div,
                                                           float* __restrict__ out, long long plane, int pitch, long long nrows) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the first layer may set up while this kernel runs
  __shared__ float tile[128][33];
  const long long r0 = (long long)blockIdx.x * 128;
  const int c0 = blockIdx.y * 32, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  long long ci[4], cj[4], kk[4];
#pragma unroll
  for (int i = 0; i < 4; i++) row_to_pos(g, r0 + i * 32 + lane < nrows ? r0 + i * 32 + lane : nrows - 1, &ci[i], &cj[i], &kk[i]);
  float v[4][4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int c = c0 + warp * 4 + k;
    const bool real = c < n_in;
    const Access a = slots[real ? c : 0];
    const float* base = (const float*)T.base[a.array] + a.off0;
#pragma unroll
    for (int i = 0; i < 4; i++) v[k][i] = real ? __ldg(base + (ci[i] * a.si + cj[i] * a.sj + kk[i] * a.sk)) : 0.f;
  }
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int c = c0 + warp * 4 + k;
    if (in_div && c < n_in) {
      const float d = __ldg(in_div + c);
#pragma unroll
      for (int i = 0; i < 4; i++) v[k][i] = __fdiv_rn(v[k][i], d);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) tile[i * 32 + lane][warp * 4 + k] = v[k][i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int rr = i * 32 + (threadIdx.x >> 3), c = (threadIdx.x & 7) * 4;
    if (r0 + rr >= nrows) continue;
    float h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; e++) split_plain(tile[rr][c + e], h[e], l[e]);
    float* o = out + (r0 + rr) * pitch + c0 + c;
    *reinterpret_cast<float4*>(o) = make_float4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<float4*>(o + plane) = make_float4(l[0], l[1], l[2], l[3]);
  }
}
// ... or from a row-major matrix
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ X, int n_in, const float* __restrict__ in_div, float* __restrict__ out,
                                                         long long plane, int pitch, long long nrows) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const long long n = nrows * (pitch / 4);
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
    const long long r = i / (pitch / 4);
    const int c = (int)(i - r * (pitch / 4)) * 4;
    float h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      float v = c + e < n_in ? __ldg(X + r * n_in + c + e) : 0.f;
      if (in_div && c + e < n_in) v = __fdiv_rn(v, __ldg(in_div + c + e));
      split_plain(v, h[e], l[e]);
    }
    *reinterpret_cast<float4*>(out + r * pitch + c) = make_float4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<float4*>(out + plane + r * pitch + c) = make_float4(l[0], l[1], l[2], l[3]);
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

int pairs_on_device() {
  static int n = 0;
  if (n) return n;
  int sms = 148, dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return n = sms / 2 > 0 ? sms / 2 : 1;
}

template <int NT>
bool launch(PairParams& P, cudaStream_t s, std::string* err) {
  if (!pair_available()) { if (err) *err = "pair kernel: shared memory or register split not available"; return false; }
  P.wait_limit = g_tc_test.wait_limit ? g_tc_test.wait_limit : kWaitLimit;
  P.test_skip_stage = g_tc_test.skip_stage;
  const long long tiles = (P.nrows + 2 * kM - 1) / (2 * kM) * P.ntn, pairs = pairs_on_device();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * (tiles < pairs ? tiles : pairs))); cfg.blockDim = dim3(kThreads); cfg.dynamicSmemBytes = Cfg<NT>::kSmem; cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  static const bool pdl = std::getenv("FORTIS_NO_PDL") == nullptr;
  cfg.attrs = at; cfg.numAttrs = pdl ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, mlp_pair_kernel<NT>, P);
  if (e != cudaSuccess) { if (err) *err = std::string("pair kernel launch: ") + cudaGetErrorString(e); return false; }
  g_launches.mlp_pair++;
  return true;
}

template <int NT>
bool available() {
  cudaFuncAttributes fa;
  const bool ok = cudaFuncSetAttribute(mlp_pair_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<NT>::kSmem) == cudaSuccess &&
                  cudaFuncGetAttributes(&fa, mlp_pair_kernel<NT>) == cudaSuccess && fa.numRegs == 168;
  if (!ok) cudaGetLastError();
  return ok;
}

}  // namespace

// The register split adds up only with what the compiler gave the kernel (168 a thread); with another compiler's number the layers stay
// on f32tc_kernel.
bool pair_available() {
  static const bool ok = available<256>() && available<128>();
  return ok;
}

// 256 features a tile, or 128 where that takes fewer rounds of tiles (a step 1536 or 900 clk) or the outputs are scattered
bool pair_wide(long long nrows, int N, bool scatter) {
  if (scatter || N <= 128) return false;
  const long long ntm = (nrows + 2 * kM - 1) / (2 * kM), pairs = pairs_on_device();
  return (ntm * ((N + 255) / 256) + pairs - 1) / pairs * 1536 <= (ntm * ((N + 127) / 128) + pairs - 1) / pairs * 900;
}

void pair_split_gathered(const Access* slots, const ArrayTable& T, const RowGeom& g, int n_in, const float* in_div, float* out, long long nrows, cudaStream_t s) {
  const int pitch = (n_in + 31) / 32 * 32;
  gather_split_kernel<<<dim3((unsigned)((nrows + 127) / 128), (unsigned)(pitch / 32)), 256, 0, s>>>(slots, T, g, n_in, in_div, out, nrows * pitch, pitch, nrows);
}
void pair_split_rows(const float* X, int n_in, const float* in_div, float* out, long long nrows, cudaStream_t s) {
  const int pitch = (n_in + 31) / 32 * 32;
  const long long blocks = (nrows * (pitch / 4) + 255) / 256;
  split_rows_kernel<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, s>>>(X, n_in, in_div, out, nrows * pitch, pitch, nrows);
}

bool pair_layer(const PairLayer& L, cudaStream_t s, std::string* err) {
  PairParams P;
  std::memset(&P, 0, sizeof P);
  const int K_pad = (L.K + 31) / 32 * 32;
  const cuuint64_t dims[3] = {(cuuint64_t)K_pad, (cuuint64_t)L.nrows, 2}, strides[2] = {(cuuint64_t)K_pad * 4, (cuuint64_t)L.nrows * K_pad * 4};
  const cuuint32_t box[3] = {kKt, kM, 2}, estr[3] = {1, 1, 1};
  EncodeFn enc = encode_fn();
  if (!enc || enc(&P.map_a, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(L.a), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
    if (err) *err = "cuTensorMapEncodeTiled failed for split activations";
    return false;
  }
  const bool wide = pair_wide(L.nrows, L.N, L.store_by_slot != nullptr);
  const int NT = wide ? 256 : 128;
  P.map_hi = *L.map_hi[wide]; P.map_lo = *L.map_lo[wide];
  P.nkt = K_pad / kKt; P.ntn = (L.N + NT - 1) / NT; P.N_real = L.N;
  P.bias = L.bias; P.act = L.act; P.slope = L.slope; P.out_mul = L.out_mul; P.relu_mask = L.relu_mask; P.nrows = L.nrows;
  P.out_pitch = (L.N + 31) / 32 * 32; P.out = L.out; P.out_plane = L.nrows * P.out_pitch;
  P.Y = L.Y; P.ldc = L.N;
  P.store_by_slot = L.store_by_slot; P.TS = L.TS; P.g = L.g;
  for (int i = 0; i < 2; i++) P.cout[i] = StrideClassP{L.cout[i][0], L.cout[i][1], L.cout[i][2]};
  P.partials = L.partials; P.sum = L.sum; P.done = L.done; P.status = L.status;
  return wide ? launch<256>(P, s, err) : launch<128>(P, s, err);
}

}  // namespace fortis
