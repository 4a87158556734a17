// Recurrent half of the LSTM layer: T sequential steps
//     gates[b, 4H] = ih[t, b, 4H] + (h_{t-1} . W_hh^T) * (s_hh[n] / 448) + bias[n]      (gate blocks i | f | g | o)
//     c_t = sigmoid(f) * c_{t-1} + sigmoid(i) * tanh(g);   h_t = sigmoid(o) * tanh(c_t)
// in ONE persistent cooperative kernel (the reference replays two launches per step from a graph,
// fly/bench_factored_lstm.py:106-121).  `ih` is the hoisted input projection for all timesteps (an FP8 GEMM of
// this library); h feeds the recurrent GEMM as E4M3 at the fixed scale 1/448 (the reference's convention for a
// value bounded by 1, fly/rdna_fp8_factored_lstm.py:321-326); c and the emitted h are fp16.
//
// Two kernels with the same arithmetic, and the same order of the sums (K = 0 .. H - 1), so that they give the same bytes:
//   lstm_tmem_kernel       what runs: W_hh in tensor memory, gates^T = W_hh . h^T, h exchanged between at most four CTAs
//   lstm_recurrent_kernel  128 batch rows x 32 hidden units per CTA, h through global memory (cooperative launch)
// The second is for a device that cannot host the first one's clusters, and the tests' second opinion (environment variables).
//
// In it, CTA (g, s) owns 128 batch rows (row group g) x 32 hidden units (slice s) = 128 gate columns.
// Its W_hh slice (128 rows x H bytes) stays in shared memory for the whole layer, c_t stays in registers.
// Batch rows are independent, so only the H/32 CTAs of a row group exchange data: each step every CTA of the cooperative
// kernel writes its 128 x 32 piece of h_t (E4M3) to a double-buffered global scratch and bumps its step counter;
// the others poll the counters (bounded), pull the full 128 x H tile into 128B-swizzled shared memory and
// run 128 x 128 x H on the tensor core (tcgen05 kind::f8f6f4, fp32 accumulators in TMEM).  The next step's ih tile
// is prefetched by TMA while the current step computes.
#include <cooperative_groups.h>
#include <cuda_fp8.h>

#include <atomic>
#include <type_traits>

#include "capi_internal.h"
#include "ptx.cuh"

namespace gsb {

constexpr int LSTM_THREADS = 256;            // 8 warps: all load / do gate math; warp 0 lane 0 also issues TMA + MMA
constexpr int LSTM_ROWS = 128;               // batch rows per CTA (UMMA M)
constexpr int LSTM_HS = 32;                  // hidden units per CTA
constexpr int LSTM_NCOL = 4 * LSTM_HS;       // gate columns per CTA (UMMA N)
constexpr int LSTM_MAX_KB = 4;               // H <= 512
constexpr int LSTM_PULLS = LSTM_ROWS * LSTM_MAX_KB * 8 / LSTM_THREADS;   // 16-byte pieces of h per thread and step (at most)
constexpr int LSTM_KB_BYTES = LSTM_ROWS * 128;                 // one 128-byte K block of a 128-row operand tile
constexpr int LSTM_IH_BYTES = LSTM_ROWS * LSTM_NCOL * 2;       // 32 KiB: four 128 x 32 fp16 boxes
constexpr int LSTM_SMEM_W = 0;
constexpr int LSTM_SMEM_H = LSTM_SMEM_W + LSTM_MAX_KB * LSTM_KB_BYTES;
constexpr int LSTM_SMEM_IH = LSTM_SMEM_H + LSTM_MAX_KB * LSTM_KB_BYTES;
constexpr int LSTM_SMEM_SC = LSTM_SMEM_IH + 2 * LSTM_IH_BYTES;   // 128 scales + 128 biases (fp32)
constexpr int LSTM_SMEM_BAR = LSTM_SMEM_SC + 1024;
constexpr int LSTM_SMEM_USED = LSTM_SMEM_BAR + 128;
constexpr int LSTM_SMEM_BYTES = LSTM_SMEM_USED + 1024;           // + alignment slack
static_assert(LSTM_SMEM_BYTES > 116 * 1024, "one CTA per SM");

struct LstmParams {
  int T, B, H;
  int reverse;                 // 1: iterate t = T-1 .. 0
  int k_blocks;                // ceil(H / 128)
  int slices;                  // H / 32
  const float* s_hh;           // [4H] per-channel scales of W_hh
  const float* bias;           // [4H] or null (b_ih + b_hh)
  const uint8_t* h0;           // [B, H] E4M3 at scale 1/448, or null (zeros)
  const __half* c0;            // [B, H] or null (zeros)
  __half* h_out;               // [T*B, H] fp16, row = t*B + b, or null
  uint8_t* h8_out;             // [T*B, H] E4M3 at scale 1/448 (input of the next layer's projection), or null
  __half* c_last;              // [B, H] final cell state, or null
  uint8_t* hbuf;               // scratch: [2][B][H] E4M3, h of the previous / current step
  unsigned int* flags;         // scratch: [row groups][slices] step counters, zero at launch
};

__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_gpu(unsigned int* p, unsigned int v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Gate functions on the hardware tanh (one special-function instruction each, relative error about 2^-11):
// sigmoid(x) = 0.5 + 0.5 * tanh(x / 2).
__device__ __forceinline__ float tanh_f(float x) { return tanh_approx(x); }
__device__ __forceinline__ float sigmoid_f(float x) { return fmaf(0.5f, tanh_approx(0.5f * x), 0.5f); }

__global__ void __launch_bounds__(LSTM_THREADS, 1)
lstm_recurrent_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_ih,
                      const LstmParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* w_s = smem + LSTM_SMEM_W;
  uint8_t* h_s = smem + LSTM_SMEM_H;
  uint8_t* ih_s = smem + LSTM_SMEM_IH;
  float* sc_s = reinterpret_cast<float*>(smem + LSTM_SMEM_SC);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + LSTM_SMEM_BAR);
  uint64_t* w_full = bars;               // W slice landed
  uint64_t* ih_full = bars + 1;          // [2] ih tile of a step landed
  uint64_t* mma_done = bars + 3;         // accumulator of this step complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);
  const AbortFlag abort_flag{smem_u32(tmem_slot + 1)};

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int grp = blockIdx.x / p.slices;        // row group
  const int slc = blockIdx.x % p.slices;        // hidden slice
  const int row0 = grp * LSTM_ROWS;
  const int hid0 = slc * LSTM_HS;
  const int H = p.H, B = p.B;

  if (tid == 0) {
    mbar_init(w_full, 1); mbar_init(&ih_full[0], 1); mbar_init(&ih_full[1], 1); mbar_init(mma_done, 1);
    abort_flag.set(0);
    fence_mbar_init();
    prefetch_tmap(&tm_w); prefetch_tmap(&tm_ih);
  }
  if (warp == 0) { tmem_alloc(tmem_slot, LSTM_NCOL); tmem_relinquish(); }
  // per-channel scale (with the 1/448 of h folded in) and bias of this CTA's 128 gate columns
  if (tid < LSTM_NCOL) {
    const int n = (tid >> 5) * H + hid0 + (tid & 31);
    sc_s[tid] = __ldg(p.s_hh + n) * (1.0f / 448.0f);
    sc_s[LSTM_NCOL + tid] = p.bias ? __ldg(p.bias + n) : 0.f;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const unsigned int budget = spin_budget();          // bound of every wait below, fetched once

  auto step_t = [&](int s) { return p.reverse ? p.T - 1 - s : s; };
  auto issue_ih = [&](int s) {   // one thread: TMA the four gate boxes of step s into buffer s & 1
    uint8_t* dst = ih_s + (s & 1) * LSTM_IH_BYTES;
    mbar_arrive_expect_tx(&ih_full[s & 1], LSTM_IH_BYTES);
    const int r = step_t(s) * B + row0;
#pragma unroll
    for (int g = 0; g < 4; ++g) tma_load_2d(dst + g * (LSTM_ROWS * LSTM_HS * 2), &tm_ih, &ih_full[s & 1], g * H + hid0, r);
  };
  if (tid == 0) {
    mbar_arrive_expect_tx(w_full, p.k_blocks * LSTM_KB_BYTES);
    for (int kb = 0; kb < p.k_blocks; ++kb)
#pragma unroll
      for (int g = 0; g < 4; ++g)
        tma_load_2d(w_s + kb * LSTM_KB_BYTES + g * (LSTM_HS * 128), &tm_w, w_full, kb * 128, g * H + hid0);
    issue_ih(0);
    if (p.T > 1) issue_ih(1);
  }

  // this thread's part of the tile: row (TMEM lane) q*32 + lane, hidden units half*16 .. +15 of the slice
  const int q = warp & 3, half = warp >> 2;
  const int r_loc = q * 32 + lane;
  const int row = row0 + r_loc;
  const bool row_ok = row < B;
  float c[16];
#pragma unroll
  for (int j = 0; j < 16; ++j)
    c[j] = (p.c0 && row_ok) ? __half2float(p.c0[(long long)row * H + hid0 + half * 16 + j]) : 0.f;

  bool ok = mbar_wait(w_full, 0, abort_flag, ST_TIMEOUT_LSTM, 0x10, budget);
  unsigned int* my_flags = p.flags + grp * p.slices;
  // The 16-byte pieces of the 128 x H tile of h this thread moves every step.  Piece i of a thread is row
  // (tid / 8) + 32 * (i % 4), 16-byte chunk tid % 8 of K block i / 4: eight neighbouring threads read one 128-byte
  // line, and both offsets are one per-thread base plus constants known at compile time (no per-piece state).
  const int pull_r = tid >> 3, pull_ck = tid & 7;
  const int pull_dst0 = pull_r * 128 + ((pull_ck ^ (pull_r & 7)) << 4);         // + kb * LSTM_KB_BYTES + j * 32 * 128
  const long long pull_src0 = (long long)(row0 + pull_r) * H + pull_ck * 16;     // + kb * 128 + j * 32 * H

  for (int s = 0; s < p.T; ++s) {
    // ---- 1. wait until every slice of this row group has published h_{s-1} -----------------------------
    const uint8_t* h_prev = (s == 0) ? p.h0 : p.hbuf + (size_t)((s + 1) & 1) * B * H;
    if (s > 0 && tid < p.slices) {
      long long t0 = clock64();
      while (ld_acquire_gpu(my_flags + tid) < (unsigned int)s) {
        if (abort_flag.get()) break;
        if (clock64() - t0 > budget) {
          abort_flag.set(1);
          atomicOr(&g_status[0], ST_TIMEOUT_LSTM);
          g_status[1] = (unsigned int)s;
          break;
        }
      }
    }
    __syncthreads();
    if (abort_flag.get() || !ok) break;
    // ---- 2. pull the 128 x H tile of h_{s-1} into the swizzled K-major operand layout ------------------
    // All of a thread's loads are issued before the first store, so their L2 latencies overlap (one after the
    // other they were the longest part of the step).
    {
      uint4 v[LSTM_PULLS];
#pragma unroll
      for (int i = 0; i < LSTM_PULLS; ++i) {
        const int kb = i >> 2, j = i & 3;
        v[i] = make_uint4(0, 0, 0, 0);
        if (h_prev && kb < p.k_blocks && row0 + pull_r + 32 * j < B && kb * 128 + pull_ck * 16 < H)
          v[i] = __ldcg(reinterpret_cast<const uint4*>(h_prev + pull_src0 + (long long)j * 32 * H + kb * 128));
      }
#pragma unroll
      for (int i = 0; i < LSTM_PULLS; ++i) {
        const int kb = i >> 2, j = i & 3;
        if (kb < p.k_blocks) *reinterpret_cast<uint4*>(h_s + pull_dst0 + kb * LSTM_KB_BYTES + j * (32 * 128)) = v[i];
      }
    }
    fence_proxy_async_smem();
    __syncthreads();
    // ---- 3. gates += h . W^T on the tensor core ----------------------------------------------------------
    if (tid == 0) {
      tc_fence_after();
      constexpr uint32_t idesc = umma_idesc(1, 0, 0, LSTM_ROWS, LSTM_NCOL);
      for (int kb = 0; kb < p.k_blocks; ++kb) {
        const uint64_t a_desc = umma_smem_desc_sw128(smem_u32(h_s + kb * LSTM_KB_BYTES));
        const uint64_t b_desc = umma_smem_desc_sw128(smem_u32(w_s + kb * LSTM_KB_BYTES));
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_f8(tmem_base, a_desc + 2 * k, b_desc + 2 * k, idesc, (kb | k) != 0);
      }
      umma_commit(mma_done);
    }
    // ---- 4. gate math on this thread's row ---------------------------------------------------------------
    ok = mbar_wait(&ih_full[s & 1], (s >> 1) & 1, abort_flag, ST_TIMEOUT_LSTM, 0x20, budget) &&
         mbar_wait(mma_done, s & 1, abort_flag, ST_TIMEOUT_LSTM, 0x30, budget);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tc_fence_after();
      uint32_t acc[4][16];
      const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16);
#pragma unroll
      for (int g = 0; g < 4; ++g) tmem_ld_32x32b_x16(t_row + g * LSTM_HS + half * 16, acc[g]);
      tmem_ld_wait(acc[0], acc[1], acc[2], acc[3]);
      const uint8_t* ihb = ih_s + (s & 1) * LSTM_IH_BYTES;
      float hv[16];
#pragma unroll
      for (int j0 = 0; j0 < 16; j0 += 8) {
        float pre[4][8];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          // 8 fp16 of gate g: one 16-byte piece of this row in the 64-byte-swizzled box
          const int piece = half * 2 + (j0 >> 3);
          const uint4 raw = *reinterpret_cast<const uint4*>(ihb + g * (LSTM_ROWS * LSTM_HS * 2) + r_loc * 64 +
                                                            ((piece ^ ((r_loc >> 1) & 3)) << 4));
          const __half2* h2 = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(h2[i]);
            const int col = g * LSTM_HS + half * 16 + j0 + 2 * i;
            pre[g][2 * i] = fmaf(__uint_as_float(acc[g][j0 + 2 * i]), sc_s[col], f.x + sc_s[LSTM_NCOL + col]);
            pre[g][2 * i + 1] = fmaf(__uint_as_float(acc[g][j0 + 2 * i + 1]), sc_s[col + 1], f.y + sc_s[LSTM_NCOL + col + 1]);
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float ig = sigmoid_f(pre[0][i]), fg = sigmoid_f(pre[1][i]), gg = tanh_f(pre[2][i]), og = sigmoid_f(pre[3][i]);
          const float cn = fmaf(fg, c[j0 + i], ig * gg);
          hv[j0 + i] = og * tanh_f(cn);
          c[j0 + i] = __half2float(__float2half_rn(cn));        // the cell state is carried in fp16
        }
      }
      uint32_t w8[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(hv[4 * i] * 448.f, hv[4 * i + 1] * 448.f), __NV_SATFINITE, __NV_E4M3);
        const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(hv[4 * i + 2] * 448.f, hv[4 * i + 3] * 448.f), __NV_SATFINITE, __NV_E4M3);
        w8[i] = lo | (hi << 16);
      }
      const size_t off = (size_t)row * H + hid0 + half * 16;
      // the piece the other slices wait for goes out first
      if (row_ok) *reinterpret_cast<uint4*>(p.hbuf + (size_t)(s & 1) * B * H + off) = make_uint4(w8[0], w8[1], w8[2], w8[3]);
      tc_fence_before();
      __syncthreads();
      // ---- 5. publish: one release store after the CTA barrier covers every thread's piece (the release is
      //         cumulative over what the barrier ordered before it); then prefetch the ih tile two steps ahead
      if (tid == 0) {
        st_release_gpu(my_flags + slc, (unsigned int)(s + 1));
        if (s + 2 < p.T) issue_ih(s + 2);
      }
      // ---- 6. the layer's outputs, off the other slices' critical path -------------------------------------
      if (row_ok) {
        const size_t toff = (size_t)step_t(s) * B * H + off;
        if (p.h8_out) *reinterpret_cast<uint4*>(p.h8_out + toff) = make_uint4(w8[0], w8[1], w8[2], w8[3]);
        if (p.h_out) {
          uint32_t w16[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) w16[i] = pack_half2(hv[2 * i], hv[2 * i + 1]);
          *reinterpret_cast<uint4*>(p.h_out + toff) = make_uint4(w16[0], w16[1], w16[2], w16[3]);
          *reinterpret_cast<uint4*>(p.h_out + toff + 8) = make_uint4(w16[4], w16[5], w16[6], w16[7]);
        }
      }
    } else {
      tc_fence_before();
      __syncthreads();
    }
    if (!ok || abort_flag.get()) break;
  }

  if (p.c_last && row_ok) {
#pragma unroll
    for (int j = 0; j < 16; ++j) p.c_last[(long long)row * H + hid0 + half * 16 + j] = __float2half_rn(c[j]);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) { tc_fence_after(); tmem_dealloc(tmem_base, LSTM_NCOL); }
}

// ---- transposed form: W_hh in tensor memory, the batch as the N dimension ------------------------------------------
// gates^T = W_hh . h^T: a CTA owns 128 hidden units and G = 4, 8, 12, 16 or 32 batch rows (N = R = 16 or 32 columns of the
// MMA; columns without a row multiply zeros).  The four gates of its hidden units are four M = 128 x N = R accumulators, so
// a cell's four gate values sit in one TMEM lane and one thread has them all.  The A operand, W_hh (4 x 128 rows x up to
// 384 bytes), is written to tensor memory once per launch (384 of its 512 columns; a fourth K block, H > 384, stays in
// shared memory).
//
// A step is latency end to end: MMAs (issue-bound: 12 per gate at H = 384), accumulator to registers, gate math, h to the
// other CTAs of the row group, MMAs.  What the split buys:
//  * a row group is ceil(H / 128) CTAs instead of H / 32, so h goes to at most three other CTAs.  (With 32 units per CTA a
//    step's all-gather was twelve bulk copies per CTA and half at 220 clocks each, all of the step's 2.7 us.)  It leaves
//    with st.async straight after the gate math, half of a warp's rows at a time, 16 bytes per lane, and reports to the
//    receiver's mbarrier; a bulk copy from a warp of its own is as fast for two receivers (1.62 us per step) and slower
//    for one, plain remote stores with a releasing arrive cost 1300 clocks (2.10 us).
//  * the batch is the small dimension, so B = 512 spreads over 129 SMs (G = 12) instead of 48: the gate math, five
//    special-function instructions per cell, is 1000 clocks for 2048 cells (G = 16), 600 for 1024.
//  * W_hh in tensor memory: an MMA from a shared-memory A operand of 128 rows takes 40 clocks, from TMEM 16.
// B = 512, H = 384: 1.03 us per step (2.57 with the 128-row tiles), H = 512: 1.74 (4.8), H = 256: 0.78 (2.29), H = 128: 0.54 (2.27).
// It was 1.34 / 1.93 / 0.93 / 0.57 before four changes to how its warps wait and issue.  An MMA warp walks its loop converged, with
// one elected lane issuing (a single thread moves the operands of every MMA to uniform registers): 1.22 / 1.84 / 0.84 / 0.56.  The
// gate warps report to it through named barriers instead of an mbarrier: 1.21 / 1.84 / 0.83 / 0.56.  The waits on the chain, for the
// accumulators and for the other CTAs' h, do not suggest to the hardware how long to stay suspended: 1.12 / 1.73 /
// 0.82 / 0.56.  The steps are unrolled by two (below): the rest.
// The K blocks are summed in ascending order on every CTA.  Starting with the CTA's own block, which is there first, takes
// 1.25 us at H = 384 and 1.81 at H = 512, but sums in an order that depends on the CTA: the last bit of a sum changes, an E4M3
// rounding of h flips with it, and after five layers of 2000 steps the outputs differ by 5e-3.  There is a
// barrier per sending CTA, so that the first blocks' MMAs do not wait for the last piece.
// Clocks of a step before that order and the converged warps (G = 16, H = 384, of ~2650): MMAs 900, wait for the others' h 300 of
// the 640 it is under way, commit to registers 300, gate math and sending 1000, hand-over to the MMA warps 130.
//   warps 0 .. CW-1   gate math.  Warp w: TMEM lane quarter w % 4 (32 hidden units, one per lane), G / (CW / 4) batch rows
//   last four warps   MMA issue, one gate each (the MMAs of a gate add to one accumulator, one after the other); the last one also
//                     issues the TMA loads of the ih tiles
// h is kept as K-major rows of 128 bytes with the 128-byte swizzle, one K block per CTA of the row group: a CTA's piece is
// one K block, written by its own gate warps where its own MMAs read it and sent from there to the others.
// h_t goes to buffer t & 1; the MMAs of step t read buffer (t + 1) & 1.  Buffer t & 1 may be written in step t: the MMAs of
// step t - 1 that read it are complete (here: this CTA has waited for them; there: the sender got our h_{t-1}, sent after
// them).
constexpr int LT_HS = 128;                                     // hidden units per CTA (UMMA M)
constexpr int LT_TMEM_KB = 3;                                  // K blocks of W_hh in tensor memory
constexpr int LT_ACC_COL = 4 * LT_TMEM_KB * 32;                // accumulator columns start here (gate g: + g * R)
constexpr int LT_MAX_SLICES = 4;                               // H <= 512
constexpr int LT_STAGES = 3;                                   // ih tiles in flight

template <int R, int G>
struct LtSmem {
  static constexpr int KB_BYTES = R * 128;                     // one K block of h
  static constexpr int HBUF = LT_MAX_SLICES * KB_BYTES;
  static constexpr int IH_GATE = G * LT_HS * 2;
  static constexpr int IH_BYTES = 4 * IH_GATE;
  static constexpr int H = 0;                                  // [2][HBUF]
  static constexpr int IH = H + 2 * HBUF;                      // [LT_STAGES][IH_BYTES]
  static constexpr int BAR = IH + LT_STAGES * IH_BYTES;
  static constexpr int W = BAR + 1024;                         // fourth K block of W_hh: four gates x 16 KiB (H > 384 only)
  static constexpr int bytes(int slices) { return W + (slices > LT_TMEM_KB ? 4 * LSTM_KB_BYTES : 0) + 1024; }
};
static_assert(LtSmem<32, 32>::bytes(4) <= 227 * 1024, "shared memory budget");

template <int R, int G, int CW>
__global__ void __launch_bounds__(32 * (CW + 4), 1)
lstm_tmem_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_ih, const uint8_t* __restrict__ w_hh,
                 long long ld_w, const LstmParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  using L = LtSmem<R, G>;
  constexpr int RPT = G / (CW / 4);                // batch rows per gate thread
  static_assert(RPT == 4 || RPT == 8, "rows per thread");
  uint8_t* h_s = smem + L::H;
  uint8_t* ih_s = smem + L::IH;
  uint8_t* w_s = smem + L::W;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR);
  uint64_t* ih_full = bars;                        // [LT_STAGES]
  uint64_t* h_ready = ih_full + LT_STAGES;         // [2][LT_MAX_SLICES] the piece of each other CTA has landed (bytes counted)
  uint64_t* mma_done = h_ready + 2 * LT_MAX_SLICES;                // the four gates' accumulators are complete
  uint64_t* w_full = mma_done + 1;                 // the fourth K block of W_hh has landed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(w_full + 1);
  const AbortFlag abort_flag{smem_u32(tmem_slot + 1)};

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int grp = blockIdx.x / p.slices;           // row group = cluster
  const int slc = blockIdx.x % p.slices;           // hidden slice = rank inside the cluster = its K block of h
  const int row0 = grp * G, hid0 = slc * LT_HS;
  const int H = p.H, B = p.B;
  const int kb_tmem = p.k_blocks < LT_TMEM_KB ? p.k_blocks : LT_TMEM_KB;
  constexpr uint32_t PIECE_BYTES = G * LT_HS;      // of h, from one CTA
  // gate warps -> MMA warps, once per step but the last: this CTA's piece of h is in the buffer, its accumulators have been read.
  // The MMA warps wait without a limit, so an exit has to keep to this:
  //  * a gate warp that gives up in step s reports for step s, then leaves; an MMA warp that gives up in step s, its barrier passed,
  //    arrives for the reports of step s, which it would have waited for next, and sets the abort flag before
  //  * whoever reports for step s has seen the barrier of step s - 2 complete (a gate warp mma_done of step s - 1, an MMA warp the
  //    barrier itself), but not that of step s - 1.  So two barriers take turns: with one, a gate warp's report for a step it gives up in
  //    could complete the step before in place of a warp that has yet to arrive, and leave that one waiting for good
  //  * nobody waits for a report that does not come: let s be the first step a gate warp gives up in.  All report for step s, and an
  //    MMA warp past that barrier finds the abort flag before it gets to the next.
  // Both loops over the steps are unrolled by two, so that which barrier and which buffer of h a step uses is a constant: the barriers
  // in turn would cost up to 2.5 % otherwise, and the gate warps' and MMA warps' addresses are constants, too.  ns per step, B x H, one
  // barrier / two / two and unrolled (gate warps alone, MMA warps alone): 512 x 384 1109 / 1118 / 1015 (1102, 1057), 64 x 384 772 / 774 / 687
  // (750, 705), 512 x 256 815 / 823 / 764, 512 x 128 560 / 572 / 531, 70 x 128 550 / 561 / 528, 512 x 512 1746 / 1751 / 1738.  An mbarrier,
  // whose wait has a limit: 4 % more than one barrier at H = 256 and 384.
  constexpr int OWN_READY = 1, OWN_THREADS = 32 * (CW + 4);

  if (tid == 0) {
    for (int i = 0; i < LT_STAGES; ++i) mbar_init(&ih_full[i], 1);
    for (int i = 0; i < 2 * LT_MAX_SLICES; ++i) mbar_init(&h_ready[i], 1);
    mbar_init(mma_done, 4); mbar_init(w_full, 1);
    // arm the first use of each buffer: h_0 arrives in buffer 0 (if there is a step 1), h_1 in buffer 1
    for (int r = 0; r < p.slices; ++r) {
      if (r == slc) continue;
      if (p.T > 1) mbar_arrive_expect_tx(&h_ready[r], PIECE_BYTES);
      if (p.T > 2) mbar_arrive_expect_tx(&h_ready[LT_MAX_SLICES + r], PIECE_BYTES);
    }
    abort_flag.set(0);
    fence_mbar_init();
    prefetch_tmap(&tm_w); prefetch_tmap(&tm_ih);
  }
  if (warp == CW) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  cluster_sync_all();                              // every CTA's barriers exist (and are armed) before anyone sends to them
  const uint32_t tmem_base = *tmem_slot;
  const unsigned int budget = spin_budget();
  const bool rank_ok = cluster_ctarank() == (uint32_t)slc;
  if (!rank_ok && tid == 0) { abort_flag.set(1); atomicOr(&g_status[0], ST_TIMEOUT_LSTM); g_status[1] = 0x50; }

  auto step_t = [&](int s) { return p.reverse ? p.T - 1 - s : s; };
  auto issue_ih = [&](int s, int st) {             // one thread: the four gate boxes of step s into stage st
    mbar_arrive_expect_tx(&ih_full[st], L::IH_BYTES);
    const int r = step_t(s) * B + row0;
#pragma unroll
    for (int g = 0; g < 4; ++g) tma_load_2d(ih_s + st * L::IH_BYTES + g * L::IH_GATE, &tm_ih, &ih_full[st], g * H + hid0, r);
  };

  // gate threads: hidden unit hid, batch rows r_lo .. r_lo + RPT - 1 of the group
  const int q = warp & 3;
  const int u = q * 32 + lane, hid = hid0 + u;
  const bool hid_ok = hid < H;
  const int r_lo = (warp >> 2) * RPT;
  const int rows_live = min(RPT, max(0, B - (row0 + r_lo)));          // rows of this thread that exist
  float c[RPT];
  if (warp < CW) {
    // W_hh -> tensor memory: lane = hidden unit, 32 columns = 128 bytes of K; the warps of a lane quarter share the K blocks.
    // A lane reads whole 32-byte sectors of its row (where base and stride allow): of 16-byte pieces the second would have to be
    // found in L1, and the shared memory that this kernel takes leaves 28 KiB of that.  us per launch of 8 steps, B = 64 / 512: 16-byte
    // pieces past L1 H = 384 24.0 / 26.9, H = 256 16.9 / 18.8, through L1 17.6 / 24.4 and 14.5 / 17.0, sectors 16.3 / 21.4 and 13.3 / 14.8.
    const bool w_sectors = ((reinterpret_cast<uintptr_t>(w_hh) | (uintptr_t)ld_w) & 31) == 0;
    for (int blk = warp >> 2; blk < 4 * kb_tmem; blk += CW / 4) {
      const int g = blk / kb_tmem, kb = blk % kb_tmem;
      uint32_t v[32];
      const uint8_t* src = w_hh + (long long)(g * H + hid) * ld_w + kb * 128;
#pragma unroll
      for (int i = 0; i < 4; ++i) {                // (H is a multiple of 32)
        uint4 lo = make_uint4(0, 0, 0, 0), hi = lo;
        if (hid_ok && kb * 128 + i * 32 < H) {
          if (w_sectors) ldg_v8(src + i * 32, lo, hi);
          else { lo = __ldca(reinterpret_cast<const uint4*>(src + i * 32)); hi = __ldca(reinterpret_cast<const uint4*>(src + i * 32 + 16)); }
        }
        v[8 * i] = lo.x; v[8 * i + 1] = lo.y; v[8 * i + 2] = lo.z; v[8 * i + 3] = lo.w;
        v[8 * i + 4] = hi.x; v[8 * i + 5] = hi.y; v[8 * i + 6] = hi.z; v[8 * i + 7] = hi.w;
      }
      tmem_st_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + (g * LT_TMEM_KB + kb) * 32, v);
    }
    tmem_st_wait();
#pragma unroll
    for (int i = 0; i < RPT; ++i)
      c[i] = (p.c0 && hid_ok && i < rows_live) ? __half2float(__ldcg(p.c0 + (long long)(row0 + r_lo + i) * H + hid)) : 0.f;
    // step 0 reads h_0 (or zeros) from buffer 1, staged by this CTA's own threads
    if constexpr (G < R)                           // the rows of the MMA that no batch row uses
      for (int id = tid; id < 2 * L::HBUF / 16; id += 32 * CW)
        if (((id >> 3) & (R - 1)) >= G) *reinterpret_cast<uint4*>(h_s + id * 16) = make_uint4(0, 0, 0, 0);
    const int chunks = H >> 4;
    for (int id = tid; id < G * chunks; id += 32 * CW) {
      const int r = id / chunks, cc = id % chunks;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (p.h0 && row0 + r < B) v = __ldcg(reinterpret_cast<const uint4*>(p.h0 + (size_t)(row0 + r) * H + cc * 16));
      *reinterpret_cast<uint4*>(h_s + L::HBUF + (cc >> 3) * L::KB_BYTES + r * 128 + (((cc & 7) ^ (r & 7)) << 4)) = v;
    }
    fence_proxy_async_smem();
  } else if (warp == CW + 3 && lane == 0) {
    if (p.slices > LT_TMEM_KB) {
      mbar_arrive_expect_tx(w_full, 4 * LSTM_KB_BYTES);
      for (int g = 0; g < 4; ++g) tma_load_2d(w_s + g * LSTM_KB_BYTES, &tm_w, w_full, LT_TMEM_KB * 128, g * H + hid0);
    }
    for (int s = 0; s < LT_STAGES && s < p.T; ++s) issue_ih(s, s);
  }
  tc_fence_before();
  __syncthreads();                                 // W_hh is in tensor memory and h_0 staged before the first MMAs read them
  tc_fence_after();

  if (warp < CW) {
    // ------------------------------ gate math ------------------------------
    // sigmoid(x) = 0.5 + 0.5 tanh(x / 2): the halving of the three sigmoid gates is folded into scale, ih and bias (exact)
    float sc[4], bi[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const float half = g == 2 ? 1.0f : 0.5f;
      sc[g] = hid_ok ? __ldcg(p.s_hh + g * H + hid) * (1.0f / 448.0f) * half : 0.f;
      bi[g] = hid_ok && p.bias ? __ldcg(p.bias + g * H + hid) * half : 0.f;
    }
    const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + LT_ACC_COL + r_lo;
    const uint8_t* ih_t = ih_s + r_lo * (LT_HS * 2) + u * 2;
    uint8_t* own = h_s + slc * L::KB_BYTES + (u & 15);               // + row * 128 + swizzled chunk
    const int ck = u >> 4;
    // all-gather: half of the warp's rows x its 32 bytes at a time, one 16-byte store per lane (peer, row, chunk)
    const bool sends = lane < (p.slices - 1) * RPT;
    const uint32_t to = (uint32_t)(lane / RPT < slc ? lane / RPT : lane / RPT + 1);
    uint32_t snd_off[2];                                              // source offset in the buffer, rows of the first / second half
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      const int r = r_lo + hf * (RPT / 2) + ((lane >> 1) & (RPT / 2 - 1));
      snd_off[hf] = slc * L::KB_BYTES + r * 128 + (((2 * q + (lane & 1)) ^ (r & 7)) << 4);
    }
    const uint32_t snd_dst = sends ? mapa_shared(smem_u32(h_s), to) : 0u, snd_bar = sends ? mapa_shared(smem_u32(h_ready + slc), to) : 0u;
    int st = 0; uint32_t st_ph = 0;
#pragma unroll 2
    for (int s = 0; s < p.T; ++s) {
      // ih + bias of this step, before the accumulators are there
      bool ok = mbar_wait(&ih_full[st], st_ph, abort_flag, ST_TIMEOUT_LSTM, 0x20, budget);
      if (!__all_sync(0xffffffffu, ok)) {            // (the MMA warps wait for this warp's report, whatever became of it)
        if (s + 1 < p.T) named_arrive<OWN_THREADS>(OWN_READY + (s & 1));
        break;
      }
      float2 x[4][RPT / 2];
      const uint8_t* ihb = ih_t + st * L::IH_BYTES;
#pragma unroll
      for (int g = 0; g < 4; ++g)
#pragma unroll
        for (int i = 0; i < RPT / 2; ++i) {
          const float half = g == 2 ? 1.0f : 0.5f;
          const float2 f = make_float2(__half2float(*reinterpret_cast<const __half*>(ihb + g * L::IH_GATE + (2 * i) * (LT_HS * 2))),
                                       __half2float(*reinterpret_cast<const __half*>(ihb + g * L::IH_GATE + (2 * i + 1) * (LT_HS * 2))));
          x[g][i] = __ffma2_rn(f, make_float2(half, half), make_float2(bi[g], bi[g]));
        }
      if (++st == LT_STAGES) { st = 0; st_ph ^= 1; }

      ok = mbar_wait<true>(mma_done, s & 1, abort_flag, ST_TIMEOUT_LSTM, 0x30, budget);
      if (!__all_sync(0xffffffffu, ok)) {
        if (s + 1 < p.T) named_arrive<OWN_THREADS>(OWN_READY + (s & 1));
        break;
      }
      tc_fence_after();
      uint32_t acc[4][RPT];
#pragma unroll
      for (int g = 0; g < 4; ++g) tmem_ld_32x32b(t_row + g * R, acc[g]);
      tmem_ld_wait(acc[0], acc[1], acc[2], acc[3]);
      uint8_t* dst = own + (s & 1) * L::HBUF;
      float2 hv[RPT / 2];
      uint32_t h8[RPT / 2];
      // half of this thread's rows at a time, so that the first half is on its way while the second is computed
      constexpr int PAIRS = RPT / 4;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
        for (int i = hf * PAIRS; i < (hf + 1) * PAIRS; ++i) {
          float2 t[4];
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const float2 pre = __ffma2_rn(make_float2(__uint_as_float(acc[g][2 * i]), __uint_as_float(acc[g][2 * i + 1])),
                                          make_float2(sc[g], sc[g]), x[g][i]);
            t[g] = make_float2(tanh_f(pre.x), tanh_f(pre.y));
            if (g != 2) t[g] = __ffma2_rn(make_float2(0.5f, 0.5f), t[g], make_float2(0.5f, 0.5f));
          }
          const float2 cn = __ffma2_rn(t[1], make_float2(c[2 * i], c[2 * i + 1]), __fmul2_rn(t[0], t[2]));
          hv[i] = __fmul2_rn(t[3], make_float2(tanh_f(cn.x), tanh_f(cn.y)));
          const float2 cr = __half22float2(__float22half2_rn(cn));        // the cell state is carried in fp16
          c[2 * i] = cr.x; c[2 * i + 1] = cr.y;
          h8[i] = __nv_cvt_float2_to_fp8x2(__fmul2_rn(hv[i], make_float2(448.f, 448.f)), __NV_SATFINITE, __NV_E4M3);
          if (!hid_ok || 2 * i >= rows_live) h8[i] = 0u;
          else if (2 * i + 1 >= rows_live) h8[i] &= 0xffu;
          const int r = r_lo + 2 * i;
          dst[r * 128 + ((ck ^ (r & 7)) << 4)] = (uint8_t)h8[i];
          dst[(r + 1) * 128 + ((ck ^ ((r + 1) & 7)) << 4)] = (uint8_t)(h8[i] >> 8);
        }
        __syncwarp();
        // (to the other CTAs first, whose MMAs wait for it longest; B = 256, H = 384 923 ns per step with the report first, 901 so)
        if (sends && s + 1 < p.T) {
          const uint32_t off = (s & 1) * L::HBUF + snd_off[hf];
          st_async_v4(snd_dst + off, *reinterpret_cast<const uint4*>(h_s + off), snd_bar + 8 * LT_MAX_SLICES * (s & 1));
        }
        if (hf == 1) {
          fence_proxy_async_smem(); tc_fence_before();                       // the stores above before this CTA's MMAs read them
          __syncwarp();
          if (s + 1 < p.T) named_arrive<OWN_THREADS>(OWN_READY + (s & 1));
        }
      }
      // the layer's outputs, off the critical path: 32 (E4M3) / 64 (fp16) contiguous bytes per warp and row
      if (hid_ok) {
        const size_t o = ((size_t)step_t(s) * B + row0 + r_lo) * H + hid;
        if (p.h8_out) {
#pragma unroll
          for (int i = 0; i < RPT; ++i)
            if (i < rows_live) p.h8_out[o + (size_t)i * H] = (uint8_t)(h8[i >> 1] >> (8 * (i & 1)));
        }
        if (p.h_out) {
#pragma unroll
          for (int i = 0; i < RPT; ++i)
            if (i < rows_live) p.h_out[o + (size_t)i * H] = __float2half_rn((i & 1) ? hv[i >> 1].y : hv[i >> 1].x);
        }
      }
    }
    if (p.c_last && hid_ok) {
#pragma unroll
      for (int i = 0; i < RPT; ++i)
        if (i < rows_live) p.c_last[(long long)(row0 + r_lo + i) * H + hid] = __float2half_rn(c[i]);
    }
  } else {
    // ------------------------------ MMA issue, one gate per warp ------------------------------
    // The whole warp walks the loop, one lane of it issues: the descriptors then stay in uniform registers.
    const int g = __shfl_sync(0xffffffffu, warp - CW, 0);
    constexpr uint32_t idesc = umma_idesc(1, 0, 0, LT_HS, R);
    const uint32_t d = tmem_base + LT_ACC_COL + g * R;
    const uint32_t a0 = tmem_base + g * LT_TMEM_KB * 32;
    const uint64_t b_base[2] = {umma_smem_desc_sw128(smem_u32(h_s)), umma_smem_desc_sw128(smem_u32(h_s + L::HBUF))};
    const uint64_t a_smem = umma_smem_desc_sw128(smem_u32(w_s + g * LSTM_KB_BYTES));
    const int ksteps = H >> 5;                     // 32 bytes of K per MMA
    bool ok = rank_ok;
    int st = 0;
    if (ok && p.slices > LT_TMEM_KB) ok = __all_sync(0xffffffffu, mbar_wait(w_full, 0, abort_flag, ST_TIMEOUT_LSTM, 0x10, budget));
    // The loop exists once per (row group size, rank): every descriptor offset is a constant of straight-line code.  Returns the step
    // it gave up in, or -1.
    auto run = [&](auto slices_tag, auto rank_tag) {
      constexpr int SLICES = decltype(slices_tag)::value, RANK = decltype(rank_tag)::value;
#pragma unroll 2
      for (int s = 0; s < p.T; ++s) {
        const int hb = (s + 1) & 1;                // h_{s-1}
        const uint32_t ph = (uint32_t)((s - 1) >> 1) & 1u;
        // (the accumulators may be overwritten and this CTA's piece read once every gate warp has reported)
        __syncwarp();
        if (s > 0) named_sync<OWN_THREADS>(OWN_READY + hb);
        tc_fence_after();
        const uint64_t b = hb ? b_base[1] : b_base[0];
        // K blocks in ascending order on every CTA (the order of the sums is part of the result), each as soon as its piece
        // of h is there
#pragma unroll
        for (int kb = 0; kb < SLICES; ++kb) {
          if (kb != RANK && s > 0) {               // another CTA's piece
            uint64_t* bar = &h_ready[hb * LT_MAX_SLICES + kb];
            if (!__all_sync(0xffffffffu, mbar_wait_cluster(bar, ph, abort_flag, ST_TIMEOUT_LSTM, 0x41, budget))) return s;
            if (g == 0 && lane == 0 && s + 2 < p.T) mbar_arrive_expect_tx(bar, PIECE_BYTES);   // its next use: h_{s+1}, read by step s + 2
            fence_proxy_async_smem();              // the peer's stores before the MMAs read them
          }
          const uint64_t bd = b + (uint64_t)(kb * (L::KB_BYTES >> 4));
          if (kb < LT_TMEM_KB && (kb < SLICES - 1 || 4 * kb + 3 < ksteps)) {
            umma_f8_ta_x4_elect(d, a0 + kb * 32, bd, idesc, kb != 0);
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              if (kb == SLICES - 1 && 4 * kb + k >= ksteps) break;
              if (kb < LT_TMEM_KB) umma_f8_ta_elect(d, a0 + kb * 32 + k * 8, bd + 2 * k, idesc, (kb | k) != 0);
              else umma_f8_elect(d, a_smem + 2 * k, bd + 2 * k, idesc, (kb | k) != 0);
            }
          }
        }
        umma_commit_elect(mma_done);
        if (__any_sync(0xffffffffu, abort_flag.get())) return s;
        // the gate warps have read the ih tile of step s - 1 (their reports above came after that): its stage is free
        if (g == 3 && s > 0) {
          if (lane == 0 && s - 1 + LT_STAGES < p.T) issue_ih(s - 1 + LT_STAGES, st);
          if (++st == LT_STAGES) st = 0;
        }
      }
      return -1;
    };
    auto run_rank = [&](auto slices_tag) {
      constexpr int SLICES = decltype(slices_tag)::value;
      if constexpr (SLICES > 3) if (slc == 3) return run(slices_tag, std::integral_constant<int, 3>{});
      if constexpr (SLICES > 2) if (slc == 2) return run(slices_tag, std::integral_constant<int, 2>{});
      if constexpr (SLICES > 1) if (slc == 1) return run(slices_tag, std::integral_constant<int, 1>{});
      return run(slices_tag, std::integral_constant<int, 0>{});
    };
    int gave_up = ok ? -1 : 0;
    if (ok) {
      if (p.slices == 1) gave_up = run_rank(std::integral_constant<int, 1>{});
      else if (p.slices == 2) gave_up = run_rank(std::integral_constant<int, 2>{});
      else if (p.slices == 3) gave_up = run_rank(std::integral_constant<int, 3>{});
      else gave_up = run_rank(std::integral_constant<int, 4>{});
    }
    if (gave_up >= 0) {                            // (before the loop: as in step 0)
      if (lane == 0) abort_flag.set(1);
      __syncwarp();
      named_arrive<OWN_THREADS>(OWN_READY + (gave_up & 1));
      if (lane == 0) {                             // loads in flight land before the CTA exits
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) { }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == CW) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
  cluster_sync_all();                              // nobody leaves while another CTA of the cluster may still copy into it
}


// ---- host -------------------------------------------------------------------------------------------------
size_t lstm_scratch_bytes(long long B, int H) {
  const size_t hbuf = ((size_t)2 * B * H + 255) & ~(size_t)255;
  const size_t flags = (size_t)((B + LSTM_ROWS - 1) / LSTM_ROWS) * (H / LSTM_HS) * sizeof(unsigned int);
  return hbuf + ((flags + 255) & ~(size_t)255);
}

using LtKernel = void (*)(const CUtensorMap, const CUtensorMap, const uint8_t*, long long, const LstmParams);
// The forms of the transposed kernel: batch rows per group, and what a step takes (ns, measured on B200) on row groups of one
// to four CTAs, i.e. at H = 128, 256, 384 and 512.  (16 rows at H = 384 as with 96 CTAs, B = 512; 1310 with 129.)  Measured before the loops were unrolled by two; now, all
// SMs taken: 4 rows 540, 623, 697, 1131; 8 700, 775, 851, 1315; 12 767, 928, 1029, 1492; 16 1109, 1206, 1252, 1746; 32 1584, 1911, 2031, 2663.  Only the order
// of the forms counts, and it is the same (but for 3 % at H = 256 with B past 1184).
struct LtForm { int rows, threads, smem[LT_MAX_SLICES + 1], step_ns[LT_MAX_SLICES + 1]; LtKernel kernel; };
template <int R, int G, int CW>
static constexpr LtForm lt_make_form(int ns1, int ns2, int ns3, int ns4) {
  LtForm f{G, 32 * (CW + 4), {}, {0, ns1, ns2, ns3, ns4}, lstm_tmem_kernel<R, G, CW>};
  // (at least 212 KiB: it takes all of tensor memory, and no CTA of another stream that wants some, a few-tile GEMM's, may sit
  // beside it waiting)
  for (int n = 1; n <= LT_MAX_SLICES; ++n) f.smem[n] = LtSmem<R, G>::bytes(n) > 212 * 1024 ? LtSmem<R, G>::bytes(n) : 212 * 1024;
  return f;
}
constexpr int LT_FORMS = 5;
static const LtForm kLtForms[LT_FORMS] = {lt_make_form<16, 4, 4>(530, 645, 775, 1180), lt_make_form<16, 8, 8>(690, 800, 920, 1330),
                                          lt_make_form<16, 12, 12>(830, 960, 1120, 1550), lt_make_form<16, 16, 8>(1045, 1150, 1240, 1740),
                                          lt_make_form<32, 32, 16>(1620, 1910, 2060, 2720)};

static cudaLaunchConfig_t lt_config(const LtForm& f, int slices, long long groups, cudaStream_t st, cudaLaunchAttribute (&attr)[2]) {
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = slices; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(groups * slices)); cfg.blockDim = dim3(f.threads);
  cfg.dynamicSmemBytes = f.smem[slices]; cfg.stream = st;
  cfg.attrs = attr; cfg.numAttrs = 2;
  return cfg;
}

// Row groups (clusters) of a form that can be resident at once on device `dev`; 0 = cannot run there.  Asked once.
static int lt_capacity(int form, int slices, int dev) {
  static std::atomic<int> cap[LT_FORMS][64][LT_MAX_SLICES + 1];
  std::atomic<int>& slot = cap[form][dev][slices];
  int c = slot.load(std::memory_order_acquire);
  if (c == 0) {
    const LtForm& f = kLtForms[form];
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = lt_config(f, slices, 1, nullptr, attr);
    // (the attribute is per kernel: it is set to what the largest row group needs)
    cudaError_t e = cudaFuncSetAttribute(f.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, f.smem[LT_MAX_SLICES]);
    int n = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, f.kernel, &cfg);
    (void)cudaGetLastError();
    c = e == cudaSuccess && n > 0 ? n : -1;
    if (getenv("GSB200_LSTM_VERBOSE") || c < 0)
      fprintf(stderr, "gigaslop_b200: LSTM, groups of %d rows on clusters of %d CTAs: %d can be resident (%s)\n", f.rows, slices, n, cudaGetErrorName(e));
    slot.store(c, std::memory_order_release);
  }
  return c > 0 ? c : 0;
}

// The form with the shortest step (times the waves it takes) if the recurrence is to leave the SMs past `max_ctas` to a
// projection beside it (0 = it has the whole GPU); -1 = none.  `max_ctas` only steers this choice, in which groups past it wait
// for a next wave: a launch brings all its row groups, and where no form holds them in `max_ctas` CTAs they take more SMs
// (lstm_layer_ctas counts what a launch does occupy).  Fewer rows per CTA make a shorter step as long as all groups are resident: B = 512, H = 384 takes 12 rows
// (43 groups, 129 CTAs), B = 512, H = 512 16 rows (128 CTAs), B = 1024, H = 384 32 rows (2.03 us per step; 12 rows in two
// waves 2.06).  *ns = the step.
static int lt_choose(long long B, int H, int dev, int max_ctas, long long* ns = nullptr) {
  const int slices = (H + LT_HS - 1) / LT_HS;
  int best = -1;
  long long best_ns = 0;
  for (int i = 0; i < LT_FORMS; ++i) {
    int cap = lt_capacity(i, slices, dev);
    if (cap > 0 && max_ctas > 0 && cap > max_ctas / slices) cap = max_ctas / slices > 0 ? max_ctas / slices : 1;
    if (cap <= 0) continue;
    const long long groups = (B + kLtForms[i].rows - 1) / kLtForms[i].rows;
    const long long t = (groups + cap - 1) / cap * kLtForms[i].step_ns[slices];
    if (best < 0 || t < best_ns) { best = i; best_ns = t; }
  }
  if (ns) *ns = best_ns;
  return best;
}

static int32_t launch_lt(const LtForm& f, const LstmLayerArgs& a, LstmParams p, cudaStream_t st) {
  p.slices = (a.H + LT_HS - 1) / LT_HS;
  CUtensorMap tw, tih;
  if (!tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.w_hh, (uint64_t)4 * a.H, (uint64_t)a.H, (uint64_t)a.ld_w, 128, LT_HS,
               CU_TENSOR_MAP_SWIZZLE_128B) ||
      !tmap_2d(&tih, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.ih, (uint64_t)a.T * a.B, (uint64_t)4 * a.H, (uint64_t)a.ld_ih, LT_HS,
               f.rows, CU_TENSOR_MAP_SWIZZLE_NONE))
    return GSB200_ERR_BAD_ARG;
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = lt_config(f, p.slices, (a.B + f.rows - 1) / f.rows, st, attr);
  return cuda_status(cudaLaunchKernelEx(&cfg, f.kernel, tw, tih, a.w_hh, a.ld_w, p), "lstm launch");
}

// GSB200_LSTM_NO_CLUSTER=1 or GSB200_LSTM_ROWS128=1 in the environment selects the cooperative kernel (128-row tiles).
static bool lstm_cooperative() {
  static std::atomic<int> env_state{-1};
  int env = env_state.load(std::memory_order_relaxed);
  if (env < 0) {
    const char* e1 = getenv("GSB200_LSTM_NO_CLUSTER");
    const char* e2 = getenv("GSB200_LSTM_ROWS128");
    env = (e1 && e1[0] == '1') || (e2 && e2[0] == '1') ? 1 : 0;
    env_state.store(env, std::memory_order_relaxed);
  }
  return env != 0;
}

// CTAs of one recurrence launch (what a projection beside it has to leave alone).
static int lstm_layer_ctas(long long B, int H, int max_ctas) {
  int dev = 0;
  cudaGetDevice(&dev);
  const int form = dev >= 0 && dev < 64 && !lstm_cooperative() ? lt_choose(B, H, dev, max_ctas) : -1;
  if (form < 0) return (int)((B + LSTM_ROWS - 1) / LSTM_ROWS) * (H / LSTM_HS);
  const int slices = (H + LT_HS - 1) / LT_HS, cap = lt_capacity(form, slices, dev);
  const long long groups = (B + kLtForms[form].rows - 1) / kLtForms[form].rows;
  return (int)(groups < cap ? groups : cap) * slices;
}

// How many launches to cut a layer's recurrence into so that the next layer's projection runs beside it (1 = not at all).
// The cut recurrence is steered to `max_ctas` CTAs, which may cost it a form with longer steps, and every launch about 12 us;
// it hides the projection up to the last block's.  Five layers, T = 2000, B = 512, H = 384: 14.3 ms one after the other, 13.4
// to 14.0 in five blocks; at B = 512, H = 512 (T = 1000, three layers) 6.8 ms against 8.0, so not cut.
static int lstm_time_blocks(long long T, long long B, int H, int max_ctas) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || lstm_cooperative()) return 8;
  long long whole = 0, limited = 0;
  if (lt_choose(B, H, dev, 0, &whole) < 0 || lt_choose(B, H, dev, max_ctas, &limited) < 0) return 8;
  const double proj = 10e3 + (double)T * (double)B * 9.0 * H / 5200.0;      // ns: fp16 [rows, 4H] written, E4M3 [rows, H] read at 5.2 TB/s
  const double rest = proj * 0.6 * sm_count_physical() / (sm_count_physical() - max_ctas);   // ... beside the recurrence
  double best = 0.98 * ((double)T * (double)whole + proj);                  // cut only for more than 2 %
  int nb = 1;
  for (int n = 2; n <= 8 && n <= T; ++n) {
    double t = (double)T * (double)limited * 1.03;                          // (the projection beside it costs the step 3 %)
    if (t < rest) t = rest;
    t += proj / n + 12e3 * n;
    if (t < best) { best = t; nb = n; }
  }
  return nb;
}

int32_t launch_lstm_layer(const LstmLayerArgs& a, void* scratch, size_t scratch_bytes, cudaStream_t st) {
  if (a.T == 0 || a.B == 0) return GSB200_OK;
  if (a.T < 0 || a.B < 0 || a.H <= 0 || a.H % LSTM_HS != 0 || a.H > LSTM_MAX_KB * 128) return GSB200_ERR_UNSUPPORTED;
  if (!a.ih || !a.w_hh || !a.s_hh || !scratch) return GSB200_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(a.ih) & 15) || (reinterpret_cast<uintptr_t>(a.w_hh) & 15) ||
      (reinterpret_cast<uintptr_t>(scratch) & 255))
    return GSB200_ERR_BAD_ARG;
  if (a.ld_ih < 4 * a.H || a.ld_ih % 8 != 0 || a.H % 16 != 0) return GSB200_ERR_BAD_ARG;
  if ((a.h_out && (reinterpret_cast<uintptr_t>(a.h_out) & 15)) || (a.h8_out && (reinterpret_cast<uintptr_t>(a.h8_out) & 15)) ||
      (a.h0 && (reinterpret_cast<uintptr_t>(a.h0) & 15)))
    return GSB200_ERR_BAD_ARG;
  if ((long long)a.T * a.B > 0x7fffffffll) return GSB200_ERR_BAD_ARG;
  if (scratch_bytes < lstm_scratch_bytes(a.B, a.H)) return GSB200_ERR_BAD_ARG;
  int32_t rc = ensure_device();
  if (rc != GSB200_OK) return rc;

  const int groups = (int)((a.B + LSTM_ROWS - 1) / LSTM_ROWS);
  const int slices = a.H / LSTM_HS;
  const int grid = groups * slices;
  // What a call may ask for, whichever kernel runs: all CTAs of the cooperative kernel resident (they wait on one another; the
  // transposed kernel's clusters could run in waves).  The grid is never capped, so the physical SM count is what bounds it, not
  // the cap a caller may have set for the GEMM grids.
  if (grid > sm_count_physical()) return GSB200_ERR_UNSUPPORTED;

  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return GSB200_ERR_DEVICE;
  if (a.ld_w < a.H || a.ld_w % 16 != 0) return GSB200_ERR_BAD_ARG;

  LstmParams p{};
  p.T = (int)a.T; p.B = (int)a.B; p.H = a.H; p.reverse = a.reverse ? 1 : 0;
  p.k_blocks = (a.H + 127) / 128; p.slices = slices;
  p.s_hh = a.s_hh; p.bias = a.bias; p.h0 = a.h0; p.c0 = a.c0;
  p.h_out = a.h_out; p.h8_out = a.h8_out; p.c_last = a.c_last;

  if (!lstm_cooperative()) {
    const int form = lt_choose(a.B, a.H, dev, a.max_ctas);
    if (form >= 0) return launch_lt(kLtForms[form], a, p, st);
  }

  static std::atomic<int> attr_done[64];
  if (!attr_done[dev].load(std::memory_order_acquire)) {
    cudaError_t e = cudaFuncSetAttribute(lstm_recurrent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LSTM_SMEM_BYTES);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(lstm)");
    attr_done[dev].store(1, std::memory_order_release);
  }
  const size_t hbuf_bytes = ((size_t)2 * a.B * a.H + 255) & ~(size_t)255;
  p.hbuf = static_cast<uint8_t*>(scratch);
  p.flags = reinterpret_cast<unsigned int*>(static_cast<uint8_t*>(scratch) + hbuf_bytes);

  CUtensorMap tw, tih;
  if (!tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.w_hh, (uint64_t)4 * a.H, (uint64_t)a.H, (uint64_t)a.ld_w, 128,
               LSTM_HS, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !tmap_2d(&tih, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.ih, (uint64_t)a.T * a.B, (uint64_t)4 * a.H,
               (uint64_t)a.ld_ih, LSTM_HS, LSTM_ROWS, CU_TENSOR_MAP_SWIZZLE_64B))
    return GSB200_ERR_BAD_ARG;
  // the cooperative kernel exchanges h through the scratch; its step counters start at zero
  cudaError_t e = cudaMemsetAsync(p.flags, 0, (size_t)grid * sizeof(unsigned int), st);
  if (e != cudaSuccess) return cuda_status(e, "lstm flags memset");
  void* args[3] = {&tw, &tih, &p};
  e = cudaLaunchCooperativeKernel(reinterpret_cast<void*>(lstm_recurrent_kernel), dim3(grid), dim3(LSTM_THREADS), args,
                                  LSTM_SMEM_BYTES, st);
  return cuda_status(e, "lstm launch");
}

// ---- variant for callers that cannot allocate device memory ------------------------------------------------
// The h exchange buffer and the step counters live in a file-scope device array instead of caller scratch.
// Limits: B <= 512 and H <= 512 (the benchmark layer is B = 512, H = 384).  Every GPU that loads the library
// holds these ~513 KiB until the process exits.
constexpr long long LSTM_STATIC_MAX_B = 512;
constexpr int LSTM_STATIC_MAX_H = 512;
constexpr size_t LSTM_STATIC_BYTES = (size_t)2 * LSTM_STATIC_MAX_B * LSTM_STATIC_MAX_H + 1024;
static __device__ __align__(256) unsigned char g_lstm_static_scratch[LSTM_STATIC_BYTES];

// In host code the array's name is only a stand-in for the symbol, not a device address: the address a kernel
// can use comes from cudaGetSymbolAddress, looked up once per device with that device current.
static void* g_lstm_static_ptr[64];

int32_t launch_lstm_layer_static(const LstmLayerArgs& a, cudaStream_t st) {
  if (a.T == 0 || a.B == 0) return GSB200_OK;
  if (a.B > LSTM_STATIC_MAX_B || a.H > LSTM_STATIC_MAX_H || lstm_scratch_bytes(a.B, a.H) > LSTM_STATIC_BYTES) {
    fprintf(stderr, "gigaslop_b200: lstm_layer_fp8_static supports B <= %lld and H <= %d (got B = %lld, H = %d); "
                    "use gsb200_lstm_layer_fp8 with caller scratch for larger shapes\n",
            LSTM_STATIC_MAX_B, LSTM_STATIC_MAX_H, a.B, a.H);
    return GSB200_ERR_UNSUPPORTED;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_status(e, "cudaGetDevice");
  if (dev < 0 || dev >= 64) return GSB200_ERR_DEVICE;
  if (!g_lstm_static_ptr[dev]) {
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_lstm_static_scratch);
    if (e != cudaSuccess || !ptr) return cuda_status(e != cudaSuccess ? e : cudaErrorInvalidSymbol, "cudaGetSymbolAddress(lstm scratch)");
    g_lstm_static_ptr[dev] = ptr;
  }
  return launch_lstm_layer(a, g_lstm_static_ptr[dev], LSTM_STATIC_BYTES, st);
}

// ---- the whole stack behind one call ---------------------------------------------------------------------------
// Per layer: the hoisted input projection (FP8 GEMM over the T*B rows) and the persistent recurrence; layers
// alternate direction and hand each other h as E4M3 at the row scale 1/448.  With an auxiliary stream the
// recurrence of a layer is cut into `time_blocks` launches (the state crosses a cut exactly: h as the E4M3 bytes
// the kernel itself feeds back, c as the fp16 it carries), and as soon as a block of layer l is done the hoisted
// projection of layer l + 1 over the same timesteps runs on the auxiliary stream, on the SMs the recurrence
// leaves idle -- ordered by events only, no kernel waits for another kernel.
//
// Workspace: [ih 0][ih 1 (overlap only)][h8 0][h8 1][T B floats, unused: the size stays what callers know it as][c 0][c 1][layer scratch]
static size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

size_t lstm_stack_workspace_bytes(long long T, long long B, int H, int overlap) {
  if (T <= 0 || B <= 0 || H <= 0) return 0;
  const size_t rows = (size_t)T * (size_t)B;
  return (overlap ? 2 : 1) * align256(rows * 4 * H * 2) + 2 * align256(rows * H) + align256(rows * 4) +
         2 * align256((size_t)B * H * 2) + align256(lstm_scratch_bytes(B, H));
}

int32_t launch_lstm_stack(const uint8_t* x, long long ldx, const float* sx, int C, const gsb200_lstm_layer_t* layers,
                          int n_layers, int reverse_first, __half* h_out, long long T, long long B, int H,
                          int time_blocks, void* ws, size_t ws_bytes, cudaStream_t st, cudaStream_t aux) {
  if (T == 0 || B == 0 || n_layers == 0) return GSB200_OK;
  if (!x || !sx || !layers || !h_out || !ws || T < 0 || B < 0 || n_layers < 0 || C <= 0) return GSB200_ERR_BAD_ARG;
  if (reinterpret_cast<uintptr_t>(ws) & 255) return GSB200_ERR_BAD_ARG;
  if (H <= 0 || H % LSTM_HS != 0 || H > LSTM_MAX_KB * 128) return GSB200_ERR_UNSUPPORTED;
  if ((long long)T * B > 0x7fffffffll) return GSB200_ERR_BAD_ARG;
  for (int l = 0; l < n_layers; ++l)
    if (!layers[l].w_ih || !layers[l].s_ih || !layers[l].w_hh || !layers[l].s_hh) return GSB200_ERR_BAD_ARG;
  bool overlap = aux != nullptr && aux != st && n_layers > 1;
  if (ws_bytes < lstm_stack_workspace_bytes(T, B, H, overlap ? 1 : 0)) return GSB200_ERR_BAD_ARG;
  int32_t rc = ensure_device();
  if (rc != GSB200_OK) return rc;

  const size_t rows = (size_t)T * (size_t)B;
  uint8_t* w = static_cast<uint8_t*>(ws);
  __half* ih[2];
  ih[0] = reinterpret_cast<__half*>(w); w += align256(rows * 4 * H * 2);
  ih[1] = ih[0];
  if (overlap) { ih[1] = reinterpret_cast<__half*>(w); w += align256(rows * 4 * H * 2); }
  uint8_t* h8[2];
  h8[0] = w; w += align256(rows * H);
  h8[1] = w; w += align256(rows * H);
  w += align256(rows * 4);
  __half* cst[2];
  cst[0] = reinterpret_cast<__half*>(w); w += align256((size_t)B * H * 2);
  cst[1] = reinterpret_cast<__half*>(w); w += align256((size_t)B * H * 2);
  void* scratch = w;
  const size_t scratch_bytes = align256(lstm_scratch_bytes(B, H));

  // hoisted projection of layer l over timesteps [t0, t1) on stream s, at most sm_cap CTAs (0 = all)
  auto project = [&](int l, long long t0, long long t1, cudaStream_t s, int sm_cap) -> int32_t {
    GemmArgs g{};
    g.kind = KIND_F8; g.epi = EPI_DEQUANT;
    if (l == 0) { g.A = x + (size_t)t0 * B * ldx; g.lda = ldx; g.scale_a = sx + (size_t)t0 * B; g.K = C; }
    else { g.A = h8[(l - 1) & 1] + (size_t)t0 * B * H; g.lda = H; g.scale_a_const = 1.0f / 448.0f; g.K = H; }
    g.B0 = layers[l].w_ih; g.ldb = layers[l].ld_w_ih;
    g.C = ih[l & 1] + (size_t)t0 * B * 4 * H; g.ldc = 4 * H;
    g.scale_b0 = layers[l].s_ih;
    g.M = (t1 - t0) * B; g.N = 4 * H;
    g.sm_cap = sm_cap;
    return launch_gemm(g, s);
  };
  rc = project(0, 0, T, st, 0);
  if (rc != GSB200_OK) return rc;

  // overlapped: the recurrence takes up to two thirds of the GPU, the projection what is left
  const int max_ctas = overlap ? sm_count_physical() * 2 / 3 : 0;
  if (!overlap) time_blocks = 1;
  else if (time_blocks <= 0) time_blocks = lstm_time_blocks(T, B, H, max_ctas);
  // launches per layer that has another one behind it; no block may be empty, the one behind it would find no state at the cut
  const int blocks_cut = time_blocks < T ? time_blocks : (int)T;
  int gemm_cap = sm_count_physical() - lstm_layer_ctas(B, H, max_ctas);
  if (gemm_cap < 8) gemm_cap = 8;
  cudaError_t ce = cudaSuccess;
  for (int l = 0; l < n_layers; ++l) {
    const bool last = l == n_layers - 1;
    const bool rev = ((l % 2) == 0) == (reverse_first != 0);
    uint8_t* h8_l = h8[l & 1];
    const int nb = last ? 1 : blocks_cut;            // (nothing runs beside the last layer: one launch on the whole GPU)
    for (int k = 0; k < nb; ++k) {
      // block k in processing order covers steps [s0, s1); in time that is [t0, t1)
      const long long s0 = T * k / nb, s1 = T * (k + 1) / nb;
      const long long t0 = rev ? T - s1 : s0, t1 = rev ? T - s0 : s1;
      LstmLayerArgs a{};
      a.ih = ih[l & 1] + (size_t)t0 * B * 4 * H; a.ld_ih = 4 * H;
      a.w_hh = layers[l].w_hh; a.ld_w = layers[l].ld_w_hh; a.s_hh = layers[l].s_hh; a.bias = layers[l].bias;
      if (k > 0) {                       // state at the cut: h of the step processed just before, c of the previous block
        const long long t_prev = rev ? t1 : t0 - 1;
        a.h0 = h8_l + (size_t)t_prev * B * H;
        a.c0 = cst[(k - 1) & 1];
      }
      a.h_out = last ? h_out + (size_t)t0 * B * H : nullptr;
      a.h8_out = h8_l + (size_t)t0 * B * H;
      a.c_last = k + 1 < nb ? cst[k & 1] : nullptr;
      a.max_ctas = nb > 1 ? max_ctas : 0;
      a.T = t1 - t0; a.B = B; a.H = H; a.reverse = rev ? 1 : 0;
      rc = launch_lstm_layer(a, scratch, scratch_bytes, st);
      if (rc != GSB200_OK) return rc;
      if (!last && k + 1 < nb) {
        cudaEvent_t ev;
        ce = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
        if (ce != cudaSuccess) return cuda_status(ce, "lstm stack: event");
        ce = cudaEventRecord(ev, st);
        if (ce == cudaSuccess) ce = cudaStreamWaitEvent(aux, ev, 0);
        cudaEventDestroy(ev);            // released by the runtime once the recorded work has completed
        if (ce != cudaSuccess) return cuda_status(ce, "lstm stack: event");
        rc = project(l + 1, t0, t1, aux, gemm_cap);
        if (rc != GSB200_OK) return rc;
      } else if (!last) {                // nothing left to run beside: the whole GPU, in `st`
        rc = project(l + 1, t0, t1, st, 0);
        if (rc != GSB200_OK) return rc;
      }
    }
    if (nb > 1) {                        // the next layer starts when its whole projection is there
      cudaEvent_t ev;
      ce = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
      if (ce != cudaSuccess) return cuda_status(ce, "lstm stack: event");
      ce = cudaEventRecord(ev, aux);
      if (ce == cudaSuccess) ce = cudaStreamWaitEvent(st, ev, 0);
      cudaEventDestroy(ev);
      if (ce != cudaSuccess) return cuda_status(ce, "lstm stack: event");
    }
  }
  return GSB200_OK;
}


}  // namespace gsb
