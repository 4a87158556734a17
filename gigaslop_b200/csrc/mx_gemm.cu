// Block-scaled MXFP8 GEMMs on tcgen05 kind::mxf8f6f4: both operands are E4M3 with one E8M0 scale per 32
// consecutive K elements (per row of A, per row of W), fp32 accumulation in TMEM, fp16 output.
//
//   plain : C[M,N]      = A . W^T                      (e.g. the down-projection fed by an MXFP8 activation)
//   dual  : C[M,N]      = silu(A . Wg^T) * (A . Wu^T)  (SwiGLU)
//
// Scale factors travel in the 128 x 4 tile order the tensor core consumes: for a matrix with R rows and
// K columns the byte for (row r, 32-block b) lives at
//     ((r / 128) * (K / 128) + b / 4) * 512 + (r % 32) * 16 + ((r % 128) / 32) * 4 + (b % 4)
// (rows padded to 128, K a multiple of 128).  One such 512-byte tile is exactly what one 128-byte K stage of
// 128 rows needs; it is bulk-copied into shared memory next to the operand tiles and moved to TMEM with
// tcgen05.cp.32x128b.warpx4 by the MMA thread, in order with the MMAs that read it.  The instruction
// descriptor's scale ids select the byte (the 32-block inside the stage) for each K = 32 MMA.
//
// Tiles are 128 rows x 128 accumulator columns (dual: gate -> columns 0..63, up -> 64..127), two accumulator
// stages.  The CTA runs TWO independent pipelines, one per accumulator stage: pipeline 0 takes the even tiles of
// the CTA, pipeline 1 the odd ones, each with its own producer thread (warps 0 / 3), its own MMA-issuing thread
// (warps 1 / 2), its own ring of operand stages and its own barriers; they share the tensor core and the eight
// epilogue warps.  The reasons, all measured on B200 with small probe kernels:
//   * an N = 128 MMA runs 64 clocks, but a tcgen05.mma costs the thread that issues it ~55 clocks, and a barrier
//     wait, a scale copy and a commit cost 60-90 each: one issuing thread leaves the tensor core idle more than half
//     the time.  Two threads can issue concurrently; the tensor core takes their MMAs in turn without loss;
//   * a producer thread that waits for a free stage and then issues its loads completes one round per ~570 clocks
//     plus ~170 per 16 KiB box, however many stages are in flight: 22 bytes per clock with one box per round, 37 with
//     two.  A second producer thread doubles that;
//   * a parity wait is only valid for a thread that sees every phase of its barrier, so no ring stage is ever shared
//     between the two threads of a role: each pipeline has its own stages.
// Two forms:
//   streaming (any K)            a stage holds one K block of A and of W and their scale tiles, three stages per
//                                pipeline; tiles are dealt round-robin; the dual form issues two N = 64 MMAs per K step
//                                so that gate and up keep their own scale tiles.
//   weight-stationary (K <= 512) CTA (group g, slice n) keeps the 128 rows of W of column slice n (dual: 64 gate + 64
//                                up) in shared memory and their scale tiles in TMEM for the whole launch and walks row
//                                blocks g, g + groups, ...; a stage holds TWO K blocks of A (one wait and one commit
//                                per 8 MMAs), two stages per pipeline.  Gate and up rows are adjacent in shared memory
//                                and are multiplied as ONE N = 128 operand whose scale tile is assembled once per CTA
//                                from the row groups of the two tiles.
// M = 65536, N = 2048, K = 512: 104 us (plain) / 276 us (dual) with one pipeline and both operands streamed, 75 / 128 us
// in the weight-stationary form.
#include <atomic>

#include "capi_internal.h"
#include "ptx.cuh"

namespace gsb {

constexpr int MX_BM = 128, MX_BN = 128, MX_BK = 128;
constexpr int MX_A_BYTES = MX_BM * MX_BK;            // 16 KiB
constexpr int MX_B_BYTES = MX_BN * MX_BK;            // 16 KiB
constexpr int MX_SF_BYTES = 512;
constexpr int MX_EPI_WARPS = 8, MX_FRONT_WARPS = 4;
constexpr int MX_THREADS = 32 * (MX_EPI_WARPS + MX_FRONT_WARPS);
constexpr int MX_OUT_BUF = 2048;                     // per epilogue warp: one 32 x 32 fp16 box
constexpr int MX_TMEM_COLS = 512;
constexpr int MX_SF_COL = 256;                       // scale-factor columns: pipeline pl uses MX_SF_COL + pl * 16 ...
constexpr int MXW_SFB_COL = MX_SF_COL + 32;          // ... and the resident W scales sit at MXW_SFB_COL + kb * 4
// streaming form: stage = A | W | SFA | SFB0 | SFB1 | pad (keeps 1 KiB alignment), three stages per pipeline
constexpr int MXS_STAGE_BYTES = MX_A_BYTES + MX_B_BYTES + 4 * MX_SF_BYTES;     // 34 KiB
constexpr int MXS_STAGES = 3;
// weight-stationary form: resident W slice (up to 4 K blocks) and its scale tiles, then stages of
// A(kb) | A(kb+1) | SFA(kb) | SFA(kb+1), two per pipeline
constexpr int MXW_MAX_KB = 4;
constexpr int MXW_KPS = 2;                                           // K blocks per stage
constexpr int MXW_W_BYTES = MXW_MAX_KB * MX_B_BYTES;                 // 64 KiB
constexpr int MXW_SFB_BYTES = MXW_MAX_KB * 2 * MX_SF_BYTES;          // 4 KiB: per K block SFB0 | SFB1
constexpr int MXW_STAGE_BYTES = MXW_KPS * (MX_A_BYTES + MX_SF_BYTES);   // 33 KiB
constexpr int MXW_STAGES = 2;
static_assert(MXW_STAGE_BYTES % 1024 == 0 && MXS_STAGE_BYTES % 1024 == 0, "swizzled tiles need 1 KiB alignment");

template <bool WST>
struct MxSmem {
  static constexpr int STAGES = WST ? MXW_STAGES : MXS_STAGES;       // per pipeline
  static constexpr int STAGE_BYTES = WST ? MXW_STAGE_BYTES : MXS_STAGE_BYTES;
  static constexpr int RING = WST ? MXW_W_BYTES + MXW_SFB_BYTES : 0;
  static constexpr int OUT = RING + 2 * STAGES * STAGE_BYTES;
  static constexpr int BAR = OUT + MX_EPI_WARPS * MX_OUT_BUF;
  static constexpr int BYTES = BAR + 256 + 1024;
  static_assert(BYTES > 116 * 1024 && BYTES <= 227 * 1024, "one CTA per SM");
};

struct MxParams {
  int M, N, K;
  int m_blocks, n_blocks, k_blocks;
  int n_groups;                      // weight-stationary: row-block groups (grid = n_groups * n_blocks)
  const uint8_t* sfa; const uint8_t* sfb0; const uint8_t* sfb1;    // tiled scale factors
};

// Shared-memory descriptor of one scale tile for tcgen05.cp: 32 rows of 16 bytes, unswizzled K-major, 8-row
// groups 128 bytes apart.
__device__ __forceinline__ uint64_t sf_smem_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);
  d |= (uint64_t)(128 >> 4) << 32;       // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;                // descriptor version
  return d;                              // layout type 0: no swizzle
}

template <bool DUAL, bool WST>
__global__ void __launch_bounds__(MX_THREADS, 1)
mx_gemm_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b0,
               const __grid_constant__ CUtensorMap tm_b1, const __grid_constant__ CUtensorMap tm_c, const MxParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  using L = MxSmem<WST>;
  constexpr int STAGES = L::STAGES, STAGE_BYTES = L::STAGE_BYTES;
  uint8_t* w_res = smem;                                   // WST: resident W slice, MX_B_BYTES per K block
  uint8_t* sfb_res = smem + MXW_W_BYTES;                   // WST: its scale tiles, 1 KiB per K block
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR);
  uint64_t* full_bar = bars;                               // [pipeline * STAGES + stage]
  uint64_t* empty_bar = bars + 2 * STAGES;
  uint64_t* acc_full = bars + 4 * STAGES;                  // [pipeline]
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* w_full = acc_empty + 2;                        // WST: resident slice landed
  uint64_t* sfb_ready = w_full + 1;                        // WST: its scale tiles are in TMEM
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sfb_ready + 1);
  const AbortFlag abort_flag{smem_u32(tmem_slot + 1)};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int OUT_COLS = DUAL ? MX_BN / 2 : MX_BN;          // output columns per tile
  const long long num_tiles = (long long)p.m_blocks * p.n_blocks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2 * STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], MX_EPI_WARPS); }
    mbar_init(w_full, 1); mbar_init(sfb_ready, 1);
    abort_flag.set(0);
    fence_mbar_init();
    prefetch_tmap(&tm_a); prefetch_tmap(&tm_b0); prefetch_tmap(&tm_b1); prefetch_tmap(&tm_c);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, MX_TMEM_COLS); tmem_relinquish(); }
  pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const unsigned int budget = spin_budget();          // bound of every wait below, fetched once
  // this CTA's tiles: streaming form t = cta, cta + grid, ... (column block fastest); weight-stationary form: a fixed
  // column block and row blocks group, group + n_groups, ...  Tile number `it` of the CTA belongs to pipeline it % 2.
  const int ws_n = WST ? (int)(blockIdx.x % p.n_blocks) : 0;
  const int ws_g = WST ? (int)(blockIdx.x / p.n_blocks) : 0;
  auto tile_at = [&](int it, int& m_blk, int& n_blk) -> bool {
    if constexpr (WST) {
      m_blk = ws_g + it * p.n_groups; n_blk = ws_n;
      return m_blk < p.m_blocks;
    } else {
      const long long t = (long long)blockIdx.x + (long long)it * gridDim.x;
      if (t >= num_tiles) return false;
      m_blk = (int)(t / p.n_blocks); n_blk = (int)(t % p.n_blocks);
      return true;
    }
  };

  if (warp == 0 || warp == 3) {
    // ------------------------------ producers: warp 0 -> pipeline 0, warp 3 -> pipeline 1 ------------------------------
    const int pl = warp == 3 ? 1 : 0;
    if (lane == 0) {
      uint8_t* ring = smem + L::RING + pl * STAGES * STAGE_BYTES;
      uint64_t* full = full_bar + pl * STAGES; uint64_t* empty = empty_bar + pl * STAGES;
      int s = 0; uint32_t ph = 0; bool ok = true;
      if (WST && pl == 0) {                                // the resident slice and its scale tiles
        const int n0 = ws_n * OUT_COLS, nb128 = n0 / 128;
        mbar_arrive_expect_tx(w_full, p.k_blocks * (MX_B_BYTES + (DUAL ? 2 : 1) * MX_SF_BYTES));
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          uint8_t* wb = w_res + kb * MX_B_BYTES;
          if constexpr (DUAL) {
            tma_load_2d(wb, &tm_b0, w_full, kb * MX_BK, n0);                     // 64 gate rows
            tma_load_2d(wb + MX_B_BYTES / 2, &tm_b1, w_full, kb * MX_BK, n0);    // 64 up rows
          } else {
            tma_load_2d(wb, &tm_b0, w_full, kb * MX_BK, n0);
          }
          bulk_load(sfb_res + kb * 2 * MX_SF_BYTES, p.sfb0 + ((size_t)nb128 * p.k_blocks + kb) * MX_SF_BYTES, MX_SF_BYTES, w_full);
          if constexpr (DUAL)
            bulk_load(sfb_res + kb * 2 * MX_SF_BYTES + MX_SF_BYTES, p.sfb1 + ((size_t)nb128 * p.k_blocks + kb) * MX_SF_BYTES, MX_SF_BYTES, w_full);
        }
      }
      int m_blk, n_blk;
      for (int it = pl; ok && tile_at(it, m_blk, n_blk); it += 2) {
        const int m0 = m_blk * MX_BM, n0 = n_blk * OUT_COLS;
        if constexpr (WST) {
          // this pipeline's next row block goes to L2 now (one CTA of the column slices asks for it)
          const int m_pf = m_blk + 2 * p.n_groups;
          if (m_pf < p.m_blocks && ws_n == m_pf % p.n_blocks)
            for (int kb = 0; kb < p.k_blocks; ++kb) tma_prefetch_l2_2d(&tm_a, kb * MX_BK, m_pf * MX_BM);
          for (int kb = 0; kb < p.k_blocks; kb += MXW_KPS) {
            if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, ST_TIMEOUT_PRODUCER, 0x600 | (pl << 4) | s, budget)) { ok = false; break; }
            uint8_t* st = ring + s * STAGE_BYTES;
            const int nk = p.k_blocks - kb < MXW_KPS ? p.k_blocks - kb : MXW_KPS;
            mbar_arrive_expect_tx(&full[s], nk * (MX_A_BYTES + MX_SF_BYTES));
            for (int j = 0; j < nk; ++j) tma_load_2d(st + j * MX_A_BYTES, &tm_a, &full[s], (kb + j) * MX_BK, m0);
            bulk_load(st + MXW_KPS * MX_A_BYTES, p.sfa + ((size_t)m_blk * p.k_blocks + kb) * MX_SF_BYTES, nk * MX_SF_BYTES, &full[s]);
            if (++s == STAGES) { s = 0; ph ^= 1; }
          }
        } else {
          const int nb128 = n0 / 128;                      // scale tile row block of W
          for (int kb = 0; kb < p.k_blocks; ++kb) {
            if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, ST_TIMEOUT_PRODUCER, 0x600 | (pl << 4) | s, budget)) { ok = false; break; }
            uint8_t* st = ring + s * STAGE_BYTES;
            mbar_arrive_expect_tx(&full[s], MX_A_BYTES + MX_B_BYTES + (DUAL ? 3 : 2) * MX_SF_BYTES);
            tma_load_2d(st, &tm_a, &full[s], kb * MX_BK, m0);
            if constexpr (DUAL) {
              tma_load_2d(st + MX_A_BYTES, &tm_b0, &full[s], kb * MX_BK, n0);                    // 64 gate rows
              tma_load_2d(st + MX_A_BYTES + MX_B_BYTES / 2, &tm_b1, &full[s], kb * MX_BK, n0);   // 64 up rows
            } else {
              tma_load_2d(st + MX_A_BYTES, &tm_b0, &full[s], kb * MX_BK, n0);
            }
            uint8_t* sf = st + MX_A_BYTES + MX_B_BYTES;
            bulk_load(sf, p.sfa + ((size_t)m_blk * p.k_blocks + kb) * MX_SF_BYTES, MX_SF_BYTES, &full[s]);
            bulk_load(sf + MX_SF_BYTES, p.sfb0 + ((size_t)nb128 * p.k_blocks + kb) * MX_SF_BYTES, MX_SF_BYTES, &full[s]);
            if constexpr (DUAL)
              bulk_load(sf + 2 * MX_SF_BYTES, p.sfb1 + ((size_t)nb128 * p.k_blocks + kb) * MX_SF_BYTES, MX_SF_BYTES, &full[s]);
            if (++s == STAGES) { s = 0; ph ^= 1; }
          }
        }
      }
      if (!ok) { long long t0 = clock64(); while (clock64() - t0 < 2000000) { } }
    }
  } else if (warp == 1 || warp == 2) {
    // ------------------------------ MMA issuers: warp 1 -> pipeline 0, warp 2 -> pipeline 1 ------------------------------
    const int pl = warp - 1;
    bool ok = true;
    if constexpr (WST) {
      // warp 1 waits for the resident slice; the dual form then builds, per K block, the scale tile of its N = 128
      // operand [64 gate rows | 64 up rows] in place: row groups sub, sub+1 of the gate tile, then of the up tile
      if (pl == 0) {
        ok = __all_sync(0xffffffffu, mbar_wait(w_full, 0, abort_flag, ST_TIMEOUT_MMA, 0xA00, budget));
        if constexpr (DUAL) {
          if (ok) {
            const int sub = ((ws_n * OUT_COLS) % 128) / 32;
            for (int kb = 0; kb < p.k_blocks; ++kb) {
              uint32_t* tg = reinterpret_cast<uint32_t*>(sfb_res + kb * 2 * MX_SF_BYTES);
              const uint32_t* tu = tg + MX_SF_BYTES / 4;
              const uint4 v = make_uint4(tg[lane * 4 + sub], tg[lane * 4 + sub + 1], tu[lane * 4 + sub], tu[lane * 4 + sub + 1]);
              *reinterpret_cast<uint4*>(tg + lane * 4) = v;
            }
            fence_proxy_async_smem();
          }
        }
        __syncwarp();
      }
    }
    if (lane == 0 && ok) {
      const uint8_t* ring = smem + L::RING + pl * STAGES * STAGE_BYTES;
      uint64_t* full = full_bar + pl * STAGES; uint64_t* empty = empty_bar + pl * STAGES;
      int s = 0; uint32_t ph = 0;
      const uint32_t sf_tmem = tmem_base + MX_SF_COL + pl * 16;    // this pipeline's scale-factor columns
      const uint32_t sfb_tmem = tmem_base + MXW_SFB_COL;
      if constexpr (WST) {
        if (pl == 0) {                                     // the slice's scale tiles go to TMEM once
          tc_fence_after();
          for (int kb = 0; kb < p.k_blocks; ++kb)
            tmem_cp_32x128b_warpx4(sfb_tmem + kb * 4, sf_smem_desc(smem_u32(sfb_res + kb * 2 * MX_SF_BYTES)));
          umma_commit(sfb_ready);
        }
        ok = mbar_wait(w_full, 0, abort_flag, ST_TIMEOUT_MMA, 0xA01, budget) &&
             mbar_wait(sfb_ready, 0, abort_flag, ST_TIMEOUT_MMA, 0xA02, budget);
        tc_fence_after();
      }
      const uint32_t d_tmem = tmem_base + pl * MX_BN;
      int m_blk, n_blk;
      for (int it = pl; ok && tile_at(it, m_blk, n_blk); it += 2) {
        const uint32_t aph = (it >> 1) & 1;
        if (!mbar_wait(&acc_empty[pl], aph ^ 1, abort_flag, ST_TIMEOUT_MMA, 0x700 | pl, budget)) { ok = false; break; }
        tc_fence_after();
        if constexpr (WST) {
          for (int kb0 = 0; kb0 < p.k_blocks; kb0 += MXW_KPS) {
            // the wait orders the TMA writes before the reads below; no tcgen05 fence is needed for that
            if (!mbar_wait(&full[s], ph, abort_flag, ST_TIMEOUT_MMA, 0x800 | (pl << 4) | s, budget)) { ok = false; break; }
            const uint32_t st = smem_u32(ring + s * STAGE_BYTES);
            const int nk = p.k_blocks - kb0 < MXW_KPS ? p.k_blocks - kb0 : MXW_KPS;
            for (int j = 0; j < nk; ++j) {
              const int kb = kb0 + j;
              const uint32_t sfa_t = sf_tmem + (kb & 3) * 4;       // a slot per K block: no copy waits for earlier MMAs
              tmem_cp_32x128b_warpx4(sfa_t, sf_smem_desc(st + MXW_KPS * MX_A_BYTES + j * MX_SF_BYTES));
              const uint64_t a_desc = umma_smem_desc_sw128(st + j * MX_A_BYTES);
              const uint64_t b_desc = umma_smem_desc_sw128(smem_u32(w_res + kb * MX_B_BYTES));
#pragma unroll
              for (int k = 0; k < 4; ++k)
                umma_mxf8(d_tmem, a_desc + 2 * k, b_desc + 2 * k, umma_idesc_mx(0, 0, MX_BM, MX_BN, k, k), sfa_t,
                          sfb_tmem + kb * 4, (kb | k) != 0);
            }
            umma_commit(&empty[s]);
            if (++s == STAGES) { s = 0; ph ^= 1; }
          }
        } else {
          const uint32_t sfb_sub = (uint32_t)(((n_blk * OUT_COLS) % 128) / 32);   // dual: which 64-row half of the scale tile
          for (int kb = 0; kb < p.k_blocks; ++kb) {
            if (!mbar_wait(&full[s], ph, abort_flag, ST_TIMEOUT_MMA, 0x800 | (pl << 4) | s, budget)) { ok = false; break; }
            const uint32_t st = smem_u32(ring + s * STAGE_BYTES);
            const uint32_t sf = st + MX_A_BYTES + MX_B_BYTES;
            tmem_cp_32x128b_warpx4(sf_tmem, sf_smem_desc(sf));
            tmem_cp_32x128b_warpx4(sf_tmem + 4, sf_smem_desc(sf + MX_SF_BYTES));
            if constexpr (DUAL) tmem_cp_32x128b_warpx4(sf_tmem + 8, sf_smem_desc(sf + 2 * MX_SF_BYTES));
            const uint32_t b_addr = st + MX_A_BYTES;
            const uint64_t a_desc = umma_smem_desc_sw128(st);
            const uint64_t b_desc = umma_smem_desc_sw128(b_addr);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint32_t acc = (kb | k) != 0;
              if constexpr (DUAL) {
                const uint64_t bu_desc = umma_smem_desc_sw128(b_addr + MX_B_BYTES / 2);
                const uint32_t idesc = umma_idesc_mx(0, 0, MX_BM, 64, k, k);
                umma_mxf8(d_tmem, a_desc + 2 * k, b_desc + 2 * k, idesc, sf_tmem, sf_tmem + 4 + sfb_sub, acc);
                umma_mxf8(d_tmem + 64, a_desc + 2 * k, bu_desc + 2 * k, idesc, sf_tmem, sf_tmem + 8 + sfb_sub, acc);
              } else {
                umma_mxf8(d_tmem, a_desc + 2 * k, b_desc + 2 * k, umma_idesc_mx(0, 0, MX_BM, MX_BN, k, k), sf_tmem, sf_tmem + 4, acc);
              }
            }
            umma_commit(&empty[s]);
            if (++s == STAGES) { s = 0; ph ^= 1; }
          }
        }
        if (ok) umma_commit(&acc_full[pl]);
      }
    }
  } else if (warp >= MX_FRONT_WARPS) {
    // ------------------------------ epilogue ------------------------------
    // Warp e: TMEM lane quarter e % 4 (32 rows) and column half e / 4 of every tile, in tile order.  The accumulator
    // stage goes back to its pipeline as soon as this warp's part is in registers; the values leave as 32 x 32
    // fp16 boxes (64-byte swizzle) through the warp's one staging buffer.
    const int e = warp - MX_FRONT_WARPS, q = warp & 3, half = e >> 2;
    uint8_t* out_buf = smem + L::OUT + e * MX_OUT_BUF;
    bool ok = true;
    int m_blk, n_blk;
    auto emit_box = [&](int n, int row_base, const uint32_t (&w)[16]) {
      if (lane == 0) tma_store_wait_read<0>();               // the previous box has left the buffer
      __syncwarp();
#pragma unroll
      for (int pc = 0; pc < 4; ++pc)
        *reinterpret_cast<uint4*>(out_buf + lane * 64 + ((pc ^ ((lane >> 1) & 3)) << 4)) = make_uint4(w[4 * pc], w[4 * pc + 1], w[4 * pc + 2], w[4 * pc + 3]);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) { tma_store_2d(&tm_c, out_buf, n, row_base); tma_store_commit(); }
    };
    for (int it = 0; ok && tile_at(it, m_blk, n_blk); ++it) {
      const int as = it & 1; const uint32_t aph = (it >> 1) & 1;
      const int n0 = n_blk * OUT_COLS;
      if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[as], aph, abort_flag, ST_TIMEOUT_EPILOGUE, 0x900 | as, budget))) { ok = false; break; }
      tc_fence_after();
      const int row_base = m_blk * MX_BM + q * 32;
      const uint32_t t_row = tmem_base + as * MX_BN + ((uint32_t)(q * 32) << 16);
      uint32_t v[2][32];                                     // plain: 64 columns; dual: 32 gate | 32 up
      tmem_ld_32x32b_x32(t_row + (DUAL ? half * 32 : half * 64), v[0]);
      tmem_ld_32x32b_x32(t_row + (DUAL ? 64 + half * 32 : half * 64 + 32), v[1]);
      tmem_ld_wait(v[0], v[1]);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[as]);
      if (row_base >= p.M) continue;
      if constexpr (DUAL) {
        const int n = n0 + half * 32;
        if (n < p.N) {
          uint32_t w[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            // silu(gate) * up with silu(g) = h + h * tanh(h), h = g / 2
            const float2 hv = __fmul2_rn(make_float2(__uint_as_float(v[0][2 * j]), __uint_as_float(v[0][2 * j + 1])), make_float2(0.5f, 0.5f));
            const float2 uv = make_float2(__uint_as_float(v[1][2 * j]), __uint_as_float(v[1][2 * j + 1]));
            w[j] = pack_half2_from(__fmul2_rn(silu_from_half2(hv), uv));
          }
          emit_box(n, row_base, w);
        }
      } else {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const int n = n0 + half * 64 + b * 32;
          if (n < p.N) {
            uint32_t w[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) w[j] = pack_half2(__uint_as_float(v[b][2 * j]), __uint_as_float(v[b][2 * j + 1]));
            emit_box(n, row_base, w);
          }
        }
      }
    }
    if (lane == 0) tma_store_wait_all<0>();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, MX_TMEM_COLS); }
}

// ---- streaming form with 256-column tiles (plain GEMM, K > 512) ---------------------------------------------------
// With both operands streamed the 128 x 128 form above waits for its operands: 33 KiB per K block and 64 tensor clocks per
// MMA, while about 55 bytes per clock arrive (600 clocks per K block).  A 128 x 256 tile brings twice the products for 1.5
// times the bytes.  Its accumulator takes 256 TMEM columns, which leaves room for the scale factors but not for a second
// stage; the epilogue hands it back once it is in registers (a few hundred clocks of the tile's >= 10^4).
//   warps 0, 3  producers: K block i of the CTA goes to ring stage i % 4, filled by warp 0 (even) or 3 (odd)
//   warp 1      MMA issue        warps 4..11  epilogue: lane quarter e % 4, column half e / 4
// M = 65536, N = 512, K = 2048: 71.8 us with 128 columns, 63.7 with 256; M = 9001 11.3 and 9.9; M = 30000 37.1 and 31.3.
constexpr int MX2_BN = 256;
constexpr int MX2_STAGES = 4;
constexpr int MX2_B_BYTES = MX2_BN * MX_BK;                                      // 32 KiB
constexpr int MX2_STAGE_BYTES = MX_A_BYTES + MX2_B_BYTES + 4 * MX_SF_BYTES;      // A | W | SFA | SFB0 | SFB1 | pad
constexpr int MX2_OUT = MX2_STAGES * MX2_STAGE_BYTES;
constexpr int MX2_BAR = MX2_OUT + MX_EPI_WARPS * MX_OUT_BUF;
constexpr int MX2_BYTES = MX2_BAR + 256 + 1024;
static_assert(MX2_STAGE_BYTES % 1024 == 0 && MX2_BYTES <= 227 * 1024, "shared memory budget");

__global__ void __launch_bounds__(MX_THREADS, 1)
mx_gemm256_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                  const __grid_constant__ CUtensorMap tm_c, const MxParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + MX2_BAR);
  uint64_t* full = bars;                                   // [MX2_STAGES]
  uint64_t* empty = bars + MX2_STAGES;                     // [MX2_STAGES]
  uint64_t* acc_full = bars + 2 * MX2_STAGES;
  uint64_t* acc_empty = acc_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);
  const AbortFlag abort_flag{smem_u32(tmem_slot + 1)};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_tiles = p.m_blocks * p.n_blocks;           // (the host keeps this below 2^31)
  const int nb128_all = (p.N + 127) / 128;                 // scale tile row blocks of W

  if (threadIdx.x == 0) {
    for (int s = 0; s < MX2_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_full, 1); mbar_init(acc_empty, MX_EPI_WARPS);
    abort_flag.set(0);
    fence_mbar_init();
    prefetch_tmap(&tm_a); prefetch_tmap(&tm_b); prefetch_tmap(&tm_c);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, MX_TMEM_COLS); tmem_relinquish(); }
  pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const unsigned int budget = spin_budget();

  if (warp == 0 || warp == 3) {
    if (lane == 0) {
      const int mine = warp == 3 ? 1 : 0;
      bool ok = true;
      int i = 0;                                           // K blocks of this CTA so far
      for (int t = blockIdx.x; ok && t < num_tiles; t += gridDim.x) {
        const int m_blk = t / p.n_blocks, n_blk = t % p.n_blocks;
        const int nb128 = 2 * n_blk;
        const bool two = nb128 + 1 < nb128_all;            // the second 128 columns have scale tiles
        for (int kb = 0; kb < p.k_blocks; ++kb, ++i) {
          if ((i & 1) != mine) continue;
          const int st_i = i & (MX2_STAGES - 1);
          if (!mbar_wait(&empty[st_i], ((uint32_t)(i / MX2_STAGES) & 1u) ^ 1u, abort_flag, ST_TIMEOUT_PRODUCER, 0xB00 | st_i, budget)) { ok = false; break; }
          uint8_t* st = smem + st_i * MX2_STAGE_BYTES;
          uint8_t* sf = st + MX_A_BYTES + MX2_B_BYTES;
          mbar_arrive_expect_tx(&full[st_i], MX_A_BYTES + MX2_B_BYTES + (two ? 3 : 2) * MX_SF_BYTES);
          tma_load_2d(st, &tm_a, &full[st_i], kb * MX_BK, m_blk * MX_BM);
          tma_load_2d(st + MX_A_BYTES, &tm_b, &full[st_i], kb * MX_BK, n_blk * MX2_BN);
          bulk_load(sf, p.sfa + ((size_t)m_blk * p.k_blocks + kb) * MX_SF_BYTES, MX_SF_BYTES, &full[st_i]);
          bulk_load(sf + MX_SF_BYTES, p.sfb0 + ((size_t)nb128 * p.k_blocks + kb) * MX_SF_BYTES, MX_SF_BYTES, &full[st_i]);
          if (two) bulk_load(sf + 2 * MX_SF_BYTES, p.sfb0 + ((size_t)(nb128 + 1) * p.k_blocks + kb) * MX_SF_BYTES, MX_SF_BYTES, &full[st_i]);
        }
      }
      if (!ok) { const long long t0 = clock64(); while (clock64() - t0 < 2000000) { } }
    }
  } else if (warp == 1) {
    // the whole warp walks the loop, one lane of it issues (a single thread: 65.2 us instead of 63.7)
    bool ok = true;
    int i = 0, it = 0;
    for (int t = blockIdx.x; ok && t < num_tiles; t += gridDim.x, ++it) {
      if (!__all_sync(0xffffffffu, mbar_wait(acc_empty, (uint32_t)(it & 1) ^ 1u, abort_flag, ST_TIMEOUT_MMA, 0xB10, budget))) { ok = false; break; }
      tc_fence_after();
      for (int kb = 0; kb < p.k_blocks; ++kb, ++i) {
        const int st_i = i & (MX2_STAGES - 1);
        if (!__all_sync(0xffffffffu, mbar_wait(&full[st_i], (uint32_t)(i / MX2_STAGES) & 1u, abort_flag, ST_TIMEOUT_MMA, 0xB20 | st_i, budget))) { ok = false; break; }
        const uint32_t st = smem_u32(smem + st_i * MX2_STAGE_BYTES);
        const uint32_t sf = st + MX_A_BYTES + MX2_B_BYTES;
        const uint32_t sfa_t = tmem_base + MX_SF_COL + st_i * 16, sfb_t = sfa_t + 4;     // a slot per stage
        tmem_cp_32x128b_warpx4_elect(sfa_t, sf_smem_desc(sf));
        tmem_cp_32x128b_warpx4_elect(sfb_t, sf_smem_desc(sf + MX_SF_BYTES));
        tmem_cp_32x128b_warpx4_elect(sfb_t + 4, sf_smem_desc(sf + 2 * MX_SF_BYTES));
        const uint64_t a_desc = umma_smem_desc_sw128(st);
        const uint64_t b_desc = umma_smem_desc_sw128(st + MX_A_BYTES);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_mxf8_elect(tmem_base, a_desc + 2 * k, b_desc + 2 * k, umma_idesc_mx(0, 0, MX_BM, MX2_BN, k, k), sfa_t, sfb_t, (kb | k) != 0);
        umma_commit_elect(&empty[st_i]);
      }
      if (ok) umma_commit_elect(acc_full);
    }
  } else if (warp >= MX_FRONT_WARPS) {
    const int e = warp - MX_FRONT_WARPS, q = warp & 3, half = e >> 2;
    uint8_t* out_buf = smem + MX2_OUT + e * MX_OUT_BUF;
    int it = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it) {
      const int m_blk = t / p.n_blocks, n0 = (t % p.n_blocks) * MX2_BN + half * 128;
      if (!__all_sync(0xffffffffu, mbar_wait(acc_full, (uint32_t)it & 1u, abort_flag, ST_TIMEOUT_EPILOGUE, 0xB30, budget))) break;
      tc_fence_after();
      const int row_base = m_blk * MX_BM + q * 32;
      const uint32_t t_row = tmem_base + half * 128 + ((uint32_t)(q * 32) << 16);
      uint32_t v[4][32];
#pragma unroll
      for (int b = 0; b < 4; ++b) tmem_ld_32x32b_x32(t_row + 32 * b, v[b]);
      tmem_ld_wait(v[0], v[1]);
      tmem_ld_wait(v[2], v[3]);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty);
      if (row_base >= p.M) continue;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int n = n0 + 32 * b;
        if (n >= p.N) break;
        if (lane == 0) tma_store_wait_read<0>();             // the previous box has left the buffer
        __syncwarp();
#pragma unroll
        for (int pc = 0; pc < 4; ++pc)
          *reinterpret_cast<uint4*>(out_buf + lane * 64 + ((pc ^ ((lane >> 1) & 3)) << 4)) =
              make_uint4(pack_half2(__uint_as_float(v[b][8 * pc]), __uint_as_float(v[b][8 * pc + 1])),
                         pack_half2(__uint_as_float(v[b][8 * pc + 2]), __uint_as_float(v[b][8 * pc + 3])),
                         pack_half2(__uint_as_float(v[b][8 * pc + 4]), __uint_as_float(v[b][8 * pc + 5])),
                         pack_half2(__uint_as_float(v[b][8 * pc + 6]), __uint_as_float(v[b][8 * pc + 7])));
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) { tma_store_2d(&tm_c, out_buf, n, row_base); tma_store_commit(); }
      }
    }
    if (lane == 0) tma_store_wait_all<0>();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, MX_TMEM_COLS); }
}

// ---- weight-stationary form with 256-column tiles (K <= 512) ---------------------------------------------------------
// The 128 x 128 weight-stationary form above is bound by shared memory: 224 KiB (dual) pass through it per tile, 1790 clocks, and
// its 32 column slices leave 20 SMs idle.  With 256 accumulator columns (dual: 128 gate | 128 up) an MMA takes 128 clocks and
// reads 12 KiB for them (96 instead of 128 bytes per clock), A passes through L2 and shared memory half as often, and N = 2048
// is 16 slices, 144 CTAs.  TMEM holds one such accumulator beside the scale factors; the next tile's MMAs begin when the
// epilogue has it in registers.
// M = 65536, us (graph of launches): dual K = 512, N = 2048 130.5 -> 120; K = 384, N = 1536 83 -> 77; K = 256, N = 1024 48.4 ->
// 41.9; K = 128, N = 512 25.3 -> 19.3; plain K = 512, N = 2048 74.7 -> 72.5.  What it is bound by: dual K = 512 takes 184 k clocks of
// which the tensor pipe is busy in 62 % (114 k: 57 tiles of 2048), plain 107 k and 53 %; with one accumulator the next tile's MMAs wait
// until the epilogue has this one in registers, about 1200 clocks a tile.  And the clock is 1.6 GHz under the power cap.  Scale tiles
// copied to TMEM a K block ahead (131), a warp of its own for them (118) and warp-converged producers (121) change little or lose.
//   warps 0, 3  producers: K block i of the CTA goes to ring stage i % 4, filled by warp 0 (even) or 3 (odd); warp 0 also loads
//               the resident slice, K block by K block
//   warp 1      MMA issue        warps 4..11  epilogue: lane quarter e % 4, column half e / 4 (of gate and up)
constexpr int MXV_BN = 256;
constexpr int MXV_STAGES = 4;
constexpr int MXV_W_KB = MXV_BN * MX_BK;                                  // 32 KiB: W rows of one K block (dual: 128 gate | 128 up)
constexpr int MXV_A = MXW_MAX_KB * MXV_W_KB;                              // ring of A blocks
constexpr int MXV_SFA = MXV_A + MXV_STAGES * MX_A_BYTES;                  // their scale tiles
constexpr int MXV_OUT = MXV_SFA + MXV_STAGES * MX_SF_BYTES;               // staging: per epilogue warp 32 rows x 64 fp16
constexpr int MXV_OUT_BUF = 4096;
// The W scale tiles (two per K block) land in the staging boxes: they are copied to TMEM before the first MMAs, whose
// completion the epilogue waits for before it writes there.
constexpr int MXV_SFB = MXV_OUT;
constexpr int MXV_BAR = MXV_OUT + MX_EPI_WARPS * MXV_OUT_BUF;
constexpr int MXV_BYTES = MXV_BAR + 256;                                  // (no room to align the base: it is 1 KiB-aligned by declaration)
constexpr int MXV_SFA_COL = 256, MXV_SFB_COL = 256 + 4 * MXV_STAGES;      // TMEM columns of the scale factors
static_assert(MXV_BYTES <= 227 * 1024 && MXV_OUT % 1024 == 0 && MXV_SFB_COL + 8 * MXW_MAX_KB <= MX_TMEM_COLS, "budget");

template <bool DUAL>
__global__ void __launch_bounds__(MX_THREADS, 1)
mx_gemm256w_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b0, const __grid_constant__ CUtensorMap tm_b1,
                   const __grid_constant__ CUtensorMap tm_c, const MxParams p) {
  extern __shared__ __align__(1024) uint8_t mxv_smem[];
  uint8_t* smem = mxv_smem;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + MXV_BAR);
  uint64_t* full = bars;                                   // [MXV_STAGES]
  uint64_t* empty = full + MXV_STAGES;                     // [MXV_STAGES]
  uint64_t* w_full = empty + MXV_STAGES;                   // [MXW_MAX_KB] a K block of the resident slice and its scale tiles
  uint64_t* acc_full = w_full + MXW_MAX_KB;
  uint64_t* acc_empty = acc_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);
  const AbortFlag abort_flag{smem_u32(tmem_slot + 1)};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int OUT_COLS = DUAL ? MXV_BN / 2 : MXV_BN;
  if ((smem_u32(smem) & 1023u) != 0) {                     // (cannot happen: the swizzled tiles need it)
    if (threadIdx.x == 0) atomicOr(&g_status[0], ST_TIMEOUT_MMA);
    return;
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < MXV_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int kb = 0; kb < MXW_MAX_KB; ++kb) mbar_init(&w_full[kb], 1);
    mbar_init(acc_full, 1); mbar_init(acc_empty, MX_EPI_WARPS);
    abort_flag.set(0);
    fence_mbar_init();
    prefetch_tmap(&tm_a); prefetch_tmap(&tm_b0); prefetch_tmap(&tm_b1); prefetch_tmap(&tm_c);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, MX_TMEM_COLS); tmem_relinquish(); }
  pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const unsigned int budget = spin_budget();
  const int ws_n = (int)(blockIdx.x % p.n_blocks), ws_g = (int)(blockIdx.x / p.n_blocks);    // column slice, row-block group
  const int n0 = ws_n * OUT_COLS;
  const bool two = DUAL || 2 * ws_n + 1 < (p.N + 127) / 128;      // the second 128 columns have scale tiles

  if (warp == 0 || warp == 3) {
    if (lane == 0) {
      const int mine = warp == 3 ? 1 : 0;
      bool ok = true;
      int i = 0;                                           // K blocks of A so far
      for (int m_blk = ws_g; ok && m_blk < p.m_blocks; m_blk += p.n_groups) {
        // the row block after this one goes to L2 now (one CTA of the column slices asks for it)
        const int m_pf = m_blk + p.n_groups;
        if (mine == 1 && m_pf < p.m_blocks && ws_n == (m_pf / p.n_groups) % p.n_blocks)
          for (int kb = 0; kb < p.k_blocks; ++kb) tma_prefetch_l2_2d(&tm_a, kb * MX_BK, m_pf * MX_BM);
        for (int kb = 0; kb < p.k_blocks; ++kb, ++i) {
          if (mine == 0 && i < p.k_blocks) {               // the slice, beside the first row block
            uint8_t* wb = smem + kb * MXV_W_KB;
            uint8_t* sf = smem + MXV_SFB + kb * 2 * MX_SF_BYTES;
            mbar_arrive_expect_tx(&w_full[kb], MXV_W_KB + (two ? 2 : 1) * MX_SF_BYTES);
            tma_load_2d(wb, &tm_b0, &w_full[kb], kb * MX_BK, n0);
            tma_load_2d(wb + MXV_W_KB / 2, &tm_b1, &w_full[kb], kb * MX_BK, DUAL ? n0 : n0 + 128);
            const size_t t0 = ((size_t)(n0 / 128) * p.k_blocks + kb) * MX_SF_BYTES;
            bulk_load(sf, p.sfb0 + t0, MX_SF_BYTES, &w_full[kb]);
            if (two) bulk_load(sf + MX_SF_BYTES, DUAL ? p.sfb1 + t0 : p.sfb0 + t0 + (size_t)p.k_blocks * MX_SF_BYTES, MX_SF_BYTES, &w_full[kb]);
          }
          if ((i & 1) != mine) continue;
          const int s = i & (MXV_STAGES - 1);
          if (!mbar_wait(&empty[s], ((uint32_t)(i / MXV_STAGES) & 1u) ^ 1u, abort_flag, ST_TIMEOUT_PRODUCER, 0xD00 | s, budget)) { ok = false; break; }
          mbar_arrive_expect_tx(&full[s], MX_A_BYTES + MX_SF_BYTES);
          tma_load_2d(smem + MXV_A + s * MX_A_BYTES, &tm_a, &full[s], kb * MX_BK, m_blk * MX_BM);
          bulk_load(smem + MXV_SFA + s * MX_SF_BYTES, p.sfa + ((size_t)m_blk * p.k_blocks + kb) * MX_SF_BYTES, MX_SF_BYTES, &full[s]);
        }
      }
      if (!ok) { const long long t0 = clock64(); while (clock64() - t0 < 2000000) { } }
    }
  } else if (warp == 1) {
    // the whole warp walks the loop, one lane of it issues
    bool ok = true;
    int i = 0, it = 0;
    for (int m_blk = ws_g; ok && m_blk < p.m_blocks; m_blk += p.n_groups, ++it) {
      if (!__all_sync(0xffffffffu, mbar_wait(acc_empty, (uint32_t)(it & 1) ^ 1u, abort_flag, ST_TIMEOUT_MMA, 0xD10, budget))) { ok = false; break; }
      tc_fence_after();
      for (int kb = 0; kb < p.k_blocks; ++kb, ++i) {
        const int s = i & (MXV_STAGES - 1);
        const uint32_t sfb_t = tmem_base + MXV_SFB_COL + kb * 8;
        if (it == 0) {                                     // the slice arrives during the first tile; its scale tiles go to TMEM once
          if (!__all_sync(0xffffffffu, mbar_wait(&w_full[kb], 0, abort_flag, ST_TIMEOUT_MMA, 0xD20 | kb, budget))) { ok = false; break; }
          const uint32_t sf = smem_u32(smem + MXV_SFB + kb * 2 * MX_SF_BYTES);
          tmem_cp_32x128b_warpx4_elect(sfb_t, sf_smem_desc(sf));
          tmem_cp_32x128b_warpx4_elect(sfb_t + 4, sf_smem_desc(sf + MX_SF_BYTES));
        }
        if (!__all_sync(0xffffffffu, mbar_wait(&full[s], (uint32_t)(i / MXV_STAGES) & 1u, abort_flag, ST_TIMEOUT_MMA, 0xD30 | s, budget))) { ok = false; break; }
        const uint32_t sfa_t = tmem_base + MXV_SFA_COL + s * 4;              // a slot per stage
        tmem_cp_32x128b_warpx4_elect(sfa_t, sf_smem_desc(smem_u32(smem + MXV_SFA + s * MX_SF_BYTES)));
        const uint64_t a_desc = umma_smem_desc_sw128(smem_u32(smem + MXV_A + s * MX_A_BYTES));
        const uint64_t b_desc = umma_smem_desc_sw128(smem_u32(smem + kb * MXV_W_KB));
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_mxf8_elect(tmem_base, a_desc + 2 * k, b_desc + 2 * k, umma_idesc_mx(0, 0, MX_BM, MXV_BN, k, k), sfa_t, sfb_t, (kb | k) != 0);
        umma_commit_elect(&empty[s]);
      }
      if (ok) umma_commit_elect(acc_full);
    }
  } else if (warp >= MX_FRONT_WARPS) {
    const int e = warp - MX_FRONT_WARPS, q = warp & 3, half = e >> 2;
    uint8_t* out_buf = smem + MXV_OUT + e * MXV_OUT_BUF;
    uint8_t* const stg_row = out_buf + lane * 128;         // this thread's 128-byte row of the box, 16-byte pieces in the 128-byte swizzle
    int it = 0;
    for (int m_blk = ws_g; m_blk < p.m_blocks; m_blk += p.n_groups, ++it) {
      if (!__all_sync(0xffffffffu, mbar_wait(acc_full, (uint32_t)it & 1u, abort_flag, ST_TIMEOUT_EPILOGUE, 0xD40, budget))) break;
      tc_fence_after();
      const int row_base = m_blk * MX_BM + q * 32;
      const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16);
      uint32_t v[4][32];                                   // dual: 64 gate columns, 64 up columns; plain: 128 columns
#pragma unroll
      for (int b = 0; b < 4; ++b) tmem_ld_32x32b_x32(t_row + (DUAL ? half * 64 + (b >> 1) * 128 + (b & 1) * 32 : half * 128 + 32 * b), v[b]);
      tmem_ld_wait(v[0], v[1]);
      tmem_ld_wait(v[2], v[3]);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty);
      if (row_base >= p.M) continue;
#pragma unroll
      for (int b = 0; b < (DUAL ? 1 : 2); ++b) {           // one 64-column box
        const int n = n0 + (DUAL ? half * 64 : half * 128 + 64 * b);
        if (n >= p.N) break;
        if (lane == 0) tma_store_wait_read<0>();           // the previous box has left the buffer
        __syncwarp();
#pragma unroll
        for (int pc = 0; pc < 8; ++pc) {                   // 8 columns
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int c = (pc & 3) * 8 + 2 * j;
            if constexpr (DUAL) {
              // silu(gate) * up with silu(g) = h + h * tanh(h), h = g / 2
              const float2 hv = __fmul2_rn(make_float2(__uint_as_float(v[pc >> 2][c]), __uint_as_float(v[pc >> 2][c + 1])), make_float2(0.5f, 0.5f));
              const float2 uv = make_float2(__uint_as_float(v[2 + (pc >> 2)][c]), __uint_as_float(v[2 + (pc >> 2)][c + 1]));
              w[j] = pack_half2_from(__fmul2_rn(silu_from_half2(hv), uv));
            } else {
              w[j] = pack_half2(__uint_as_float(v[2 * b + (pc >> 2)][c]), __uint_as_float(v[2 * b + (pc >> 2)][c + 1]));
            }
          }
          *reinterpret_cast<uint4*>(stg_row + ((pc ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) { tma_store_2d(&tm_c, out_buf, n, row_base); tma_store_commit(); }
      }
    }
    if (lane == 0) tma_store_wait_all<0>();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, MX_TMEM_COLS); }
}

// ---- row-major [rows, K/32] scales -> the 128 x 4 tile order --------------------------------------------------
// A thread moves the four scales of one row and one 128-wide K tile: one word of the tile, four neighbouring source bytes
// (K % 128 == 0, so a row holds whole groups of four).  Consecutive threads write consecutive words; the 32 rows of a
// lane group lie ld bytes apart, and the other words of their sectors are picked up from L1 by the threads of the
// neighbouring tiles.  With a thread per byte the launch took 10.5 us (mean of 65536 x 512 and x 2048; 4.3 us now).
__global__ void mx_scales_to_tiled_kernel(const uint8_t* src, long long ld, long long rows, int kt,
                                          uint8_t* __restrict__ dst, unsigned words, bool word_loads, bool word_stores) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_trigger();
  pdl_wait();
  if (i >= words) return;
  const unsigned tile = i >> 7, in = i & 127;              // 128 words per tile
  const unsigned rb = tile / (unsigned)kt, kb = tile % (unsigned)kt;
  const long long row = (long long)rb * 128 + (in >> 2) + 32 * (in & 3);
  uint32_t v = 0x7f7f7f7fu;                                // padding rows: scale 1.0 on zero data
  if (row < rows) {
    const uint8_t* s = src + row * ld + kb * 4;
    if (word_loads) v = __ldcg(reinterpret_cast<const uint32_t*>(s));
    else v = s[0] | (uint32_t)s[1] << 8 | (uint32_t)s[2] << 16 | (uint32_t)s[3] << 24;
  }
  uint8_t* d = dst + (size_t)i * 4;
  if (word_stores) *reinterpret_cast<uint32_t*>(d) = v;
  else { d[0] = (uint8_t)v; d[1] = (uint8_t)(v >> 8); d[2] = (uint8_t)(v >> 16); d[3] = (uint8_t)(v >> 24); }
}

size_t mx_tiled_scale_bytes(long long rows, int K) {
  return (size_t)((rows + 127) / 128) * (size_t)(K / 128) * 512;
}

int32_t launch_mx_scales_to_tiled(const uint8_t* src, long long ld, long long rows, int K, uint8_t* dst, cudaStream_t st) {
  if (rows == 0) return GSB200_OK;
  if (!src || !dst || rows < 0 || K <= 0 || K % 128 != 0 || ld < K / 32) return GSB200_ERR_BAD_ARG;
  const long long words = (long long)mx_tiled_scale_bytes(rows, K) / 4;
  if (words > 0xffffff00ll) return GSB200_ERR_BAD_ARG;
  const bool word_loads = ld % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 3) == 0;
  const bool word_stores = (reinterpret_cast<uintptr_t>(dst) & 3) == 0;
  const cudaError_t e = launch_dependent(mx_scales_to_tiled_kernel, (unsigned)((words + 255) / 256), 256, 0, st, src, ld, rows,
                                         K / 128, dst, (unsigned)words, word_loads, word_stores);
  return cuda_status(e, "mx scale re-tiling launch");
}

int32_t launch_mx_gemm(bool dual, const uint8_t* A, long long lda, const uint8_t* sfa, const uint8_t* B0,
                       const uint8_t* B1, long long ldb, const uint8_t* sfb0, const uint8_t* sfb1, void* C,
                       long long ldc, long long M, int N, int K, cudaStream_t st) {
  if (M == 0) return GSB200_OK;
  if (M < 0 || M > 0x7fffff00ll || N <= 0 || K <= 0) return GSB200_ERR_BAD_ARG;
  if (!A || !sfa || !B0 || !sfb0 || !C || (dual && (!B1 || !sfb1))) return GSB200_ERR_BAD_ARG;
  const uintptr_t al = reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(sfa) | reinterpret_cast<uintptr_t>(B0) |
                       reinterpret_cast<uintptr_t>(sfb0) | reinterpret_cast<uintptr_t>(C) |
                       (dual ? (reinterpret_cast<uintptr_t>(B1) | reinterpret_cast<uintptr_t>(sfb1)) : 0);
  if (al & 15) return GSB200_ERR_BAD_ARG;
  if (K % 128 != 0 || lda < K || ldb < K || lda % 16 != 0 || ldb % 16 != 0) return GSB200_ERR_BAD_ARG;
  if (N % 32 != 0 || ldc < N || ldc % 8 != 0) return GSB200_ERR_BAD_ARG;
  int32_t rc = ensure_device();
  if (rc != GSB200_OK) return rc;
  static std::atomic<int> attr_done[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return GSB200_ERR_DEVICE;
  if (!attr_done[dev].load(std::memory_order_acquire)) {
    cudaError_t e1 = cudaFuncSetAttribute(mx_gemm_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, MxSmem<false>::BYTES);
    cudaError_t e2 = cudaFuncSetAttribute(mx_gemm_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, MxSmem<false>::BYTES);
    cudaError_t e3 = cudaFuncSetAttribute(mx_gemm_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, MxSmem<true>::BYTES);
    cudaError_t e4 = cudaFuncSetAttribute(mx_gemm_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, MxSmem<true>::BYTES);
    if (e1 != cudaSuccess || e2 != cudaSuccess) return cuda_status(e1 != cudaSuccess ? e1 : e2, "cudaFuncSetAttribute(mx gemm)");
    cudaError_t e5 = cudaFuncSetAttribute(mx_gemm256_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MX2_BYTES);
    if (e5 != cudaSuccess) return cuda_status(e5, "cudaFuncSetAttribute(mx gemm)");
    cudaError_t e6 = cudaFuncSetAttribute(mx_gemm256w_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, MXV_BYTES);
    if (e6 == cudaSuccess) e6 = cudaFuncSetAttribute(mx_gemm256w_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, MXV_BYTES);
    if (e6 != cudaSuccess) return cuda_status(e6, "cudaFuncSetAttribute(mx gemm)");
    if (e3 != cudaSuccess || e4 != cudaSuccess) return cuda_status(e3 != cudaSuccess ? e3 : e4, "cudaFuncSetAttribute(mx gemm)");
    attr_done[dev].store(1, std::memory_order_release);
  }
  auto map2d = [&](CUtensorMap* m, CUtensorMapDataType dt, int esz, const void* base, uint64_t rows, uint64_t cols,
                   uint64_t ld, uint32_t bc, uint32_t br, CUtensorMapSwizzle sw) {
    return tmap_2d(m, dt, esz, base, rows, cols, ld, bc, br, sw);
  };
  CUtensorMap ta, tb0, tb1, tc;
  if (!map2d(&ta, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, 128, 128, CU_TENSOR_MAP_SWIZZLE_128B)) return GSB200_ERR_BAD_ARG;
  // W in boxes of `rows` rows, the output in 32 x 32 boxes
  auto map_w = [&](uint32_t rows) {
    if (!map2d(&tb0, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, B0, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 128, rows, CU_TENSOR_MAP_SWIZZLE_128B)) return false;
    if (!dual) { tb1 = tb0; return true; }
    return map2d(&tb1, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, B1, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 128, rows, CU_TENSOR_MAP_SWIZZLE_128B);
  };
  auto map_c = [&]() {
    return map2d(&tc, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, C, (uint64_t)M, (uint64_t)N, (uint64_t)ldc, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B);
  };
  const bool wst = K / MX_BK <= MXW_MAX_KB && (N + (dual ? 64 : 128) - 1) / (dual ? 64 : 128) <= sm_count();
  MxParams p{};
  p.M = (int)M; p.N = N; p.K = K;
  const int out_cols = dual ? 64 : 128;
  p.m_blocks = (int)((M + MX_BM - 1) / MX_BM);
  p.n_blocks = (N + out_cols - 1) / out_cols;
  p.k_blocks = K / MX_BK;
  p.sfa = sfa; p.sfb0 = sfb0; p.sfb1 = sfb1;
  const long long tiles = (long long)p.m_blocks * p.n_blocks;
  cudaError_t e;
  // 256-column weight-stationary tiles where their rounds are cheaper: a tile takes about 1.5 times what a 128-column one does
  // (dual, K = 512, N = 2048: M = 4096 12.5 us with 128 columns, 11.9 with 256; M = 1024 6.8 and 5.9; M = 128, one round of either,
  // 5.3 and 5.5).  Where the 128-column slices are more than the SMs, the other side is the streaming kernel, which deals its tiles
  // to all SMs while this form leaves idle what its slices do not fill; a tile here takes 1.5 (dual 1.25) times what a round of 128
  // columns does there (us, streaming / this one; M = 5000, K = 512: plain N = 18976, 75 slices, 60.0 / 79.0, N = 22016, 86, 68.6 / 81.4, N =
  // 30016, 118, 92.0 / 84.1; dual N = 9504, 75, 65.5 / 77.8, N = 12000, 94, 80.4 / 81.4, N = 18944, 148, 122 / 87; K = 128: plain N = 22016
  // 42.2 / 56.1, dual N = 10016 40.8 / 44.9; M = 100, plain N = 22016, a second round there, 6.1 / 6.1, dual N = 9504 6.4 / 5.8).
  if (K / MX_BK <= MXW_MAX_KB) {
    const int out256 = dual ? 128 : 256, nb = (N + out256 - 1) / out256, sms = sm_count();
    const int g256 = sms / nb, g128 = wst ? sms / p.n_blocks : 0;
    const long long r256 = g256 > 0 ? (p.m_blocks + g256 - 1) / g256 : 0;
    const bool better = g128 > 0 ? r256 * 15 < (p.m_blocks + g128 - 1) / g128 * 10ll : r256 * (dual ? 25 : 30) < (tiles + sms - 1) / sms * 20;
    if (g256 > 0 && better) {
      if (!map_w(128) || !map2d(&tc, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, C, (uint64_t)M, (uint64_t)N, (uint64_t)ldc, 64, 32, CU_TENSOR_MAP_SWIZZLE_128B))
        return GSB200_ERR_BAD_ARG;
      p.n_blocks = nb;
      p.n_groups = g256 < p.m_blocks ? g256 : p.m_blocks;
      const int grid = p.n_groups * nb;
      e = dual ? launch_dependent(mx_gemm256w_kernel<true>, grid, MX_THREADS, MXV_BYTES, st, ta, tb0, tb1, tc, p)
               : launch_dependent(mx_gemm256w_kernel<false>, grid, MX_THREADS, MXV_BYTES, st, ta, tb0, tb1, tc, p);
      return cuda_status(e, "mx gemm launch");
    }
  }
  if (wst) {                                                        // weight-stationary form
    if (!map_w(dual ? 64 : 128) || !map_c()) return GSB200_ERR_BAD_ARG;
    int groups = sm_count() / p.n_blocks;
    if (groups > p.m_blocks) groups = p.m_blocks;
    p.n_groups = groups;
    const int grid = groups * p.n_blocks;
    if (dual) e = launch_dependent(mx_gemm_kernel<true, true>, grid, MX_THREADS, MxSmem<true>::BYTES, st, ta, tb0, tb1, tc, p);
    else e = launch_dependent(mx_gemm_kernel<false, true>, grid, MX_THREADS, MxSmem<true>::BYTES, st, ta, tb0, tb1, tc, p);
    return cuda_status(e, "mx gemm launch");
  }
  // 256-column tiles where their rounds are cheaper: a K block takes about 1.65 times what it takes with 128 columns, so few
  // tiles and an N just above a multiple of 256 stay with 128 (M = 65536, N = 384, K = 1536: 45.1 us, with 256 columns 46.3).
  const long long sms = sm_count(), tiles256 = (long long)p.m_blocks * ((N + MX2_BN - 1) / MX2_BN);
  if (!dual && (tiles256 + sms - 1) / sms * 33 < (tiles + sms - 1) / sms * 20 && tiles256 <= 0x7fffffffll) {
    if (!map_w(MX2_BN) || !map_c()) return GSB200_ERR_BAD_ARG;
    p.n_blocks = (N + MX2_BN - 1) / MX2_BN;
    e = launch_dependent(mx_gemm256_kernel, (int)(tiles256 < sms ? tiles256 : sms), MX_THREADS, MX2_BYTES, st, ta, tb0, tc, p);
    return cuda_status(e, "mx gemm launch");
  }
  if (!map_w(dual ? 64 : 128) || !map_c()) return GSB200_ERR_BAD_ARG;
  const int grid = (int)(tiles < sm_count() ? tiles : sm_count());
  if (dual) e = launch_dependent(mx_gemm_kernel<true, false>, grid, MX_THREADS, MxSmem<false>::BYTES, st, ta, tb0, tb1, tc, p);
  else e = launch_dependent(mx_gemm_kernel<false, false>, grid, MX_THREADS, MxSmem<false>::BYTES, st, ta, tb0, tb1, tc, p);
  return cuda_status(e, "mx gemm launch");
}

}  // namespace gsb
