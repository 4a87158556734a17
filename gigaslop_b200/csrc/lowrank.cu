// Low-rank input projection of a factored LSTM in one launch:
//     x_down = f16((x . dn^T) * sx[m] * s_dn)            FP8, [M, C] x [R, C], R = 64 or 128
//     ih     = f16(x_down . up^T + bias)                 fp16, [M, R] x [N, R]
// with x_down kept on chip (fly/rdna_fp8_factored_gemm.py:86-435 keeps it in LDS).  What bounds it is writing ih: 1.07 GB at
// M = 131072, N = 4096.  As two launches the 134 MB of x were read first, by themselves, and x_down made a round trip through the
// output rows; here the reads of the next row block run beside the writes of this one.  And as x_down is no longer where the output
// goes, the column tiles of a row block can be shared out: a CTA that takes some of them computes the row block's x_down for
// itself, which costs about as much as one and a half column tiles.
//   unit     a row block (128 rows) and a range of its 256-column tiles; a CTA's units come in rounds, the last, incomplete round
//            cut into shares so that all SMs have some (TileWalk's rule for the rotary GEMM)
//   item     D(u): x_down of unit u, C / 128 K blocks of x and dn;  U(u, n): column tile n, R / 64 K blocks of up
//   order    D(first); then the U items of unit after unit, with D of the next unit three items before the unit's end, so that its
//            x_down is in shared memory when the next unit's first MMAs want it
//   warp 0 producer (one thread), warp 1 MMA issue (one thread), warps 4..11 epilogue; two accumulator stages of 256 columns, items
//   take them in turn.  x_down lies in two buffers (units in turn) as the K-major, 128-byte-swizzled A operand of the U items.
// Same sums in the same order and the same roundings as the two launches: same bytes.  us (graph of launches), two launches -> one:
//   C = 1024, R = 128, N = 4096: M = 64 33.4 -> 7.6, 1000 36.4 -> 8.3, 4096 36.5 -> 13.1, 20000 72.0 -> 42.7, 65536 143.7 -> 127.0,
//   131072 249 -> 249 (seven rounds of 2.2 us per column tile: its epilogue and 4.3 TB/s of writes beside 0.5 of reads)
//   C = 512, N = 1536: M = 64 18.1 -> 6.9, 20000 34.1 -> 19.5, 131072 113.6 -> 97.5      C = 256, R = 64, N = 1024: 13.4 -> 5.8, 22.1 ->
//   13.3, 74.6 -> 59.1
#include <atomic>

#include "capi_internal.h"
#include "gemm_kernel.cuh"

namespace gsb {

constexpr int LR_STAGES = 3;
constexpr int LR_STAGE_BYTES = B_STAGE_BYTES;                  // 32 KiB: x 16 | dn up to 16, or 256 rows of up
constexpr int LR_XD_BYTES = 2 * A_STAGE_BYTES;                 // one x_down buffer: up to two K blocks of 64 fp16
constexpr int LR_OUT_BUFS = 3;
constexpr int LR_BIAS_BUFS = 6;                                // as SmemMap::SCALE_BUFS (an item is at most three ahead of the MMAs)
constexpr int LR_XD = LR_STAGES * LR_STAGE_BYTES;
constexpr int LR_OUT = LR_XD + 2 * LR_XD_BYTES;
constexpr int LR_BIAS = LR_OUT + EPI_WARPS * LR_OUT_BUFS * OUT_BUF_BYTES;
constexpr int LR_BAR = LR_BIAS + LR_BIAS_BUFS * BN * 4;
constexpr int LR_SMEM = LR_BAR + 256 + 1024;
static_assert(LR_SMEM <= 227 * 1024 && LR_OUT % 1024 == 0, "shared memory budget");

struct LrParams {
  int M, N, m_blocks, n_blocks, kb_d, kb_u, R;
  int split;                   // shares of each row block of the last round
  const float* sx; const float* s_dn; const float* bias;
};

struct LrUnit { int m, lo, hi; };
struct LrWalk {
  LrUnit cur, nxt;
  int n, visit;                // column tile of cur; which unit of the CTA cur is
  bool is_d, started, placed;  // the item is a D; the first D is behind us; D(nxt) is behind us
  __device__ __forceinline__ static LrUnit unit(const LrParams& p, int visit) {
    const int grid = (int)gridDim.x, cta = (int)blockIdx.x, full = p.m_blocks / grid, rem = p.m_blocks - full * grid;
    LrUnit u{-1, 0, p.n_blocks};
    if (visit < full) u.m = cta + visit * grid;
    else {
      const int per = (p.n_blocks + p.split - 1) / p.split, k = cta + (visit - full) * grid;
      if (k < rem * p.split) {
        u.m = full * grid + k / p.split;
        u.lo = (k % p.split) * per;
        u.hi = u.lo + per < p.n_blocks ? u.lo + per : p.n_blocks;
      }
    }
    return u;
  }
  __device__ __forceinline__ void start(const LrParams& p) {
    visit = 0; cur = unit(p, 0); nxt = unit(p, 1); n = cur.lo; is_d = true; started = false; placed = false;
  }
  __device__ __forceinline__ bool valid() const { return cur.m >= 0; }
  __device__ __forceinline__ const LrUnit& d_unit() const { return started ? nxt : cur; }       // of a D item
  __device__ __forceinline__ int buf() const { return (is_d && started ? visit + 1 : visit) & 1; }      // x_down buffer of the item
  __device__ __forceinline__ void next(const LrParams& p) {
    if (is_d) {
      if (started) placed = true;
      started = true;
    } else if (++n == cur.hi) {
      cur = nxt; ++visit; nxt = unit(p, visit + 1); n = cur.lo; placed = false;
    }
    is_d = !placed && nxt.m >= 0 && n == (cur.hi - 3 > cur.lo ? cur.hi - 3 : cur.lo);
  }
};

__global__ void __launch_bounds__(GEMM_THREADS, 1)
lowrank_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_dn, const __grid_constant__ CUtensorMap tm_up,
               const __grid_constant__ CUtensorMap tm_c, const LrParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + LR_BAR);     // [LR_STAGES]
  uint64_t* empty = full + LR_STAGES;                              // [LR_STAGES]
  uint64_t* acc_full = empty + LR_STAGES;                          // [ACC_STAGES]
  uint64_t* acc_empty = acc_full + ACC_STAGES;                     // [ACC_STAGES]
  uint64_t* xd_full = acc_empty + ACC_STAGES;                      // [2] x_down of a unit is in its buffer
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(xd_full + 2);
  float* bias_s = reinterpret_cast<float*>(smem + LR_BIAS);
  const AbortFlag abort_flag{smem_u32(tmem_slot + 1)};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < LR_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < ACC_STAGES; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], EPI_WARPS); mbar_init(&xd_full[s], EPI_WARPS); }
    abort_flag.set(0);
    fence_mbar_init();
    prefetch_tmap(&tm_x); prefetch_tmap(&tm_dn); prefetch_tmap(&tm_up); prefetch_tmap(&tm_c);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
  pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const unsigned int budget = spin_budget();

  if (warp == 0) {
    // ------------------------------ producer ------------------------------
    if (lane == 0) {
      int s = 0, bb = 0; uint32_t ph = 0; bool ok = true;
      LrWalk w; w.start(p);
      for (; ok && w.valid(); w.next(p)) {
        const int m0 = w.d_unit().m * BM, n0 = w.n * BN;
        // the next unit's rows of x come from HBM: ask for them in L2 a few items before they are loaded
        if (!w.is_d && w.nxt.m >= 0 && w.n == (w.cur.hi - 5 > w.cur.lo ? w.cur.hi - 5 : w.cur.lo))
          for (int kb = 0; kb < p.kb_d; ++kb) tma_prefetch_l2_2d(&tm_x, kb * BK, w.nxt.m * BM);
        const int kbs = w.is_d ? p.kb_d : p.kb_u;
        for (int kb = 0; kb < kbs; ++kb) {
          if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, ST_TIMEOUT_PRODUCER, 0xE00 | s, budget)) { ok = false; break; }
          uint8_t* st = smem + s * LR_STAGE_BYTES;
          if (w.is_d) {
            mbar_arrive_expect_tx(&full[s], A_STAGE_BYTES + p.R * BK);
            tma_load_2d(st, &tm_x, &full[s], kb * BK, m0);
            tma_load_2d(st + A_STAGE_BYTES, &tm_dn, &full[s], kb * BK, 0);
          } else {
            const uint32_t bias_bytes = kb == 0 ? (uint32_t)(min(BN, p.N - n0) * 4) : 0u;
            mbar_arrive_expect_tx(&full[s], LR_STAGE_BYTES + bias_bytes);
            if (bias_bytes) bulk_load(bias_s + bb * BN, p.bias + n0, bias_bytes, &full[s]);
            tma_load_2d(st, &tm_up, &full[s], kb * 64, n0);                  // (x counts fp16 elements)
            tma_load_2d(st + (BN / 2) * BK, &tm_up, &full[s], kb * 64, n0 + BN / 2);
          }
          if (++s == LR_STAGES) { s = 0; ph ^= 1; }
        }
        if (!w.is_d && ++bb == LR_BIAS_BUFS) bb = 0;
      }
      if (!ok) { const long long t0 = clock64(); while (clock64() - t0 < 2000000) { } }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issue ------------------------------
    if (lane == 0) {
      const uint32_t idesc_d = umma_idesc(1, 0, 0, BM, p.R);               // e4m3 x e4m3 -> f32, N = R
      constexpr uint32_t idesc_u = umma_idesc(1, 0, 0, BM, BN);            // f16 x f16 -> f32
      int s = 0; uint32_t ph = 0; bool ok = true;
      LrWalk w; w.start(p);
      for (int it = 0; ok && w.valid(); ++it, w.next(p)) {
        const int as = it & 1; const uint32_t aph = (it >> 1) & 1;
        if (!mbar_wait(&acc_empty[as], aph ^ 1, abort_flag, ST_TIMEOUT_MMA, 0xE10 | as, budget)) { ok = false; break; }
        // the first item of a unit reads its x_down (the others come after it)
        if (!w.is_d && w.n == w.cur.lo &&
            !mbar_wait(&xd_full[w.buf()], (uint32_t)(w.visit >> 1) & 1u, abort_flag, ST_TIMEOUT_MMA, 0xE20 | w.buf(), budget)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d = tmem_base + as * BN;
        const uint32_t xd = smem_u32(smem + LR_XD + w.buf() * LR_XD_BYTES);
        const int kbs = w.is_d ? p.kb_d : p.kb_u;
        for (int kb = 0; kb < kbs; ++kb) {
          if (!mbar_wait(&full[s], ph, abort_flag, ST_TIMEOUT_MMA, 0xE30 | s, budget)) { ok = false; break; }
          tc_fence_after();
          const uint32_t st = smem_u32(smem + s * LR_STAGE_BYTES);
          if (w.is_d) {
            const uint64_t a = umma_smem_desc_sw128(st), b = umma_smem_desc_sw128(st + A_STAGE_BYTES);
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_f8(d, a + 2 * k, b + 2 * k, idesc_d, (kb | k) != 0);
          } else {
            const uint64_t a = umma_smem_desc_sw128(xd + kb * A_STAGE_BYTES), b = umma_smem_desc_sw128(st);
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_f16(d, a + 2 * k, b + 2 * k, idesc_u, (kb | k) != 0);
          }
          umma_commit(&empty[s]);
          if (++s == LR_STAGES) { s = 0; ph ^= 1; }
        }
        if (ok) umma_commit(&acc_full[as]);
      }
    }
  } else if (warp >= FRONT_WARPS) {
    // ------------------------------ epilogue ------------------------------
    // warp e: TMEM lane quarter e % 4 (32 rows), column half e / 4 of the item
    const int e = warp - FRONT_WARPS, q = warp & 3, half = e >> 2;
    uint8_t* out_buf = smem + LR_OUT + e * LR_OUT_BUFS * OUT_BUF_BYTES;
    const int rl = q * 32 + lane;
    const float2 sdn2 = pk2(ldg_f_here(p.s_dn), 0.f);
    int obuf = 0, bb = 0;
    LrWalk w; w.start(p);
    float sx = 0.f;
    if (w.valid() && w.cur.m * BM + rl < p.M) sx = ldg_f_here(p.sx + w.cur.m * BM + rl);
    for (int it = 0; w.valid(); ++it, w.next(p)) {
      const int as = it & 1; const uint32_t aph = (it >> 1) & 1;
      const bool got = mbar_wait(&acc_full[as], aph, abort_flag, ST_TIMEOUT_EPILOGUE, 0xE40 | as, budget);
      uint32_t agreed = __all_sync(0xffffffffu, got) ? 1u : 0u;
      if (!agreed) break;
      asm volatile("" : "+r"(agreed));                 // the bias address below stays dependent on the wait
      tc_fence_after();
      const uint32_t t_row = tmem_base + as * BN + ((uint32_t)(q * 32) << 16);
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[as]);
      };
      if (w.is_d) {
        // this warp's R / 2 columns of x_down, 32 at a time, into the operand layout of the U items: column c of row r is fp16
        // element c % 64 of K block c / 64, its 16-byte chunk XOR-ed with r % 8.  (Rows past M: x was read as zeros.)
        const float2 sa2 = pk2(sx, sx), sd2 = pk2(sdn2.x, sdn2.x);
        uint8_t* xd = smem + LR_XD + w.buf() * LR_XD_BYTES + rl * 128;
        const int c0 = half * (p.R / 2);
        for (int c = c0; c < c0 + p.R / 2; c += 32) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(t_row + c, v);
          tmem_ld_wait(v);
          if (c + 32 >= c0 + p.R / 2) release();
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint4 o;
            o.x = pack_half2_from(dequant2<KIND_F8>(v[8 * j], v[8 * j + 1], sa2, sd2));
            o.y = pack_half2_from(dequant2<KIND_F8>(v[8 * j + 2], v[8 * j + 3], sa2, sd2));
            o.z = pack_half2_from(dequant2<KIND_F8>(v[8 * j + 4], v[8 * j + 5], sa2, sd2));
            o.w = pack_half2_from(dequant2<KIND_F8>(v[8 * j + 6], v[8 * j + 7], sa2, sd2));
            const int ck = ((c & 63) >> 3) + j;
            *reinterpret_cast<uint4*>(xd + (c >> 6) * A_STAGE_BYTES + ((ck ^ (rl & 7)) << 4)) = o;
          }
        }
        fence_proxy_async_smem();                      // the stores above before the MMAs read them
        __syncwarp();
        if (lane == 0) mbar_arrive(&xd_full[w.buf()]);
        // the token scales of the unit after this one
        const LrUnit after = LrWalk::unit(p, w.started ? w.visit + 2 : 1);
        sx = after.m >= 0 && after.m * BM + rl < p.M ? ldg_f_here(p.sx + after.m * BM + rl) : 0.f;
        continue;
      }
      const int row_base = w.cur.m * BM + q * 32, nw = w.n * BN + half * (BN / 2);
      const uint32_t sc = smem_u32(bias_s + bb * BN + half * (BN / 2)) + ((agreed - 1u) << 2);
      if (++bb == LR_BIAS_BUFS) bb = 0;
      if (row_base >= p.M) { release(); continue; }
      const float2 one2 = pk2(1.f, 1.f);
      const uint32_t t = t_row + half * (BN / 2);
      int buf_a = 0, buf_b = 0;
      // a pair of boxes of 16 rows x 64 columns, 128-byte swizzle (gemm_kernel.cuh)
      auto begin = [&]() {
        buf_a = obuf; buf_b = obuf + 1 == LR_OUT_BUFS ? 0 : obuf + 1;
        if (lane == 0) tma_store_wait_read<LR_OUT_BUFS - 2>();
        __syncwarp();
      };
      auto emit = [&](const uint32_t (&v)[32], int c, int which) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          *reinterpret_cast<uint4*>(out_buf + (lane < 16 ? buf_a : buf_b) * OUT_BUF_BYTES + (lane & 15) * 128 + (((which * 4 + j) ^ (lane & 7)) << 4)) =
              bias_piece<KIND_F16>(&v[8 * j], one2, lds_f4_ro(sc + 4 * c + 32 * j), lds_f4_ro(sc + 4 * c + 32 * j + 16));
      };
      auto end = [&](int n) {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_2d(&tm_c, out_buf + buf_a * OUT_BUF_BYTES, n, row_base); tma_store_commit();
          if (row_base + OUT_BOX_ROWS < p.M) tma_store_2d(&tm_c, out_buf + buf_b * OUT_BUF_BYTES, n, row_base + OUT_BOX_ROWS);
          tma_store_commit();                          // two groups per pair (the second may be empty): begin counts groups
        }
        obuf = buf_b + 1 == LR_OUT_BUFS ? 0 : buf_b + 1;
      };
      uint32_t va[32], vb[32];
      tmem_ld_32x32b_x32(t, va);
#pragma unroll
      for (int c = 0; c < BN / 2; c += 64) {
        const bool live = nw + c < p.N;
        tmem_ld_wait(va);
        tmem_ld_32x32b_x32(t + c + 32, vb);
        if (live) { begin(); emit(va, c, 0); }
        tmem_ld_wait(vb);
        if (c + 64 < BN / 2) tmem_ld_32x32b_x32(t + c + 64, va); else release();
        if (live) { emit(vb, c + 32, 1); end(nw + c); }
      }
    }
    if (lane == 0) tma_store_wait_all<0>();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, TMEM_COLS); }
}

// ih = f16(f16((x . dn^T) * sx * s_dn) . up^T + bias), R = 64 or 128.  The arguments have passed gsb200_fac_gemm_fp8_f16's checks
// and those of launch_gemm for the two products.
int32_t launch_lowrank(const uint8_t* x, long long ldx, const float* sx, const uint8_t* dn, long long lddn, const float* s_dn, const void* up,
                       long long ldup, const float* bias, void* ih, long long ldih, long long M, int C, int R, int N, cudaStream_t st) {
  int32_t rc = ensure_device();
  if (rc != GSB200_OK) return rc;
  static std::atomic<int> attr_done[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return GSB200_ERR_DEVICE;
  if (!attr_done[dev].load(std::memory_order_acquire)) {
    const cudaError_t e = cudaFuncSetAttribute(lowrank_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LR_SMEM);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(low-rank projection)");
    attr_done[dev].store(1, std::memory_order_release);
  }
  LrParams p{};
  p.M = (int)M; p.N = N; p.R = R;
  p.m_blocks = (int)((M + BM - 1) / BM);
  p.n_blocks = (N + BN - 1) / BN;
  p.kb_d = (C + BK - 1) / BK;
  p.kb_u = R / 64;
  p.sx = sx; p.s_dn = s_dn; p.bias = bias;
  // The last, incomplete round (with few row blocks the only one): as many shares per row block as let it end soonest, a share
  // charged 1.5 column tiles for its x_down at C = 1024.
  const int sms = sm_count(), rem = p.m_blocks % sms;
  int grid = p.m_blocks < sms ? p.m_blocks : sms;
  p.split = 1;
  if (rem > 0) {
    const long long d4 = 2 + p.kb_d / 2;                         // x_down in quarters of a column tile
    long long best = 4 * p.n_blocks + d4;
    for (int S = 2; S <= p.n_blocks && S <= sms; ++S) {
      const int per = (p.n_blocks + S - 1) / S, shares = (p.n_blocks + per - 1) / per;
      const long long t = ((long long)rem * shares + sms - 1) / sms * (4 * per + d4);
      if (shares == S && t < best) { best = t; p.split = S; }
    }
    if (p.m_blocks < sms) grid = rem * p.split < sms ? rem * p.split : sms;
  }
  CUtensorMap tx, td, tu, tc;
  const CUtensorMapDataType u8 = CU_TENSOR_MAP_DATA_TYPE_UINT8, f16 = CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  if (!tmap_2d(&tx, u8, 1, x, (uint64_t)M, (uint64_t)C, (uint64_t)ldx, BK, BM, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !tmap_2d(&td, u8, 1, dn, (uint64_t)R, (uint64_t)C, (uint64_t)lddn, BK, (uint32_t)R, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !tmap_2d(&tu, f16, 2, up, (uint64_t)N, (uint64_t)R, (uint64_t)ldup, 64, BN / 2, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !tmap_2d(&tc, f16, 2, ih, (uint64_t)M, (uint64_t)N, (uint64_t)ldih, OUT_BOX_COLS, OUT_BOX_ROWS, CU_TENSOR_MAP_SWIZZLE_128B))
    return GSB200_ERR_BAD_ARG;
  return cuda_status(launch_dependent(lowrank_kernel, (unsigned)grid, GEMM_THREADS, LR_SMEM, st, tx, td, tu, tc, p), "low-rank projection launch");
}

}  // namespace gsb
