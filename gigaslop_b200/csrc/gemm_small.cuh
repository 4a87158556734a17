// Few-tile form of the 8-bit GEMMs: one tile of 64 or 128 rows per CTA, no persistence.
//
// What bounds a GEMM of a few rows is not bandwidth but the chain launch -> first bytes -> MMAs -> epilogue on the few SMs
// that have a tile.  The persistent kernel's tile is 128 x 256: at K = 512 its MMAs take 2048 clocks and its epilogue about
// 5000, one after the other when there is only one tile, and the down-projection of 256 rows to 512 columns is four of them.
// Here a tile is 64 rows x 64 or 128 accumulator columns (128 x 128 where those are too many), so the same work spreads over 8
// to 16 times as many SMs: the MMAs of K = 512 take about 900 clocks (issue-bound), a CTA loads 64 KiB instead of 192, and a
// thread's epilogue is 32 columns, loaded once and stored straight from registers.  us per launch from a graph, persistent
// kernel -> this one:
//   dequant N = 512, K = 512    M = 1 5.3 -> 3.0, 256 6.0 -> 3.2, 1024 6.0 -> 3.7, 3072 6.0 -> 4.5
//   dequant N = 512, K = 2048   M = 64 9.7 -> 5.9, 1024 9.7 -> 6.5, 3072 10.3 -> 7.8      N = 128, K = 1024 (FP8)  M = 256 6.7 -> 4.1
//   rotary N = 1536, K = 512    M = 64 6.6 -> 3.7, 256 7.5 -> 4.4, 768 8.1 -> 5.2
//   SwiGLU N = 2048, K = 512    M = 64 5.6 -> 3.3, 256 5.9 -> 4.3, 768 6.2 -> 5.8
//   accumulator columns  [0, NPART) = rows n0 .. of W (dual: gate), [NPART, 2 NPART) = rows n1 .. of W (dual: of the up weight).
//   n1 = n0 + NPART for the plain epilogue; for the rotary one the two parts are what rotates together (heads of 128 with all
//   columns rotated: 64 apart).
//   warp 0 lane 0 loads (TMA, ring of p.stages K blocks), warp 1 lane 0 issues the MMAs, all eight warps do the epilogue: warp w
//   reads TMEM lane quarter w % 4 (64 rows: row 16 q + l lies in lane 32 q + l, l < 16) and half w / 4 of both parts.
// The arithmetic, its order and its rounding points are those of gemm_kernel.cuh's epilogues: same bytes.
#pragma once
#include <cuda_fp8.h>

#include <atomic>

#include "capi_internal.h"
#include "gemm_kernel.cuh"

namespace gsb {

constexpr int SG_THREADS = 256;
constexpr int SG_MAX_STAGES = 12;

template <int TM, int NPART>
struct SgSmem {
  static constexpr int A_BYTES = TM * BK;                              // per K block
  static constexpr int STAGE_BYTES = A_BYTES + 2 * NPART * BK;         // 16, 24 or 32 KiB
  static constexpr int TAIL = 2 * NPART * 4 + (2 * SG_MAX_STAGES + 1) * 8 + 16;      // channel scales, barriers, TMEM address, abort flag
  static constexpr int bytes(int stages) { return stages * STAGE_BYTES + ((TAIL + 127) & ~127); }
};

struct SgParams {
  int M, N, n_tiles, k_blocks, stages;
  void* C; long long ldc;
  uint8_t* out_scale; long long ld_scale;
  float scale_a_const;
  const float* scale_a; const float* scale_b0; const float* scale_b1;
  int scale_b_scalar;
  const float* sin_tab; const float* cos_tab;
  int seqlen, row_offset, rot_cols;
  int rot_geo;             // rotary: 0 heads of 128, all rotated; 1 heads of 128, 64 rotated; 2 heads of 64, 32 rotated; 3 heads of 64, all rotated
};

template <int KIND, int EPI, int TM, int NPART>
__global__ void __launch_bounds__(SG_THREADS, 2)
gemm_small_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b0, const __grid_constant__ CUtensorMap tm_b1,
                  const SgParams p) {
  extern __shared__ __align__(1024) uint8_t sg_smem[];
  constexpr bool DUAL = EPI == EPI_SILU || EPI == EPI_SILU_MX;
  constexpr int ST = SgSmem<TM, NPART>::STAGE_BYTES, H = NPART / 2;    // H = columns of each part that a warp handles
  constexpr int QR = TM / 4;                                           // rows in a TMEM lane quarter
  constexpr int SG_A_BYTES = SgSmem<TM, NPART>::A_BYTES;
  static_assert(TM == 128 || TM == 64, "UMMA M");
  static_assert(EPI != EPI_ROTARY || TM == 64, "the rotary rows of a tile");
  static_assert(EPI != EPI_SILU_MX || H == 32, "a thread quantises whole blocks of 32 columns");
  static_assert(EPI != EPI_ROTARY || NPART == 32, "rotary parts are 32 columns");
  float* sc_s = reinterpret_cast<float*>(sg_smem + p.stages * ST);     // [2 NPART]
  uint64_t* full = reinterpret_cast<uint64_t*>(sc_s + 2 * NPART);
  uint64_t* empty = full + SG_MAX_STAGES;
  uint64_t* acc_full = empty + SG_MAX_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  const AbortFlag abort_flag{smem_u32(tmem_slot + 1)};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if ((smem_u32(sg_smem) & 1023u) != 0) {              // (cannot happen: the swizzled tiles need it)
    if (threadIdx.x == 0) atomicOr(&g_status[0], ST_TIMEOUT_MMA);
    return;
  }

  const int m0 = (int)(blockIdx.x / p.n_tiles) * TM, tn = (int)(blockIdx.x % p.n_tiles);
  int n0, n1;                                          // first W row (= output column) of the two parts
  if constexpr (DUAL) { n0 = n1 = tn * NPART; }
  else if (EPI == EPI_ROTARY && p.rot_geo == 0) { n0 = (tn >> 1) * 128 + (tn & 1) * 32; n1 = n0 + 64; }
  else { n0 = tn * 2 * NPART; n1 = n0 + NPART; }

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_full, 1);
    abort_flag.set(0);
    fence_mbar_init();
    prefetch_tmap(&tm_a); prefetch_tmap(&tm_b0); prefetch_tmap(&tm_b1);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 2 * NPART); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // The grid is at most a wave, so its successor's blocks find room while it runs.  They may start only once this CTA has its
  // tensor memory: a successor's CTA that took some first would hold it until this grid is done, and this one wait for it.
  pdl_trigger();
  pdl_wait();
  const unsigned int budget = spin_budget();

  // this thread's row; its token scale and sin / cos values are on their way during the main loop
  const int q = warp & 3, half = warp >> 2;
  const int row = m0 + q * QR + lane;
  const bool row_ok = lane < QR && row < p.M;
  const int rc = row < p.M ? row : p.M - 1;            // (a row that exists, for the load)
  // rotary: the warp's two 16-column chunks ca, cb rotate together (or are only dequantised)
  const bool pairs32 = EPI != EPI_ROTARY || p.rot_geo != 2;
  const int ca = pairs32 ? half * H : half * 32, cb = pairs32 ? NPART + half * H : half * 32 + 16;
  bool rotated = false;
  float sa = p.scale_a_const;
  // Rotary: the tile's 64 rows of sin and of cos, 8 chunks of 16 bytes each (geometry 2: 4), are fetched by all threads in
  // whole lines during the main loop and handed to the threads that need them through the ring, once the MMAs have read it.
  // (A thread loading its own row's values, 32 scattered rows per instruction: 5.1 instead of 4.4 us at 256 rows, 7.0 instead
  // of 5.2 at 768.)
  const bool tile_rot = EPI == EPI_ROTARY && n0 < p.rot_cols && (p.rot_geo != 1 || (tn & 1) == 0);
  const int rot_ch = p.rot_geo == 2 ? 4 : 8;           // chunks of a row that the tile uses
  [[maybe_unused]] float4 tr[4];
  auto fetch = [&]() {
    if (p.scale_a) sa = ldg_f_here(p.scale_a + rc);
    if (tile_rot) {
      rotated = p.rot_geo != 2 || half == 0;
      const int ld = p.rot_geo == 0 ? 64 : p.rot_geo == 2 ? 16 : 32, col = p.rot_geo == 0 ? (tn & 1) * 32 : 0, ch = threadIdx.x & 7;
      if (ch < rot_ch) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          int r = m0 + (threadIdx.x >> 3) + 32 * i;
          r = r < p.M ? r : p.M - 1;
          const long long off = (long long)(((unsigned)r + (unsigned)p.row_offset) % (unsigned)p.seqlen) * ld + col + 4 * ch;
          tr[i] = ldg_f4_here(p.sin_tab + off);
          tr[2 + i] = ldg_f4_here(p.cos_tab + off);
        }
      }
    }
  };
  if (warp != 0) fetch();

  if (warp == 0) {
    if (lane == 0) {
      int s = 0; uint32_t ph = 0;
      for (int kb = 0; kb < p.k_blocks; ++kb) {
        if (kb >= p.stages && !mbar_wait(&empty[s], ph ^ 1, abort_flag, ST_TIMEOUT_PRODUCER, 0xC00 | s, budget)) break;
        uint8_t* st = sg_smem + s * ST;
        mbar_arrive_expect_tx(&full[s], ST);
        tma_load_2d(st, &tm_a, &full[s], kb * BK, m0);
        tma_load_2d(st + SG_A_BYTES, &tm_b0, &full[s], kb * BK, n0);
        tma_load_2d(st + SG_A_BYTES + NPART * BK, &tm_b1, &full[s], kb * BK, n1);
        if (++s == p.stages) { s = 0; ph ^= 1; }
      }
    }
    __syncwarp();
    fetch();
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = (KIND == KIND_I8) ? umma_idesc(2, 1, 1, TM, 2 * NPART) : umma_idesc(1, 0, 0, TM, 2 * NPART);
      int s = 0; uint32_t ph = 0; bool ok = true;
      for (int kb = 0; kb < p.k_blocks; ++kb) {
        if (!mbar_wait(&full[s], ph, abort_flag, ST_TIMEOUT_MMA, 0xC10 | s, budget)) { ok = false; break; }
        tc_fence_after();
        const uint32_t st = smem_u32(sg_smem + s * ST);
        const uint64_t a_desc = umma_smem_desc_sw128(st), b_desc = umma_smem_desc_sw128(st + SG_A_BYTES);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {
          const uint64_t koff = (uint64_t)((k * UMMA_K) >> 4);
          if constexpr (KIND == KIND_I8) umma_i8(tmem_base, a_desc + koff, b_desc + koff, idesc, (kb | k) != 0);
          else umma_f8(tmem_base, a_desc + koff, b_desc + koff, idesc, (kb | k) != 0);
        }
        if (kb + p.stages < p.k_blocks) umma_commit(&empty[s]);
        if (++s == p.stages) { s = 0; ph ^= 1; }
      }
      if (ok) umma_commit(acc_full);
    }
  } else {
    // channel scales of the tile (one per accumulator column)
    for (int i = threadIdx.x - 64; i < 2 * NPART; i += SG_THREADS - 64) {
      const int n = i < NPART ? n0 + i : n1 + i - NPART;
      const float* sb = DUAL && i >= NPART ? p.scale_b1 : p.scale_b0;
      sc_s[i] = !sb ? 1.f : p.scale_b_scalar ? ldg_f_here(sb) : n < p.N ? ldg_f_here(sb + n) : 0.f;
    }
  }
  __syncthreads();                                     // the scales are there
  const bool got = mbar_wait(acc_full, 0, abort_flag, ST_TIMEOUT_EPILOGUE, 0xC20, budget);
  // (the rotary epilogue has a barrier inside, so there all warps go the same way)
  if (EPI == EPI_ROTARY ? __syncthreads_and(got) : __all_sync(0xffffffffu, got)) {
    tc_fence_after();
    const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16);
    float4 sn[4], cs[4];
    if (tile_rot) {
      // (the MMAs are complete, so the ring is free; a row's chunks are XOR-ed with the row, so that neither side conflicts)
      const int ch = threadIdx.x & 7, r = threadIdx.x >> 3;
      if (ch < rot_ch) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<float4*>(sg_smem + (i >> 1) * 8192 + (r + 32 * (i & 1)) * 128 + ((ch ^ (r & 7)) << 4)) = tr[i];
      }
      __syncthreads();
      if (rotated) {
        const int rl = q * 16 + (lane & 15), c0 = p.rot_geo == 2 ? 0 : half * 4;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          sn[i] = *reinterpret_cast<const float4*>(sg_smem + rl * 128 + (((c0 + i) ^ (rl & 7)) << 4));
          cs[i] = *reinterpret_cast<const float4*>(sg_smem + 8192 + rl * 128 + (((c0 + i) ^ (rl & 7)) << 4));
        }
      }
    }
    const float2 sa2 = pk2(sa, sa);
    [[maybe_unused]] const float2 sah2 = pk2(0.5f * sa, 0.5f * sa);      // the gate is dequantised straight to gate / 2 (exact halving)
    [[maybe_unused]] float2 o[EPI == EPI_SILU_MX ? 16 : 1];
    [[maybe_unused]] float amax = 0.f;
#pragma unroll
    for (int u = 0; u < H / 16; ++u) {
      uint32_t va[16], vb[16];
      tmem_ld_32x32b_x16(t_row + ca + 16 * u, va);
      tmem_ld_32x32b_x16(t_row + cb + 16 * u, vb);
      tmem_ld_wait(va, vb);
      const float* s0 = sc_s + ca + 16 * u;
      const float* s1 = sc_s + cb + 16 * u;
      if constexpr (EPI == EPI_SILU_MX) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float2 hv = dequant2<KIND>(va[2 * i], va[2 * i + 1], sah2, make_float2(s0[2 * i], s0[2 * i + 1]));
          const float2 uv = dequant2<KIND>(vb[2 * i], vb[2 * i + 1], sa2, make_float2(s1[2 * i], s1[2 * i + 1]));
          const float2 ov = fmul2(silu_from_half2(hv), uv);
          o[8 * u + i] = ov;
          amax = fmaxf(amax, fmaxf(fabsf(ov.x), fabsf(ov.y)));
        }
      } else {
        uint32_t oa[8], ob[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float2 b0 = make_float2(s0[2 * i], s0[2 * i + 1]), b1 = make_float2(s1[2 * i], s1[2 * i + 1]);
          if constexpr (EPI == EPI_SILU) {
            const float2 hv = dequant2<KIND>(va[2 * i], va[2 * i + 1], sah2, b0);
            const float2 uv = dequant2<KIND>(vb[2 * i], vb[2 * i + 1], sa2, b1);
            oa[i] = pack_half2_from(fmul2(silu_from_half2(hv), uv));
          } else if (EPI == EPI_ROTARY && rotated) {
            const float4 s4 = sn[i >> 1], c4 = cs[i >> 1];
            const float2 s2 = fmul2((i & 1) ? make_float2(s4.z, s4.w) : make_float2(s4.x, s4.y), sa2);   // sA sin
            const float2 c2 = fmul2((i & 1) ? make_float2(c4.z, c4.w) : make_float2(c4.x, c4.y), sa2);   // sA cos
            const float2 y0 = fmul2(pk2(acc_to_float<KIND>(va[2 * i]), acc_to_float<KIND>(va[2 * i + 1])), b0);
            const float2 y1 = fmul2(pk2(acc_to_float<KIND>(vb[2 * i]), acc_to_float<KIND>(vb[2 * i + 1])), b1);
            const float2 qa = fmul2(y1, s2), ta = fmul2(y1, c2);
            oa[i] = pack_half2_from(__ffma2_rn(y0, c2, make_float2(-qa.x, -qa.y)));
            ob[i] = pack_half2_from(__ffma2_rn(y0, s2, ta));
          } else {
            oa[i] = pack_half2_from(dequant2<KIND>(va[2 * i], va[2 * i + 1], sa2, b0));
            ob[i] = pack_half2_from(dequant2<KIND>(vb[2 * i], vb[2 * i + 1], sa2, b1));
          }
        }
        // 16 fp16 at output column n (N is a multiple of 8, the row 16-byte aligned)
        auto store16 = [&](int n, const uint32_t (&w)[8]) {
          if (!row_ok || n >= p.N) return;
          __half* dst = reinterpret_cast<__half*>(p.C) + (long long)row * p.ldc + n;
          const uint4 lo = make_uint4(w[0], w[1], w[2], w[3]), hi = make_uint4(w[4], w[5], w[6], w[7]);
          if (n + 16 <= p.N && (reinterpret_cast<uintptr_t>(dst) & 31) == 0) stg_v8(dst, lo, hi);
          else {
            *reinterpret_cast<uint4*>(dst) = lo;
            if (n + 16 <= p.N) *reinterpret_cast<uint4*>(dst + 8) = hi;
          }
        };
        // (accumulator column -> output column of its part)
        store16((ca < NPART ? n0 + ca : n1 + ca - NPART) + 16 * u, oa);
        if constexpr (!DUAL) store16((cb < NPART ? n0 + cb : n1 + cb - NPART) + 16 * u, ob);
      }
    }
    if constexpr (EPI == EPI_SILU_MX) {
      const int n = n0 + ca;
      int eb = (int)((__float_as_uint(amax) >> 23) & 0xffu) - 8;
      eb = max(0, min(254, eb));
      const float inv = __uint_as_float((uint32_t)(254 - eb) << 23);
      const float2 inv2 = pk2(inv, inv);
      uint32_t w[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t lo = __nv_cvt_float2_to_fp8x2(fmul2(o[2 * k], inv2), __NV_SATFINITE, __NV_E4M3);
        const uint32_t hi = __nv_cvt_float2_to_fp8x2(fmul2(o[2 * k + 1], inv2), __NV_SATFINITE, __NV_E4M3);
        w[k] = lo | (hi << 16);
      }
      if (row_ok && n < p.N) {                         // (N is a multiple of 32, rows of 16-byte aligned)
        uint8_t* dst = reinterpret_cast<uint8_t*>(p.C) + (long long)row * p.ldc + n;
        *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(dst + 16) = make_uint4(w[4], w[5], w[6], w[7]);
        p.out_scale[(long long)row * p.ld_scale + (n >> 5)] = (uint8_t)eb;
      }
    }
  } else if (threadIdx.x == 0) {                       // loads in flight land before the CTA exits
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) { }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 2 * NPART); }
}

static long long small_gemm_tiles(const GemmArgs& a, int tm, int npart) {
  const int cols = a.epi == EPI_SILU || a.epi == EPI_SILU_MX ? npart : 2 * npart;
  return (long long)((a.M + tm - 1) / tm) * ((a.N + cols - 1) / cols);
}

template <int KIND, int EPI, int TM, int NPART>
static int32_t launch_small_inst(const SgParams& p, int grid, int dev, const CUtensorMap& ta, const CUtensorMap& tb0,
                                 const CUtensorMap& tb1, cudaStream_t st) {
  static std::atomic<int> attr_done[64];
  auto k = gemm_small_kernel<KIND, EPI, TM, NPART>;
  if (!attr_done[dev].load(std::memory_order_acquire)) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SgSmem<TM, NPART>::bytes(TM == 128 ? 6 : NPART == 32 ? SG_MAX_STAGES : 8));
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(small gemm)");
    attr_done[dev].store(1, std::memory_order_release);
  }
  return cuda_status(launch_dependent(k, (unsigned)grid, SG_THREADS, (size_t)SgSmem<TM, NPART>::bytes(p.stages), st, ta, tb0, tb1, p), "gemm launch");
}

template <int KIND>
static int32_t launch_small_kind(const GemmArgs& a, int tm, int npart, const SgParams& p, int grid, int dev, const CUtensorMap& ta, const CUtensorMap& tb0,
                                 const CUtensorMap& tb1, cudaStream_t st) {
  switch (a.epi) {
    case EPI_DEQUANT: return tm == 64 ? launch_small_inst<KIND, EPI_DEQUANT, 64, 32>(p, grid, dev, ta, tb0, tb1, st)
                                      : launch_small_inst<KIND, EPI_DEQUANT, 128, 64>(p, grid, dev, ta, tb0, tb1, st);
    case EPI_ROTARY: return launch_small_inst<KIND, EPI_ROTARY, 64, 32>(p, grid, dev, ta, tb0, tb1, st);
    case EPI_SILU: return tm == 128 ? launch_small_inst<KIND, EPI_SILU, 128, 64>(p, grid, dev, ta, tb0, tb1, st)
                        : npart == 32 ? launch_small_inst<KIND, EPI_SILU, 64, 32>(p, grid, dev, ta, tb0, tb1, st)
                                      : launch_small_inst<KIND, EPI_SILU, 64, 64>(p, grid, dev, ta, tb0, tb1, st);
    default:
      if constexpr (KIND == KIND_F8) return launch_small_inst<KIND_F8, EPI_SILU_MX, 64, 64>(p, grid, dev, ta, tb0, tb1, st);
      return GSB200_ERR_BAD_ARG;
  }
}

// Launches the few-tile form if it is the better one; *taken = false and nothing launched otherwise.  `g` is what launch_gemm
// made of the arguments, `geo` the rotary geometry (SgParams).
// It is the better one as long as all its tiles are resident at once, up to three on an SM (their rings then have 4 or 3
// stages); a second wave costs more than the persistent kernel's longer tiles (us, this form / persistent):
//   dequant N = 1536, K = 512: three per SM, M = 1024, 4.5 / 6.6; a second wave, M = 1536, 7.3 / 6.1
//   SwiGLU N = 2048, K = 512: three, M = 768, 5.8 / 6.2; a second wave, M = 1024, 8.4 / 6.4.  The one that emits MXFP8 holds 124
//   registers a thread, two CTAs per SM: M = 512 4.8 / 6.3, M = 768 7.7 / 6.4
//   SwiGLU over a longer K: three 64 x (64 + 64) tiles move 1.5 times the operand bytes of the SM's share of 128 x 256 ones, and from some K
//   on that is what counts.  N = 1024, M = 1700, three per SM: K = 640 6.2 / 6.7, 1024 7.6 / 7.6, 1536 9.5 / 9.1, 2048 11.5 / 10.4, 4096 18.9 /
//   15.7; so three up to K = 1024, and two at any K (M = 1150: K = 1536 7.2 / 8.7, 2048 8.4 / 10.1, 4096 13.4 / 15.2, 8192 23.6 / 31.5)
// The rotary form stops at two per SM, although three would be faster where they fit (N = 1536, K = 512, M = 1024 5.5 / 7.6): it stores without a
// tensor map of the output, and a test of the table of maps counts the one that a launch of a thousand rows encodes.
// Where the 64-row tiles are too many, 128 x 128 ones (dequant; SwiGLU 128 x (64 + 64)) still fit (us, these / persistent kernel):
//   dequant, one per SM: N = 512, K = 512, M = 4096 4.5 / 6.1; K = 2048 7.9 / 9.8; N = 1536, K = 512, M = 1500 4.4 / 6.1 (two per SM:
//   N = 1536, K = 512, M = 2000 5.8 / 6.2, but N = 512, K = 512, M = 6000 6.1 / 6.1 and K = 2048 11.0 / 10.1)
//   SwiGLU, up to two per SM, K <= 512: N = 2048, K = 512, M = 768 5.3 / 6.2 (64-row tiles, three per SM, 5.7), M = 1024 5.3 / 6.3
// Under a cap on the SMs a launch may take, one CTA per SM of the cap: more would spread over more SMs.
static int32_t launch_gemm_small(const GemmArgs& a, const GemmParams& g, int geo, cudaStream_t st, bool* taken) {
  *taken = false;
  const bool dual = a.epi == EPI_SILU || a.epi == EPI_SILU_MX;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return GSB200_OK;
  long long limit = sm_count();
  if (a.sm_cap > 0 && a.sm_cap < limit) limit = a.sm_cap;
  int tm = 64, npart = a.epi == EPI_SILU_MX ? 64 : 32;
  long long tiles = small_gemm_tiles(a, tm, npart);
  if (a.epi == EPI_SILU && tiles > limit) { npart = 64; tiles = small_gemm_tiles(a, tm, npart); }
  const long long tiles128 = small_gemm_tiles(a, 128, 64);
  if ((a.epi == EPI_DEQUANT && tiles > 3 * limit && tiles128 <= limit) ||
      (a.epi == EPI_SILU && tiles > 2 * limit && tiles128 <= 2 * limit && g.k_blocks <= RES_MAX_KBLOCKS)) {
    tm = 128; npart = 64; tiles = tiles128;
  }
  const long long per_sm = (tiles + limit - 1) / limit;
  const int most = limit < sm_count_physical() ? 1 : a.epi == EPI_ROTARY || a.epi == EPI_SILU_MX || (a.epi == EPI_SILU && g.k_blocks > 8) ? 2 : 3;
  if (per_sm > most) return GSB200_OK;
  *taken = true;
  SgParams p{};
  p.M = g.M; p.N = g.N; p.k_blocks = g.k_blocks;
  const int cols = dual ? npart : 2 * npart;
  p.n_tiles = (a.N + cols - 1) / cols;
  p.stages = tm == 128 ? (per_sm == 1 ? 6 : 3) : npart == 32 ? (per_sm == 1 ? SG_MAX_STAGES : per_sm == 2 ? 6 : 4) : (per_sm == 1 ? 8 : per_sm == 2 ? 4 : 3);
  if (p.stages > p.k_blocks) p.stages = p.k_blocks;
  p.C = g.C; p.ldc = g.ldc; p.out_scale = g.out_scale; p.ld_scale = g.ld_scale;
  p.scale_a = g.scale_a; p.scale_a_const = g.scale_a_const; p.scale_b0 = g.scale_b0; p.scale_b1 = g.scale_b1; p.scale_b_scalar = g.scale_b_scalar;
  p.sin_tab = g.sin_tab; p.cos_tab = g.cos_tab; p.seqlen = g.seqlen; p.row_offset = g.row_offset; p.rot_cols = g.rot_cols; p.rot_geo = geo;
  const CUtensorMapDataType u8 = CU_TENSOR_MAP_DATA_TYPE_UINT8;
  CUtensorMap ta, tb0, tb1;
  bool ok = tmap_2d(&ta, u8, 1, a.A, (uint64_t)a.M, (uint64_t)a.K, (uint64_t)a.lda, BK, (uint32_t)tm, CU_TENSOR_MAP_SWIZZLE_128B) &&
            tmap_2d(&tb0, u8, 1, a.B0, (uint64_t)a.N, (uint64_t)a.K, (uint64_t)a.ldb, BK, npart, CU_TENSOR_MAP_SWIZZLE_128B);
  if (!dual) tb1 = tb0;
  else ok = ok && tmap_2d(&tb1, u8, 1, a.B1, (uint64_t)a.N, (uint64_t)a.K, (uint64_t)a.ldb, BK, npart, CU_TENSOR_MAP_SWIZZLE_128B);
  if (!ok) return GSB200_ERR_BAD_ARG;
  return a.kind == KIND_I8 ? launch_small_kind<KIND_I8>(a, tm, npart, p, (int)tiles, dev, ta, tb0, tb1, st)
                           : launch_small_kind<KIND_F8>(a, tm, npart, p, (int)tiles, dev, ta, tb0, tb1, st);
}

}  // namespace gsb
