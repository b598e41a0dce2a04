// The W8 GEMM for many tokens: a persistent kernel of CTA pairs, one CTA per SM.
//
// Same product as w8_gemm.cu (e4m3 weight tile on the UMMA's M side, activation planes on its N side,
// fp32 accumulation in tensor memory), built for launches that the tensor pipe bounds:
//   * a pair (tcgen05 cta_group::2) works on 256 weight rows x up to 256 tokens, or, for the forms that
//     need two values per output (gate / up, rotary partners), on 2 x 256 weight rows x up to 128 tokens.
//     The planes of a K slice accumulate into the SAME columns, so a token costs one column whatever the
//     plane count.  Operand fill per CTA and 128-wide K block: 16 KB of weights + np x 16 KB of planes for
//     np x 512 clocks of tensor work = 48 (np = 2) or 43 (np = 3) bytes per clock, under the ~50-60 that
//     an SM draws from L2; the 128 x 80-token tiles used before needed 70 and were bound by it.
//   * two accumulators of 256 columns take turns: sixteen epilogue warps, 16 tokens at a time, empty one while the next
//     tile's products fill the other.  (Eight warps with 32 tokens each did not keep up where a tile's K is short and its epilogue
//     long: four warps per scheduler instead of two hide the latencies of its chains, results are rounded to bf16 in
//     pairs, and half the registers do.  DiT denoiser at 106 tokens 16.65 -> 16.21 ms, same bits.)  Before, each tile's epilogue ran on a second resident CTA, which halved the
//     ring (two 46 KB stages in flight per CTA).  Now the ring has 4 (np = 2) or 3 stages of 48 / 64 KB.
//   * an epilogue thread holds one channel (its tensor-memory lane) of 16 tokens, so scale, bias and gate
//     are per-thread scalars; results turn into four channels per thread by a 4 x 4 transpose across
//     four lanes (two shuffles per 16 values), without a trip through shared memory.
//   * one CTA per SM that takes all 512 tensor-memory columns: nothing else that allocates tensor memory
//     can be resident beside it (its shared memory leaves no room), so allocation never waits.
// Token tiles differ by 32 tokens at most (two tensor maps), so ragged token counts waste under one step.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "../../include/tybok_b200.h"
#include "host_util.h"
#include "ptx.cuh"
#include "split3.cuh"
#include "w8_gemm.h"

namespace tb {

namespace {

constexpr int P_BK = 128;             // K per stage
constexpr int P_WTILE = 128 * P_BK;   // weight bytes of one 128-row tile and stage
constexpr int P_MAX_STAGES = 8;
constexpr int P_EPI_WARPS = 16;
constexpr int P_CHUNK = 16;           // tokens that an epilogue warp finishes at a time
constexpr int P_THREADS = 32 * (2 + P_EPI_WARPS);
constexpr int P_SMEM = 226 * 1024;
constexpr int P_ACC_COLS = 256;       // tensor-memory columns of one accumulator (two per CTA)

struct PairParams {
  int M, N, K, n_out;
  int np;
  int packed;            // gate / up and rotary forms: 1 = interleaved blocks of 64 rows, 0 = two matrices
  int kb;                // K blocks
  int splits, kb_split;  // split form: pairs of a cluster that share a tile, K blocks of each
  int merge;             // 1: every plane has its own columns and the epilogue adds them (one accumulator, M <= 128)
  int nstages, stage_bytes;
  int ch_tiles, tok_tiles, group;  // tiles; token tiles per L2 group
  int n_big, bt_big, bt_small;     // the first n_big token tiles hold bt_big tokens, the others bt_small
  int pdl;
  float out_scale, plane_scale;
  const float* row_scale;
  const float* s0;
  const float* s1;
  const __nv_bfloat16* bias;
  __nv_bfloat16* y;
  long long ldy;
  uint8_t* y_planes;
  const __nv_bfloat16* res;
  long long ldres;
  const void* gate;
  long long ldgate;
  int rows_per_gate, gate_bf16;
  int* status;
  long long wait_limit;
  RopeEpi rope;
};

struct __align__(8) PairBars {
  uint64_t full[P_MAX_STAGES];   // even CTA: both CTAs' operand bytes of a stage have landed
  uint64_t empty[P_MAX_STAGES];  // each CTA: the pair's products have read the stage
  uint64_t acc_full[2];          // each CTA: accumulator complete
  uint64_t acc_empty[2];         // even CTA: the epilogue warps of both CTAs have read the accumulator
  uint64_t mma_done;             // every product this pair issued has retired
  uint32_t tmem_base;
  volatile int issued;           // stages whose copies this CTA's producer has requested, once it is through; -1 before
  volatile int abort;
};

// Gives up for the whole cluster, whose CTAs wait for one another's operands, products and parts.
__device__ __noinline__ void pair_fail(PairBars* b, int* status, int code) {
  if (status) atomicCAS(status, 0, code);
  uint32_t n;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
  const uint32_t flag = smem_u32(const_cast<int*>(&b->abort));
  for (uint32_t r = 0; r < n; ++r) st_dsmem(dsmem_addr(flag, r), 1u);
}
// One arrival on the barrier at shared::cluster address `addr` (this CTA's or its partner's).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}

struct Tile {
  int ch, m0, bt;
};
__device__ __forceinline__ Tile tile_at(const PairParams& p, int t) {
  const int per_group = p.group * p.ch_tiles;
  const int g = t / per_group, r = t - g * per_group;
  const int gs = min(p.group, p.tok_tiles - g * p.group);
  const int ch = r / gs, tok = g * p.group + (r - ch * gs);
  Tile o;
  o.ch = ch;
  if (tok < p.n_big) {
    o.m0 = tok * p.bt_big;
    o.bt = p.bt_big;
  } else {
    o.m0 = p.n_big * p.bt_big + (tok - p.n_big) * p.bt_small;
    o.bt = p.bt_small;
  }
  return o;
}

// Unwinding after a failed wait, in the even CTA, whose barriers count the copies of both: neither CTA may leave while its own
// copies can still land in its shared memory.  Once both producers have stopped (the abort flag is the whole cluster's), a
// stage that only one of them has requested is completed for the other, and the newest copies of every ring slot are
// waited for.  Every wait is bounded.
__device__ __forceinline__ void see_copies_land(const PairParams& p, PairBars* b, int pair, int npairs, int nkb, int na, uint32_t odd) {
  const uint32_t theirs = dsmem_addr(smem_u32(const_cast<int*>(&b->issued)), odd);
  const long long t0 = clock64();
  int n0, n1;
  do {
    n0 = b->issued;
    asm volatile("ld.relaxed.cluster.shared::cluster.s32 %0, [%1];" : "=r"(n1) : "r"(theirs) : "memory");
  } while ((n0 < 0 || n1 < 0) && clock64() - t0 <= kWaitLimitCycles);
  const int hi = max(n0, n1);
  if (n0 >= 0 && n1 >= 0) {
#pragma unroll 1
    for (int i = min(n0, n1); i < hi; ++i) {
      const Tile tl = tile_at(p, pair + i / nkb * npairs);
      const uint32_t half = na * P_WTILE + p.np * (tl.bt >> 1) * P_BK;  // one CTA's bytes of the stage
      uint64_t* bar = &b->full[i % p.nstages];
      if (n1 > n0) mbar_arrive_expect_tx(bar, half);
      else mbar_complete_tx(bar, half);
    }
  }
#pragma unroll 1
  for (int i = max(0, hi - p.nstages); i < hi; ++i) mbar_wait(&b->full[i % p.nstages], (i / p.nstages) & 1);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&t);
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// 4 x 4 transpose of 16-bit values across the four lanes of a quad.  Lane j holds channel j: a = tokens (0, 1),
// b = tokens (2, 3).  Afterwards lane j holds token j: x = channels (0, 1), y = channels (2, 3).
__device__ __forceinline__ uint2 quad_transpose(uint32_t a, uint32_t b, int lane) {
  const bool b1 = lane & 2, b0 = lane & 1;
  const uint32_t keep = b1 ? b : a;
  const uint32_t recv = __shfl_xor_sync(0xffffffffu, b1 ? a : b, 2);
  const uint32_t lo = b1 ? recv : keep, hi = b1 ? keep : recv;  // channels (j & 1) and (j & 1) + 2
  const uint32_t even = __byte_perm(lo, hi, 0x5410), odd = __byte_perm(lo, hi, 0x7632);
  const uint32_t mine = b0 ? odd : even;
  const uint32_t other = __shfl_xor_sync(0xffffffffu, b0 ? even : odd, 1);
  const uint32_t c02 = b0 ? other : mine, c13 = b0 ? mine : other;
  return make_uint2(__byte_perm(c02, c13, 0x5410), __byte_perm(c02, c13, 0x7632));
}

// EPI: EPI_NONE, EPI_GELU, EPI_RESIDUAL, EPI_GEGLU (both layouts of gate and up, p.packed) or EPI_QKV_ROPE.
// SPLIT: long K and too few tiles for the device: a cluster of 2 * splits CTAs works on ONE tile, each pair on its part of
// K.  Once all of them are through (their rings are idle then), every pair sends the token chunks it does not own
// into the owners' shared memory, and a chunk's owner adds the parts in split order and finishes it.
template <int EPI, bool SPLIT>
__global__ void __launch_bounds__(P_THREADS, 1)
w8_gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_w0, const __grid_constant__ CUtensorMap tm_w1,
                    const __grid_constant__ CUtensorMap tm_big, const __grid_constant__ CUtensorMap tm_small,
                    const PairParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ PairBars bars;
  constexpr int NA = (EPI == EPI_GEGLU || EPI == EPI_QKV_ROPE) ? 2 : 1;  // accumulators (of <= 256 / NA tokens) per tile
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t crank = cluster_ctarank(), rank = crank & 1u, lead = crank & ~1u;  // the even CTA issues the pair's products
  const int split = SPLIT ? static_cast<int>(crank >> 1) : 0;
  const int tiles = p.ch_tiles * p.tok_tiles;
  const int pair = SPLIT ? blockIdx.x / (2 * p.splits) : blockIdx.x >> 1, npairs = SPLIT ? tiles : gridDim.x >> 1;
  const int kb0 = SPLIT ? split * p.kb_split : 0, nkb = SPLIT ? min(p.kb_split, p.kb - kb0) : p.kb;
  const uint16_t both = static_cast<uint16_t>(3u << lead);

  if (tid == 0) {
    for (int i = 0; i < P_MAX_STAGES; ++i) {
      mbar_init(&bars.full[i], 1);
      mbar_init(&bars.empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars.acc_full[i], 1);
      mbar_init(&bars.acc_empty[i], 2 * P_EPI_WARPS);
    }
    mbar_init(&bars.mma_done, 1);
    bars.abort = 0;
    bars.issued = -1;
    fence_barrier_init();
    tma_prefetch_desc(&tm_w0);
    tma_prefetch_desc(&tm_big);
  }
  if (warp == 1) {
    tmem_alloc_pair(&bars.tmem_base, 2 * P_ACC_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncwarp();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem = bars.tmem_base;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      if (p.pdl) pdl_launch_dependents();
      auto load_w = [&](int ch, int kb, uint8_t* st, uint32_t bar) {
        const int k0 = (kb0 + kb) * P_BK;
        if (NA == 1) {
          tma_load_2d_pair(st, &tm_w0, bar, k0, ch * 256 + static_cast<int>(rank) * 128);
        } else if (p.packed) {  // blocks of 64 + 64 rows: the first halves to one tile, the partners to the other
          const int r0 = (ch * 4 + static_cast<int>(rank) * 2) * 128;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            tma_load_2d_pair(st + (i & 1) * P_WTILE + (i >> 1) * (P_WTILE / 2), &tm_w0, bar, k0, r0 + i * 64);
        } else {
          const int r0 = ch * 256 + static_cast<int>(rank) * 128;
          tma_load_2d_pair(st, &tm_w0, bar, k0, r0);
          tma_load_2d_pair(st + P_WTILE, &tm_w1, bar, k0, r0);
        }
      };
      int s = 0, n = 0;  // ring slot, loads issued
      uint32_t par = 1;  // parity of the slot's `empty` barrier to wait for (fresh barriers pass at 1)
      bool ok = true, waited = false;
      for (int t = pair; t < tiles && ok; t += npairs) {
        const Tile tl = tile_at(p, t);
        const CUtensorMap* tx = tl.bt == p.bt_big ? &tm_big : &tm_small;
        const int hrows = tl.bt >> 1;
        const uint32_t bytes = 2u * (NA * P_WTILE + p.np * hrows * P_BK);
        if (!waited) {
          // Weights depend on nothing that runs before this kernel: fill the ring's weight tiles first.
          const int pre = min(p.nstages, nkb);
          for (int i = 0; i < pre; ++i) {
            if (rank == 0) mbar_arrive_expect_tx(&bars.full[i], bytes);
            load_w(tl.ch, i, smem + i * p.stage_bytes, dsmem_addr(smem_u32(&bars.full[i]), lead));
          }
          if (p.pdl) pdl_wait();
        }
        for (int k = 0; k < nkb; ++k) {
          const bool primed = !waited && k < p.nstages;
          uint8_t* st = smem + s * p.stage_bytes;
          const uint32_t bar = dsmem_addr(smem_u32(&bars.full[s]), lead);
          if (!primed) {
            if (!wait_or_abort(&bars.empty[s], par, &bars.abort)) {
              pair_fail(&bars, p.status, TYBOK_DEV_TIMEOUT_PRODUCER);
              ok = false;
              break;
            }
            if (rank == 0) mbar_arrive_expect_tx(&bars.full[s], bytes);
            load_w(tl.ch, k, st, bar);
          }
          for (int pl = 0; pl < p.np; ++pl)
            tma_load_3d_pair(st + NA * P_WTILE + pl * hrows * P_BK, tx, bar, (kb0 + k) * P_BK,
                             tl.m0 + static_cast<int>(rank) * hrows, pl);
          ++n;
          if (++s == p.nstages) {
            s = 0;
            par ^= 1;
          }
        }
        waited = true;
      }
      bars.issued = n;
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (even CTA)
    const bool leader = elect_one();
    bool ok = true;
    if (rank == 0) {
      int s = 0, it = 0;
      uint32_t par = 0;
      for (int t = pair; t < tiles && ok; t += npairs, ++it) {
        const Tile tl = tile_at(p, t);
        const int a = it & 1;
        const uint32_t plane16 = static_cast<uint32_t>(tl.bt * (P_BK / 2)) >> 4;
        const uint32_t idesc = p.np == 2 ? idesc_e4m3_e4m3_f32(256, tl.bt) : idesc_e4m3_e5m2_f32(256, tl.bt);
        ok = __all_sync(0xffffffffu, wait_or_abort(&bars.acc_empty[a], ((it >> 1) & 1) ^ 1, &bars.abort));
        tc_fence_after();
        for (int k = 0; k < nkb && ok; ++k) {
          ok = __all_sync(0xffffffffu, wait_or_abort(&bars.full[s], par, &bars.abort));
          if (!ok) break;
          tc_fence_after();
          const uint64_t wd = smem_desc_sw128(smem_u32(smem + s * p.stage_bytes)), xd = wd + NA * (P_WTILE >> 4);
          for (int pl = 0; pl < p.np; ++pl) {
#pragma unroll
            for (int w = 0; w < NA; ++w) {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const uint64_t ad = wd + w * (P_WTILE >> 4) + j * 2;
                const uint64_t bd = xd + pl * plane16 + j * 2;
                if (leader) umma_ss_f8_pair(tmem + a * P_ACC_COLS + (p.merge ? pl : w) * tl.bt, ad, bd, idesc,
                                            (k | (p.merge ? 0 : pl) | j) ? 1u : 0u);
              }
            }
          }
          if (leader) tc_commit_pair(&bars.empty[s], both);
          __syncwarp();
          if (++s == p.nstages) {
            s = 0;
            par ^= 1;
          }
        }
        if (ok && leader) tc_commit_pair(&bars.acc_full[a], both);
        __syncwarp();
      }
      // Both CTAs free their tensor memory at the end: first every product issued has to retire.  (The commit comes while the
      // warp is still together: behind the branch below it reached one of the two CTAs only.)
      if (leader) tc_commit_pair(&bars.mma_done, both);
      __syncwarp();
      if (!ok && lane == 0) {
        pair_fail(&bars, p.status, TYBOK_DEV_TIMEOUT_MMA);
        see_copies_land(p, &bars, pair, npairs, nkb, NA, lead + 1);
      }
      __syncwarp();
    }
    // The odd CTA's wait spans the whole launch: it only gives up once something else has failed.
    bool done = false;
    for (int tries = 0; tries < 16 && !done; ++tries) {
      done = mbar_wait(&bars.mma_done, 0);
      if (bars.abort) break;
    }
    if (!done) done = mbar_wait(&bars.mma_done, 0);
    if (!done && lane == 0) pair_fail(&bars, p.status, TYBOK_DEV_TIMEOUT_MMA);
  } else {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3, part = (warp - 2) >> 2;  // tensor-memory lane quadrant; which of its four warps
    const int row = q * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    const int g4 = (lane >> 2) * 4, j4 = lane & 3;   // after the transpose: first channel of four, token of four
    const long long plane = static_cast<long long>(p.M) * p.n_out;
    const uint32_t acc_empty0 = dsmem_addr(smem_u32(&bars.acc_empty[0]), lead);
    if (p.pdl) pdl_wait();
    bool ok = true;
    int it = 0;
    for (int t = pair; t < tiles; t += npairs, ++it) {
      const Tile tl = tile_at(p, t);
      const int a = it & 1;
      // ---- per-channel constants of this lane
      int rows[2];  // weight row(s) of this lane
      int n_first;  // output channel (head dimension for the rotary form) of this lane's quad after the transpose
      bool live;
      int blk = 0, col = 0;
      if (NA == 1) {
        rows[0] = rows[1] = tl.ch * 256 + static_cast<int>(rank) * 128 + row;
        live = rows[0] < p.N;
        n_first = tl.ch * 256 + static_cast<int>(rank) * 128 + q * 32 + g4;
      } else if (p.packed) {
        blk = tl.ch * 4 + static_cast<int>(rank) * 2 + (row >> 6);
        col = row & 63;
        rows[0] = blk * 128 + col;
        rows[1] = rows[0] + 64;
        live = blk * 128 < p.N;
        n_first = blk * 64 + ((q & 1) * 32) + g4;
      } else {
        rows[0] = rows[1] = tl.ch * 256 + static_cast<int>(rank) * 128 + row;
        live = rows[0] < p.N;
        n_first = tl.ch * 256 + static_cast<int>(rank) * 128 + q * 32 + g4;
      }
      float sc0 = 0.f, sc1 = 0.f, bi = 0.f, gt = 1.f;
      int gate_group = -1;
      if (live) {
        sc0 = p.s0[rows[0]] * p.out_scale;
        if (NA == 2) sc1 = (p.packed ? p.s0 : p.s1)[rows[1]] * p.out_scale;
        if (NA == 1 && p.bias) bi = __bfloat162float(p.bias[rows[0]]);
        if (EPI == EPI_RESIDUAL && p.gate) {
          gate_group = tl.m0 / p.rows_per_gate;
          const long long gi = static_cast<long long>(gate_group) * p.ldgate + rows[0];
          gt = p.gate_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.gate)[gi])
                           : bf16_round(static_cast<const float*>(p.gate)[gi]);
        }
      }
      const bool one_group = gate_group < 0 || (min(tl.m0 + tl.bt, p.M) - 1) / p.rows_per_gate == gate_group;
      const bool quad_live = NA == 1 || !p.packed ? n_first < p.N : live;

      if (ok && !__all_sync(0xffffffffu, wait_or_abort(&bars.acc_full[a], (it >> 1) & 1, &bars.abort, p.wait_limit))) {
        ok = false;
        if (lane == 0) pair_fail(&bars, p.status, TYBOK_DEV_TIMEOUT_EPILOGUE);
      }
      if (!ok && !SPLIT) break;
      tc_fence_after();
      const int nchunk = (tl.bt + P_CHUNK - 1) / P_CHUNK, m_end = min(p.M, tl.m0 + tl.bt);
      // Accumulator values of chunk c (16 tokens from mc on; v, and u of the second accumulator) -> outputs.  The
      // residual rows are requested first.
      auto residual_rows = [&](int mc, uint2 (&rr)[EPI == EPI_RESIDUAL ? 4 : 1]) {
        if (EPI == EPI_RESIDUAL) {  // 4 token rows per lane after the transpose: m = mc + 4 k + j4
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int m = mc + 4 * k + j4;
            if (m < m_end && quad_live) rr[EPI == EPI_RESIDUAL ? k : 0] = *reinterpret_cast<const uint2*>(p.res + m * p.ldres + n_first);
          }
        }
      };
      auto finish = [&](int mc, uint32_t (&v)[16], uint32_t (&u)[NA == 2 ? 16 : 1], uint2 (&rr)[EPI == EPI_RESIDUAL ? 4 : 1]) {
        float rs = 1.0f;
        if (p.row_scale) rs = p.row_scale[min(mc + (lane & 15), p.M - 1)];
        uint32_t pk[8], pw[EPI == EPI_QKV_ROPE ? 8 : 1];  // bf16 results of two tokens each (and of the rotary partners)
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          float o[2], w[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int i = 2 * k + e;
            float x = __uint_as_float(v[i]);
            float r = 1.0f;
            if (p.row_scale) {
              r = __shfl_sync(0xffffffffu, rs, i);
              x *= r;
            }
            o[e] = x * sc0;
            if constexpr (NA == 2) w[e] = __uint_as_float(u[i]) * r * sc1;
            if (NA == 1) o[e] += bi;
          }
          // Rounding points of the reference's bf16 modules: linear output, GELU output, product, gated value, sum.
          if (EPI == EPI_GELU || EPI == EPI_GEGLU || (EPI == EPI_RESIDUAL && p.gate)) {
            const uint32_t lin = pack_bf16(o[0], o[1]);
            o[0] = bf16_lo(lin);
            o[1] = bf16_hi(lin);
          }
          if (EPI == EPI_GELU) {
            o[0] = gelu_tanh_fast(o[0]);
            o[1] = gelu_tanh_fast(o[1]);
          } else if (EPI == EPI_RESIDUAL && p.gate) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              float gv = gt;
              if (!one_group) {
                const int m = min(mc + 2 * k + e, p.M - 1);
                const long long gi = static_cast<long long>(m / p.rows_per_gate) * p.ldgate + rows[0];
                gv = !live ? 0.f : p.gate_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.gate)[gi])
                                               : bf16_round(static_cast<const float*>(p.gate)[gi]);
              }
              o[e] *= gv;
            }
          } else if (EPI == EPI_GEGLU) {
            const uint32_t g = pack_bf16(gelu_tanh_fast(o[0]), gelu_tanh_fast(o[1])), uw = pack_bf16(w[0], w[1]);
            o[0] = bf16_lo(g) * bf16_lo(uw);
            o[1] = bf16_hi(g) * bf16_hi(uw);
          }
          pk[k] = pack_bf16(o[0], o[1]);
          if constexpr (EPI == EPI_QKV_ROPE) pw[k] = pack_bf16(w[0], w[1]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          uint2 t0 = quad_transpose(pk[2 * k], pk[2 * k + 1], lane);
          const int m = mc + 4 * k + j4;
          if constexpr (EPI == EPI_QKV_ROPE) {
            const uint2 t1 = quad_transpose(pw[2 * k], pw[2 * k + 1], lane);
            if (m < m_end && quad_live) {
              const RopeEpi& rp = p.rope;
              const int tps = rp.D >> 7, slot = blk / tps, hd2 = rp.D >> 1;
              const int d = (blk - slot * tps) * 64 + (q & 1) * 32 + g4;
              uint2 lo = t0, hi = t1;
              if (slot < rp.H + rp.G) {
                const long long tbl = static_cast<long long>(rp.pos[m]) * rp.D + d;
                const uint2 c0 = *reinterpret_cast<const uint2*>(rp.cos + tbl), c1 = *reinterpret_cast<const uint2*>(rp.cos + tbl + hd2);
                const uint2 n0 = *reinterpret_cast<const uint2*>(rp.sin + tbl), n1 = *reinterpret_cast<const uint2*>(rp.sin + tbl + hd2);
                const float l[4] = {bf16_lo(t0.x), bf16_hi(t0.x), bf16_lo(t0.y), bf16_hi(t0.y)};
                const float h[4] = {bf16_lo(t1.x), bf16_hi(t1.x), bf16_lo(t1.y), bf16_hi(t1.y)};
                const float fc0[4] = {bf16_lo(c0.x), bf16_hi(c0.x), bf16_lo(c0.y), bf16_hi(c0.y)};
                const float fc1[4] = {bf16_lo(c1.x), bf16_hi(c1.x), bf16_lo(c1.y), bf16_hi(c1.y)};
                const float fn0[4] = {bf16_lo(n0.x), bf16_hi(n0.x), bf16_lo(n0.y), bf16_hi(n0.y)};
                const float fn1[4] = {bf16_lo(n1.x), bf16_hi(n1.x), bf16_lo(n1.y), bf16_hi(n1.y)};
                float ol[4], oh[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {  // rotate_half(x) = (-x2, x1)
                  ol[e] = rope1(l[e], -h[e], fc0[e], fn0[e]);
                  oh[e] = rope1(h[e], l[e], fc1[e], fn1[e]);
                }
                lo = make_uint2(pack_bf16(ol[0], ol[1]), pack_bf16(ol[2], ol[3]));
                hi = make_uint2(pack_bf16(oh[0], oh[1]), pack_bf16(oh[2], oh[3]));
              }
              __nv_bfloat16* dst;
              if (slot < rp.H) {
                dst = rp.q + (static_cast<long long>(m) * rp.H + slot) * rp.D;
              } else {
                const int g = (slot - rp.H) % rp.G;
                const int b = m / rp.L, tk = m - b * rp.L;
                dst = (slot < rp.H + rp.G ? rp.kcache : rp.vcache) +
                      ((static_cast<long long>(b) * rp.G + g) * rp.Lcap + rp.key_off + tk) * rp.D;
              }
              *reinterpret_cast<uint2*>(dst + d) = lo;
              *reinterpret_cast<uint2*>(dst + hd2 + d) = hi;
            }
          } else {
            if (m < m_end && quad_live) {
              if (EPI == EPI_RESIDUAL) {
                const uint2 r2 = rr[EPI == EPI_RESIDUAL ? k : 0];
                t0 = make_uint2(pack_bf16(bf16_lo(t0.x) + bf16_lo(r2.x), bf16_hi(t0.x) + bf16_hi(r2.x)),
                                pack_bf16(bf16_lo(t0.y) + bf16_lo(r2.y), bf16_hi(t0.y) + bf16_hi(r2.y)));
              }
              if (p.y) *reinterpret_cast<uint2*>(p.y + m * p.ldy + n_first) = t0;
              if (p.y_planes) {
                const float xs[4] = {bf16_lo(t0.x) * p.plane_scale, bf16_hi(t0.x) * p.plane_scale,
                                     bf16_lo(t0.y) * p.plane_scale, bf16_hi(t0.y) * p.plane_scale};
                uint32_t w1, w2, w3;
                split3_quad(xs, w1, w2, w3);
                uint8_t* dst = p.y_planes + static_cast<long long>(m) * p.n_out + n_first;
                *reinterpret_cast<uint32_t*>(dst) = w1;
                *reinterpret_cast<uint32_t*>(dst + plane) = w2;
                *reinterpret_cast<uint32_t*>(dst + 2 * plane) = w3;
              }
            }
          }
        }
      };
      if constexpr (SPLIT) {
        cluster_sync_all();  // every pair of the cluster has its part (all rings are idle), or has given up
        const bool whole = !bars.abort;  // the same in every CTA: nobody gives up after this point
        const int nown = (nchunk + p.splits - 1) / p.splits;
        const uint32_t buf = smem_u32(smem);
        for (int c = part; c < nchunk && whole; c += 4) {
          const int owner = c % p.splits;
          if (owner == split || tl.m0 + c * P_CHUNK >= m_end) continue;
          uint32_t v[16];
          tmem_ld16(tmem + lane_addr + c * P_CHUNK, v);
          const uint32_t dst = dsmem_addr(buf + (((split * nown + c / p.splits) * P_CHUNK) * 128 + row) * 4, owner * 2 + rank);
          tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e)
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + e * 512), "f"(__uint_as_float(v[e])));
        }
        __syncwarp();
        cluster_sync_all();  // every part has arrived
        const float* parts = reinterpret_cast<const float*>(smem);
        for (int i = part; i < nown && whole; i += 4) {
          const int c = i * p.splits + split, mc = tl.m0 + c * P_CHUNK;
          if (c >= nchunk || mc >= m_end) break;
          uint32_t v[16], t[16], u[NA == 2 ? 16 : 1];
          uint2 rr[EPI == EPI_RESIDUAL ? 4 : 1];
          residual_rows(mc, rr);
          tmem_ld16(tmem + lane_addr + c * P_CHUNK, t);
          tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) v[e] = 0u;
          for (int sp = 0; sp < p.splits; ++sp) {  // split order: bit-reproducible
            const float* src = parts + ((sp * nown + i) * P_CHUNK) * 128 + row;
#pragma unroll
            for (int e = 0; e < 16; ++e)
              v[e] = __float_as_uint(__uint_as_float(v[e]) + (sp == split ? __uint_as_float(t[e]) : src[e * 128]));
          }
          finish(mc, v, u, rr);
        }
      } else {
        for (int c = part; c < nchunk; c += 4) {
          const int mc = tl.m0 + c * P_CHUNK;  // first token of this chunk
          if (mc >= m_end) break;
          uint32_t v[16];
          uint32_t u[NA == 2 ? 16 : 1];
          tmem_ld16(tmem + a * P_ACC_COLS + lane_addr + c * P_CHUNK, v);
          if constexpr (NA == 2) tmem_ld16(tmem + a * P_ACC_COLS + lane_addr + tl.bt + c * P_CHUNK, u);
          uint2 rr[EPI == EPI_RESIDUAL ? 4 : 1];
          residual_rows(mc, rr);
          tc_wait_ld();
          if (NA == 1 && p.merge) {
            for (int pl = 1; pl < p.np; ++pl) {
              uint32_t v2[16];
              tmem_ld16(tmem + a * P_ACC_COLS + lane_addr + pl * tl.bt + c * P_CHUNK, v2);
              tc_wait_ld();
#pragma unroll
              for (int e = 0; e < 16; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) + __uint_as_float(v2[e]));
            }
          }
          finish(mc, v, u, rr);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc_empty0 + a * 8);
    }
  }

  if (SPLIT && warp < 2) {  // the two meeting points of the epilogue warps' exchange
    __syncwarp();
    cluster_sync_all();
    cluster_sync_all();
  }
  // The pair leaves together: both have read their accumulators, every remote arrival has been made.
  tc_fence_before();
  __syncwarp();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, 2 * P_ACC_COLS);
  }
}

struct PairPlan {
  int ch_tiles, tok_tiles, n_big, bt_big, bt_small, nstages, stage_bytes, group, kb, merge, splits, kb_split;
  double cost;  // SM clocks
};

// Token tiles are whole steps of 32 tokens, at most 256 / na, and differ by one step.  Cost of a tile and K block:
// tensor time against operand fill at 52 bytes per clock and SM (measured for this kernel's access pattern).
PairPlan plan_pair(int M, int rows, int K, int na, int np) {
  PairPlan best{};
  best.cost = -1.0;
  // Up to 128 tokens the planes keep their own columns, as in the one-tile kernel: the sum over K and planes then has
  // the same order in both, so such a call's result does not depend on which of them the tile count selects.
  best.merge = (na == 1 && M <= 128) ? 1 : 0;
  const int pairs = std::max(1, host::sm_count() / 2);
  const int ch = (rows + 256 * na - 1) / (256 * na);
  const int units = (M + 31) / 32;
  // Those columns are a token tile's planes times its tokens: one accumulator takes 256 of them, and the whole of tensor
  // memory (384 for three planes of 128 tokens) where no pair has a second tile.  One token tile reads the weights once
  // (106 x 14336 x 3072: two tiles of 64 tokens 25.2 us, one of 128 20.7 us).
  const int umax = best.merge ? (ch <= pairs ? 16 / np : 8 / np) : 8 / na;
  const int kb = (K + P_BK - 1) / P_BK;
  auto tile_cost = [&](int u) {
    const double mma = 64.0 * u * na * np, fill = (na * 16384.0 + np * 2048.0 * u) / 52.0;
    return std::max(kb * std::max(mma, fill), 700.0 + 32.0 * u * 24.0 * na);
  };
  for (int tt = (units + umax - 1) / umax; tt <= units; ++tt) {
    const int ub = (units + tt - 1) / tt, us = units % tt == 0 ? ub : ub - 1;
    const int nb = units % tt == 0 ? tt : units % tt;
    const long long tiles = static_cast<long long>(ch) * tt;
    const double avg = (nb * tile_cost(ub) + (tt - nb) * tile_cost(us)) / tt;
    const double cost = static_cast<double>(tiles / pairs) * avg + (tiles % pairs ? tile_cost(ub) : 0.0);
    if (best.cost < 0 || cost < best.cost) {
      best.cost = cost;
      best.ch_tiles = ch; best.tok_tiles = tt; best.n_big = nb; best.bt_big = 32 * ub; best.bt_small = 32 * us; best.kb = kb;
    }
  }
  best.splits = 1;
  best.kb_split = best.kb;
  best.stage_bytes = na * P_WTILE + np * (best.bt_big / 2) * P_BK;
  best.nstages = std::min(P_MAX_STAGES, (P_SMEM - 1024) / best.stage_bytes);
  // L2 groups: as many token tiles as keep the group's planes within a quarter of L2
  const double tile_bytes = static_cast<double>(best.bt_big) * K * np;
  best.group = std::max(1, std::min(best.tok_tiles, static_cast<int>(32.0e6 / tile_bytes)));
  return best;
}

// Clusters of 2 * splits CTAs that the device holds at once.
int resident_clusters(int splits) {
  static host::DeviceCache cache[5];
  return host::per_device(cache[splits], [splits] {
    auto* k = w8_gemm_pair_kernel<EPI_RESIDUAL, true>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, P_SMEM);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * splits);
    cfg.blockDim = dim3(P_THREADS);
    cfg.dynamicSmemBytes = P_SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = host::sm_count() / (2 * splits + 2);
    }
    return n;
  });
}

// Split form: one wave of clusters.  The exchange moves (splits - 1) / splits of a 128-channel fp32 tile through
// distributed shared memory (about 18 bytes per clock and SM) between two cluster meetings.
PairPlan plan_split(int M, int rows, int K, int np) {
  PairPlan best{};
  best.cost = -1.0;
  const int units = (M + 31) / 32, ch = (rows + 255) / 256, kb = (K + P_BK - 1) / P_BK;
  for (int sp = 2; sp <= 4; ++sp) {
    const int cap = resident_clusters(sp), kbs = (kb + sp - 1) / sp;
    if ((sp - 1) * kbs >= kb) continue;  // no empty split
    for (int tt = (units + 7) / 8; tt <= units && static_cast<long long>(ch) * tt <= cap; ++tt) {
      const int ub = (units + tt - 1) / tt;
      const int stage = P_WTILE + np * 16 * ub * P_BK, ns = std::min(P_MAX_STAGES, (P_SMEM - 1024) / stage);
      if (sp * ((2 * ub + sp - 1) / sp) * P_CHUNK * 512 > ns * stage) continue;  // the parts land in the idle ring
      const double mma = 64.0 * ub * np, fill = (16384.0 + np * 2048.0 * ub) / 36.0;  // one tile per pair: latency shows
      const double cost = kbs * std::max(mma, fill) + 32.0 * ub * 512.0 * (sp - 1) / sp / 18.0 + 4000.0;
      if (best.cost < 0 || cost < best.cost) {
        best.cost = cost;
        best.ch_tiles = ch; best.tok_tiles = tt; best.kb = kb; best.splits = sp; best.kb_split = kbs;
        best.n_big = units % tt == 0 ? tt : units % tt;
        best.bt_big = 32 * ub;
        best.bt_small = units % tt == 0 ? 32 * ub : 32 * (ub - 1);
        best.stage_bytes = stage;
        best.nstages = ns;
        best.group = tt;
      }
    }
  }
  return best;
}

}  // namespace

double gemm_pair_split_cost(int M, int N, int K, int np) { return plan_split(M, N, K, np).cost; }

// The pair form takes what the one-tile-per-CTA form (w8_gemm.cu) would run in more than one wave: more than one
// 128-row x 80-token (three planes) or 128-token (two planes) tile per SM.  Within one wave that form is ahead, since
// its CTAs set up beside the previous kernel's last ones (800 x 2048 x 2048: three planes, 160 tiles, 28.1 -> 18.8 us;
// two planes, 112 tiles, 15.5 against 17.3 us; one token x 32768 x 2048: 256 tiles, 19.3 -> 16.7 us).
bool gemm_pair_suits(int M, int N, int nw, int np) {
  const int cap = np == 2 ? 128 : 80;
  const long long tiles = static_cast<long long>((M + cap - 1) / cap) * ((static_cast<long long>(nw) * N + 127) / 128);
  return tiles > host::sm_count();
}

int launch_gemm_pair(const GemmCall& c) {
  const int na = (c.epi == EPI_QKV_ROPE || c.epi == EPI_GEGLU || c.epi == EPI_GEGLU_PACKED) ? 2 : 1;
  const bool packed = c.epi == EPI_GEGLU_PACKED || c.epi == EPI_QKV_ROPE;
  const PairPlan pl = c.split ? plan_split(c.M, c.N, c.K, c.np) : plan_pair(c.M, c.w1 ? 2 * c.N : c.N, c.K, na, c.np);

  CUtensorMap tm_w0, tm_w1, tm_big, tm_small;
  if (int rc = host::tensor_map_2d(&tm_w0, c.w0, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, c.K, c.N, c.K, P_BK, packed ? 64 : 128)) return rc;
  tm_w1 = tm_w0;
  if (c.w1)
    if (int rc = host::tensor_map_2d(&tm_w1, c.w1, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, c.K, c.N, c.K, P_BK, 128)) return rc;
  const uint64_t pitch2 = static_cast<uint64_t>(c.M) * c.K;
  if (int rc = host::tensor_map_3d(&tm_big, c.planes, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, c.K, c.M, c.np, c.K, pitch2, P_BK, pl.bt_big / 2, 1)) return rc;
  tm_small = tm_big;
  if (pl.bt_small != pl.bt_big)
    if (int rc = host::tensor_map_3d(&tm_small, c.planes, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, c.K, c.M, c.np, c.K, pitch2, P_BK, pl.bt_small / 2, 1)) return rc;

  PairParams p{};
  p.M = c.M; p.N = c.N; p.K = c.K; p.n_out = c.n_out; p.np = c.np; p.packed = packed ? 1 : 0;
  p.kb = pl.kb; p.splits = pl.splits; p.kb_split = pl.kb_split; p.merge = pl.merge; p.nstages = pl.nstages; p.stage_bytes = pl.stage_bytes;
  p.ch_tiles = pl.ch_tiles; p.tok_tiles = pl.tok_tiles; p.group = pl.group;
  p.n_big = pl.n_big; p.bt_big = pl.bt_big; p.bt_small = pl.bt_small;
  p.pdl = host::pdl_enabled() ? 1 : 0;
  p.out_scale = c.out_scale; p.plane_scale = c.plane_scale; p.row_scale = c.row_scale;
  p.s0 = c.s0; p.s1 = c.s1; p.bias = c.bias; p.y = c.y; p.ldy = c.ldy; p.y_planes = c.y_planes;
  p.res = c.res; p.ldres = c.ldres; p.gate = c.gate; p.ldgate = c.ldgate;
  p.rows_per_gate = c.rows_per_gate > 0 ? c.rows_per_gate : 1; p.gate_bf16 = c.gate_bf16;
  p.status = c.status;
  p.wait_limit = host::epilogue_wait_limit() > 0 ? host::epilogue_wait_limit() : kWaitLimitCycles;
  if (c.rope) p.rope = *c.rope;

  static host::DeviceCache attr_set;
  if (!host::per_device(attr_set, [] {
        for (auto* k : {w8_gemm_pair_kernel<EPI_NONE, false>, w8_gemm_pair_kernel<EPI_GELU, false>, w8_gemm_pair_kernel<EPI_RESIDUAL, false>,
                        w8_gemm_pair_kernel<EPI_GEGLU, false>, w8_gemm_pair_kernel<EPI_QKV_ROPE, false>, w8_gemm_pair_kernel<EPI_NONE, true>,
                        w8_gemm_pair_kernel<EPI_GELU, true>, w8_gemm_pair_kernel<EPI_RESIDUAL, true>})
          if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, P_SMEM) != cudaSuccess) return 0;
        return 1;
      }))
    return host::fail_cuda("cudaFuncSetAttribute(w8_gemm_pair_kernel)");
  cudaLaunchConfig_t cfg{};
  const int tiles = pl.ch_tiles * pl.tok_tiles;
  const int pairs = c.split ? tiles * pl.splits : std::min(tiles, std::max(1, host::sm_count() / 2));
  cfg.gridDim = dim3(2 * pairs);
  cfg.blockDim = dim3(P_THREADS);
  cfg.dynamicSmemBytes = P_SMEM;  // always the whole SM: no other user of tensor memory beside this CTA
  cfg.stream = c.stream;
  cudaLaunchAttribute attr[2];
  int n_attr = 0;
  if (p.pdl) {
    attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
    ++n_attr;
  }
  attr[n_attr].id = cudaLaunchAttributeClusterDimension;
  attr[n_attr].val.clusterDim.x = 2 * pl.splits;
  attr[n_attr].val.clusterDim.y = 1;
  attr[n_attr].val.clusterDim.z = 1;
  ++n_attr;
  cfg.attrs = attr;
  cfg.numAttrs = n_attr;
  auto* k = c.split ? w8_gemm_pair_kernel<EPI_NONE, true> : w8_gemm_pair_kernel<EPI_NONE, false>;
  switch (c.epi) {
    case EPI_GELU: k = c.split ? w8_gemm_pair_kernel<EPI_GELU, true> : w8_gemm_pair_kernel<EPI_GELU, false>; break;
    case EPI_RESIDUAL: k = c.split ? w8_gemm_pair_kernel<EPI_RESIDUAL, true> : w8_gemm_pair_kernel<EPI_RESIDUAL, false>; break;
    case EPI_GEGLU:
    case EPI_GEGLU_PACKED: k = w8_gemm_pair_kernel<EPI_GEGLU, false>; break;
    case EPI_QKV_ROPE: k = w8_gemm_pair_kernel<EPI_QKV_ROPE, false>; break;
    default: break;
  }
  if (cudaLaunchKernelEx(&cfg, k, tm_w0, tm_w1, tm_big, tm_small, p) != cudaSuccess) return host::fail_cuda("launch w8_gemm_pair_kernel");
  host::count_launch();
  return TYBOK_OK;
}

}  // namespace tb
