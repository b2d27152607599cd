// Subset-sum hash H = A * B (pcs/src/subset_sum.rs:43-67, called at pcs/src/ligesis.rs:302) on
// the 5th-generation tensor cores, fused with the Merkle leaf hashes of H's columns
// (pcs/src/ligesis.rs:306-313).
//
// Exactness: A's canonical 64-bit entries are split into byte limbs, Alimb[8r + l][k] = byte l of
// A[r][k], and B[64 i + b][j] = bit b of the RS codeword word F'[i][j].  S_l = Alimb_l * B is an
// exact int32 sum (terms <= 255, at most 64 * 2^13 of them), and H[r][j] = sum_l 2^(8l) S_l mod p
// is recombined exactly in 128-bit arithmetic.  K is stored permuted inside each aligned group of
// 32 (the same permutation in A's limb columns and B's rows, so the products are unchanged): it
// lets the producers spread a word's bits into bytes with a shift and a mask per 4 bytes.
//
// Persistent CTA pairs (clusters of two, one CTA per SM) walk the 256-column tiles with
// tcgen05.mma.cta_group::2: M = 256 codeword columns, 128 per CTA, by N = 256 limb rows, K in stages
// of two chunks of 128 bytes (two codeword rows each).  Each CTA stages the bits of its own 128
// columns and half of the limb rows (32 KB each, three stages), and its TMEM holds its columns'
// accumulators: 128 lanes by 256 limb sums, twice, so a tile's epilogue runs under the next tile's
// MMAs.
//   warp 0      TMA producer: 128 x 128 bytes of A's limbs per chunk, SWIZZLE_128B, no multicast
//   warp 1      TMEM allocation; in the leader (rank 0) one thread issues the pair's MMAs (M256 N256
//               K32).  The tensor pipe queues little ahead, so what this thread waits for is lost:
//               it waits on one barrier per stage and looks at it before it sleeps
//   warps 2-5   bit producers: expand 4 x 128 codeword words into 128 x 128-byte K-major
//               SWIZZLE_128B bit tiles
//   warps 6-13  epilogue, two sets of four warps taking alternate tiles: a thread owns a column,
//               reads its 256 limb sums with tcgen05.ld, recombines mod p, writes H (coalesced) and
//               hashes the 256-byte column leaf with BLAKE3 from registers.
//   warp 14     word loader: bulk copies of the codeword words into a ring of four stages.  The
//               producers must not have loads of their own in flight: their fence to the async
//               proxy waits for those too, a DRAM latency per stage
//   warp 15     passes the arrival of this CTA's limbs on to the leader's stage barrier
// What bounds it: the tensor pipe, and what the issuing thread adds to it.  The MMAs of a stage take
// 1032-1067 clocks at the pipe's peak and a stage passes in about 1200 (counted over 2^7 x 2^17
// with the codeword random, at the 1.77 GHz that the chip then holds); with all loads and bit
// stores left out it is 1090, so the rest is the wait, the fence, the descriptors and the
// commit between two stages.  A CTA alone on a tile (M = 128 limb rows twice, N = 256 columns)
// moved 154 bytes per clock through a shared memory that gives 128 and ran at 0.64 of peak; the
// pair reads each operand byte once per SM, 123 bytes per clock.  2^7 x 2^17: 0.41 -> 0.316 ms,
// 2^7 x 2^19: 1.53 -> 1.21, 2^12 x 2^12: 0.42 -> 0.31, 2^10 x 2^10: 0.103 -> 0.048 (the last two
// with K split, whose combine read its slices with too few threads as well).
// Every mbarrier wait is bounded by a clock budget and watches a CTA-wide failure flag; on a
// timeout the CTA records an error code, every role stops issuing work, the MMA thread waits
// (bounded) for the MMAs it issued, the TMA thread waits (bounded) for the A-limb copies it
// issued (each stage's copy completes on its own barrier, so this wait does not depend on the
// other roles); then the two CTAs meet, and the TMEM is freed before they exit.  The budget of
// the role waits is a kernel argument (lgs_set_wait_budget shortens it to test this path); the
// two drain waits always keep the long default.
#include <cuda.h>
#include <cudaTypedefs.h>

#include "blake3.cuh"
#include "kernels.cuh"
#include "tcgen05.cuh"

namespace lgs {

namespace {
constexpr int TC_N = 256;      // columns of a tile (two CTAs)
constexpr int TC_COLS = 128;   // columns of a CTA
constexpr int H_ROWS = 32;     // digest rows (C)
constexpr int TC_KB = 128;
constexpr int TC_STAGES = 3;
constexpr int TC_SUB = 2;  // K chunks of a stage
constexpr int BIT_TILE = TC_COLS * TC_KB;
constexpr int LIMB_TILE = 128 * TC_KB;  // half of the 256 limb rows
constexpr int STAGE_BYTES = TC_SUB * (BIT_TILE + LIMB_TILE);  // bit tiles, then limb tiles
constexpr int NPROD = 128;
constexpr int NEPI = 256;  // epilogue threads: two sets of four warps, one per TMEM lane quarter
constexpr int NTHREADS = 64 + NPROD + NEPI + 64;
constexpr int TMEM_COLS = 512;
constexpr int W_STAGES = 4;  // ring of codeword words: two rows per chunk
constexpr int W_ROW = TC_COLS * 8, W_BYTES = 2 * TC_SUB * W_ROW;
// full, empty, tma; word full, word empty; acc_full[2], acc_empty[2], drain
constexpr int NBARS = 3 * TC_STAGES + 2 * W_STAGES + 5;
constexpr int SMEM_BYTES =
    TC_STAGES * STAGE_BYTES + W_STAGES * W_BYTES + 1024 /*align*/ + 512 /*barriers*/;
static_assert(NBARS * 8 + 4 <= 512, "barrier space");
static_assert(TC_SUB == 2, "the MMA loop issues a stage's two chunks");
constexpr long long WAIT_CYCLES = tc::DRAIN_CYCLES;  // ~2 s at 1.9 GHz (default budget)
constexpr uint32_t IDESC_PAIR = tc::idesc_u8(256, 256);
constexpr uint32_t IDESC = tc::idesc_u8(128, 256);  // the peak microbenchmark's MMA

using tc::flag_failure;
using tc::mbar_arrive;
using tc::mbar_arrive_tx;
using tc::mbar_init;
using tc::mbar_peek;
using tc::mbar_wait;
using tc::mbar_wait_drain;
using tc::mma_commit;
using tc::smem_u32;
using tc::sw128_desc;
using tc::tmem_wait_ld;
__device__ __forceinline__ void mma_i8(uint32_t dtmem, uint64_t adesc, uint64_t bdesc,
                                       uint32_t accumulate) {
  tc::mma_i8(dtmem, adesc, bdesc, IDESC, accumulate);
}
// 16 bytes of 0/1 from bits 0-3 and 8-11, 16-19, 24-27 of x: byte k of word p is bit 8k + p.
// Applied to x and x >> 4, the 32 bits of a codeword word land in 32 K positions in the order
// alimb_kernel stores A's limb columns, two instructions per word instead of a nibble multiply
// per word.
__device__ __forceinline__ uint4 bit_spread(uint32_t x) {
  constexpr uint32_t M = 0x01010101u;
  return make_uint4(x & M, (x >> 1) & M, (x >> 2) & M, (x >> 3) & M);
}
}  // namespace

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NTHREADS, 1)
    hash_tc_kernel(const __grid_constant__ CUtensorMap tmap_a, const u64* __restrict__ cw,
                   u64* __restrict__ H, u32* __restrict__ leaves, unsigned m, size_t two_n,
                   int* __restrict__ err, long long budget, unsigned c0, unsigned nck,
                   int mode, unsigned splits) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* words = smem + TC_STAGES * STAGE_BYTES;
  uint64_t* bars = (uint64_t*)(words + W_STAGES * W_BYTES);
  uint32_t* tmem_holder = (uint32_t*)(bars + NBARS);
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[TC_STAGES]);
  const uint32_t tma0 = smem_u32(&bars[2 * TC_STAGES]);
  const uint32_t acc_full0 = smem_u32(&bars[3 * TC_STAGES]);
  const uint32_t acc_empty0 = smem_u32(&bars[3 * TC_STAGES + 2]);
  const uint32_t drain = smem_u32(&bars[3 * TC_STAGES + 4]);
  const uint32_t wfull0 = smem_u32(&bars[3 * TC_STAGES + 5]);
  const uint32_t wempty0 = smem_u32(&bars[3 * TC_STAGES + 5 + W_STAGES]);
  const unsigned tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned rank = tc::cluster_rank(), pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  // K chunks (pairs of codeword rows) c0 .. c0 + nck - 1 of this launch; mode bit 0: add the
  // partial digest to H (else write it), bit 1: hash the leaves of the finished H.
  // Work units: (tile, split) with unit u = tile + ntiles * split, walked by the pair as u = pair,
  // pair + npairs, ..; split sp sums its share of the K chunks into its own digest slice
  // H + sp * 32 * two_n (the host sums the slices when splits > 1).
  const unsigned ntiles = (unsigned)(two_n / TC_N), nunits = ntiles * splits;
  struct Unit {
    unsigned tile, split, c, end;
  };
  auto unit_at = [&](unsigned u) {
    Unit x;
    x.tile = u % ntiles, x.split = u / ntiles;
    x.c = c0 + nck * x.split / splits;
    x.end = c0 + nck * (x.split + 1) / splits;
    return x;
  };
  __shared__ volatile int s_fail;

  if (tid == 0) {
    s_fail = 0;
    for (int s = 0; s < TC_STAGES; ++s) {
      // the leader's: four producer warps and the limbs of each CTA
      mbar_init(full0 + 8 * s, 2 * (NPROD / 32 + 1));
      mbar_init(empty0 + 8 * s, 1);
      mbar_init(tma0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full0 + 8 * b, 1);
      mbar_init(acc_empty0 + 8 * b, 2 * 4);  // a set's four warps of each CTA
    }
    for (int s = 0; s < W_STAGES; ++s) {
      mbar_init(wfull0 + 8 * s, 1);
      mbar_init(wempty0 + 8 * s, NPROD / 32);
    }
    mbar_init(drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // The pair's TMEM instructions want the other CTA launched and alive: the first meeting comes
  // before the allocation, the last one after the deallocation.  Without them, allocations under
  // launches from several streams have been seen to block for good, the pair's other half done.
  tc::cluster_sync();
  if (warp == 1)
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_holder)),
                 "r"(TMEM_COLS)
                 : "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  tc::cluster_sync();  // both CTAs' barriers are initialised and both hold their TMEM
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 1)
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  const uint32_t tmem = *tmem_holder;
  const uint32_t lead_full0 = tc::map_to_rank(full0, 0);
  const uint32_t lead_acc_empty0 = tc::map_to_rank(acc_empty0, 0);

  if (warp == 0) {
    // ---- TMA producer: this CTA's half of the A-limb rows ----
    if (lane == 0) {
      unsigned f = 0;
      bool ok = true;
      for (unsigned u = pair; u < nunits && ok; u += npairs) {
        const Unit x = unit_at(u);
        for (unsigned c = x.c; c < x.end; c += TC_SUB, ++f) {
          const unsigned ns = min((unsigned)TC_SUB, x.end - c);
          const unsigned s = f % TC_STAGES;
          if (f >= TC_STAGES &&
              !mbar_wait(empty0 + 8 * s, ((f / TC_STAGES) - 1) & 1, &s_fail, budget)) {
            if (!s_fail) flag_failure(&s_fail, err, 1);
            ok = false;
            break;
          }
          const uint32_t bar = tma0 + 8 * s;
          mbar_arrive_tx(bar, ns * LIMB_TILE);
          const uint32_t dst = smem_u32(smem + s * STAGE_BYTES + TC_SUB * BIT_TILE);
          const int y = (int)(rank * 128);
          for (unsigned h = 0; h < ns; ++h)
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                "[%0], [%1, {%2, %3}], [%4];" ::"r"(dst + h * LIMB_TILE),
                "l"((uint64_t)&tmap_a), "r"((int)((c + h) * TC_KB)), "r"(y), "r"(bar)
                : "memory");
        }
      }
      // Only the newest copy of each stage can still be in flight (an older one was consumed
      // before its stage was refilled): wait for those before the CTA may exit.
      for (unsigned g = f > TC_STAGES ? f - TC_STAGES : 0; g < f; ++g)
        if (!mbar_wait_drain(tma0 + 8 * (g % TC_STAGES), (g / TC_STAGES) & 1)) atomicExch(err, 6);
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      // ---- MMA issuer ----  (descriptors by addition and the next stage's barrier looked at
      // before the commit: the thread's own instructions cost tensor time)
      const uint64_t ad0 = sw128_desc(smem_u32(smem));
      const uint64_t bd0 = sw128_desc(smem_u32(smem) + TC_SUB * BIT_TILE);
      unsigned s = 0, ph = 0, t = 0;
      bool ok = true, ready = false;
      for (unsigned u = pair; u < nunits && ok; u += npairs, ++t) {
        const Unit x = unit_at(u);
        const uint32_t d = tmem + (t & 1) * 256;
        if (t >= 2 && !mbar_wait(acc_empty0 + 8 * (t & 1), ((t >> 1) - 1) & 1, &s_fail, budget)) {
          if (!s_fail) flag_failure(&s_fail, err, 2);
          ok = false;
          break;
        }
        for (unsigned c = x.c; c < x.end; c += TC_SUB) {
          if (!ready && !mbar_wait(full0 + 8 * s, ph, &s_fail, budget)) {
            if (!s_fail) flag_failure(&s_fail, err, 3);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t ad = ad0 + s * (STAGE_BYTES >> 4), bd = bd0 + s * (STAGE_BYTES >> 4);
          const uint32_t bar = empty0 + 8 * s;
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            tc::mma_i8_pair(d, ad + 2 * ks, bd + 2 * ks, IDESC_PAIR, c > x.c || ks > 0);
          if (c + 1 < x.end)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              tc::mma_i8_pair(d, ad + (BIT_TILE >> 4) + 2 * ks, bd + (LIMB_TILE >> 4) + 2 * ks,
                              IDESC_PAIR, 1);
          if (++s == TC_STAGES) s = 0, ph ^= 1;
          ready = mbar_peek(full0 + 8 * s, ph);
          tc::mma_commit_both(bar);
        }
        if (ok) tc::mma_commit_both(acc_full0 + 8 * (t & 1));
      }
      // Every MMA issued so far has completed once this arrives; wait for it before the TMEM
      // is freed (also after a failure).
      tc::mma_commit_leader(drain);
      if (!mbar_wait_drain(drain, 0)) atomicExch(err, 7);
    }
  } else if (warp < 6) {
    // ---- bit producers (128 threads): a column each ----
    const unsigned j = tid - 64;
    unsigned f = 0;
    bool ok = true;
    for (unsigned u = pair; u < nunits && ok; u += npairs) {
      const Unit x = unit_at(u);
      for (unsigned c = x.c; c < x.end; c += TC_SUB, ++f) {
        const unsigned ns = min((unsigned)TC_SUB, x.end - c);
        const unsigned s = f % TC_STAGES, ws = f % W_STAGES;
        ok = mbar_wait(wfull0 + 8 * ws, (f / W_STAGES) & 1, &s_fail, budget);
        u64 wv[2 * TC_SUB];
        if (ok) {
          const u64* wp = (const u64*)(words + ws * W_BYTES) + j;
#pragma unroll
          for (unsigned r = 0; r < 2 * TC_SUB; ++r)  // rows past the last are zero
            wv[r] = r < 2 * ns && 2 * c + r < m ? wp[r * TC_COLS] : 0;
          if (f >= TC_STAGES)
            ok = mbar_wait(empty0 + 8 * s, ((f / TC_STAGES) - 1) & 1, &s_fail, budget);
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (!s_fail) flag_failure(&s_fail, err, 4);
          break;
        }
#pragma unroll
        for (unsigned h = 0; h < TC_SUB; ++h) {
          uint8_t* bt = smem + s * STAGE_BYTES + h * BIT_TILE + j * TC_KB;
          const uint32_t x4[4] = {(uint32_t)wv[2 * h], (uint32_t)(wv[2 * h] >> 32),
                                  (uint32_t)wv[2 * h + 1], (uint32_t)(wv[2 * h + 1] >> 32)};
          if (h < ns)
#pragma unroll
            for (int q = 0; q < 4; ++q) {  // 32 bits -> chunks 2q, 2q + 1 (bit_spread's order)
              *(uint4*)(bt + (((2 * q) ^ (j & 7)) << 4)) = bit_spread(x4[q]);
              *(uint4*)(bt + (((2 * q + 1) ^ (j & 7)) << 4)) = bit_spread(x4[q] >> 4);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(wempty0 + 8 * ws);
          tc::mbar_arrive_cluster(lead_full0 + 8 * s);
        }
      }
    }
  } else if (warp == 14) {
    // ---- word loader: the stage's rows of this CTA's 128 columns ----
    if (lane == 0) {
      unsigned f = 0;
      bool ok = true;
      for (unsigned u = pair; u < nunits && ok; u += npairs) {
        const Unit x = unit_at(u);
        const u64* col = cw + (size_t)x.tile * TC_N + rank * TC_COLS;
        for (unsigned c = x.c; c < x.end; c += TC_SUB, ++f) {
          const unsigned ns = min((unsigned)TC_SUB, x.end - c);
          const unsigned ws = f % W_STAGES;
          if (f >= W_STAGES &&
              !mbar_wait(wempty0 + 8 * ws, ((f / W_STAGES) - 1) & 1, &s_fail, budget)) {
            if (!s_fail) flag_failure(&s_fail, err, 9);
            ok = false;
            break;
          }
          const unsigned nrow = min(2 * ns, m - 2 * c);
          const uint32_t bar = wfull0 + 8 * ws, dst = smem_u32(words + ws * W_BYTES);
          mbar_arrive_tx(bar, nrow * W_ROW);
          for (unsigned r = 0; r < nrow; ++r)
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes "
                "[%0], [%1], %2, [%3];" ::"r"(dst + r * W_ROW),
                "l"((uint64_t)__cvta_generic_to_global(col + (size_t)(2 * c + r) * two_n)),
                "r"((uint32_t)W_ROW), "r"(bar)
                : "memory");
        }
      }
      for (unsigned g = f > W_STAGES ? f - W_STAGES : 0; g < f; ++g)  // the copies still in flight
        if (!mbar_wait_drain(wfull0 + 8 * (g % W_STAGES), (g / W_STAGES) & 1)) atomicExch(err, 10);
    }
  } else if (warp == 15) {
    // ---- this CTA's limbs of a stage have landed: tell the leader ----
    if (lane == 0) {
      unsigned f = 0;
      bool ok = true;
      for (unsigned u = pair; u < nunits && ok; u += npairs) {
        const Unit x = unit_at(u);
        for (unsigned c = x.c; c < x.end; c += TC_SUB, ++f) {
          const unsigned ns = min((unsigned)TC_SUB, x.end - c);
          const unsigned s = f % TC_STAGES;
          if (!mbar_wait(tma0 + 8 * s, (f / TC_STAGES) & 1, &s_fail, budget)) {
            if (!s_fail) flag_failure(&s_fail, err, 8);
            ok = false;
            break;
          }
          tc::mbar_arrive_cluster(lead_full0 + 8 * s);
        }
      }
    }
  } else {
    // ---- epilogue: set (warps 6-9, 10-13) takes every other tile; a thread owns TMEM lane =
    // column 32 (warp mod 4) + lane of this CTA's 128 and reads its 256 limb sums
    const unsigned set = (warp - 6) >> 2, quarter = warp & 3;
    const unsigned jc = 32 * quarter + lane;
    const uint32_t acc = tmem + ((32 * quarter) << 16) + set * 256;
    unsigned t = 0;
    for (unsigned u = pair; u < nunits; u += npairs, ++t) {
      if ((t & 1) != set) continue;
      const Unit x = unit_at(u);
      const bool got = mbar_wait(acc_full0 + 8 * set, (t >> 1) & 1, &s_fail, budget);
      if (!__all_sync(0xffffffffu, got)) {
        if (!s_fail) flag_failure(&s_fail, err, 5);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const size_t j = (size_t)x.tile * TC_N + rank * TC_COLS + jc;
      u64* hp = H + (size_t)x.split * H_ROWS * two_n + j;
      u32 cv[8];
      b3_init(cv);
#pragma unroll 1
      for (int blk = 0; blk < 4; ++blk) {
        u32 wd[16];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t r[32];
          tc::tmem_ld32(acc + blk * 64 + half * 32, r);
          tmem_wait_ld();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t* l = r + 8 * q;
            const u64 a = (u64)l[0] + ((u64)l[1] << 8) + ((u64)l[2] << 16) + ((u64)l[3] << 24);
            const u64 b = (u64)l[4] + ((u64)l[5] << 8) + ((u64)l[6] << 16) + ((u64)l[7] << 24);
            const u64 lo = a + (b << 32);
            const u64 hi = (b >> 32) + (lo < a ? 1 : 0);
            u64* h = hp + (size_t)(blk * 8 + half * 4 + q) * two_n;
            u64 v = gl_reduce(lo, hi);
            if (mode & 1) v = gl_add(__ldcg(h), v);
            *h = v;
            wd[8 * half + 2 * q] = (u32)v;
            wd[8 * half + 2 * q + 1] = (u32)(v >> 32);
          }
        }
        if (blk == 3) {  // accumulators read: the MMAs of the tile after next may start
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) tc::mbar_arrive_cluster(lead_acc_empty0 + 8 * set);
        }
        if (mode & 2)  // the leaf hash of the 256-byte column (C = 32 canonical u64)
          b3_compress(cv, wd, 64,
                      (blk == 0 ? B3_CHUNK_START : 0) | (blk == 3 ? (B3_CHUNK_END | B3_ROOT) : 0));
      }
      if (mode & 2) {
        uint4* lp = (uint4*)(leaves + j * 8);
        lp[0] = make_uint4(cv[0], cv[1], cv[2], cv[3]);
        lp[1] = make_uint4(cv[4], cv[5], cv[6], cv[7]);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  tc::cluster_sync();  // neither CTA's shared memory, barriers or TMEM are in use any more
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(TMEM_COLS)
                 : "memory");
  }
  tc::cluster_sync();
}

// ---- the int8 tensor-core peak this hash is measured against ----------------------------------
// One CTA per SM; one thread issues `iters` x 4 back-to-back tcgen05.mma.kind::i8 M128 N256 K32
// on a fixed 128 x 128-byte A tile and 256 x 128-byte B tile in shared memory (the shape and
// layout the hash uses), accumulating into TMEM; one commit at the end, waited with a bound.
constexpr int PK_SMEM = 128 * TC_KB + 256 * TC_KB + 1024 + 64;

__global__ void __launch_bounds__(128, 1) i8_peak_kernel(unsigned iters, int* __restrict__ err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bar = (uint64_t*)(smem + 128 * TC_KB + 256 * TC_KB);
  uint32_t* tmem_holder = (uint32_t*)(bar + 1);
  const unsigned tid = threadIdx.x, warp = tid >> 5;
  for (unsigned i = tid; i < (128 + 256) * TC_KB / 16; i += blockDim.x)
    ((uint4*)smem)[i] = make_uint4(0x01020304u * (i & 7), i, 0x80808080u, 0x7f7f7f7fu);
  if (tid == 0) {
    mbar_init(smem_u32(bar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_holder)),
                 "r"(256)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_holder;
  if (tid == 0) {
    const uint32_t a_base = smem_u32(smem), b_base = a_base + 128 * TC_KB;
    for (unsigned i = 0; i < iters; ++i)
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        mma_i8(tmem, sw128_desc(a_base + ks * 32), sw128_desc(b_base + ks * 32),
               (i > 0 || ks > 0) ? 1u : 0u);
    mma_commit(smem_u32(bar));
    if (!mbar_wait_drain(smem_u32(bar), 0)) atomicExch(err, 8);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256)
                 : "memory");
  }
}

double i8_tensor_peak_tops(unsigned iters, int* err, cudaStream_t st) {
  int dev = 0, sms = 0;
  LGS_CUDA(cudaGetDevice(&dev));
  LGS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  LGS_CUDA(cudaFuncSetAttribute(i8_peak_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                PK_SMEM));
  cudaEvent_t e0, e1;
  LGS_CUDA(cudaEventCreate(&e0));
  LGS_CUDA(cudaEventCreate(&e1));
  double best = 0.0;
  for (int rep = 0; rep < 4; ++rep) {  // the first launch warms up; keep the best
    LGS_CUDA(cudaEventRecord(e0, st));
    i8_peak_kernel<<<sms, 128, PK_SMEM, st>>>(iters, err);
    LGS_LAUNCH_CHECK();
    LGS_CUDA(cudaEventRecord(e1, st));
    LGS_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    LGS_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    const double ops = 2.0 * 128 * 256 * 32 * 4.0 * iters * sms;
    if (rep > 0 && ms > 0) best = std::max(best, ops / (ms * 1e-3) / 1e12);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return best;
}

// Alimb[8r + l][kperm(k)] = byte l of A[r][k] (the 256 x W limb matrix the TMA descriptor
// covers), with the K order of the B tiles the hash's producers write: inside each aligned group
// of 32 columns, bit t of a codeword word sits at position 16 ((t >> 2) & 1) + 4 (t & 3) + (t >> 3).
__global__ void alimb_kernel(const u64* __restrict__ A, uint8_t* __restrict__ alimb, size_t W) {
  size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned r = blockIdx.y;
  if (k >= W) return;
  u64 v = A[(size_t)r * W + k];
  const unsigned t = (unsigned)(k & 31);
  const size_t kp = (k & ~(size_t)31) | (16 * ((t >> 2) & 1) + 4 * (t & 3) + (t >> 3));
#pragma unroll
  for (int l = 0; l < 8; ++l) alimb[(size_t)(r * 8 + l) * W + kp] = (uint8_t)(v >> (8 * l));
}

void alimb_from_a(const u64* A, uint8_t* alimb, size_t W, cudaStream_t st) {
  alimb_kernel<<<dim3(cdiv(W, 256), 32), 256, 0, st>>>(A, alimb, W);
  LGS_LAUNCH_CHECK();
}

// ---- host side -----------------------------------------------------------------------------
namespace {
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    LGS_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
    if (!p || q != cudaDriverEntryPointSuccess)
      throw CudaError("cuTensorMapEncodeTiled is not available from the driver");
    fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  }
  return fn;
}
}  // namespace

// The TMA descriptor of the 256 x W byte matrix of A's limbs: boxes of 128 rows x 128 bytes,
// 128-byte swizzle (the K-major layout tcgen05 reads).  W must be a multiple of 64.
void make_alimb_tmap(const uint8_t* alimb, size_t W, void* tmap_out) {
  if (W % 64 || ((uintptr_t)alimb & 15)) throw ShapeError("hash: A-limb matrix misaligned");
  CUtensorMap* tm = (CUtensorMap*)tmap_out;
  cuuint64_t dims[2] = {(cuuint64_t)W, 256};
  cuuint64_t strides[1] = {(cuuint64_t)W};
  cuuint32_t box[2] = {TC_KB, 128};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode_fn()(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)alimb, dims, strides, box,
                           estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    throw CudaError("cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
}

// The TMA descriptor of a row-major rows x inner matrix of 64-bit integers (inner even, base
// 16-byte aligned): boxes of box_rows rows x 16 values (128 bytes), 128-byte swizzle, zeros
// outside the matrix.
void make_i64_tmap(const int64_t* base, size_t rows, size_t inner, unsigned box_rows,
                   void* tmap_out) {
  if (inner % 2 || ((uintptr_t)base & 15)) throw ShapeError("TMA: int64 matrix misaligned");
  CUtensorMap* tm = (CUtensorMap*)tmap_out;
  cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)inner * 8};
  cuuint32_t box[2] = {16, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode_fn()(tm, CU_TENSOR_MAP_DATA_TYPE_INT64, 2, (void*)base, dims, strides, box,
                           estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    throw CudaError("cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
}

size_t tensor_map_bytes() { return sizeof(CUtensorMap); }

namespace {
// Sums the split slices of the digest (H = sum of slices, plus the old H in mode bit 0) and, in
// mode bit 1, hashes each finished column as its Merkle leaf.  A thread sums 4 rows of a column: the
// slices are read in few long chains, and one thread per column left 2^13 columns on 32 SMs
// (2^12 x 2^12, 9 slices: 63 -> 9 us).
__global__ void __launch_bounds__(256) hash_combine_kernel(const u64* __restrict__ Hp,
                                                           unsigned splits, u64* __restrict__ H,
                                                           u32* __restrict__ leaves, size_t two_n,
                                                           int mode) {
  constexpr int RT = H_ROWS / 8;  // rows of a thread
  __shared__ u64 sv[H_ROWS][32];
  const unsigned lane = threadIdx.x & 31, r0 = (threadIdx.x >> 5) * RT;
  const size_t j = (size_t)blockIdx.x * 32 + lane;  // two_n is a multiple of 256
  u64 acc[RT];
#pragma unroll
  for (int r = 0; r < RT; ++r) acc[r] = (mode & 1) ? H[(r0 + r) * two_n + j] : 0;
  for (unsigned sp = 0; sp < splits; ++sp) {
    const u64* h = Hp + ((size_t)sp * H_ROWS + r0) * two_n + j;
#pragma unroll
    for (int r = 0; r < RT; ++r) acc[r] = gl_add(acc[r], __ldcs(h + r * two_n));
  }
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    H[(r0 + r) * two_n + j] = acc[r];
    sv[r0 + r][lane] = acc[r];
  }
  if (!(mode & 2)) return;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  u32 cv[8];
  b3_init(cv);
#pragma unroll
  for (int blk = 0; blk < 4; ++blk) {
    u32 wd[16];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const u64 x = sv[blk * 8 + q][lane];
      wd[2 * q] = (u32)x;
      wd[2 * q + 1] = (u32)(x >> 32);
    }
    const u32 flags = (blk == 0 ? B3_CHUNK_START : 0) | (blk == 3 ? (B3_CHUNK_END | B3_ROOT) : 0);
    b3_compress(cv, wd, 64, flags);
  }
  uint4* lp = (uint4*)(leaves + j * 8);
  lp[0] = make_uint4(cv[0], cv[1], cv[2], cv[3]);
  lp[1] = make_uint4(cv[4], cv[5], cv[6], cv[7]);
}

// CTA pairs of a launch: max_ctas / 2 (at least one), or as many as the GPU's SMs hold.
unsigned hash_pairs_for(unsigned max_ctas) {
  int dev = 0, sms = 0;
  LGS_CUDA(cudaGetDevice(&dev));
  LGS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const unsigned all = std::max(1u, (unsigned)sms / 2);
  return max_ctas ? std::min(std::max(1u, max_ctas / 2), all) : all;
}
}  // namespace

// Work units are (tile, K share): time ~ rounds over the pairs x (chunks of a unit + a fixed cost).
// Splitting costs a second kernel that sums the slices, so the unsplit plan wins unless a split is
// clearly shorter; the constants are in K chunks (0.27 us each): 16 for a unit's start and
// epilogue, 40 for the second launch.
unsigned subset_sum_hash_splits(size_t two_n, unsigned rows, unsigned max_ctas) {
  const size_t ntiles = two_n / TC_N, pairs = hash_pairs_for(max_ctas);
  const unsigned nck = (rows + 1) / 2;
  unsigned best = 1;
  size_t best_cost = (size_t)-1;
  for (unsigned sp = 1; sp <= 16 && nck / sp >= 8 - (sp == 1 ? 7 : 0); ++sp) {
    const size_t rounds = (ntiles * sp + pairs - 1) / pairs;
    const size_t cost = rounds * ((nck + sp - 1) / sp + 16) + (sp > 1 ? 40 : 0);
    if (cost < best_cost) best = sp, best_cost = cost;
  }
  return best;
}

void subset_sum_hash_tc(const void* tmap, const u64* cw, u64* H, u32* leaves, unsigned m,
                        size_t two_n, int* err, cudaStream_t st, uint64_t wait_cycles,
                        unsigned max_ctas, unsigned row0, unsigned rows, int mode,
                        u64* split_scratch) {
  if (two_n % TC_N) throw ShapeError("hash: 2n must be a multiple of 256");
  if (m == 0 || m > 8192) throw ShapeError("hash: 1 <= m <= 8192");
  if (rows == 0) rows = m - row0;
  if (row0 % 2 || (rows % 2 && row0 + rows != m) || row0 + rows > m || mode < 0 || mode > 3)
    throw ShapeError("hash: row range must start and end on chunks of two rows");
  LGS_CUDA(cudaFuncSetAttribute(hash_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                SMEM_BYTES));
  const size_t ntiles = two_n / TC_N;
  const unsigned nck = (rows + 1) / 2;
  // Few column tiles (square shapes): split K over the pairs into digest slices, summed afterwards
  const unsigned splits = split_scratch ? subset_sum_hash_splits(two_n, rows, max_ctas) : 1;
  // no more pairs than the rounds need: the SMs left over run the prove's kernels beside the hash
  const size_t units = ntiles * splits, all = hash_pairs_for(max_ctas);
  const unsigned grid = 2 * (unsigned)cdiv(units, cdiv(units, all));
  const long long budget =
      wait_cycles ? (long long)std::min<uint64_t>(wait_cycles, (uint64_t)WAIT_CYCLES) : WAIT_CYCLES;
  if (splits == 1) {
    hash_tc_kernel<<<grid, NTHREADS, SMEM_BYTES, st>>>(*(const CUtensorMap*)tmap, cw, H, leaves,
                                                       m, two_n, err, budget, row0 / 2, nck, mode,
                                                       1u);
    LGS_LAUNCH_CHECK();
    return;
  }
  hash_tc_kernel<<<grid, NTHREADS, SMEM_BYTES, st>>>(*(const CUtensorMap*)tmap, cw, split_scratch,
                                                     leaves, m, two_n, err, budget, row0 / 2, nck,
                                                     0, splits);
  LGS_LAUNCH_CHECK();
  hash_combine_kernel<<<(unsigned)(two_n / 32), 256, 0, st>>>(split_scratch, splits, H,
                                                                 leaves, two_n, mode);
  LGS_LAUNCH_CHECK();
}

}  // namespace lgs
