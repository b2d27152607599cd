// Product sumcheck prover (utils/src/sumcheck.rs:37-84) on the device.
//
// Round t sends g_t(q) = sum_{i < half} prod_j (lo_j + q (hi_j - lo_j)), q = 0..d, with
// lo = P[i], hi = P[i + half] (the HIGH variable is bound first), then folds every factor with
// the round challenge r_t: P[i] = P[i] + r_t (P[i + half] - P[i]).  All challenges come from the
// pre-drawn oracle (utils/src/oracle.rs:10-64), so no round depends on a message: the folds form a
// chain, and every round's sum is a sum over a level of that chain that nothing waits for.
//
// One kernel, sc_tile_kernel, does both the passes over long vectors and the end of every
// sumcheck.  A tile is c consecutive low positions with all 2^r of their high parts (T = c 2^r
// entries per factor): the pairs of r rounds lie inside it.  A CTA loads a tile, one pair per
// thread, sums round 0 from registers and folds into shared memory, folds on, keeping every level,
// and then sums the other rounds at once, again one pair per thread.  Persistent CTAs walk the tiles
// and leave one partial sum per round.
// Vectors of at most 2^SC_LOG_T entries finish in one CTA, which also adds the earlier passes'
// partials and fills in their g(1): g_t(1) = claim_t - g_t(0), claim_{t+1} = g_t(r_t), an affine
// recurrence run as a scan.  What bounds a short vector is the chain of folds, one product and one
// barrier each; a long one is bound by its products on the integer pipes.  Passes of two rounds
// with a one-CTA end of ten sequential rounds took 38 us for that end and 473 us for three factors
// of 2^22; tiles take 20 us and 406 us.
// One or two factors have few products per entry, and a tile's high parts are runs of 2^(10 - r)
// entries, which DRAM reads badly once the vector is longer than L2: sc_stream_kernel halves such
// vectors twice per pass, in registers.
//
// Binary variant (the B_I check of pcs/src/ligesis.rs:423-428, factors [b, b - 1, eq]): the
// middle factor is always the first minus one (folding is affine), so only b and eq are stored
// and folded; the products, round messages and final evaluations are those of the 3-factor run.
#include "kernels.cuh"
#include "limb_sums.cuh"

namespace lgs {

namespace {
constexpr unsigned SC_THREADS = 512;
constexpr unsigned SC_LOG_T = 10;   // tile entries per factor
constexpr unsigned SC_MAX_R = 8;    // rounds per pass: at least 64-byte runs of global memory
constexpr unsigned SC_MAX_K = 30;   // as the C ABI
// Vectors of one or two factors are streamed from 2^23 entries on (134 MB a factor, against an L2
// of 126 MB), two rounds per pass.  Device time with tiles alone and as it is: one factor 2^23 208
// and 125 us, 2^24 377 and 218, 2^27 2663 and 1115; two factors 2^23 402 and 291, 2^24 748 and 535,
// 2^27 5599 and 3431.  Three factors are bound by their products in tiles too (2^24: 1249 us).
constexpr unsigned SC_STREAM_LOG = 23, SC_STREAM_R = 2, SC_STREAM_THREADS = 256;
constexpr unsigned SC_MAX_PASSES = 6;  // 2^30: four streamed passes to 2^22, then two of tiles

__device__ __forceinline__ ef2 shfl_xor_ef(ef2 v, int m) {
  ef2 r;
  r.c0 = __shfl_xor_sync(0xffffffffu, v.c0, m);
  r.c1 = __shfl_xor_sync(0xffffffffu, v.c1, m);
  return r;
}

// Stored factor count: the binary variant keeps [b, eq] for the logical [b, b - 1, eq].
template <int D, bool BIN>
struct Fac {
  static constexpr int S = BIN ? D - 1 : D;
};

// Out-of-line F_p2 products for code that runs a few times per launch: one shared copy is less to
// fetch than one inlined copy per use.
__device__ __noinline__ ef2 ef_mul_ol(ef2 a, ef2 b) { return ef_mul(a, b); }

// Lagrange weights of the nodes 0..D at r: g(r) = sum_q L[q] g(q).
template <int D>
__device__ void interp_weights(ef2 r, ef2 (&L)[D + 1]) {
  const u64 inv2 = 0x7FFFFFFF80000001ULL, inv6 = 0xD555555480000001ULL;
  const ef2 r1 = ef_sub(r, ef_from(1)), r2 = ef_sub(r, ef_from(2));
  if (D == 1) {
    L[0] = ef_sub(ef_one(), r);
    L[1] = r;
  } else if (D == 2) {
    L[0] = ef_scale(ef_mul_ol(r1, r2), inv2);
    L[1] = ef_sub(ef_zero(), ef_mul_ol(r, r2));
    L[D] = ef_scale(ef_mul_ol(r, r1), inv2);
  } else {
    const ef2 r3 = ef_sub(r, ef_from(3));
    const ef2 r12 = ef_mul_ol(r1, r2), rr1 = ef_mul_ol(r, r1);
    L[0] = ef_sub(ef_zero(), ef_scale(ef_mul_ol(r12, r3), inv6));
    L[1] = ef_scale(ef_mul_ol(ef_mul_ol(r, r2), r3), inv2);
    L[D - 1] = ef_sub(ef_zero(), ef_scale(ef_mul_ol(rr1, r3), inv2));
    L[D] = ef_scale(ef_mul_ol(rr1, r2), inv6);
  }
}

// One sumcheck: factors read from src (factor 0 as base-field words if bf0, in the first pass) and
// folded into dst (which may be src), its challenges, results and partial sums.
template <int S>
struct ScOne {
  const void* src[S];
  ef2* dst[S];
  const ef2* ch;
  ef2 *rounds, *fin, *part;
};
template <int S>
struct ScJobs {
  ScOne<S> j[SC_MAX_JOBS];
};
// The block's sumcheck, field by field: indexing the parameters with blockIdx.y would copy them
// to local memory first.
template <int S>
__device__ __forceinline__ ScOne<S> my_job(const ScJobs<S>& jobs) {
  static_assert(SC_MAX_JOBS == 2, "two candidates");
  const bool y = blockIdx.y != 0;
  ScOne<S> o;
#pragma unroll
  for (int j = 0; j < S; ++j) {
    o.src[j] = y ? jobs.j[1].src[j] : jobs.j[0].src[j];
    o.dst[j] = y ? jobs.j[1].dst[j] : jobs.j[0].dst[j];
  }
  o.ch = y ? jobs.j[1].ch : jobs.j[0].ch;
  o.rounds = y ? jobs.j[1].rounds : jobs.j[0].rounds;
  o.fin = y ? jobs.j[1].fin : jobs.j[0].fin;
  o.part = y ? jobs.j[1].part : jobs.j[0].part;
  return o;
}
// The passes before this launch: pass p ran nb[p] CTAs and ended before round t[p].
struct ScPasses {
  unsigned n, t[SC_MAX_PASSES], nb[SC_MAX_PASSES];
};

template <int D, bool BIN>
struct TileSmem {
  static constexpr int S = Fac<D, BIN>::S;
  ef2 sv[S][1u << SC_LOG_T];  // level l >= 1 of the tile at T - (2T >> l)
  ef2 ch[SC_LOG_T];
  uint32_t acc[SC_LOG_T][D + 1][6];
};
// The last CTA's use of sv once the tile is summed: the passes' round sums and weights.
template <int D>
struct ChainSmem {
  ef2 g[SC_MAX_K][D + 1], w[SC_MAX_K][D + 1];
};

// Rounds t0 .. t0 + r - 1 of blockIdx.y's sumcheck on vectors of `len` entries in tiles of
// 2^log_t.  final: one tile, r = log_t, and the sumcheck ends.
template <int D, bool BIN>
__global__ void __launch_bounds__(SC_THREADS, 2)
    sc_tile_kernel(const ScJobs<Fac<D, BIN>::S> jobs, size_t len, unsigned log_t, unsigned r,
                   unsigned t0, int bf0, int final, size_t stride, const ScPasses prev) {
  constexpr int S = Fac<D, BIN>::S;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TileSmem<D, BIN>& sm = *reinterpret_cast<TileSmem<D, BIN>*>(smem_raw);
  ChainSmem<D>& cs = *reinterpret_cast<ChainSmem<D>*>(smem_raw + sizeof(TileSmem<D, BIN>));
  const ScOne<S> jb = my_job(jobs);
  const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned T = 1u << log_t, log_c = log_t - r, c = 1u << log_c;
  const size_t ntiles = len >> log_t, hstep = len >> r;
  if (tid < r) sm.ch[tid] = jb.ch[t0 + tid];
  for (unsigned i = tid; i < sizeof(sm.acc) / 4; i += SC_THREADS) (&sm.acc[0][0][0])[i] = 0;
  if (final) {
    // the passes' rounds 0 .. t0 - 1: one warp per sum, and the weights of their claim chain
    constexpr unsigned NW = SC_THREADS / 32;
    for (unsigned x = warp; x < t0 * (D + 1); x += NW) {
      const unsigned t = x / (D + 1), q = x % (D + 1);
      unsigned nb = prev.nb[0];
#pragma unroll
      for (unsigned p = 1; p < SC_MAX_PASSES; ++p)
        if (p < prev.n && t >= prev.t[p - 1]) nb = prev.nb[p];
      const ef2* src = jb.part + (size_t)t * stride + q;
      ef2 s = ef_zero();
#pragma unroll 4
      for (unsigned b = lane; b < nb; b += 32) s = ef_add(s, src[(size_t)b * (D + 1)]);
#pragma unroll
      for (int m = 16; m; m >>= 1) s = ef_add(s, shfl_xor_ef(s, m));
      if (lane == 0) cs.g[t][q] = s;
    }
    if (warp == NW - 1)
      for (unsigned t = lane; t < t0; t += 32) {
        ef2 L[D + 1];
        interp_weights<D>(jb.ch[t], L);
#pragma unroll
        for (int q = 0; q <= D; ++q) cs.w[t][q] = L[q];
      }
  }
  ef2 run = ef_zero();  // thread (round, q) of the first r (D + 1): its sum over the CTA's tiles
  for (size_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const size_t i0 = tile << log_c;
    __syncthreads();  // the previous tile is summed; sm.ch is visible
    // phase 0: the tile's first round, pair tid, from global memory; phase 1: all later rounds
#pragma unroll 1
    for (unsigned ph = 0; ph < 2; ++ph) {
      const unsigned npairs = ph ? (T >> 1) - c : T >> 1;
      const bool act = tid < npairs;
      unsigned rd = 0;
      ef2 v[S], df[S];
      if (ph == 0) {
        if (act) {
          const ef2 rt = sm.ch[0];
          const unsigned ih = tid + (T >> 1);
          const size_t gl = i0 + (tid & (c - 1)) + (size_t)(tid >> log_c) * hstep;
          const size_t gh = i0 + (ih & (c - 1)) + (size_t)(ih >> log_c) * hstep;
#pragma unroll
          for (int j = 0; j < S; ++j) {
            if (j == 0 && bf0) {
              const u64* src = (const u64*)jb.src[0];
              v[0] = ef_from(src[gl]), df[0] = ef_from(gl_sub(src[gh], src[gl]));
            } else {
              const ef2* src = (const ef2*)jb.src[j];
              v[j] = src[gl], df[j] = ef_sub(src[gh], v[j]);
            }
          }
#pragma unroll
          for (int j = 0; j < S; ++j)
            sm.sv[j][tid] = ef_add(v[j], j == 0 && bf0 ? ef_scale(rt, df[0].c0)
                                                       : ef_mul(rt, df[j]));
        }
      } else {
        for (unsigned l = 1; l < r; ++l) {
          __syncthreads();
          const ef2 rt = sm.ch[l];
          const unsigned lh = log_t - 1 - l, half = 1u << lh, off = T - (2 * T >> l);
          for (unsigned x = tid; x < (unsigned)S << lh; x += SC_THREADS) {
            ef2* e = sm.sv[x >> lh] + off + (x & (half - 1));  // level l + 1 at off + 2 half
            e[2 * half] = ef_lerp(e[0], e[half], rt);
          }
        }
        __syncthreads();
        if (!final) {
          const unsigned off = T - (2 * T >> r);
          for (unsigned x = tid; x < (unsigned)S << log_c; x += SC_THREADS) {
            const unsigned j = x >> log_c, i = x & (c - 1);
            ef2* dst = jb.dst[0];
#pragma unroll
            for (int y = 1; y < S; ++y)
              if (j == (unsigned)y) dst = jb.dst[y];
            dst[i0 + i] = sm.sv[j][off + i];
          }
        }
        if (act) {  // T / 2 >= u > c: the round with T >> (rd + 1) < u <= T >> rd
          const unsigned u = (T >> 1) - tid;
          rd = log_t - (32 - __clz(u - 1));
          const unsigned lo = T - (2 * T >> rd) + tid - ((T >> 1) - (T >> rd));
#pragma unroll
          for (int j = 0; j < S; ++j) {
            v[j] = sm.sv[j][lo];
            df[j] = ef_sub(sm.sv[j][lo + (T >> (rd + 1))], v[j]);
          }
        }
      }
      if ((tid & ~31u) >= npairs) continue;  // the whole warp
      // 32 consecutive pairs lie in one round, except the last 32 of phase 1
      const bool mixed = ph ? (tid & ~31u) + 64 > T >> 1 : T < 64;
      const bool first = t0 + rd == 0;
      // b of the binary check is 0 or 1 in round 0: b (b - 1) is 0 at q = 0, 1 and, where lo != hi,
      // 2 and 6 at q = 2, 3
      const bool bin0 = BIN && first, scale0 = ph == 0 && bf0;
      const bool diff = df[0].c0 != 0;
#pragma unroll 1
      for (int q = 0; q <= D; ++q) {
        if (q != 1 || first || final) {
          ef2 pr;
          if (bin0) {
            pr = ef_zero();
            if (diff && q >= 2) {
              pr = ef_add(v[S - 1], v[S - 1]);
              if (q == 3) pr = ef_add(pr, ef_add(pr, pr));
            }
          } else {
            if (BIN) {
              pr = ef_mul(v[0], ef_sub(v[0], ef_one()));
            } else {
              pr = v[0];
            }
#pragma unroll
            for (int j = 1; j < S; ++j)
              pr = j == 1 && !BIN && scale0 ? ef_scale(v[1], pr.c0) : ef_mul(pr, v[j]);
          }
          if (!mixed) {
            warp_add(pr, sm.acc[rd][q], lane);
          } else if (act) {
            uint32_t l[6];
            limbs22(pr, l);
#pragma unroll
            for (int y = 0; y < 6; ++y) atomicAdd(&sm.acc[rd][q][y], l[y]);
          }
        }
#pragma unroll
        for (int j = 0; j < S; ++j) v[j] = ef_add(v[j], df[j]);
      }
    }
    __syncthreads();
    if (tid < r * (D + 1)) {
      uint32_t* a = &sm.acc[0][0][0] + 6 * tid;
      run = ef_add(run, acc_value(a));
#pragma unroll
      for (int y = 0; y < 6; ++y) a[y] = 0;
    }
  }
  if (!final) {
    if (tid < r * (D + 1))
      jb.part[(size_t)(t0 + tid / (D + 1)) * stride + (size_t)blockIdx.x * (D + 1) +
              tid % (D + 1)] = run;
    return;
  }
  if (tid < r * (D + 1)) jb.rounds[(size_t)t0 * (D + 1) + tid] = run;
  if (tid == 0) {
    const unsigned off = T - 2;
    if (BIN) {
      jb.fin[0] = sm.sv[0][off];
      jb.fin[1] = ef_sub(sm.sv[0][off], ef_one());
#pragma unroll
      for (int j = 1; j < S; ++j) jb.fin[j + 1] = sm.sv[j][off];
    } else {
#pragma unroll
      for (int j = 0; j < S; ++j) jb.fin[j] = sm.sv[j][off];
    }
  }
  if (warp != 0 || t0 == 0) return;
  // The claim chain of the passes' rounds: with g_t(r) = sum_q L_q(r) g_t(q), claim_{t+1} = A_t +
  // L_1(r_t) claim_t, A_t collecting the other terms (and A_0 = g_0(r_0), whose g(1) is summed).
  // Lane t prepares round t's map and an inclusive scan of the compositions gives every lane
  // claim_{t+1}; claim_t is the previous lane's.
  static_assert(SC_MAX_K - SC_LOG_T <= 32, "a lane per round of the passes");
  const unsigned t = lane;
  ef2 a = ef_zero(), w1 = ef_one(), g0 = ef_zero();
  if (t < t0) {
    g0 = cs.g[t][0];
    w1 = t ? cs.w[t][1] : ef_zero();
    a = ef_mul_ol(ef_sub(cs.w[t][0], w1), g0);
    for (int q = t ? 2 : 1; q <= D; ++q) a = ef_add(a, ef_mul_ol(cs.w[t][q], cs.g[t][q]));
  }
  for (unsigned off = 1; off < t0; off <<= 1) {
    const ef2 pa = ef_make(__shfl_up_sync(0xffffffffu, a.c0, off),
                           __shfl_up_sync(0xffffffffu, a.c1, off));
    const ef2 pw = ef_make(__shfl_up_sync(0xffffffffu, w1.c0, off),
                           __shfl_up_sync(0xffffffffu, w1.c1, off));
    if (lane >= off) {
      a = ef_add(a, ef_mul_ol(w1, pa));
      w1 = ef_mul_ol(w1, pw);
    }
  }
  const ef2 claim = ef_make(__shfl_up_sync(0xffffffffu, a.c0, 1),
                            __shfl_up_sync(0xffffffffu, a.c1, 1));  // claim_t, from t = 1 on
  if (t < t0) {
    ef2* out = jb.rounds + (size_t)t * (D + 1);
    out[0] = g0;
    out[1] = t ? ef_sub(claim, g0) : cs.g[0][1];
#pragma unroll
    for (int q = 2; q <= D; ++q) out[q] = cs.g[t][q];
  }
}

// Rounds t0, .. of blockIdx.y's sumcheck on vectors of `len` entries: a thread owns the entries
// i + m len / 2^R whose folds meet, holds them in registers, and keeps its sums there to the end.
// What bounds it is its products again (first pass over two factors of 2^24: 345 us, ALU pipe 66 %
// busy, DRAM 23 %).
template <int D>
__global__ void __launch_bounds__(SC_STREAM_THREADS, 2)
    sc_stream_kernel(const ScJobs<D> jobs, size_t len, unsigned t0, size_t stride) {
  constexpr int R = SC_STREAM_R;
  __shared__ uint32_t acc[R][D + 1][6];
  const ScOne<D> jb = my_job(jobs);
  const unsigned tid = threadIdx.x, lane = tid & 31;
  if (tid < sizeof(acc) / 4) (&acc[0][0][0])[tid] = 0;
  ef2 run[R][D + 1];
#pragma unroll
  for (int l = 0; l < R; ++l)
#pragma unroll
    for (int q = 0; q <= D; ++q) run[l][q] = ef_zero();
  const size_t step = len >> R;
  for (size_t i = (size_t)blockIdx.x * SC_STREAM_THREADS + tid; i < step;
       i += (size_t)gridDim.x * SC_STREAM_THREADS) {
    ef2 x[D][1 << R];
#pragma unroll
    for (int j = 0; j < D; ++j)
#pragma unroll
      for (int m = 0; m < 1 << R; ++m) x[j][m] = ((const ef2*)jb.src[j])[i + m * step];
#pragma unroll
    for (int l = 0; l < R; ++l) {
      const ef2 rt = jb.ch[t0 + l];
      const int h = 1 << (R - 1 - l);
#pragma unroll
      for (int m = 0; m < h; ++m) {
        ef2 v[D], df[D];
#pragma unroll
        for (int j = 0; j < D; ++j) {
          v[j] = x[j][m], df[j] = ef_sub(x[j][m + h], v[j]);
          x[j][m] = ef_add(v[j], ef_mul(rt, df[j]));
        }
#pragma unroll
        for (int q = 0; q <= D; ++q) {
          if (q != 1 || t0 + l == 0) {  // later rounds' g(1): from the claim chain
            ef2 pr = v[0];
#pragma unroll
            for (int j = 1; j < D; ++j) pr = ef_mul(pr, v[j]);
            run[l][q] = ef_add(run[l][q], pr);
          }
          if (q < D)
#pragma unroll
            for (int j = 0; j < D; ++j) v[j] = ef_add(v[j], df[j]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < D; ++j) jb.dst[j][i] = x[j][0];
  }
  __syncthreads();  // acc is clear
#pragma unroll
  for (int l = 0; l < R; ++l)
#pragma unroll
    for (int q = 0; q <= D; ++q) warp_add(run[l][q], acc[l][q], lane);
  __syncthreads();
  if (tid < R * (D + 1))
    jb.part[(size_t)(t0 + tid / (D + 1)) * stride + (size_t)blockIdx.x * (D + 1) +
            tid % (D + 1)] = acc_value(&acc[0][0][0] + 6 * tid);
}

template <int D, bool BIN>
void sumcheck_run(const ScJob* js, unsigned njobs, unsigned k, cudaStream_t st,
                  unsigned max_blocks) {
  constexpr int S = Fac<D, BIN>::S;
  const unsigned cap = (max_blocks && max_blocks < SC_MAX_BLOCKS) ? max_blocks : SC_MAX_BLOCKS;
  const size_t stride = (size_t)SC_MAX_BLOCKS * (D + 1);
  ScJobs<S> jobs;
  for (unsigned y = 0; y < njobs; ++y) {
    for (int j = 0; j < S; ++j) {
      jobs.j[y].src[j] = js[y].src[j];
      jobs.j[y].dst[j] = js[y].dst[j];
    }
    jobs.j[y].ch = js[y].ch;
    jobs.j[y].rounds = js[y].rounds;
    jobs.j[y].fin = js[y].fin;
    jobs.j[y].part = js[y].partials;
  }
  auto kern = sc_tile_kernel<D, BIN>;
  static_assert(SC_THREADS == 1u << (SC_LOG_T - 1), "one pair of a tile per thread");
  static_assert(SC_MAX_PASSES >= (SC_MAX_K - SC_STREAM_LOG + SC_STREAM_R) / SC_STREAM_R +
                                     (SC_STREAM_LOG - 1 - SC_LOG_T + SC_MAX_R - 1) / SC_MAX_R &&
                    SC_MAX_PASSES >= (SC_MAX_K - SC_LOG_T + SC_MAX_R - 1) / SC_MAX_R,
                "every plan fits ScPasses");
  constexpr size_t smem = sizeof(TileSmem<D, BIN>), smem_end = smem + sizeof(ChainSmem<D>);
  LGS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_end));
  ScPasses prev{};
  int bf0 = js[0].bf0;
  unsigned t = 0;
  while (k - t > SC_LOG_T) {
    const size_t len = (size_t)1 << (k - t);
    unsigned r = 0, nb = 0;
    if constexpr (D <= 2 && !BIN)
      if (k - t >= SC_STREAM_LOG && !bf0) {
        r = SC_STREAM_R;
        nb = cap;  // far fewer than the vector's threads
        sc_stream_kernel<D><<<dim3(nb, njobs), SC_STREAM_THREADS, 0, st>>>(jobs, len, t, stride);
      }
    if (!r) {  // passes of about equally many rounds, down to one tile
      const unsigned left = k - t - SC_LOG_T, np = (left + SC_MAX_R - 1) / SC_MAX_R;
      r = (left + np - 1) / np;
      nb = (unsigned)std::min<size_t>(cap, len >> SC_LOG_T);
      kern<<<dim3(nb, njobs), SC_THREADS, smem, st>>>(jobs, len, SC_LOG_T, r, t, bf0, 0, stride,
                                                      prev);
    }
    LGS_LAUNCH_CHECK();
    t += r;
    prev.t[prev.n] = t;
    prev.nb[prev.n++] = nb;
    for (unsigned y = 0; y < njobs; ++y)
      for (int j = 0; j < S; ++j) jobs.j[y].src[j] = jobs.j[y].dst[j];
    bf0 = 0;
  }
  tl_mark("sc_passes_end", st);
  kern<<<dim3(1, njobs), SC_THREADS, smem_end, st>>>(jobs, (size_t)1 << (k - t), k - t, k - t, t,
                                                     bf0, 1, stride, prev);
  LGS_LAUNCH_CHECK();
}
}  // namespace

size_t sumcheck_partials_elems(unsigned k, unsigned d) {
  return (size_t)(k ? k : 1) * SC_MAX_BLOCKS * (d + 1);
}

void sumcheck_jobs_dev(const ScJob* jobs, unsigned njobs, unsigned d, unsigned k, cudaStream_t st,
                       unsigned max_blocks) {
  if (k == 0) throw ShapeError("sumcheck: zero variables");
  if (k > SC_MAX_K) throw ShapeError("sumcheck: too many variables");
  if (njobs < 1 || njobs > SC_MAX_JOBS) throw ShapeError("sumcheck: too many at once");
  for (unsigned y = 1; y < njobs; ++y)
    if (jobs[y].bf0 != jobs[0].bf0 || jobs[y].binary != jobs[0].binary)
      throw ShapeError("sumcheck: sumchecks of one launch must be alike");
  if (jobs[0].binary) {
    if (d != 3) throw ShapeError("sumcheck: the binary check has three factors");
    return sumcheck_run<3, true>(jobs, njobs, k, st, max_blocks);
  }
  switch (d) {
    case 1: return sumcheck_run<1, false>(jobs, njobs, k, st, max_blocks);
    case 2: return sumcheck_run<2, false>(jobs, njobs, k, st, max_blocks);
    case 3: return sumcheck_run<3, false>(jobs, njobs, k, st, max_blocks);
    default: throw ShapeError("sumcheck: 1 to 3 factors supported");
  }
}

void sumcheck_prove_dev(ef2* const* polys, unsigned d, unsigned k, const ef2* ch, ef2* rounds_out,
                        ef2* final_out, ef2* partials, cudaStream_t st, unsigned max_blocks) {
  if (d < 1 || d > 3) throw ShapeError("sumcheck: 1 to 3 factors supported");
  ScJob j{};
  for (unsigned i = 0; i < d; ++i) j.src[i] = j.dst[i] = polys[i];
  j.ch = ch, j.rounds = rounds_out, j.fin = final_out, j.partials = partials;
  sumcheck_jobs_dev(&j, 1, d, k, st, max_blocks);
}

}  // namespace lgs
