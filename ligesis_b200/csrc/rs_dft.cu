// Batched Reed-Solomon encoding of the commitment rows: out[j] = sum_k in[k] g_N^(jk) for every
// row (p3-dft's `Radix2Dit::dft` in natural order, pcs/src/ligesis.rs:222-235), for
// N = 2^12 .. 2^20 with the row zero-padded from N/2 (rate 1/2), N/4 or N/8 values, or full.
//
// Four-step split N = 4096 * N2, k = k1 N2 + k2, j = j1 + 4096 j2:
//   X[j1 + 4096 j2] = sum_k2 w_N2^(j2 k2) w_N^(j1 k2) sum_k1 x[k1 N2 + k2] w_4096^(j1 k1)
// pass A  the 4096-point DFTs over k1 of 1, 2 or 4 consecutive columns k2 per CTA, as 64 x 64, each
//         64-point DFT as radix-8 x radix-8 shared by 8 warps (one radix-8 per thread, a
//         shared-memory exchange between the two), written as Z[k2][j1] (contiguous in j1).
//         Global reads are 32-byte runs with 4 columns; the zeros of a padded row are never
//         read.  N = 2^12 is finished here, and N = 2^13 too: a thread holds both columns of its row
//         at the end and does the last radix-2.
// pass B  the four-step twiddle w_N^(j1 k2) from a table laid out [k2][j1], then the N2-point
//         DFT over k2; reads Z and writes X in 256-byte runs per warp.  N2 <= 32: one thread per
//         column, in registers.  N2 = 64: 8 warps on 32 columns, an exchange between two radix-8.
//         N2 = 128, 256: N2 / 64 such 64-point DFTs and a radix-2 or -4 over them in registers.
// A radix-8 runs on 24-bit limbs (limb.cuh), so its roots of unity cost nothing.  Roots of order
// 64 and less between radix-8 digits are powers of two too, applied as shifts while the limbs are
// packed: the shift is a compile-time constant, so the warps of an exchange run one copy of it
// each.  Values in between are any representative below 2^64; the encoded row is canonical.
// What bounds both passes is the integer pipes (ALU and wide-multiply pipes about 70 % busy each).
#include <type_traits>

#include "kernels.cuh"
#include "limb.cuh"

namespace lgs {

namespace {

// w_64 = 2^RS_W64 mod p (the reference generator's order-64 root).
constexpr unsigned RS_W64 = 39;

// The second half of a 64-point DFT's first digit: ex[j][W][lane] = y[j] w_64^(j W), the twiddle
// after the radix-8 of warp W.
template <int W, int J = 0>
__device__ __forceinline__ void tw64_store(const Limbs (&y)[8], u64* ex) {
  if constexpr (J < 8) {
    ex[(J * 8 + W) * 32] = limb_pack_shl<(RS_W64 * J * W) % 192>(y[J]);
    tw64_store<W, J + 1>(y, ex);
  }
}
// Radix-8 of v by warp w of 8, the order-64 twiddles, and the exchange buffer (ex at this lane).
template <bool ZH>
__device__ __forceinline__ void dft64_first(const u64 (&v)[8], unsigned w, u64* ex) {
  Limbs y[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) y[i] = limb_unpack(v[ZH ? i % 4 : i]);
  limb_dft<8, ZH>(y);
  switch (w) {
    case 0: tw64_store<0>(y, ex); break;
    case 1: tw64_store<1>(y, ex); break;
    case 2: tw64_store<2>(y, ex); break;
    case 3: tw64_store<3>(y, ex); break;
    case 4: tw64_store<4>(y, ex); break;
    case 5: tw64_store<5>(y, ex); break;
    case 6: tw64_store<6>(y, ex); break;
    default: tw64_store<7>(y, ex); break;
  }
}

// ---- pass A: the 4096-point column DFTs of COLS columns, COLS groups of 8 warps ----------------
// k1 = a + 64 b, a = a0 + 8 a1, b = b0 + 8 b1 (all digits < 8).  Phase 1, per group and round:
// 32 lane-columns (c, a) with lane = c + COLS (a mod 32/COLS); warp w holds b0 = w and does the
// radix-8 over b1, multiplies by w_64^(jb1 b0), and exchanges through shared memory so that warp w
// then holds jb1 = w and does the radix-8 over b0: j' = jb1 + 8 jb0 is the 64-point output over b.
// After the w_4096^(j' a) twiddle the values go to the column tile big[c][j'][a].  Phase 2 does
// the same over a for lane-columns (c, j') and writes j1 = j' + 64 (ja1 + 8 ja0).  Two rounds per
// group in each phase; a CTA of 4 columns has 32 warps (64 registers each): with 16 warps of 128
// registers the passes' loads and barriers were less covered (2^18: 0.292 -> 0.265 ms).
constexpr int PA_JS = 65;    // big[] stride of j' (odd: conflict-free phase-2 reads)
constexpr int PA_CS = 4164;  // big[] stride of a column (= 4 mod 16: conflict-free phase-1 stores)
constexpr size_t pa_smem(int cols) { return (size_t)cols * (PA_CS + 2048) * 8; }
// where the column DFTs go: Z, the finished rows of N = 2^12, or through the last radix-2 of 2^13
enum PaTail { PA_Z, PA_ROW, PA_ROW2 };

__device__ __forceinline__ void group_sync(unsigned grp) {
  asm volatile("bar.sync %0, 256;" ::"r"(1 + grp) : "memory");
}

template <bool HALF, int COLS, PaTail TAIL>
__global__ void __launch_bounds__(256 * COLS, 4 / COLS)
    rs_pass_a_kernel(const u64* __restrict__ in, size_t ld_in, u64* __restrict__ z, size_t ld_out,
                     unsigned log_n2, size_t ncols, unsigned nb1,
                     const u64* __restrict__ tw4096, const u64* __restrict__ t4) {
  extern __shared__ u64 sm[];
  u64* big = sm;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned grp = warp >> 3, w = warp & 7;
  u64* ex = sm + COLS * PA_CS + grp * 2048 + lane;  // [jb][w][lane]
  const size_t g0 = (size_t)blockIdx.x * COLS;      // columns are numbered row N2 + k2
  constexpr int APR = 32 / COLS;                    // values of a per round and group

  // phase 1 inputs of this thread's two rounds, loaded up front (b1 < nb1 <= NB1 are not zero)
  constexpr int NB1 = HALF ? 4 : 8;
  const unsigned c = lane % COLS, al = lane / COLS;
  u64 pre[2][NB1];
  {
    const size_t g = min(g0 + c, ncols - 1);  // a ragged last CTA repeats the last column
    const u64* src = in + (g >> log_n2) * ld_in + (g & (((size_t)1 << log_n2) - 1));
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const unsigned a = APR * (grp + COLS * i) + al;
      const u64* s = src + ((size_t)(a + 64 * w) << log_n2);
#pragma unroll
      for (int b1 = 0; b1 < NB1; ++b1)
        pre[i][b1] = !HALF || b1 < (int)nb1 ? __ldg(s + ((size_t)b1 << (9 + log_n2))) : 0;
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const unsigned a = APR * (grp + COLS * i) + al;
    u64 v[8];
#pragma unroll
    for (int b1 = 0; b1 < 8; ++b1) v[b1] = pre[i][b1 % NB1];
    dft64_first<HALF>(v, w, ex);
    group_sync(grp);
#pragma unroll
    for (int b0 = 0; b0 < 8; ++b0) v[b0] = ex[(w * 8 + b0) * 32];
    dft_lazy<8>(v);
#pragma unroll
    for (int j0 = 0; j0 < 8; ++j0) {
      const unsigned jp = w + 8 * j0;
      big[c * PA_CS + jp * PA_JS + a] = gl_mul_lazy(v[j0], __ldg(tw4096 + jp * a));
    }
    group_sync(grp);
  }
  __syncthreads();
  u64 first[TAIL == PA_ROW2 ? 8 : 1];
#pragma unroll 1
  for (unsigned i = 0; i < 2; ++i) {
    // (column, half of j') of this round; the two columns of a 2^13-point row go to one thread
    const unsigned r = TAIL == PA_ROW2 ? (grp & ~1u) * 2 + 2 * i + (grp & 1) : grp + COLS * i;
    const unsigned cc = r >> 1, jp = 32 * (r & 1) + lane;
    u64 v[8];
    const u64* s = big + cc * PA_CS + jp * PA_JS + w;
#pragma unroll
    for (int a1 = 0; a1 < 8; ++a1) v[a1] = s[8 * a1];
    dft64_first<false>(v, w, ex);
    group_sync(grp);
#pragma unroll
    for (int a0 = 0; a0 < 8; ++a0) v[a0] = ex[(w * 8 + a0) * 32];
    dft_lazy<8>(v);
    const size_t g = g0 + cc;
    if constexpr (TAIL == PA_Z) {
      u64* dst = z + g * 4096 + jp + 64 * w;
      if (g < ncols)
#pragma unroll
        for (int j0 = 0; j0 < 8; ++j0) dst[512 * j0] = v[j0];
    } else if constexpr (TAIL == PA_ROW) {
      u64* dst = z + g * ld_out + jp + 64 * w;
      if (g < ncols)
#pragma unroll
        for (int j0 = 0; j0 < 8; ++j0) dst[512 * j0] = gl_canon(v[j0]);
    } else {
      if (i == 0) {
#pragma unroll
        for (int j0 = 0; j0 < 8; ++j0) first[j0] = v[j0];
      } else if (g < ncols) {
        u64* dst = z + (g >> 1) * ld_out + jp + 64 * w;
        const u64* t = t4 + 4096 + jp + 64 * w;
#pragma unroll
        for (int j0 = 0; j0 < 8; ++j0) {
          const u64 x = gl_canon(first[j0]), y = gl_mul(v[j0], __ldg(t + 512 * j0));
          dst[512 * j0] = gl_add(x, y);
          dst[512 * j0 + 4096] = gl_sub(x, y);
        }
      }
    }
    group_sync(grp);
  }
}

// ---- pass B, N2 = 64 R: 8 warps on 32 consecutive j1 of one row --------------------------------
// k2 = c + R k', j2 = j' + 64 jc.  For each c < R the 64-point DFT over k' = ka + 8 kb: warp w = ka
// loads Z[k2][j1] (256-byte rows), applies w_N^(j1 k2), does the radix-8 over kb, multiplies by
// w_64^(jb ka), exchanges, and as jb = w does the radix-8 over ka: it then holds j' = w + 8 j0.
// With R > 1 the outputs are multiplied by w_N2^(c j') and all but the last kept in the thread's
// own slots of shared memory; a thread holds one j' for every c, so the radix-R over c needs no
// exchange.  The loop over c is not unrolled: four copies of the eight warps' code missed the
// instruction cache (2^20, 32 rows: 0.341 ms unrolled, 0.210 ms as it is).
constexpr size_t pb64_smem(int r) { return (size_t)(8 * 8 * 32 + (r - 1) * 8 * 256) * 8; }
template <int R>
__global__ void __launch_bounds__(256, R <= 2 ? 4 : 3)
    rs_pass_b64_kernel(const u64* __restrict__ z, u64* __restrict__ out, size_t ld_out,
                       const u64* __restrict__ t4, const u64* __restrict__ tw4096) {
  extern __shared__ u64 sm[];
  const unsigned lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  u64* ex = sm + lane;
  u64* keep = sm + 2048 + threadIdx.x;  // [c][j0][thread]
  const unsigned j1 = blockIdx.x * 32 + lane;
  const size_t row = blockIdx.y;
  const u64* src = z + row * ((size_t)64 * R * 4096) + j1;
  u64 v[8];
#pragma unroll 1
  for (int c = 0; c < R; ++c) {
#pragma unroll
    for (int kb = 0; kb < 8; ++kb) v[kb] = src[(size_t)(c + R * (w + 8 * kb)) * 4096];
#pragma unroll
    for (int kb = 0; kb < 8; ++kb)
      v[kb] = gl_mul_lazy(v[kb], __ldg(t4 + (c + R * (w + 8 * kb)) * 4096 + j1));
    if (c > 0) __syncthreads();
    dft64_first<false>(v, w, ex);
    __syncthreads();
#pragma unroll
    for (int ka = 0; ka < 8; ++ka) v[ka] = ex[(w * 8 + ka) * 32];
    dft_lazy<8>(v);
    if constexpr (R > 1) {
#pragma unroll
      for (int j0 = 0; j0 < 8; ++j0)
        v[j0] = gl_mul_lazy(v[j0], __ldg(tw4096 + (64 / R) * c * (w + 8 * j0)));
      if (c + 1 < R)
#pragma unroll
        for (int j0 = 0; j0 < 8; ++j0) keep[(c * 8 + j0) * 256] = v[j0];
    }
  }
  u64* dst = out + row * ld_out + j1;
  if constexpr (R == 1) {
#pragma unroll
    for (int j0 = 0; j0 < 8; ++j0) dst[(size_t)(w + 8 * j0) * 4096] = gl_canon(v[j0]);
  } else {
#pragma unroll
    for (int j0 = 0; j0 < 8; ++j0) {
      u64 x[R];
#pragma unroll
      for (int c = 0; c + 1 < R; ++c) x[c] = keep[(c * 8 + j0) * 256];
      x[R - 1] = v[j0];
      dft_lazy<R>(x);
#pragma unroll
      for (int jc = 0; jc < R; ++jc)
        dst[(size_t)(w + 8 * j0 + 64 * jc) * 4096] = gl_canon(x[jc]);
    }
  }
}

// ---- pass B for N2 = 4 .. 32: one thread per column, in registers ------------------------------
// N2 = A B, k2 = c + B k', j2 = j' + A jc: an A-point DFT over k' for each c, its outputs times
// w_N2^(c j') (a power of two: a shift as the limbs are packed), then a B-point DFT over c.
constexpr int PB_THREADS = 128;

template <int A, int B, int C, unsigned EL, int J = 0>
__device__ __forceinline__ void tw_pack(const Limbs (&y)[A], u64 (&r)[A][B]) {
  if constexpr (J < A) {
    r[J][C] = limb_pack_shl<(EL * C * J) % 192>(y[J]);
    tw_pack<A, B, C, EL, J + 1>(y, r);
  }
}
template <int A, int B, unsigned EL, int C = 0>
__device__ __forceinline__ void pass_b_first(const u64* src, const u64* t4, u64 (&r)[A][B]) {
  if constexpr (C < B) {
    Limbs y[A];
#pragma unroll
    for (int k = 0; k < A; ++k) {
      const size_t o = (size_t)(C + B * k) * 4096;
      y[k] = limb_unpack(C + B * k == 0 ? src[0] : gl_mul_lazy(src[o], __ldg(t4 + o)));
    }
    limb_dft<A>(y);
    tw_pack<A, B, C, EL>(y, r);
    pass_b_first<A, B, EL, C + 1>(src, t4, r);
  }
}

template <int LOGL>
__global__ void __launch_bounds__(PB_THREADS)
    rs_pass_b_kernel(const u64* __restrict__ z, u64* __restrict__ out, size_t ld_out,
                     const u64* __restrict__ t4) {
  constexpr int L = 1 << LOGL, A = LOGL == 2 ? 4 : 8, B = L / A;
  constexpr unsigned EL = LOGL == 5 ? 78 : 156;  // w_32, w_16 = 2^EL
  const unsigned j1 = blockIdx.x * PB_THREADS + threadIdx.x;
  const size_t row = blockIdx.y;
  u64 r[A][B];
  pass_b_first<A, B, EL>(z + row * ((size_t)L * 4096) + j1, t4 + j1, r);
  u64* dst = out + row * ld_out + j1;
#pragma unroll
  for (int j = 0; j < A; ++j) {
    if constexpr (B > 1) dft_lazy<B>(r[j]);
#pragma unroll
    for (int jc = 0; jc < B; ++jc) dst[(size_t)(j + A * jc) * 4096] = gl_canon(r[j][jc]);
  }
}

// tables[0 .. 4096) = w_4096^e; the four-step table of each logN at rs_table_offset(logN):
// T[k2 * 4096 + j1] = w_N^(j1 k2) for k2 < N / 4096.
__global__ void rs_tables_kernel(u64* tables, const u64* __restrict__ tw, size_t total) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  if (i < 4096) {
    tables[i] = tw[i << (TW_LOG - 12)];
    return;
  }
  unsigned logN = RS_LOGN_MIN + 1;
  size_t off = 4096;
  while (off + ((size_t)1 << logN) <= i) off += (size_t)1 << logN++;
  const size_t e = i - off, k2 = e >> 12, j1 = e & 4095;
  tables[i] = tw[(j1 * k2) << (TW_LOG - logN)];
}

template <bool HALF, int COLS, PaTail TAIL>
void launch_a(const u64* in, size_t ld_in, u64* z, size_t ld_out, unsigned log_n2, size_t ncols,
              unsigned nb1, const u64* tw4096, const u64* t4, cudaStream_t st) {
  auto k = rs_pass_a_kernel<HALF, COLS, TAIL>;
  LGS_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)pa_smem(COLS)));
  k<<<cdiv(ncols, COLS), 256 * COLS, pa_smem(COLS), st>>>(in, ld_in, z, ld_out, log_n2, ncols,
                                                          nb1, tw4096, t4);
  LGS_LAUNCH_CHECK();
}
// 4 columns per CTA read 32-byte runs; fewer columns make more, smaller CTAs, for transforms that
// would otherwise leave SMs idle.
template <bool HALF, PaTail TAIL>
void launch_a_cols(const u64* in, size_t ld_in, u64* z, size_t ld_out, unsigned log_n2,
                   size_t ncols, unsigned nb1, const u64* tw4096, const u64* t4,
                   cudaStream_t st) {
  if (ncols >= 4 * 148)
    launch_a<HALF, 4, TAIL>(in, ld_in, z, ld_out, log_n2, ncols, nb1, tw4096, t4, st);
  else if (ncols >= 2 * 148 || TAIL == PA_ROW2)
    launch_a<HALF, 2, TAIL>(in, ld_in, z, ld_out, log_n2, ncols, nb1, tw4096, t4, st);
  else if constexpr (TAIL != PA_ROW2)
    launch_a<HALF, 1, TAIL>(in, ld_in, z, ld_out, log_n2, ncols, nb1, tw4096, t4, st);
}

template <int LOGL>
void launch_b(const u64* z, u64* out, size_t ld_out, size_t rows, const u64* t4, cudaStream_t st) {
  dim3 grid(4096 / PB_THREADS, (unsigned)rows);
  rs_pass_b_kernel<LOGL><<<grid, PB_THREADS, 0, st>>>(z, out, ld_out, t4);
  LGS_LAUNCH_CHECK();
}
template <int R>
void launch_b64(const u64* z, u64* out, size_t ld_out, size_t rows, const u64* t4,
                const u64* tw4096, cudaStream_t st) {
  auto k = rs_pass_b64_kernel<R>;
  LGS_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)pb64_smem(R)));
  dim3 grid(4096 / 32, (unsigned)rows);
  k<<<grid, 256, pb64_smem(R), st>>>(z, out, ld_out, t4, tw4096);
  LGS_LAUNCH_CHECK();
}

// ---- the arithmetic floor of the encoding: its operations with no memory traffic -------------
// op 0: one radix-8 DFT (dft_lazy, as every stage of both passes) per iteration; op 1: eight
// independent twiddle multiplications (gl_mul_lazy) per iteration.  Eight values per thread, a
// checksum to `sink` so nothing is optimised away.
__global__ void __launch_bounds__(256) rs_alu_floor_kernel(unsigned iters, int op, u64* sink) {
  const u64 seed = 0x9E3779B97F4A7C15ull * (blockIdx.x * blockDim.x + threadIdx.x + 1);
  u64 v[8], t[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[j] = gl_canon(seed + 0x632BE59BD9B4E019ull * j);
    t[j] = gl_canon(seed ^ (0xD1B54A32D192ED03ull * (j + 3)));
  }
  if (op == 0) {
#pragma unroll 1
    for (unsigned i = 0; i < iters; ++i) dft_lazy<8>(v);
  } else {
#pragma unroll 1
    for (unsigned i = 0; i < iters; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = gl_mul_lazy(v[j], t[j]);
  }
  u64 acc = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) acc ^= v[j];
  if (acc == 0x0123456789ABCDEFull) *sink = acc;  // practically never: keeps v live
}

}  // namespace

double rs_alu_rate(int op, unsigned iters, u64* sink, cudaStream_t st) {
  int dev = 0, sms = 0;
  LGS_CUDA(cudaGetDevice(&dev));
  LGS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  int per_sm = 1;
  LGS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, rs_alu_floor_kernel, 256, 0));
  const unsigned blocks = (unsigned)(sms * std::max(1, per_sm));
  cudaEvent_t e0, e1;
  LGS_CUDA(cudaEventCreate(&e0));
  LGS_CUDA(cudaEventCreate(&e1));
  double best = 0.0;
  for (int rep = 0; rep < 4; ++rep) {  // the first launch warms up; keep the best
    LGS_CUDA(cudaEventRecord(e0, st));
    rs_alu_floor_kernel<<<blocks, 256, 0, st>>>(iters, op, sink);
    LGS_LAUNCH_CHECK();
    LGS_CUDA(cudaEventRecord(e1, st));
    LGS_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    LGS_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    const double ops = (double)blocks * 256 * iters * (op == 0 ? 1.0 : 8.0);
    if (rep > 0 && ms > 0) best = std::max(best, ops / (ms * 1e-3));
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return best;
}

size_t rs_table_offset(unsigned logN) {
  size_t off = 4096;
  for (unsigned l = RS_LOGN_MIN + 1; l < logN; ++l) off += (size_t)1 << l;
  return off;
}
size_t rs_tables_elems() { return rs_table_offset(RS_LOGN_MAX + 1); }

void build_rs_tables(u64* tables, const u64* tw, cudaStream_t st) {
  const size_t total = rs_tables_elems();
  rs_tables_kernel<<<cdiv(total, 256), 256, 0, st>>>(tables, tw, total);
  LGS_LAUNCH_CHECK();
}

bool rs_dft_supported(unsigned logN, size_t n_in) {
  const size_t N = (size_t)1 << logN;
  return logN >= RS_LOGN_MIN && logN <= RS_LOGN_MAX &&
         (n_in == N || 2 * n_in == N || 4 * n_in == N || 8 * n_in == N);
}

void rs_dft_rows(const u64* in, size_t ld_in, size_t n_in, u64* out, size_t ld_out,
                 unsigned logN, size_t rows, u64* z, const u64* tables, cudaStream_t st) {
  if (!rs_dft_supported(logN, n_in)) throw ShapeError("rs_dft_rows: unsupported size");
  if (rows == 0) return;
  if (logN > 13 && rows > 65535) throw ShapeError("rs_dft_rows: too many rows");
  const size_t N = (size_t)1 << logN;
  const unsigned log_n2 = logN - 12;
  const size_t ncols = rows << log_n2;
  const u64* t4 = log_n2 ? tables + rs_table_offset(logN) : nullptr;
  const bool half = n_in < N;
  const unsigned nb1 = (unsigned)(8 * n_in / N);  // nonzero values per radix-8 of the first stage
  auto pass_a = [&](auto tail, u64* dst) {
    constexpr PaTail T = decltype(tail)::value;
    if (half)
      launch_a_cols<true, T>(in, ld_in, dst, ld_out, log_n2, ncols, nb1, tables, t4, st);
    else
      launch_a_cols<false, T>(in, ld_in, dst, ld_out, log_n2, ncols, nb1, tables, t4, st);
  };
  if (log_n2 == 0) return pass_a(std::integral_constant<PaTail, PA_ROW>{}, out);
  if (log_n2 == 1) return pass_a(std::integral_constant<PaTail, PA_ROW2>{}, out);
  pass_a(std::integral_constant<PaTail, PA_Z>{}, z);
  switch (log_n2) {
    case 2: launch_b<2>(z, out, ld_out, rows, t4, st); break;
    case 3: launch_b<3>(z, out, ld_out, rows, t4, st); break;
    case 4: launch_b<4>(z, out, ld_out, rows, t4, st); break;
    case 5: launch_b<5>(z, out, ld_out, rows, t4, st); break;
    case 6: launch_b64<1>(z, out, ld_out, rows, t4, tables, st); break;
    case 7: launch_b64<2>(z, out, ld_out, rows, t4, tables, st); break;
    case 8: launch_b64<4>(z, out, ld_out, rows, t4, tables, st); break;
    default: throw ShapeError("rs_dft_rows: unsupported size");
  }
}

}  // namespace lgs
