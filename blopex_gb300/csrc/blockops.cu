// blockops.cu -- tall-skinny block kernels on column-major multivectors
// (CUDA-core versions, FP64 and FP32 storage):
//   Gram        G = X' Y          (serial_Multi_VectorInnerProd, multi_vector.c:354-406);
//               X' X of one block on the lower triangle only, bit-identical
//   X*C update  Y = X C [+ Z]     (serial_Multi_VectorByMatrix, multi_vector.c:474-524);
//               C upper triangular: the zero triangle skipped, bit-identical
//   axpby, column scaling, column dots, residual, precision conversion,
//   drand48 fill (multi_vector.c:165-184).
// Columns are addressed through blk_cols pointer tables, so masked
// (non-contiguous) columns and concatenated blocks [X R P] cost nothing.
// Split-k partial sums are reduced in a fixed order: results are
// deterministic run to run.
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>
#include <string.h>

#include "internal.h"
#include "pdl.cuh"
#include "blas32.cuh"

#define CUDA_LAUNCH_CHECK(ctx, what) gb_cuda_check((ctx), (int)cudaGetLastError(), (what))

static inline cudaStream_t S(gpu_Context* ctx) { return (cudaStream_t)ctx->stream; }

// ------------------------------------------------------------------------
// Gram: partial[s][j*h + i] = sum over rows of split s of X(r,i) * Y(r,j)
// 256 threads as 16 x 16; each thread owns a TM x TN register tile with
// rows ty + 16*a and columns tx + 16*b; rows are staged 32 at a time.
// FP32 inputs accumulate in FP32 over 128-row blocks, flushed to FP64.
// ------------------------------------------------------------------------
template <typename T, int TM, int TN>
__global__ void __launch_bounds__(256) gram_partial_kernel(blk_cols X, int h, blk_cols Y, int w,
                                                           long n, long rows_per_split,
                                                           double* __restrict__ partial)
{
  gb_pdl_entry();
  constexpr int BM = 16 * TM, BN = 16 * TN, RK = 32;
  __shared__ T xs[RK][BM + 1];
  __shared__ T ys[RK][BN + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int i0 = blockIdx.x * BM, j0 = blockIdx.y * BN;
  const long r_begin = (long)blockIdx.z * rows_per_split;
  const long r_end = min(n, r_begin + rows_per_split);

  double acc[TM][TN];
  T accs[TM][TN];
#pragma unroll
  for (int a = 0; a < TM; a++)
#pragma unroll
    for (int b = 0; b < TN; b++) {
      acc[a][b] = 0.0;
      accs[a][b] = T(0);
    }

  int chunk = 0;
  for (long r0 = r_begin; r0 < r_end; r0 += RK) {
    // stage rows r0..r0+RK of the BM columns of X and BN columns of Y
    for (int e = threadIdx.x; e < RK * BM; e += 256) {
      int rr = e % RK, cc = e / RK;
      long r = r0 + rr;
      int c = i0 + cc;
      T v = T(0);
      if (r < r_end && c < h) v = ((const T*)X.col[c])[r];
      xs[rr][cc] = v;
    }
    for (int e = threadIdx.x; e < RK * BN; e += 256) {
      int rr = e % RK, cc = e / RK;
      long r = r0 + rr;
      int c = j0 + cc;
      T v = T(0);
      if (r < r_end && c < w) v = ((const T*)Y.col[c])[r];
      ys[rr][cc] = v;
    }
    __syncthreads();
#pragma unroll 8
    for (int rr = 0; rr < RK; rr++) {
      T xv[TM], yv[TN];
#pragma unroll
      for (int a = 0; a < TM; a++) xv[a] = xs[rr][ty + 16 * a];
#pragma unroll
      for (int b = 0; b < TN; b++) yv[b] = ys[rr][tx + 16 * b];
#pragma unroll
      for (int a = 0; a < TM; a++)
#pragma unroll
        for (int b = 0; b < TN; b++) accs[a][b] = fma(xv[a], yv[b], accs[a][b]);
    }
    __syncthreads();
    if (sizeof(T) == 8 || (++chunk & 3) == 0) {
#pragma unroll
      for (int a = 0; a < TM; a++)
#pragma unroll
        for (int b = 0; b < TN; b++) {
          acc[a][b] += (double)accs[a][b];
          accs[a][b] = T(0);
        }
    }
  }
  double* out = partial + (size_t)blockIdx.z * h * w;
#pragma unroll
  for (int a = 0; a < TM; a++)
#pragma unroll
    for (int b = 0; b < TN; b++) {
      int i = i0 + ty + 16 * a, j = j0 + tx + 16 * b;
      if (i < h && j < w) out[(size_t)j * h + i] = acc[a][b] + (double)accs[a][b];
    }
}

// G from the partials, in a fixed order: 32 entries per CTA; 64 splits at a time
// are loaded by all its threads, then added in order by one thread an entry.
// A split's value is the sum of its `chunks` partials in order (nparts in all;
// chunks = 1: the split's own sum).  One thread an entry loading as it adds took
// 44 us for 304 splits of 8 x 8, a chain of loads and FP64 additions; this takes 20.
//   mode 0: entries e = j h + i of a full product
//   mode 1: e = i (i + 1) / 2 + j, the packed lower triangle of X'X
//   mode 2: the lower triangle of X'X at e = j h + i
static __device__ __forceinline__ void tri_index(int e, int* i, int* j)
{
  int r = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
  while (r * (r + 1) / 2 > e) r--;
  while ((r + 1) * (r + 2) / 2 <= e) r++;
  *i = r;
  *j = e - r * (r + 1) / 2;
}

__global__ void __launch_bounds__(256) gram_reduce_kernel(const double* __restrict__ partial, int splits, int chunks,
                                                          long nparts, int E, int h, int mode,
                                                          double* __restrict__ G, int ldg)
{
  gb_pdl_entry();
  __shared__ double sm[64][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int e0 = blockIdx.x * 32 + x;
  const int e = min(e0, E - 1);
  double s = 0.0;
  for (int base = 0; base < splits; base += 64) {
    const int cnt = min(64, splits - base);
    if (chunks == 1) {
#pragma unroll 8
      for (int q = y; q < cnt; q += 8) sm[q][x] = partial[(size_t)(base + q) * E + e];
    } else {
      for (int q = y; q < cnt; q += 8) {
        const long p0 = (long)(base + q) * chunks, p1 = min(p0 + chunks, nparts);
        double v = 0.0;
#pragma unroll 4
        for (long c = p0; c < p1; c++) v += partial[(size_t)c * E + e];
        sm[q][x] = v;
      }
    }
    __syncthreads();
    if (y == 0) {
#pragma unroll 8
      for (int q = 0; q < cnt; q++) s += sm[q][x];
    }
    __syncthreads();
  }
  if (y || e0 >= E) return;
  int i, j;
  if (mode == 1) {
    tri_index(e, &i, &j);
  } else {
    i = e % h;
    j = e / h;
    if (mode == 2 && i < j) return;
  }
  G[(size_t)j * ldg + i] = s;
  if (mode) G[(size_t)i * ldg + j] = s;
}

// FP64 Gram of narrow blocks: E <= 512 entries -- h w, or for X'X the h (h + 1) / 2
// of the lower triangle -- one to a thread, packed onto whole warps, since a
// warp-wide FP64 instruction occupies the pipe 16 cycles whatever its lane
// count: ceil(E / 32) of them per row, where a padded 32 x 32 tile spends 32.
// The threads left over form groups that take different 32-row chunks, each
// chunk's sum (32 FMAs in row order) being added to its entry's in chunk order
// afterwards.  With few splits the CTAs of a split (`sub` of them) leave that
// to the reduction, so that every SM has work.  Splits, chunks and the order of
// all sums are those of gram_partial_kernel: the results are its bits.  (Above
// 512 entries a thread's register tile wins: 32 x 32 65,536 rows 135 us against
// 160 with two packed entries a thread.)
//   8,000 x 10 x 10: 16 us with the reduction against 96 (padded tile, 28 CTAs);
//   262,144 x 8 x 8: 60 us against 504.
#define GRAMP_T 512
#define GRAMP_ROWS_SMEM (64 * 1024)                   // most of the staged rows (one group of 128 columns: 33 KB)
#define GRAMP_SMEM (GRAMP_ROWS_SMEM + 8 * GRAMP_T)  // and the groups' sums
template <bool SYM>
__global__ void __launch_bounds__(GRAMP_T) gram_packed_kernel(blk_cols X, int h, blk_cols Y, int w, long n,
                                                              long rows_per_split, int sub, int groups,
                                                              double* __restrict__ partial)
{
  gb_pdl_entry();
  extern __shared__ double sm[];  // [32 groups][h (+ w), odd stride], then [groups][E32]
  const int E = SYM ? h * (h + 1) / 2 : h * w, E32 = (E + 31) & ~31;
  const int nc = SYM ? h : h + w, ld = nc | 1, RS = 32 * groups;
  double* red = sm + RS * ld;
  const int t = threadIdx.x, g = t / E32, e = t - g * E32;
  const long chunks = rows_per_split / 32, per = (chunks + sub - 1) / sub;  // per split, per CTA
  const long split = blockIdx.x / sub;
  const long c0 = (long)(blockIdx.x % sub) * per, c1 = min(c0 + per, chunks);
  const long r_end = min(n, (split + 1) * rows_per_split);
  int xi, yj;
  if (SYM) {
    tri_index(min(e, E - 1), &xi, &yj);
  } else {
    xi = min(e, E - 1) % h;
    yj = h + min(e, E - 1) / h;
  }
  const bool live = g < groups && e < E;
  double acc = 0.0;
  for (long c = c0; c < c1; c += groups) {
    const long r0 = split * rows_per_split + 32 * c;
    if (r0 >= r_end) break;
    for (int q = t; q < RS * nc; q += GRAMP_T) {
      const int rr = q % RS, cc = q / RS;
      const double* col = (const double*)(cc < h ? X.col[cc] : Y.col[cc - h]);
      const long r = r0 + rr;
      sm[rr * ld + cc] = r < r_end ? col[r] : 0.0;
    }
    __syncthreads();
    if (live) {
      double a = 0.0;
      const double* row = sm + 32 * g * ld;
#pragma unroll 8
      for (int rr = 0; rr < 32; rr++, row += ld) a = fma(row[xi], row[yj], a);
      if (sub > 1) {
        if (c + g < c1 && r0 + 32 * g < r_end) partial[(size_t)(split * chunks + c + g) * E + e] = a;
      } else {
        red[g * E32 + e] = a;
      }
    }
    __syncthreads();
    if (sub == 1 && live && g == 0)
      for (int k = 0; k < groups && c + k < c1 && r0 + 32 * k < r_end; k++) acc += red[k * E32 + e];
  }
  if (sub == 1 && live && g == 0) partial[(size_t)split * E + e] = acc;
}

// Symmetric Gram X'X (h <= 64) on the lower triangle only.  Thread t owns
// the BS x BS block (bi, bj), bi >= bj, of the triangular numbering t =
// bi (bi + 1) / 2 + bj, so whole warps drop out of the upper triangle (a
// warp-wide FP64 instruction costs the same whatever its lane count).  Row
// splits, staging, the order of the multiply-adds into each entry and the
// flushes to FP64 are those of gram_partial_kernel, so every entry (and its
// mirror, as x_i x_j = x_j x_i exactly) is bit-identical to the full
// product's.
template <typename T, int BS>
__global__ void __launch_bounds__(544) gram_sym_partial_kernel(blk_cols X, int h, long n,
                                                               long rows_per_split,
                                                               double* __restrict__ partial)
{
  gb_pdl_entry();
  constexpr int BM = 32 * BS, RK = 32;
  __shared__ T xs[RK][BM + 1];
  const int t = threadIdx.x;
  const int nb = (h + BS - 1) / BS;
  const bool active = t < nb * (nb + 1) / 2;
  int bi = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
  while (bi * (bi + 1) / 2 > t) bi--;
  while ((bi + 1) * (bi + 2) / 2 <= t) bi++;
  const int bj = t - bi * (bi + 1) / 2;
  const long r_begin = (long)blockIdx.z * rows_per_split;
  const long r_end = min(n, r_begin + rows_per_split);

  double acc[BS][BS];
  T accs[BS][BS];
#pragma unroll
  for (int a = 0; a < BS; a++)
#pragma unroll
    for (int b = 0; b < BS; b++) {
      acc[a][b] = 0.0;
      accs[a][b] = T(0);
    }

  int chunk = 0;
  for (long r0 = r_begin; r0 < r_end; r0 += RK) {
    for (int e = t; e < RK * BM; e += blockDim.x) {
      int rr = e % RK, cc = e / RK;
      long r = r0 + rr;
      T v = T(0);
      if (r < r_end && cc < h) v = ((const T*)X.col[cc])[r];
      xs[rr][cc] = v;
    }
    __syncthreads();
    if (active) {
#pragma unroll 8
      for (int rr = 0; rr < RK; rr++) {
        T xv[BS], yv[BS];
#pragma unroll
        for (int a = 0; a < BS; a++) xv[a] = xs[rr][BS * bi + a];
#pragma unroll
        for (int b = 0; b < BS; b++) yv[b] = xs[rr][BS * bj + b];
#pragma unroll
        for (int a = 0; a < BS; a++)
#pragma unroll
          for (int b = 0; b < BS; b++) accs[a][b] = fma(xv[a], yv[b], accs[a][b]);
      }
    }
    __syncthreads();
    if (sizeof(T) == 8 || (++chunk & 3) == 0) {
#pragma unroll
      for (int a = 0; a < BS; a++)
#pragma unroll
        for (int b = 0; b < BS; b++) {
          acc[a][b] += (double)accs[a][b];
          accs[a][b] = T(0);
        }
    }
  }
  if (!active) return;
  double* out = partial + (size_t)blockIdx.z * h * h;
#pragma unroll
  for (int a = 0; a < BS; a++)
#pragma unroll
    for (int b = 0; b < BS; b++) {
      const int i = BS * bi + a, j = BS * bj + b;
      if (i < h && j <= i) out[(size_t)j * h + i] = acc[a][b] + (double)accs[a][b];
    }
}

// the row splits of gram_launch for a single (gx = gy = 1) output tile
static long gram_splits(gpu_Context* ctx, long n, long* rows)
{
  long splits = 2 * ctx->num_sms;
  long max_splits = (n + 255) / 256;
  if (splits > max_splits) splits = max_splits;
  if (splits < 1) splits = 1;
  long r = (n + splits - 1) / splits;
  r = (r + 31) / 32 * 32;
  splits = (n + r - 1) / r;
  if (splits < 1) splits = 1;
  *rows = r;
  return splits;
}

template <typename T, int BS>
static int gram_sym_launch(gpu_Context* ctx, long n, const blk_cols* X, int h, double* G, int ldg)
{
  long rows;
  const long splits = gram_splits(ctx, n, &rows);
  double* partial = (double*)gb_workspace(ctx, sizeof(double) * (size_t)splits * h * h);
  if (!partial) return -1;
  const int nb = (h + BS - 1) / BS;
  const int threads = (nb * (nb + 1) / 2 + 31) / 32 * 32;
  dim3 grid(1, 1, (unsigned)splits);
  gb_prof_rec pr;
  gb_prof_begin(ctx, &pr, sizeof(T) == 8 ? GB_K_GRAM : GB_K_GRAM32);
  gb_pdl(gram_sym_partial_kernel<T, BS>, grid, threads, 0, S(ctx), *X, h, n, rows, partial);
  gb_pdl(gram_reduce_kernel, (h * h + 31) / 32, 256, 0, S(ctx), partial, (int)splits, 1, splits, h * h, h, 2, G, ldg);
  gb_prof_end(ctx, &pr, (double)sizeof(T) * n * h, (double)n * h * (h + 1));
  gb_count_launch(2);
  return CUDA_LAUNCH_CHECK(ctx, "gram_sym");
}

template <typename T, int TM, int TN>
static int gram_launch(gpu_Context* ctx, long n, const blk_cols* X, int h, const blk_cols* Y,
                       int w, double* G, int ldg)
{
  constexpr int BM = 16 * TM, BN = 16 * TN;
  int gx = (h + BM - 1) / BM, gy = (w + BN - 1) / BN;
  int target = 2 * ctx->num_sms;
  long splits = target / (gx * gy);
  if (splits < 1) splits = 1;
  long max_splits = (n + 255) / 256;
  if (splits > max_splits) splits = max_splits;
  if (splits < 1) splits = 1;
  long rows = (n + splits - 1) / splits;
  rows = (rows + 31) / 32 * 32;
  splits = (n + rows - 1) / rows;
  if (splits < 1) splits = 1;
  double* partial = (double*)gb_workspace(ctx, sizeof(double) * (size_t)splits * h * w);
  if (!partial) return -1;
  dim3 grid(gx, gy, (unsigned)splits);
  gb_prof_rec pr;
  gb_prof_begin(ctx, &pr, sizeof(T) == 8 ? GB_K_GRAM : GB_K_GRAM32);
  gb_pdl(gram_partial_kernel<T, TM, TN>, grid, 256, 0, S(ctx), *X, h, *Y, w, n, rows, partial);
  int tot = h * w;
  gb_pdl(gram_reduce_kernel, (tot + 31) / 32, 256, 0, S(ctx), partial, (int)splits, 1, splits, tot, h, 0, G, ldg);
  gb_prof_end(ctx, &pr, (double)sizeof(T) * n * (h + w), 2.0 * n * h * w);
  gb_count_launch(2);
  return CUDA_LAUNCH_CHECK(ctx, "gram");
}

template <bool SYM>
static int gram_packed(gpu_Context* ctx, long n, const blk_cols* X, int h, const blk_cols* Y, int w, double* G, int ldg)
{
  long rows;
  const long splits = gram_splits(ctx, n, &rows), chunks = rows / 32;
  const int E = SYM ? h * (h + 1) / 2 : h * w, E32 = (E + 31) & ~31, nc = SYM ? h : h + w;
  int groups = GRAMP_T / E32;
  if (groups > chunks) groups = (int)chunks;
  while (groups > 1 && 32 * groups * (nc | 1) * 8 > GRAMP_ROWS_SMEM) groups /= 2;
  // few splits: several CTAs a split, each leaving its chunks' sums
  int sub = 1;
  if (splits <= ctx->num_sms) {
    const long most = (chunks + groups - 1) / groups, want = 4L * ctx->num_sms / splits;
    sub = (int)(want < most ? want : most);
  }
  const long nparts = sub > 1 ? (n + 31) / 32 : splits;
  double* partial = (double*)gb_workspace(ctx, sizeof(double) * (size_t)nparts * E);
  if (!partial) return -1;
  const int smem = 8 * (32 * groups * (nc | 1) + groups * E32);
  if (smem > 40 * 1024 &&  // (always the most: the limit is the function's, for all threads)
      cudaFuncSetAttribute(gram_packed_kernel<SYM>, cudaFuncAttributeMaxDynamicSharedMemorySize, GRAMP_SMEM) !=
          cudaSuccess)
    return gb_fail(ctx, "gram: cannot reserve %d bytes of shared memory", smem);
  gb_prof_rec pr;
  gb_prof_begin(ctx, &pr, GB_K_GRAM);
  gb_pdl(gram_packed_kernel<SYM>, (unsigned)(splits * sub), GRAMP_T, smem, S(ctx), *X, h, *Y, w, n, rows, sub, groups,
                                                                               partial);
  gb_pdl(gram_reduce_kernel, (E + 31) / 32, 256, 0, S(ctx), partial, (int)splits, sub > 1 ? (int)chunks : 1, nparts, E, h,
                                                        SYM ? 1 : 0, G, ldg);
  gb_prof_end(ctx, &pr, 8.0 * n * nc, SYM ? (double)n * h * (h + 1) : 2.0 * n * h * w);
  gb_count_launch(2);
  return CUDA_LAUNCH_CHECK(ctx, "gram_packed");
}

extern "C" int gb_gram(gpu_Context* ctx, int dtype, long n, const blk_cols* X, int h,
                       const blk_cols* Y, int w, double* G, int ldg)
{
  if (h <= 0 || w <= 0) return 0;
  // X'X with h <= 64 (one output tile): the lower triangle only
  const int sym = h == w && h <= 64 && memcmp(X->col, Y->col, sizeof(void*) * (size_t)h) == 0;
  if (dtype == GPU_MV_FLOAT64) {
    if (sym && h * (h + 1) / 2 <= GRAMP_T) return gram_packed<true>(ctx, n, X, h, Y, w, G, ldg);
    if (!sym && h * w <= GRAMP_T && h <= 64 && w <= 64) return gram_packed<false>(ctx, n, X, h, Y, w, G, ldg);
    if (sym)
      return h <= 32 ? gram_sym_launch<double, 1>(ctx, n, X, h, G, ldg)
                     : gram_sym_launch<double, 2>(ctx, n, X, h, G, ldg);
    if (h <= 32 && w <= 32) return gram_launch<double, 2, 2>(ctx, n, X, h, Y, w, G, ldg);
    return gram_launch<double, 4, 4>(ctx, n, X, h, Y, w, G, ldg);
  }
  if (sym)
    return h <= 32 ? gram_sym_launch<float, 1>(ctx, n, X, h, G, ldg)
                   : gram_sym_launch<float, 2>(ctx, n, X, h, G, ldg);
  if (h <= 32 && w <= 32) return gram_launch<float, 2, 2>(ctx, n, X, h, Y, w, G, ldg);
  return gram_launch<float, 4, 4>(ctx, n, X, h, Y, w, G, ldg);
}

// A caller's products (the interpreter's entry): large FP64 ones on the tensor cores
// (oz_gram64.cu), checked there against the bound of multiply-adds.  Those cost a
// row as much for all blocks whose 8-column units its eight producer warps hold at
// once (0.27 ns a row, 0.6 with two units a warp), the multiply-adds what their
// entries take (2.0 ps each; X'X half).  Measured, 2,097,152 rows, multiply-adds and
// tensor cores: 8 x 8 287 and 545 us, 16 x 8 552 and 561, 12 x 12 690 and 560, 16 x 16
// 1058 and 568 (X'X 676 and 556), 32 x 4 555 and 642, 32 x 32 5.5 ms and 696, 64 x 4 1102
// and 1221, 64 x 8 2138 and 1243, 64 x 64 14.6 ms and 1755.  The three launches take 30 us:
// 262,144 x 16 x 16 147 and 91, 20,000 x 32 x 32 89 and 40, x 64 x 4 31 and 49.  The solver
// keeps gb_gram: the signs of its Ritz vectors follow the last bits of these sums,
// and a solve returns the same iterates, bit for bit, as it always did.
#define GRAM_TENSOR_MIN 1e8
#define GRAM_TENSOR_ENTRIES 132

static int gram_on_tensor_cores(long n, int h, int w, int sym)
{
  const int units = (h + 7) / 8 + (sym ? 0 : (w + 7) / 8);
  return (double)n * h * w >= GRAM_TENSOR_MIN &&
         (sym ? h * (h + 1) / 2 : h * w) >= GRAM_TENSOR_ENTRIES * ((units + 7) / 8);
}

extern "C" int gb_gram_large(gpu_Context* ctx, int dtype, long n, const blk_cols* X, int h,
                             const blk_cols* Y, int w, double* G, int ldg, int* verdict)
{
  if (h <= 0 || w <= 0) return 0;
  const int sym = h == w && memcmp(X->col, Y->col, sizeof(void*) * (size_t)h) == 0;
  if (dtype != GPU_MV_FLOAT64 || !gram_on_tensor_cores(n, h, w, sym))
    return gb_gram(ctx, dtype, n, X, h, Y, w, G, ldg);
  gb_prof_rec pr;
  gb_prof_begin(ctx, &pr, GB_K_GRAM);
  const int rc = gb_oz_gram64(ctx, n, X, h, Y, w, sym, G, ldg, verdict);
  gb_prof_end(ctx, &pr, 8.0 * n * (sym ? h : h + w), sym ? (double)n * h * (h + 1) : 2.0 * n * h * w);
  return rc ? -1 : 1;
}

// ------------------------------------------------------------------------
// X*C update: Y(:, j0:j0+32) for 64 rows per CTA; thread t owns row t%64
// and 8 columns (t/64)*8 ... ; K staged 32 at a time in shared memory.
// tri: C is upper triangular with explicit zeros below the diagonal (a
// Cholesky-QR factor); a warp stops at its last column's diagonal, skipping
// only terms that add an exact zero, so Y is bit-identical to the full
// product.
// ------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) bymat_kernel(blk_cols X, int h, const double* __restrict__ C,
                                                    int ldc, blk_cols Y, int w, blk_cols Z,
                                                    int has_z, long n, int tri)
{
  gb_pdl_entry();
  constexpr int BM = 64, BN = 32, KC = 32;
  __shared__ T xs[KC][BM];
  __shared__ T cs[KC][BN];
  const int t = threadIdx.x;
  const int rl = t & 63, cg = t >> 6;
  const long r0 = (long)blockIdx.x * BM;
  const int j0 = blockIdx.y * BN;
  T acc[8];
#pragma unroll
  for (int b = 0; b < 8; b++) acc[b] = T(0);

  const int kmax = tri ? min(h, j0 + BN) : h;
  for (int k0 = 0; k0 < kmax; k0 += KC) {
    const int kc = min(KC, h - k0);  // (narrow blocks: no work on padding)
    for (int e = t; e < kc * BM; e += 256) {
      int rr = e % BM, kk = e / BM;
      long r = r0 + rr;
      T v = T(0);
      if (r < n) v = ((const T*)X.col[k0 + kk])[r];
      xs[kk][rr] = v;
    }
    for (int e = t; e < KC * BN; e += 256) {
      int kk = e % KC, jj = e / KC;
      T v = T(0);
      if (k0 + kk < h && j0 + jj < w) v = (T)C[(size_t)(j0 + jj) * ldc + k0 + kk];
      cs[kk][jj] = v;
    }
    __syncthreads();
    const int nb = min(8, w - j0 - cg * 8);  // this warp's columns
    const int kk_end = nb <= 0 ? 0 : (tri ? max(0, min(kc, j0 + cg * 8 + 8 - k0)) : kc);
#pragma unroll 8
    for (int kk = 0; kk < kk_end; kk++) {
      T xv = xs[kk][rl];
#pragma unroll
      for (int b = 0; b < 8; b++)
        if (b < nb) acc[b] = fma(xv, cs[kk][cg * 8 + b], acc[b]);
    }
    __syncthreads();
  }
  long r = r0 + rl;
  if (r < n) {
#pragma unroll
    for (int b = 0; b < 8; b++) {
      int j = j0 + cg * 8 + b;
      if (j < w) {
        T v = acc[b];
        if (has_z) v += ((const T*)Z.col[j])[r];
        ((T*)Y.col[j])[r] = v;
      }
    }
  }
}

static int bymat_launch(gpu_Context* ctx, int dtype, long n, const blk_cols* X, int h,
                        const double* C, int ldc, const blk_cols* Y, int w, const blk_cols* Z,
                        int tri)
{
  if (w <= 0 || n <= 0) return 0;
  dim3 grid((unsigned)((n + 63) / 64), (w + 31) / 32);
  blk_cols empty;
  const blk_cols* z = Z ? Z : &empty;
  const double es = dtype == GPU_MV_FLOAT64 ? 8.0 : 4.0;
  gb_prof_rec pr;
  gb_prof_begin(ctx, &pr, dtype == GPU_MV_FLOAT64 ? GB_K_XC : GB_K_XC32);
  if (dtype == GPU_MV_FLOAT64)
    gb_pdl(bymat_kernel<double>, grid, 256, 0, S(ctx), *X, h, C, ldc, *Y, w, *z, Z != NULL, n, tri);
  else
    gb_pdl(bymat_kernel<float>, grid, 256, 0, S(ctx), *X, h, C, ldc, *Y, w, *z, Z != NULL, n, tri);
  // a triangular C: sum over j of min(j + 1, h) products per row
  const double kw = tri ? (double)w * (w + 1) / 2 - (w > h ? (double)(w - h) * (w - h + 1) / 2 : 0.0)
                        : (double)h * w;
  gb_prof_end(ctx, &pr, es * n * (h + w + (Z ? w : 0)), 2.0 * n * kw);
  gb_count_launch(1);
  return CUDA_LAUNCH_CHECK(ctx, "bymat");
}

extern "C" int gb_bymat(gpu_Context* ctx, int dtype, long n, const blk_cols* X, int h,
                        const double* C, int ldc, const blk_cols* Y, int w, const blk_cols* Z)
{
  return bymat_launch(ctx, dtype, n, X, h, C, ldc, Y, w, Z, 0);
}

// Callers' updates (the interpreter's entries): large FP64 ones on the tensor cores
// (oz_xc64.cu), within the bound of multiply-adds.  Measured, 2,097,152 rows,
// multiply-adds and tensor cores: 4 x 16 336 and 899 us, 8 x 8 355 and 343, 10 x 10 614 and 333,
// 12 x 12 718 and 294, 16 x 4 534 and 243, 16 x 16 881 and 295, 32 x 32 3454 and 509, 64 x 4
// 2148 and 500, 64 x 64 13.8 ms and 1302; 65,536 x 12 x 12 35 and 20, 20,000 x 16 x 16 17 and 14, x 32 x 32
// 54 and 19.  From 12 input columns on, few of random entries are summed directly
// (8 columns: 3%, 12: 1%, 16: 0.3%); summed directly an entry costs up to three times its
// multiply-adds (32 x 32, C triangular, 3.1 ms; identity 5.8; 16 x 16 triangular
// 1.4; X's columns graded over 18 decades 3.9).  Hence the look at C: at most one column
// in eight may be of few values (its 1-norm below h / 8 of its largest).  And a launch
// of 64 x 64 columns takes 20 us at least, C's digits above all, 36 of them for 384 x
// 384: 3000 x 200 x 200 263 and 322, 6000 rows 576 and 330; 3000 x 384 x 384 1038 and 879,
// 1500 rows 411 and 878.  The solver keeps gb_bymat, for the reason given at
// gb_gram_large.
#define XC_TENSOR_MIN 1.6e7
#define XC_TENSOR_H 12
#define XC_TENSOR_ROWS 5000

static int update_on_tensor_cores(long n, int h, int w, const double* C, int ldc)
{
  if (h < XC_TENSOR_H || n < XC_TENSOR_ROWS || (double)n * h * w < XC_TENSOR_MIN) return 0;
  int sparse = 0;
  for (int j = 0; j < w; j++) {
    double sum = 0.0, big = 0.0;
    for (int i = 0; i < h; i++) {
      const double a = fabs(C[i + (size_t)j * ldc]);
      sum += a;
      big = a > big ? a : big;
    }
    sparse += !(sum * 8 >= big * h && big > 0.0);  // (zeros and NaN count as sparse)
  }
  return sparse * 8 <= w;
}

// whether a column of X shares memory with a column of Y (`bytes` long each)
extern "C" int gb_cols_overlap(const blk_cols* X, int h, const blk_cols* Y, int w, size_t bytes)
{
  uintptr_t lo = UINTPTR_MAX, hi = 0;  // Y's columns
  for (int j = 0; j < w; j++) {
    const uintptr_t y = (uintptr_t)Y->col[j];
    lo = y < lo ? y : lo;
    hi = y > hi ? y : hi;
  }
  for (int i = 0; i < h; i++) {
    const uintptr_t x = (uintptr_t)X->col[i];
    if (x >= hi + bytes || lo >= x + bytes) continue;
    for (int j = 0; j < w; j++) {
      const uintptr_t y = (uintptr_t)Y->col[j];
      if (x < y + bytes && y < x + bytes) return 1;
    }
  }
  return 0;
}

extern "C" int gb_bymat_large(gpu_Context* ctx, int dtype, long n, const blk_cols* X, int h,
                              const double* C, int ldc, const double* C_host, int ldch,
                              const blk_cols* Y, int w, const blk_cols* Z)
{
  if (w <= 0 || n <= 0) return 0;
  // (in place: gb_bymat, whose CTAs read all of their rows of X before they write;
  // the tensor-core kernel comes back to X for the entries that it sums directly)
  if (dtype != GPU_MV_FLOAT64 || h <= 0 || !update_on_tensor_cores(n, h, w, C_host, ldch) ||
      gb_cols_overlap(X, h, Y, w, sizeof(double) * (size_t)n))
    return gb_bymat(ctx, dtype, n, X, h, C, ldc, Y, w, Z);
  gb_prof_rec pr;
  gb_prof_begin(ctx, &pr, GB_K_XC);
  const int rc = gb_oz_bymat64(ctx, n, X, h, C, ldc, Y, w, Z);
  gb_prof_end(ctx, &pr, 8.0 * n * (h + w + (Z ? w : 0)), 2.0 * n * h * w);
  return rc ? -1 : 1;
}

extern "C" int gb_bymat_tri(gpu_Context* ctx, int dtype, long n, const blk_cols* X, int h,
                            const double* C, int ldc, const blk_cols* Y, int w)
{
  return bymat_launch(ctx, dtype, n, X, h, C, ldc, Y, w, NULL, 1);
}

// ------------------------------------------------------------------------
// elementwise column kernels: grid.y = column, grid-stride over rows
// ------------------------------------------------------------------------
template <typename T>
__global__ void axpby_kernel(blk_cols X, double alpha, blk_cols Y, double beta, long n)
{
  gb_pdl_entry();
  const T* x = (const T*)X.col[blockIdx.y];
  T* y = (T*)Y.col[blockIdx.y];
  const T a = (T)alpha, b = (T)beta;
  for (long r = blockIdx.x * (long)blockDim.x + threadIdx.x; r < n; r += (long)gridDim.x * blockDim.x) {
    if (beta == 0.0)
      y[r] = a * x[r];
    else
      y[r] = a * x[r] + b * y[r];
  }
}

static unsigned row_blocks(gpu_Context* ctx, long n, int w)
{
  long want = (n + 255) / 256;
  long cap = (long)ctx->num_sms * 8 / (w > 0 ? w : 1);
  if (cap < 4) cap = 4;
  if (want > cap) want = cap;
  if (want < 1) want = 1;
  return (unsigned)want;
}

extern "C" int gb_axpby(gpu_Context* ctx, int dtype, long n, double alpha, const blk_cols* X,
                        double beta, const blk_cols* Y, int w)
{
  if (w <= 0 || n <= 0) return 0;
  dim3 grid(row_blocks(ctx, n, w), w);
  gb_prof_rec pr;
  gb_prof_begin(ctx, &pr, GB_K_BLAS1);
  if (dtype == GPU_MV_FLOAT64)
    gb_pdl(axpby_kernel<double>, grid, 256, 0, S(ctx), *X, alpha, *Y, beta, n);
  else
    gb_pdl(axpby_kernel<float>, grid, 256, 0, S(ctx), *X, alpha, *Y, beta, n);
  gb_prof_end(ctx, &pr, (dtype == GPU_MV_FLOAT64 ? 8.0 : 4.0) * n * w * (beta == 0.0 ? 2 : 3), 0.0);
  gb_count_launch(1);
  return CUDA_LAUNCH_CHECK(ctx, "axpby");
}

struct idx_table {
  int v[BLK_MAXCOLS];
};

template <typename T>
__global__ void scale_cols_kernel(blk_cols X, const double* __restrict__ d, idx_table idx,
                                  blk_cols Y, long n)
{
  gb_pdl_entry();
  const T* x = (const T*)X.col[blockIdx.y];
  T* y = (T*)Y.col[blockIdx.y];
  const T a = (T)d[idx.v[blockIdx.y]];
  for (long r = blockIdx.x * (long)blockDim.x + threadIdx.x; r < n; r += (long)gridDim.x * blockDim.x)
    y[r] = a * x[r];
}

static void fill_idx(idx_table* t, const int* idx, int w)
{
  for (int j = 0; j < w; j++) t->v[j] = idx ? idx[j] : j;
}

extern "C" int gb_scale_cols(gpu_Context* ctx, int dtype, long n, const blk_cols* X,
                             const double* d, const int* idx, const blk_cols* Y, int w)
{
  if (w <= 0 || n <= 0) return 0;
  idx_table t;
  fill_idx(&t, idx, w);
  dim3 grid(row_blocks(ctx, n, w), w);
  gb_prof_rec pr;
  gb_prof_begin(ctx, &pr, GB_K_BLAS1);
  if (dtype == GPU_MV_FLOAT64)
    gb_pdl(scale_cols_kernel<double>, grid, 256, 0, S(ctx), *X, d, t, *Y, n);
  else
    gb_pdl(scale_cols_kernel<float>, grid, 256, 0, S(ctx), *X, d, t, *Y, n);
  gb_prof_end(ctx, &pr, (dtype == GPU_MV_FLOAT64 ? 8.0 : 4.0) * n * w * 2, 0.0);
  gb_count_launch(1);
  return CUDA_LAUNCH_CHECK(ctx, "scale_cols");
}

// column dot products: per-CTA partial sums, then a fixed-order reduction
template <typename T>
__global__ void dot_partial_kernel(blk_cols X, blk_cols Y, long n, double* __restrict__ partial)
{
  gb_pdl_entry();
  const T* x = (const T*)X.col[blockIdx.y];
  const T* y = (const T*)Y.col[blockIdx.y];
  double s = 0.0;
  for (long r = blockIdx.x * (long)blockDim.x + threadIdx.x; r < n; r += (long)gridDim.x * blockDim.x)
    s += (double)x[r] * (double)y[r];
  s = block_sum256(s);
  if (threadIdx.x == 0) partial[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = s;
}

__global__ void dot_reduce_kernel(const double* __restrict__ partial, int nb, idx_table idx,
                                  double* __restrict__ out)
{
  gb_pdl_entry();
  const double s = ordered_sum256(partial + (size_t)blockIdx.x * nb, nb);
  if (threadIdx.x == 0) out[idx.v[blockIdx.x]] = s;
}

// FP32 blocks with 16-byte aligned columns: float4 loads, exact products in
// a compensated FP32 sum flushed to FP64 every 64 terms (blas32.cuh)
__global__ void __launch_bounds__(256) dot32_partial_kernel(blk_cols X, blk_cols Y, long n,
                                                            double* __restrict__ partial)
{
  gb_pdl_entry();
  const float4* x = (const float4*)X.col[blockIdx.y];
  const float4* y = (const float4*)Y.col[blockIdx.y];
  const long n4 = n >> 2, stride = (long)gridDim.x * blockDim.x;
  double acc = 0.0;
  float s = 0.f, c = 0.f;
  // the flush stands outside the inner loop: predicated off inside it, its four
  // FP64 instructions still held the FP64 pipe (16 cycles each)
  for (long v = blockIdx.x * (long)blockDim.x + threadIdx.x; v < n4;) {
    if (v + 15 * stride < n4) {
#pragma unroll 4
      for (int i = 0; i < 16; i++, v += stride) acc_prod32x4(s, c, x[v], y[v]);
      acc += (double)s + (double)c;
      s = c = 0.f;
    } else {
#pragma unroll 4
      for (; v < n4; v += stride) acc_prod32x4(s, c, x[v], y[v]);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {  // the last n % 4 rows
    const long r = 4 * n4 + threadIdx.x;
    acc_prod32(s, c, ((const float*)x)[r], ((const float*)y)[r]);
  }
  acc += (double)s + (double)c;
  const double t = block_sum256(acc);
  if (threadIdx.x == 0) partial[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = t;
}

extern "C" int gb_dot_cols(gpu_Context* ctx, int dtype, long n, const blk_cols* X,
                           const blk_cols* Y, int w, double* out, const int* idx)
{
  if (w <= 0) return 0;
  idx_table t;
  fill_idx(&t, idx, w);
  unsigned nb = row_blocks(ctx, n, w);
  double* partial = (double*)gb_workspace(ctx, sizeof(double) * (size_t)nb * w);
  if (!partial) return -1;
  dim3 grid(nb, w);
  gb_prof_rec pr;
  gb_prof_begin(ctx, &pr, GB_K_BLAS1);
  if (dtype == GPU_MV_FLOAT64)
    gb_pdl(dot_partial_kernel<double>, grid, 256, 0, S(ctx), *X, *Y, n, partial);
  else if (cols_aligned16(X->col, w) && cols_aligned16(Y->col, w))
    gb_pdl(dot32_partial_kernel, grid, 256, 0, S(ctx), *X, *Y, n, partial);
  else
    gb_pdl(dot_partial_kernel<float>, grid, 256, 0, S(ctx), *X, *Y, n, partial);
  gb_pdl(dot_reduce_kernel, w, 256, 0, S(ctx), partial, nb, t, out);
  gb_prof_end(ctx, &pr, (dtype == GPU_MV_FLOAT64 ? 8.0 : 4.0) * n * w * 2, 2.0 * n * w);
  gb_count_launch(2);
  return CUDA_LAUNCH_CHECK(ctx, "dot_cols");
}

// fused residual R = lambda*BX - AX with squared column norms
template <typename T, int OUT32>
struct rr_out {
  typedef T type;
};
template <>
struct rr_out<double, 1> {
  typedef float type;
};

template <typename T, int OUT32 = 0>
__global__ void residual_partial_kernel(blk_cols BX, blk_cols AX, const double* __restrict__ lambda,
                                        idx_table idx, blk_cols R, long n,
                                        double* __restrict__ partial)
{
  gb_pdl_entry();
  // T: arithmetic and input type; the residual is stored as TO (FP32 for the
  // FP64-accumulated explicit phase: its norm is taken before the rounding)
  using TO = typename rr_out<T, OUT32>::type;
  const T* bx = (const T*)BX.col[blockIdx.y];
  const T* ax = (const T*)AX.col[blockIdx.y];
  TO* rr = (TO*)R.col[blockIdx.y];
  const T lam = (T)lambda[idx.v[blockIdx.y]];
  double s = 0.0;
  for (long r = blockIdx.x * (long)blockDim.x + threadIdx.x; r < n; r += (long)gridDim.x * blockDim.x) {
    T v = lam * bx[r] - ax[r];
    rr[r] = (TO)v;
    s += (double)v * (double)v;
  }
  s = block_sum256(s);
  if (threadIdx.x == 0) partial[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = s;
}

extern "C" int gb_residual(gpu_Context* ctx, int dtype, long n, const blk_cols* BX,
                           const blk_cols* AX, const double* lambda, const int* idx,
                           const blk_cols* R, int w, double* norm2)
{
  if (w <= 0) return 0;
  idx_table t;
  fill_idx(&t, idx, w);
  unsigned nb = row_blocks(ctx, n, w);
  double* partial = (double*)gb_workspace(ctx, sizeof(double) * (size_t)nb * w);
  if (!partial) return -1;
  dim3 grid(nb, w);
  gb_prof_rec pr;
  gb_prof_begin(ctx, &pr, GB_K_RESID);
  if (dtype == GPU_MV_FLOAT64)
    gb_pdl(residual_partial_kernel<double>, grid, 256, 0, S(ctx), *BX, *AX, lambda, t, *R, n, partial);
  else if (dtype == GPU_MV_FLOAT32)
    gb_pdl(residual_partial_kernel<float>, grid, 256, 0, S(ctx), *BX, *AX, lambda, t, *R, n, partial);
  else  // FP64 inputs, FP32 residual
    gb_pdl(residual_partial_kernel<double, 1>, grid, 256, 0, S(ctx), *BX, *AX, lambda, t, *R, n, partial);
  gb_pdl(dot_reduce_kernel, w, 256, 0, S(ctx), partial, nb, t, norm2);
  gb_prof_end(ctx, &pr, (dtype == GPU_MV_FLOAT32 ? 12.0 : (dtype == GPU_MV_FLOAT64 ? 24.0 : 20.0)) * n * w,
              4.0 * n * w);
  gb_count_launch(2);
  return CUDA_LAUNCH_CHECK(ctx, "residual");
}

// Y64 = X64 + D (D FP32), and D <- (float) Y64: the FP64-accumulated block
// update of the explicit phase (the correction carries FP32 rounding
// relative to its own size) and its FP32 shadow
__global__ void acc64_kernel(blk_cols X, blk_cols D, blk_cols Y, long n)
{
  gb_pdl_entry();
  const double* x = (const double*)X.col[blockIdx.y];
  float* d = (float*)D.col[blockIdx.y];
  double* y = (double*)Y.col[blockIdx.y];
  for (long r = blockIdx.x * (long)blockDim.x + threadIdx.x; r < n; r += (long)gridDim.x * blockDim.x) {
    const double v = x[r] + (double)d[r];
    y[r] = v;
    d[r] = (float)v;
  }
}

extern "C" int gb_accumulate64(gpu_Context* ctx, long n, const blk_cols* X64, const blk_cols* D32,
                               const blk_cols* Y64, int w)
{
  if (w <= 0 || n <= 0) return 0;
  dim3 grid(row_blocks(ctx, n, w), w);
  gb_prof_rec pr;
  gb_prof_begin(ctx, &pr, GB_K_BLAS1);
  gb_pdl(acc64_kernel, grid, 256, 0, S(ctx), *X64, *D32, *Y64, n);
  gb_prof_end(ctx, &pr, 24.0 * n * w, (double)n * w);
  gb_count_launch(1);
  return CUDA_LAUNCH_CHECK(ctx, "accumulate64");
}

// The explicit pencil (G, H) of [X R P] from the exact Gram products of the
// split mode.  Inputs (column-major FP64):
//   Hx = X'[X R P]          (k x m, ld k)
//   Hr = R'[R P AR AP]      (nR x (2 nR + 2 nP), ld nR)
//   Hp = P'[P AP]           (nP x 2 nP, ld nP)
//   Gt(c, i) = S_c' RS_i    (ld ld; column i < k of the tensor-core product
//                            [X R P]'[RS AR AP]), RS = lambda X - A X
// with lambda the Rayleigh quotients of X.  The X rows of G are formed in
// residual form, G(i, c) = X_i' A S_c = lambda_i X_i' S_c - RS_i' S_c, so that
// A X (whose norm is the spectrum's scale) never enters a product and the
// rounding of RS'S scales with the residual (TF32 products suffice there);
// the other blocks are R'AR, R'AP, P'AP.  Symmetric blocks are averaged with
// their transposes.
__global__ void split_pencil_kernel(const double* __restrict__ Hx, const double* __restrict__ Hr,
                                    const double* __restrict__ Hp, const double* __restrict__ Gt,
                                    double* G, double* H, int ld, const double* __restrict__ lam,
                                    int k, int nR, int nP)
{
  gb_pdl_entry();
  const int m = k + nR + nP;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m * m) return;
  const int a = e % m, b = e / m;
  double g, h;
  if (a < k || b < k) {
    // Gt = RS' [RS S] (k x (k + m), leading dimension k): S_c' RS_i at
    // Gt[i + (k + c) k]
    if (a < k && b < k) {
      const double h1 = Hx[a + (size_t)b * k], h2 = Hx[b + (size_t)a * k];
      h = 0.5 * (h1 + h2);
      g = 0.5 * ((lam[a] * h1 - Gt[a + (size_t)(k + b) * k]) + (lam[b] * h2 - Gt[b + (size_t)(k + a) * k]));
    } else {
      const int i = a < k ? a : b, c = a < k ? b : a;
      h = Hx[i + (size_t)c * k];
      g = lam[i] * h - Gt[i + (size_t)(k + c) * k];
    }
  } else {
    const int ra = a - k, rb = b - k;  // offsets in [R P]
    if (ra < nR && rb < nR) {
      h = 0.5 * (Hr[ra + (size_t)rb * nR] + Hr[rb + (size_t)ra * nR]);
      const size_t o = (size_t)(nR + nP) * nR;
      g = 0.5 * (Hr[o + ra + (size_t)rb * nR] + Hr[o + rb + (size_t)ra * nR]);
    } else if (ra < nR || rb < nR) {
      const int r = ra < nR ? ra : rb, p = (ra < nR ? rb : ra) - nR;
      h = Hr[r + (size_t)(nR + p) * nR];
      g = Hr[r + (size_t)(2 * nR + nP + p) * nR];
    } else {
      const int pa = ra - nR, pb = rb - nR;
      h = 0.5 * (Hp[pa + (size_t)pb * nP] + Hp[pb + (size_t)pa * nP]);
      g = 0.5 * (Hp[pa + (size_t)(nP + pb) * nP] + Hp[pb + (size_t)(nP + pa) * nP]);
    }
  }
  G[a + (size_t)b * ld] = g;
  H[a + (size_t)b * ld] = h;
}

extern "C" int gb_split_pencil(gpu_Context* ctx, const double* Hx, const double* Hr, const double* Hp,
                               const double* Gt, double* G, double* H, int ld, const double* lam, int k,
                               int nR, int nP)
{
  const int m = k + nR + nP;
  gb_pdl(split_pencil_kernel, (m * m + 255) / 256, 256, 0, S(ctx), Hx, Hr, Hp, Gt, G, H, ld, lam, k, nR, nP);
  gb_count_launch(1);
  return CUDA_LAUNCH_CHECK(ctx, "split pencil");
}

__global__ void rayleigh_kernel(int w, const double* num, const double* den, double* lam)
{
  gb_pdl_entry();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < w) lam[i] = den[i] > 0.0 ? num[i] / den[i] : 0.0;
}

extern "C" int gb_rayleigh_quotients(gpu_Context* ctx, int dtype, long n, const blk_cols* X,
                                     const blk_cols* AX, int w, double* scratch, double* lam)
{
  int idx[BLK_MAXCOLS];
  for (int c = 0; c < w; c++) idx[c] = c;
  if (gb_dot_cols(ctx, dtype, n, X, AX, w, scratch, idx)) return -1;
  if (gb_dot_cols(ctx, dtype, n, X, X, w, scratch + w, idx)) return -1;
  gb_pdl(rayleigh_kernel, (w + 127) / 128, 128, 0, S(ctx), w, scratch, scratch + w, lam);
  gb_count_launch(1);
  return CUDA_LAUNCH_CHECK(ctx, "rayleigh quotients");
}

template <typename TI, typename TO>
__global__ void convert_kernel(blk_cols X, blk_cols Y, long n)
{
  gb_pdl_entry();
  const TI* x = (const TI*)X.col[blockIdx.y];
  TO* y = (TO*)Y.col[blockIdx.y];
  for (long r = blockIdx.x * (long)blockDim.x + threadIdx.x; r < n; r += (long)gridDim.x * blockDim.x)
    y[r] = (TO)x[r];
}

extern "C" int gb_convert(gpu_Context* ctx, long n, int dtype_x, const blk_cols* X, int dtype_y,
                          const blk_cols* Y, int w)
{
  if (w <= 0 || n <= 0) return 0;
  dim3 grid(row_blocks(ctx, n, w), w);
  gb_prof_rec pr;
  gb_prof_begin(ctx, &pr, GB_K_BLAS1);
  if (dtype_x == GPU_MV_FLOAT64 && dtype_y == GPU_MV_FLOAT32)
    gb_pdl(convert_kernel<double, float>, grid, 256, 0, S(ctx), *X, *Y, n);
  else if (dtype_x == GPU_MV_FLOAT32 && dtype_y == GPU_MV_FLOAT64)
    gb_pdl(convert_kernel<float, double>, grid, 256, 0, S(ctx), *X, *Y, n);
  else if (dtype_x == GPU_MV_FLOAT64)
    gb_pdl(convert_kernel<double, double>, grid, 256, 0, S(ctx), *X, *Y, n);
  else
    gb_pdl(convert_kernel<float, float>, grid, 256, 0, S(ctx), *X, *Y, n);
  gb_prof_end(ctx, &pr, ((dtype_x == GPU_MV_FLOAT64 ? 8.0 : 4.0) + (dtype_y == GPU_MV_FLOAT64 ? 8.0 : 4.0)) * n * w, 0.0);
  gb_count_launch(1);
  return CUDA_LAUNCH_CHECK(ctx, "convert");
}

// ------------------------------------------------------------------------
// drand48: state_{t+1} = a*state_t + c mod 2^48 with a = 0x5DEECE66D,
// c = 0xB, state_0 = (seed << 16) | 0x330E, value = state / 2^48.
// Element e of the fill (column-major over the listed columns) uses state
// e+1; each thread jumps ahead with the affine-map powers (mod 2^64
// arithmetic is exact mod 2^48).
// ------------------------------------------------------------------------
struct lcg_table {
  unsigned long long a[48], c[48];  // map for 2^b steps
};

__device__ __forceinline__ unsigned long long lcg_jump(const lcg_table& t, unsigned long long s,
                                                       unsigned long long steps)
{
  const unsigned long long M = (1ULL << 48) - 1;
  for (int b = 0; b < 48 && steps; b++, steps >>= 1)
    if (steps & 1) s = (t.a[b] * s + t.c[b]) & M;
  return s;
}

template <typename T>
__global__ void drand48_kernel(T* data, long n, long ld, idx_table idx, int w,
                               unsigned long long state0, lcg_table tab)
{
  gb_pdl_entry();
  const unsigned long long M = (1ULL << 48) - 1;
  const unsigned long long A = 0x5DEECE66DULL, Cc = 0xBULL;
  long total = n * (long)w;
  long per = 64;  // consecutive values per thread
  long first = (blockIdx.x * (long)blockDim.x + threadIdx.x) * per;
  if (first >= total) return;
  unsigned long long s = lcg_jump(tab, state0, (unsigned long long)first);
  long last = min(total, first + per);
  for (long e = first; e < last; e++) {
    s = (A * s + Cc) & M;
    double v = (double)s * (1.0 / 281474976710656.0);
    long c = e / n, r = e - c * n;
    data[(long)idx.v[c] * ld + r] = (T)(2.0 * v - 1.0);
  }
}

extern "C" int gb_drand48_fill(gpu_Context* ctx, int dtype, void* data, long n, long ld,
                               const int* idx, int w, unsigned int seed)
{
  if (w <= 0 || n <= 0) return 0;
  idx_table t;
  fill_idx(&t, idx, w);
  lcg_table tab;
  const unsigned long long M = (1ULL << 48) - 1;
  unsigned long long a = 0x5DEECE66DULL, c = 0xBULL;
  for (int b = 0; b < 48; b++) {
    tab.a[b] = a;
    tab.c[b] = c;
    // compose the map with itself: s -> a(a s + c) + c
    unsigned long long a2 = (a * a) & M, c2 = (a * c + c) & M;
    a = a2;
    c = c2;
  }
  unsigned long long state0 = (((unsigned long long)seed) << 16) | 0x330EULL;
  long total = n * (long)w;
  long threads = (total + 63) / 64;
  unsigned blocks = (unsigned)((threads + 255) / 256);
  if (dtype == GPU_MV_FLOAT64)
    gb_pdl(drand48_kernel<double>, blocks, 256, 0, S(ctx), (double*)data, n, ld, t, w, state0, tab);
  else
    gb_pdl(drand48_kernel<float>, blocks, 256, 0, S(ctx), (float*)data, n, ld, t, w, state0, tab);
  gb_count_launch(1);
  return CUDA_LAUNCH_CHECK(ctx, "drand48_fill");
}

// ------------------------------------------------------------------------
// Gram product that allocates nothing (gpu_GramNoAlloc in lobpcg_gb300.h).
// The split-k partial sums live in this file-scope device array instead of
// the context's cudaMalloc'ed workspace.  Host code must not pass the
// array's name to a kernel (on the host it is only a stand-in symbol); its
// device address is looked up once per device with cudaGetSymbolAddress.
// ------------------------------------------------------------------------
#define GRAM_NOALLOC_SCRATCH_DOUBLES (512 * 1024) /* 4 MiB per device */
static __device__ __align__(256) double g_gram_noalloc_scratch[GRAM_NOALLOC_SCRATCH_DOUBLES];

#define GRAM_NOALLOC_MAX_DEVICES 64
static double* g_noalloc_addr[GRAM_NOALLOC_MAX_DEVICES];

static double* noalloc_scratch(int device)
{
  if (device < 0 || device >= GRAM_NOALLOC_MAX_DEVICES) return NULL;
  if (!g_noalloc_addr[device]) {
    void* p = NULL;
    // the caller's device is current here (cudaGetDevice above)
    if (cudaGetSymbolAddress(&p, g_gram_noalloc_scratch) != cudaSuccess || !p) return NULL;
    g_noalloc_addr[device] = (double*)p;
  }
  return g_noalloc_addr[device];
}

template <typename T, int TM, int TN>
static int gram_noalloc_launch(long n, const blk_cols* X, int h, const blk_cols* Y, int w,
                               double* G, int ldg, double* partial, cudaStream_t stream, int sms)
{
  constexpr int BM = 16 * TM, BN = 16 * TN;
  int gx = (h + BM - 1) / BM, gy = (w + BN - 1) / BN;
  long splits = 2L * sms / (gx * gy);
  long cap = GRAM_NOALLOC_SCRATCH_DOUBLES / ((long)h * w);  // splits that fit the array
  if (splits > cap) splits = cap;
  long max_splits = (n + 255) / 256;
  if (splits > max_splits) splits = max_splits;
  if (splits < 1) splits = 1;
  long rows = (n + splits - 1) / splits;
  rows = (rows + 31) / 32 * 32;
  splits = (n + rows - 1) / rows;
  if (splits < 1) splits = 1;
  dim3 grid(gx, gy, (unsigned)splits);
  // an error left pending by earlier work on this thread is not ours to
  // clear: report it (-3) and leave it for its owner to read
  if (cudaPeekAtLastError() != cudaSuccess) return -3;
  // every partial element of the used splits is written before the
  // reduction reads it, so stale contents from an earlier call never leak
  gram_partial_kernel<T, TM, TN><<<grid, 256, 0, stream>>>(*X, h, *Y, w, n, rows, partial);
  if (cudaGetLastError() != cudaSuccess) return -3;
  gram_reduce_kernel<<<(h * w + 31) / 32, 256, 0, stream>>>(partial, (int)splits, 1, splits, h * w, h, 0, G, ldg);
  gb_count_launch(2);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

extern "C" int gpu_GramNoAlloc(int dtype, long n, const void* X, long ldx, int h, const void* Y,
                               long ldy, int w, double* G, int ldg, void* stream)
{
  if (n <= 0 || h <= 0 || w <= 0 || !X || !Y || !G || ldx < n || ldy < n || ldg < h ||
      (dtype != GPU_MV_FLOAT64 && dtype != GPU_MV_FLOAT32))
    return -1;
  if (h > BLK_MAXCOLS || w > BLK_MAXCOLS || (long)h * w > GRAM_NOALLOC_SCRATCH_DOUBLES) return -2;
  int device = -1;
  if (cudaGetDevice(&device) != cudaSuccess) return -3;
  double* partial = noalloc_scratch(device);
  if (!partial) return -3;
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0)
    sms = 152;
  const size_t es = dtype == GPU_MV_FLOAT64 ? 8 : 4;
  blk_cols xc, yc;
  for (int c = 0; c < h; c++) xc.col[c] = (const char*)X + es * (size_t)ldx * c;
  for (int c = 0; c < w; c++) yc.col[c] = (const char*)Y + es * (size_t)ldy * c;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == GPU_MV_FLOAT64) {
    if (h <= 32 && w <= 32) return gram_noalloc_launch<double, 2, 2>(n, &xc, h, &yc, w, G, ldg, partial, s, sms);
    return gram_noalloc_launch<double, 4, 4>(n, &xc, h, &yc, w, G, ldg, partial, s, sms);
  }
  if (h <= 32 && w <= 32) return gram_noalloc_launch<float, 2, 2>(n, &xc, h, &yc, w, G, ldg, partial, s, sms);
  return gram_noalloc_launch<float, 4, 4>(n, &xc, h, &yc, w, G, ldg, partial, s, sms);
}
