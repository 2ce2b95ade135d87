// oz_xc64.cu -- block update Y = X C (+ Z) with the accuracy of FP64 arithmetic on
// the tensor cores, by error-free splitting (oz8_common.cuh): X an FP64 block of
// n rows and h <= 64 columns, C the FP64 h x w coordinate block (w <= 64) on the
// device, Z an optional FP32 or FP64 block, Y FP64.  It is
// serial_Multi_VectorByMatrix (blopex_serial_double/multivector/multi_vector.c:
// 474-524), for callers' large FP64 blocks (gb_bymat_large) and gpu_BlockUpdate's
// mode 2.
//
// Scales: each row of X (its h values) and each column of C share one power of
// two; both are cut into 7 8-bit digits (55 fraction bits).  Level L = t + u of
// the digit products is accumulated exactly in FP32 in TMEM (at most 7 products
// of 2^14 over 64 columns: below 2^23); the epilogue recombines the eight levels
// into one 64-bit integer, rounds it to FP64 with integer operations and adds Z.
//
// Accuracy.  The digits alone (gpu_BlockUpdate's mode 2) are off by up to
// 2^-55 S S' (|x/S| + |c/S'| + 1.3) (1-norms; S, S' the scales: every value cut
// below 2^-55 of its scale, products of levels 8 and up left out, T rounded): less
// than the roundings of fused multiply-adds on random blocks (6e-17 against 2.0e-16
// relative, h = 32), and more, or everything, where a row's large values meet
// zeros or small values of C.  Callers' products (BOUND) are held to the bound of
// the multiply-adds, m 2^-53 sum |x_i c_ij| with the m nonzeros of column j of C
// (+ the rounding of Z), in every entry: the magnitudes of the top digits are
// multiplied as well (an eighth slice, a ninth accumulator).  D = sum |d_0(x)|
// |d_0(c)| bounds sum |x_i c_ij| / (S S') from below by (D - 0.502 (N + N')) 2^-14,
// N and N' being the sums of the top digits, which bound the 1-norms from above
// by (N + h / 2) / 128.  The digits serve where
//   2^-55 ((N + N' + h) / 128 + 1.3) <= (m - 1) 2^-53 (D - 0.502 (N + N')) 2^-14,
// the last of the m roundings being that of the sum.  Other entries are summed
// directly with FP64 FMAs by the epilogue, in the order of bymat_kernel: 1 in 10^5
// of random blocks of 32 columns; all of a column of C with one nonzero (a copy of
// X's column comes back as it is), most where X's large columns meet C's zeros.  So
// are rows or columns whose scale the digits cannot carry (infinities, NaN,
// values below 2^-960), and products whose scale is below 2^-924.
//
// What bounds it: instructions, ~17 integer ones per X value in the producers and
// ~30 per Y value in the epilogue (32 x 32: 63% of the issue slots, 52% of the ALU
// pipe, 17 warps to cover their latencies); FP64 FMAs instead would need h w / 2
// cycles per row and SM (2 per cycle), 2,048 at h = w = 64.  With D the narrower
// units cost more MMAs, each of which reads its 4 KB of A.  Measured, 2,097,152 rows,
// with D (without; FMAs): 16 x 16 0.29 ms (-; 0.88), 32 x 32 0.51 (0.46; 3.45), 64 x 64
// 1.30 (0.88; 13.8); 32 x 32 with X's columns graded over 18 decades 3.9 ms.  Hence no
// shared-memory staging of X: its columns are read by coalesced 8-byte loads
// straight into registers (any alignment and spacing of the columns), all 32 of
// a thread in flight at once, while the MMAs of the previous tile run.
//
// Per CTA (one per SM, persistent over 128-row tiles; a tile's output columns
// are taken 32 at a time, "units", into two alternating TMEM accumulator sets --
// with D 16 at a time, three sets -- so that the MMAs of one unit overlap the
// epilogue of the ones before):
//   warps 8-15  producers: warp p holds rows 32 (p mod 4) .. + 31 (lane = row)
//               of 32 columns in registers, finds the rows' scales and writes
//               the digit slices in the 128-byte-swizzled K-major layout;
//   warp 16     allocates TMEM; one thread issues tcgen05.mma.kind::f16
//               (M = 128, K = 16): for X slice t one MMA per K step against the
//               C slices stacked along N, so that level t + u lands at TMEM
//               column 32 (16) (t + u), and D behind them;
//   warps 0-7   read a unit's accumulators (lane = row; warps w and w + 4 share
//               TMEM lanes and take half of the unit's columns each), recombine
//               and store Y.
// Every wait is bounded; a timeout sets an error word, the outputs become NaN and
// all roles finish.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "internal.h"
#include "oz8_common.cuh"

#define OZY_S OZ8_S
#define OZY_THREADS 544
#define OZY_NPROD 256
#define OZY_ASLICE 16384          // 128 rows x 128 bytes
#define OZY_TILES 8               // tiles whose rows' scales and sums are kept

// BOUND: every entry held to the bound of FP64 FMAs
template <bool BOUND>
struct ozy_cfg {
  static constexpr int SLICES = BOUND ? OZY_S + 1 : OZY_S;  // the digits' and, last, the magnitudes of the top digits
  static constexpr int UNIT = BOUND ? 16 : 32;              // output columns per unit
  static constexpr int SETS = BOUND ? 3 : 2;
  static constexpr int LEVELS = BOUND ? 9 : 8;              // accumulators of a column: levels 0-7 (and D)
  static constexpr int SET = LEVELS * UNIT;                 // TMEM columns of one accumulator set
  static constexpr int BSLICE = UNIT * 128;                 // one unit's columns of one slice
  static constexpr int C_BYTES = 64 * 128 * SLICES;         // [unit][slice][UNIT rows][128 B]
  static constexpr int SMEM = C_BYTES + SLICES * OZY_ASLICE + 1024;
  static_assert(SETS * SET <= 512, "accumulators exceed TMEM");
};

struct ozy_params {
  const void *x[64], *z[64];
  void* y[64];
  const double* C;
  int ldc, h, w, z_kind;  // z_kind: 0 none, 1 FP32, 2 FP64
  long n;
  long polls;  // limit of one pipeline wait
  int* err;
};

// global loads and stores through pointers kept in shared memory (the compiler
// would take them for generic addresses, which cost several times as much)
static __device__ __forceinline__ double ozy_ld(const void* p, long i)
{
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(__cvta_generic_to_global((const double*)p + i)));
  return v;
}
static __device__ __forceinline__ uint32_t ozy_ld32(const void* p, long i)
{
  uint32_t v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(__cvta_generic_to_global((const uint32_t*)p + i)));
  return v;
}
static __device__ __forceinline__ void ozy_st(void* p, long i, double v)
{
  asm volatile("st.global.f64 [%0], %1;" ::"l"(__cvta_generic_to_global((double*)p + i)), "d"(v) : "memory");
}

// the Z values of one row in columns j0 .. j0 + 3 (bit patterns; 0 outside)
static __device__ __forceinline__ void ozy_load_z(int z_kind, const void* const* s_z, int j0, int w, long row,
                                                  long n, unsigned long long (&zb)[4])
{
#pragma unroll
  for (int jj = 0; jj < 4; jj++) {
    const int j = j0 + jj;
    zb[jj] = 0;
    if (row < n && j < w) {
      if (z_kind == 1)
        zb[jj] = ozy_ld32(s_z[j], row);
      else if (z_kind == 2)
        zb[jj] = (unsigned long long)__double_as_longlong(ozy_ld(s_z[j], row));
    }
  }
}

// the accumulators of four output columns of this warp's rows (not waited for)
template <int UNIT, int LEVELS>
static __device__ __forceinline__ void ozy_tmem_ld(uint32_t taddr, uint32_t (&v)[LEVELS][4])
{
#pragma unroll
  for (int L = 0; L < LEVELS; L++)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v[L][0]), "=r"(v[L][1]), "=r"(v[L][2]), "=r"(v[L][3])
                 : "r"(taddr + (uint32_t)(L * UNIT)));
}

// one entry of X C by FP64 FMAs, in column order
static __device__ __noinline__ double ozy_direct(const void* const* s_x, const double* C, int ldc, int h, int j,
                                                 long row)
{
  double acc = 0.0;
#pragma unroll 8
  for (int i = 0; i < h; i++) acc = fma(ozy_ld(s_x[i], row), C[i + (size_t)j * ldc], acc);
  return acc;
}

// a group's largest exponent, raised to 1 (unsafe) when it holds nothing but
// subnormals
static __device__ __forceinline__ int ozy_group_exp(uint32_t mag, bool nonzero)
{
  const int e = (int)(mag >> 20);
  return e == 0 && nonzero ? 1 : e;
}

template <bool BOUND>
__global__ void __launch_bounds__(OZY_THREADS, 1) oz_xc64_kernel(const __grid_constant__ ozy_params prm)
{
  using K = ozy_cfg<BOUND>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = smem_align1024(smem_raw);
  unsigned char* cdig = smem;               // [unit][slice][UNIT rows][128 B]
  unsigned char* adig = smem + K::C_BYTES;  // [slice][128 rows][128 B]
  __shared__ uint64_t a_full[4], a_empty[4], acc_full[K::SETS], acc_empty[K::SETS], done_bar;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  __shared__ __align__(16) int colexp[64];
  // the digits serve where D >= kappa (N + N') + const: by column, kappa and the rest
  __shared__ __align__(16) float colkappa[BOUND ? 64 : 4], colneed[BOUND ? 64 : 4];
  __shared__ int coltop[64], colnnz[64];  // N' and m
  __shared__ uint32_t colpart[8][64];      // per (8-row group of C, column) largest magnitude word
  __shared__ unsigned char colnz[8][64];   // and whether any value is not zero
  // by tile modulo OZY_TILES (read by the epilogue): scales, and N by column half
  // (two FP16 sums).  Written for tile i once the MMAs of tile i - 2 are done, hence
  // the epilogue with every unit two or three before that tile's last: tile i - 5
  __shared__ int rowexp[OZY_TILES][128];
  __shared__ uint32_t rowtop[BOUND ? OZY_TILES : 1][2][128];
  __shared__ int rowpart[2][2][128];       // by tile modulo 2: per (column half, row) exponent
  // column pointers: shared memory serves a runtime index in a few cycles,
  // where the kernel-parameter table behind it does not
  __shared__ const void* s_x[64];
  __shared__ void* s_y[64];
  __shared__ const void* s_z[64];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = prm.h, w = prm.w;
  const int ksteps = (h + 15) >> 4;
  const int nh = (w + K::UNIT - 1) / K::UNIT;  // units per tile
  const long ntiles = (prm.n + 127) / 128;
  const long my_tiles = (long)blockIdx.x < ntiles ? (ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;

  if (tid == 0) {
    abort_flag = 0;
    for (int k = 0; k < 4; k++) {
      mbar_init(&a_full[k], OZY_NPROD);
      mbar_init(&a_empty[k], 1);
    }
    for (int b = 0; b < K::SETS; b++) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 256);
    }
    mbar_init(&done_bar, 1);
  }
  if (tid < 64) {
    coltop[tid] = colnnz[tid] = 0;
    s_x[tid] = tid < h ? prm.x[tid] : nullptr;
    s_y[tid] = tid < w ? prm.y[tid] : nullptr;
    s_z[tid] = (tid < w && prm.z_kind) ? prm.z[tid] : nullptr;
  }
  // C: one scale per column, digits as the B operand (row j = output column,
  // K = input column); rows j >= w and columns i >= h are zero
  for (int e = tid; e < 64 * 8; e += OZY_THREADS) {
    const int j = e & 63, cg = e >> 6;
    uint32_t mag = 0;
    bool nz = false;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const int i = cg * 8 + c;
      const double v = (j < w && i < h) ? prm.C[i + (size_t)j * prm.ldc] : 0.0;
      mag = max(mag, (uint32_t)__double2hiint(v) & 0x7FFFFFFFu);
      nz |= v != 0.0;
    }
    colpart[cg][j] = mag;
    colnz[cg][j] = nz;
  }
  if (warp == 16) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  for (int e = tid; e < 64 * 8; e += OZY_THREADS) {  // (column j, 8-row group cg)
    const int j = e & 63, cg = e >> 6;
    uint32_t mag = 0;
    bool nz = false;
#pragma unroll
    for (int g = 0; g < 8; g++) {
      mag = max(mag, colpart[g][j]);
      nz |= colnz[g][j] != 0;
    }
    const int E = ozy_group_exp(mag, nz);
    if (cg == 0) colexp[j] = oz8_code(E);
    uint32_t lo[8], hi[8], pk[OZY_S][4];
    int nnz = 0;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const int i = cg * 8 + c;
      const double v = (j < w && i < h) ? prm.C[i + (size_t)j * prm.ldc] : 0.0;
      nnz += v != 0.0;
      lo[c] = (uint32_t)__double2loint(v);
      hi[c] = (uint32_t)__double2hiint(v);
    }
    oz8_digits8(lo, hi, oz8_scale(E), pk);
    // a unit's slices of 16 output columns are stacked, so one MMA takes several
    // of them as a single operand
    const int jr = j & (K::UNIT - 1);
    unsigned char* dst = cdig + (j / K::UNIT) * K::SLICES * K::BSLICE + jr * 128 + ((cg ^ (jr & 7)) << 4);
#pragma unroll
    for (int t = 0; t < OZY_S; t++)
      *(uint4*)(dst + t * K::BSLICE) = make_uint4(pk[t][0], pk[t][1], pk[t][2], pk[t][3]);
    if (BOUND) {
      uint32_t m[4];
      const uint32_t top = oz8_magnitudes(pk[0], m);
      *(uint4*)(dst + OZY_S * K::BSLICE) = make_uint4(m[0], m[1], m[2], m[3]);
      atomicAdd(&coltop[j], (int)oz8_both(top));
      atomicAdd(&colnnz[j], nnz);
    }
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;

  if (warp >= 8 && warp < 16) {
    // ------------------------------------------------------- digit slices
    // (every producer runs every iteration: the named barrier of a pair of
    // warps must be reached by both; an abort only skips the work)
    // A thread holds the 8-column groups 2k + half of its row, so that K step
    // k (columns 16 k .. + 15) is complete, and its MMAs start, while the next
    // steps are still being cut.
    const int pw = warp - 8, r = 32 * (pw & 3) + lane, half = pw >> 2;
    for (long i = 0; i < my_tiles; i++) {
      const long row = (blockIdx.x + i * gridDim.x) * 128 + r;
      uint32_t lo[32], hi[32];
#pragma unroll
      for (int c = 0; c < 32; c++) {
        const int col = 16 * (c >> 3) + 8 * half + (c & 7);
        double v = 0.0;
        if (row < prm.n && col < h) v = ozy_ld(s_x[col], row);
        lo[c] = (uint32_t)__double2loint(v);
        hi[c] = (uint32_t)__double2hiint(v);
      }
      if (i + 1 < my_tiles) {
        // the next tile's X and Z (1 KB, 8 lines, of a column) on their way
        // into L2
        const long r1 = (blockIdx.x + (i + 1) * gridDim.x) * 128 + 16 * (lane & 7);
        if (r1 < prm.n) {
          for (int q = 4 * pw + (lane >> 3); q < h; q += 32)
            asm volatile("prefetch.global.L2 [%0];" ::"l"((const char*)s_x[q] + 8 * r1));
          if (prm.z_kind)
            for (int q = 4 * pw + (lane >> 3); q < w; q += 32)
              asm volatile("prefetch.global.L2 [%0];" ::"l"((const char*)s_z[q] + (prm.z_kind == 2 ? 8 : 4) * r1));
        }
      }
      uint32_t mag = 0;
#pragma unroll
      for (int c = 0; c < 32; c++) mag = max(mag, hi[c] & 0x7FFFFFFFu);
      int e = (int)(mag >> 20);
      if (e == 0) {
        uint32_t any = 0;
#pragma unroll
        for (int c = 0; c < 32; c++) any |= lo[c] | (hi[c] << 1);
        e = any != 0;
      }
      rowpart[i & 1][half][r] = e;
      // the rows' other half is warp pw ^ 4's; a slot is rewritten two tiles
      // later, after another passage through this barrier
      named_bar(1 + (pw & 3), 64);
      const int E = max(rowpart[i & 1][0][r], rowpart[i & 1][1][r]);
      const uint32_t es = oz8_scale(E);
      if (half == 0) rowexp[i % OZY_TILES][r] = oz8_code(E);
      uint32_t top = 0;  // the sums of the magnitudes of the top digits: integers up to 2048
#pragma unroll
      for (int k = 0; k < 4; k++) {
        if (k >= ksteps) break;
        // the step's part of the A slices is free once the previous tile's
        // MMAs on it have completed
        if (i >= 1 && !abort_flag && !mbar_wait_n(&a_empty[k], (uint32_t)((i - 1) & 1), &abort_flag, prm.polls)) {
          abort_flag = 1;
          atomicExch(prm.err, 13);
        }
        if (!abort_flag) {
          tc_fence_after();
          uint32_t pk[OZY_S][4];
          oz8_digits8(lo + 8 * k, hi + 8 * k, es, pk);
          // eight consecutive lanes (rows) write eight different 16-byte
          // bank groups
          const uint32_t off = (uint32_t)r * 128u + ((uint32_t)((2 * k + half) ^ (r & 7)) << 4);
#pragma unroll
          for (int t = 0; t < OZY_S; t++)
            *(uint4*)(adig + t * OZY_ASLICE + off) = make_uint4(pk[t][0], pk[t][1], pk[t][2], pk[t][3]);
          if (BOUND) {
            uint32_t m[4];
            top = oz8_hadd2(top, oz8_magnitudes(pk[0], m));
            *(uint4*)(adig + OZY_S * OZY_ASLICE + off) = make_uint4(m[0], m[1], m[2], m[3]);
            if (k + 1 == ksteps) rowtop[i % OZY_TILES][half][r] = top;
          }
          fence_proxy_async();
          mbar_arrive(&a_full[k]);
        }
      }
    }
  } else if (warp == 16) {
    if (lane == 0) {
      // ------------------------------------------------------- MMA issuer
      const uint32_t abase = smem_u32(adig), cbase = smem_u32(cdig);
      long u = 0;  // units issued
      for (long i = 0; i < my_tiles && !abort_flag; i++) {
        for (int hf = 0; hf < nh; hf++, u++) {
          const int set = (int)(u % K::SETS);
          if (u >= K::SETS &&
              !mbar_wait_n(&acc_empty[set], (uint32_t)((u / K::SETS - 1) & 1), &abort_flag, prm.polls)) {
            abort_flag = 1;
            atomicExch(prm.err, 15);
            break;
          }
          const uint32_t d = tmem + (uint32_t)(set * K::SET);
          for (int ks = 0; ks < ksteps; ks++) {
            if (hf == 0 && !mbar_wait_n(&a_full[ks], (uint32_t)(i & 1), &abort_flag, prm.polls)) {
              abort_flag = 1;
              atomicExch(prm.err, 14);
              break;
            }
            tc_fence_after();
            const uint32_t ab = abase + ks * 32, cb = cbase + hf * K::SLICES * K::BSLICE + ks * 32;
            // slice t against C slices u0 .. u0 + nu - 1 (levels t + u0 ..).
            // t = 1 first: in the first K step its seven levels 1-7 start from
            // zero, level 0 from t = 0, u = 0, and everything else accumulates
            auto mma_at = [&](int level, int t, int u0, int nu, bool fresh) {
              mma_bf16(d + (uint32_t)(level * K::UNIT), sw128_desc(ab + t * OZY_ASLICE),
                       sw128_desc(cb + u0 * K::BSLICE), f16_idesc(128, K::UNIT * nu),
                       (!fresh || ks > 0) ? 1u : 0u);
            };
            auto mma = [&](int t, int u0, int nu, bool fresh) { mma_at(t + u0, t, u0, nu, fresh); };
            if (BOUND) mma_at(8, OZY_S, OZY_S, 1, true);  // D
            mma(1, 0, 7, true);
            if (ks == 0) {
              mma(0, 0, 1, true);
              mma(0, 1, 6, false);
            } else {
              mma(0, 0, 7, false);
            }
            for (int t = 2; t < OZY_S; t++) mma(t, 0, 8 - t, false);
            if (hf + 1 == nh) mma_commit(&a_empty[ks]);
          }
          if (abort_flag) break;
          mma_commit(&acc_full[set]);
        }
      }
      mma_commit(&done_bar);
    }
  } else {
    // ------------------------------------------------------- epilogue
    const int quarter = warp & 3, chalf = warp >> 2;
    const int r = 32 * quarter + lane;
    if (BOUND && tid < 64) {
      const float inv = 1.0f / (float)(colnnz[tid] - 1);
      const bool sums = colnnz[tid] > 1;  // (at most one product: none but the direct ones)
      colkappa[tid] = sums ? 0.503f + 32.01f * inv : 0.f;
      colneed[tid] = sums ? colkappa[tid] * (float)coltop[tid] + (32.01f * (float)h + 5330.f) * inv : HUGE_VALF;
    }
    if (BOUND) named_bar(5, 256);
    long u = 0;
    bool stop = false;
    for (long i = 0; i < my_tiles && !stop; i++) {
      const long row = (blockIdx.x + i * gridDim.x) * 128 + r;
      for (int hf = 0; hf < nh; hf++, u++) {
        const int set = (int)(u % K::SETS);
        const int jbase = hf * K::UNIT + K::UNIT / 2 * chalf;  // this warp's columns
        unsigned long long zn[4];  // Z, four columns ahead
        ozy_load_z(prm.z_kind, s_z, jbase, w, row, prm.n, zn);
        const bool got = mbar_wait_n(&acc_full[set], (uint32_t)((u / K::SETS) & 1), &abort_flag, prm.polls);
        if (!__all_sync(0xffffffffu, got)) {  // tcgen05.ld needs the whole warp
          abort_flag = 1;
          atomicExch(prm.err, 16);
          stop = true;
          // nothing is left as it was: NaN in this warp's part of the units to come
          for (long i1 = i; i1 < my_tiles; i1++) {
            const long row1 = (blockIdx.x + i1 * gridDim.x) * 128 + r;
            for (int h1 = i1 == i ? hf : 0; h1 < nh; h1++)
              for (int c = 0; c < K::UNIT / 2; c++) {
                const int j = h1 * K::UNIT + K::UNIT / 2 * chalf + c;
                if (row1 < prm.n && j < w) ozy_st(s_y[j], row1, __longlong_as_double(0x7ff8000000000000LL));
              }
          }
          break;
        }
        tc_fence_after();
        const int er = rowexp[i % OZY_TILES][r];
        float top = 0.f;
        if (BOUND) top = oz8_both(rowtop[i % OZY_TILES][0][r]) + oz8_both(rowtop[i % OZY_TILES][1][r]);
        const uint32_t tl = tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(set * K::SET + K::UNIT / 2 * chalf);
        double yp[4];
        int jp = -1;
        auto put = [&](const double(&y)[4], int j0) {
#pragma unroll
          for (int jj = 0; jj < 4; jj++)
            if (row < prm.n && j0 + jj < w) ozy_st(s_y[j0 + jj], row, y[jj]);
        };
        // (not unrolled: the roles of a scheduler's warps share its instruction
        // cache)
#pragma unroll 1
        for (int g = 0; g < K::UNIT / 8; g++) {
          const int j0 = jbase + 4 * g;
          if (j0 >= w) break;
          __syncwarp();  // (the branches below are taken by single lanes; tcgen05.ld needs the whole warp)
          uint32_t x[K::LEVELS][4];  // the eight levels (and D) of four columns
          ozy_tmem_ld<K::UNIT, K::LEVELS>(tl + (uint32_t)(4 * g), x);
          // the previous four columns go out only now: their conversions and
          // additions have had this group's start to finish in
          if (g > 0) put(yp, jp);
          unsigned long long zb[4];
#pragma unroll
          for (int jj = 0; jj < 4; jj++) zb[jj] = zn[jj];
          if (g + 1 < K::UNIT / 8) ozy_load_z(prm.z_kind, s_z, j0 + 4, w, row, prm.n, zn);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          // (no branch among the entries: their integer chains overlap)
          double y[4];
          long long T[4];
          // out of the ordinary: the general conversion, or the direct sum
          const int4 ec4 = *(const int4*)&colexp[j0];
          const float4 kp = *(const float4*)&colkappa[BOUND ? j0 : 0], nd4 = *(const float4*)&colneed[BOUND ? j0 : 0];
          const int ec[4] = {ec4.x, ec4.y, ec4.z, ec4.w};
          const float nd[4] = {fmaf(kp.x, top, nd4.x), fmaf(kp.y, top, nd4.y), fmaf(kp.z, top, nd4.z),
                               fmaf(kp.w, top, nd4.w)};
          bool odd = false, weak[4];
#pragma unroll
          for (int jj = 0; jj < 4; jj++) {
            T[jj] = oz8_combine<false>(x[0][jj], x[1][jj], x[2][jj], x[3][jj], x[4][jj], x[5][jj], x[6][jj], x[7][jj]);
            weak[jj] = BOUND && !(__uint_as_float(x[K::LEVELS - 1][jj]) >= nd[jj]);
            // (|T| < 2^32: cancellation, a zero)
            odd |= !oz8_ordinary(er + ec[jj]) || (uint32_t)((T[jj] >> 32) + 1) <= 1u || weak[jj];
          }
          if (odd) {
#pragma unroll
            for (int jj = 0; jj < 4; jj++) {
              y[jj] = oz8_scaled(T[jj], er + ec[jj] - OZ8_BASE);
              // (of a row or column of zeros T is 0)
              if (row < prm.n && j0 + jj < w &&
                  (oz8_direct(er, ec[jj]) || (er && ec[jj] && weak[jj])))
                y[jj] = ozy_direct(s_x, prm.C, prm.ldc, h, j0 + jj, row);
            }
          } else {
#pragma unroll
            for (int jj = 0; jj < 4; jj++) y[jj] = oz8_scaled_fast(T[jj], er + ec[jj] - OZ8_BASE);
          }
          if (prm.z_kind == 1) {
            bool cvt = false;
#pragma unroll
            for (int jj = 0; jj < 4; jj++) cvt |= (((uint32_t)zb[jj] & 0x7FFFFFFFu) - 0x00800000u) >= 0x7F000000u;
            if (cvt) {
#pragma unroll
              for (int jj = 0; jj < 4; jj++) y[jj] += (double)__uint_as_float((uint32_t)zb[jj]);
            } else {
              // a normal FP32 number widened on its bits: the conversion
              // instruction would occupy the FP64 pipe as long as the addition
#pragma unroll
              for (int jj = 0; jj < 4; jj++) {
                const uint32_t z = (uint32_t)zb[jj];
                const uint32_t hi = (z & 0x80000000u) | (((z & 0x7FFFFFFFu) >> 3) + 0x38000000u);
                y[jj] += __hiloint2double((int)hi, (int)(z << 29));
              }
            }
          } else if (prm.z_kind == 2) {
#pragma unroll
            for (int jj = 0; jj < 4; jj++) y[jj] += __longlong_as_double((long long)zb[jj]);
          }
#pragma unroll
          for (int jj = 0; jj < 4; jj++) yp[jj] = y[jj];
          jp = j0;
        }
        __syncwarp();
        tc_fence_before();
        mbar_arrive(&acc_empty[set]);
        if (jp >= 0) put(yp, jp);
      }
    }
  }
  // TMEM is freed only after the last MMA has completed (done_bar is always
  // committed by the issuer) and every epilogue read has finished
  if (warp == 16) {
    mbar_drain(&done_bar, 0);
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 16) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

__global__ void ozy_check_kernel(const int* err, int* status)
{
  if (*err) *status = *err;
}

// columns [0, h) x [0, w) of the tables, h, w <= 64; polls <= 0: the default limit
template <bool BOUND>
static int ozy_launch(gpu_Context* ctx, long n, const void* const* X, int h, const double* C, int ldc,
                      const void* const* Y, int w, const void* const* Z, int z_kind, int polls, int* err)
{
  ozy_params prm;
  memset(&prm, 0, sizeof(prm));
  for (int c = 0; c < h; c++) prm.x[c] = X[c];
  for (int j = 0; j < w; j++) {
    prm.y[j] = (void*)Y[j];
    if (z_kind) prm.z[j] = Z[j];
  }
  prm.C = C;
  prm.ldc = ldc;
  prm.h = h;
  prm.w = w;
  prm.z_kind = z_kind;
  prm.n = n;
  prm.polls = polls > 0 ? (long)polls : TC_WAIT_LIMIT;
  prm.err = err;
  const int smem = ozy_cfg<BOUND>::SMEM;
  if (cudaFuncSetAttribute(oz_xc64_kernel<BOUND>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return gb_fail(ctx, "oz_xc64: cannot reserve %d bytes of shared memory", smem);
  const long ntiles = (n + 127) / 128;
  const unsigned nctas = (unsigned)(ntiles < ctx->num_sms ? ntiles : ctx->num_sms);
  oz_xc64_kernel<BOUND><<<nctas, OZY_THREADS, smem, (cudaStream_t)ctx->stream>>>(prm);
  gb_count_launch(1);
  return gb_cuda_check(ctx, (int)cudaGetLastError(), "oz_xc64");
}

extern "C" int gb_oz_xc64(gpu_Context* ctx, long n, const blk_cols* X, int h, const double* C, int ldc,
                        const blk_cols* Y, int w, const blk_cols* Z, int z_dtype)
{
  if (n <= 0 || w <= 0) return 0;
  if (h < 1 || h > 64 || w > 64)
    return gb_fail(ctx, "oz_xc64: block widths (%d -> %d) not supported", h, w);
  for (int c = 0; c < h; c++)
    if ((uintptr_t)X->col[c] & 15) return gb_fail(ctx, "oz_xc64: input column %d not 16-byte aligned", c);
  int* err = (int*)gb_workspace(ctx, 256);
  if (!err) return -1;
  if (cudaMemsetAsync(err, 0, sizeof(int), (cudaStream_t)ctx->stream) != cudaSuccess)
    return gb_fail(ctx, "oz_xc64: memset failed");
  const int zk = Z ? (z_dtype == GPU_MV_FLOAT64 ? 2 : 1) : 0;
  gb_prof_rec pr;
  gb_prof_begin(ctx, &pr, GB_K_OZ_XC);
  const int rc = ozy_launch<false>(ctx, n, X->col, h, C, ldc, Y->col, w, Z ? Z->col : NULL, zk, ctx->opt.wait_polls, err);
  const double zb = zk == 2 ? 8.0 * w : (zk == 1 ? 4.0 * w : 0.0);
  gb_prof_end(ctx, &pr, (double)n * (8.0 * h + 8.0 * w + zb),
              2.0 * n * h * w);
  if (rc) return rc;
  ozy_check_kernel<<<1, 1, 0, (cudaStream_t)ctx->stream>>>(err, ctx->dcount + 5);
  gb_count_launch(1);
  return gb_cuda_check(ctx, (int)cudaGetLastError(), "oz_xc64_check");
}

// The FP64 block update of gb_bymat for any widths: 64 output columns at a
// time, and within them up to 64 input columns at a time, the later ones added to
// the sum so far.  (The parts' nonzeros add up to the column's, so that the
// roundings of the parts and of the additions stay within its bound.)  A wait that
// gives up is reported in the device error word.
extern "C" int gb_oz_bymat64(gpu_Context* ctx, long n, const blk_cols* X, int h, const double* C, int ldc,
                             const blk_cols* Y, int w, const blk_cols* Z)
{
  // (input columns in equal parts: a part of one or two columns would be summed directly)
  const int hc = (h + (h + 63) / 64 - 1) / ((h + 63) / 64);
  for (int j0 = 0; j0 < w; j0 += 64) {
    const int wj = w - j0 < 64 ? w - j0 : 64;
    for (int i0 = 0; i0 < h; i0 += hc) {
      const int hi = h - i0 < hc ? h - i0 : hc;
      const void* const* z = i0 ? Y->col + j0 : (Z ? Z->col + j0 : NULL);
      if (ozy_launch<true>(ctx, n, X->col + i0, hi, C + i0 + (size_t)j0 * ldc, ldc, Y->col + j0, wj, z, z ? 2 : 0,
                           ctx->opt.wait_polls, ctx->dcount + 5))
        return -1;
    }
  }
  return 0;
}
