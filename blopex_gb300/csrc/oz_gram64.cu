// oz_gram64.cu -- Gram products G = X' Y of FP64 blocks with the accuracy of
// FP64 arithmetic on the tensor cores, by error-free splitting (oz8_common.cuh).
// It is serial_Multi_VectorInnerProd (blopex_serial_double/multivector/
// multi_vector.c:354-406) for callers' large FP64 blocks (gb_gram_large,
// blockops.cu).
//
// Rows are taken in groups of R = 128 or 256.  Within a group every column
// shares one power of two and is cut into 7 8-bit digits (55 fraction bits);
// the digit products of a level are summed exactly in FP32 in TMEM, recombined
// into one 64-bit integer per group and entry, rounded once to FP64 and added
// into the entry's FP64 sum: one FP64 addition per group where fused
// multiply-adds spend one per row, on a pipe that takes 16 cycles for a warp.
// Each CTA (one per SM) covers every gridDim.x-th group of a tile of up to 64 x
// 64 entries; gram64_finish_kernel adds the CTAs' sums, 32 chains and a tree (X'X
// from its lower triangle, so that it comes out symmetric).
//
// Operands.  B: the digit slices of the tile's X columns, stacked along N.  A:
// the slices of its Y columns, wpad = 16, 32 or 64 rows each, stacked along M so
// that all 128 rows of an MMA work: block a holds the f = 128 / wpad slices t =
// f a .. f a + f - 1.  Against X slice u they land in TMEM column block c = f a
// + u: row block q of the accumulators then holds level c + q, whatever a.
// 19 (f = 2), 11 (f = 4) or 7 (f = 8) MMA columns per X column instead of 34.
// Row block q's sums carry the weight 2^(-8 q); they are added up at the end.
//
// What bounds it: the producers' instructions and latency, ~17 instructions per value
// cut and ~30 per entry and group recombined (32 x 32: 50% of the issue slots, 54% of
// the ALU pipe), and with h > 32 the epilogue, whose 512 TMEM columns leave no second
// set.  So the values are read straight into registers by coalesced loads (four
// lanes a column, any alignment), not staged; a group's scales are found one group
// ahead from the same columns (the second read of a value comes from L2).  Measured,
// 2,097,152 rows, all three kernels: 32 x 32 0.70 ms (FP64 FMAs 3.9 to 5.5; HBM 0.16),
// 64 x 64 1.75 (14.6), X'X of 64 1.42 (7.9).  Error against 64 bits on random blocks 3.0
// to 8.3e-16 of the norm (FMAs 3.8e-16 to 1.2e-15).
//
// Accuracy.  Within a group of R rows, scales S and S', the digits are off by up to
// 2^-55 S S' (|x/S| + |y/S'| + 4) (1-norms: every value cut below 2^-55 of its
// scale, products of levels 8 and up left out, T rounded), which is small beside the
// roundings of multiply-adds only where sum |x_r y_r| is not far below S S' -- not,
// say, for columns that are large in different rows.  So the result is checked.
// The producers sum the groups' Q = sum S^2 and P = sum (S |x/S|)^2 of every column
// (1-norms from the top digits), which bound the error of an entry by
// 2^-55 (sqrt(P Q') + sqrt(Q P') + 4 sqrt(Q Q')); gram64_cover_kernel adds up
// |x_r y_r| over an eighth of the rows in FP32, rounded down, a lower bound of
// sum |x_r y_r|; and gram64_finish_kernel asks for an error of at most
// OZH_ROUNDINGS 2^-53 of it.  Together with the additions over groups and CTAs that
// is within (32 + n / 9728 + 310) 2^-53 sum |x_r y_r|, the bound of the kernels of
// blockops.cu.  Random blocks pass with a factor of 20 to spare; when an entry does
// not, the caller takes the product again with FP64 multiply-adds.
//
// Columns whose scale the digits cannot carry in some group (infinities, NaN,
// values below 2^-960) and pairs of columns whose product's scale is below 2^-924
// are summed directly there with FP64 FMAs.
//
// Per CTA:
//   warps 8-15  producers: a warp cuts 8 columns (a unit) of a 32-row stage at a
//               time into the 64-byte-swizzled K-major slices of a ring;
//   warp 16     allocates TMEM; one thread issues tcgen05.mma.kind::f16
//               (M = 128, N <= 256, K = 16);
//   warps 0-7   recombine a group's accumulators (lane = row; warps w and w + 4
//               share TMEM lanes and halve the columns) into FP64 sums in
//               shared memory.
// Every wait is bounded; a timeout sets the device error word and the outputs
// become NaN.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "internal.h"
#include "oz8_common.cuh"
#include "pdl.cuh"

#define OZH_THREADS 544
#define OZH_PROD 8               // producer warps
#define OZH_STAGE 32             // rows per stage
#define OZH_MAXST 4              // stages of the ring
#define OZH_SMEM_MAX 225280
#define OZH_ROUNDINGS 128        // units of 2^-53 sum |x y| that the digits may be off
#define OZH_SAMPLE 256           // one chunk of 32 rows in so many is covered

struct ozh_params {
  const void *x[BLK_MAXCOLS], *y[BLK_MAXCOLS];
  int h, w, tx, sym;       // tx: tiles along x; sym: X and Y are the same columns
  int nst, acc_off, smem;  // ring stages, offset of the FP64 sums, bytes
  long n;
  long polls;              // limit of one pipeline wait
  double* partial;         // [CTA][w][h]
  double* norms;           // [CTA][Q, P][h + w]
  int* err;
};

// shared-memory descriptor: K-major, 64-byte swizzle, 8-row groups 512 B apart
static __device__ __forceinline__ uint64_t sw64_desc(uint32_t saddr)
{
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)4 << 61;
}

static __device__ __forceinline__ double ozh_ld(const void* p, long i)
{
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(__cvta_generic_to_global((const double*)p + i)));
  return v;
}
static __device__ __forceinline__ uint2 ozh_ld2(const void* p, long i)
{
  uint2 v;
  asm volatile("ld.global.v2.u32 {%0, %1}, [%2];"
               : "=r"(v.x), "=r"(v.y)
               : "l"(__cvta_generic_to_global((const double*)p + i)));
  return v;
}

// the sum over rows r0 .. r1 of one entry by FP64 FMAs
static __device__ __noinline__ double ozh_direct(const void* x, const void* y, long r0, long r1)
{
  double acc = 0.0;
  for (long r = r0; r < r1; r++) acc = fma(ozh_ld(x, r), ozh_ld(y, r), acc);
  return acc;
}

template <int F>  // slices of A stacked in an MMA: 2, 4, 8 (wpad = 64, 32, 16)
__global__ void __launch_bounds__(OZH_THREADS, 1) oz_gram64_kernel(const __grid_constant__ ozh_params prm)
{
  constexpr int WPAD = 128 / F;
  constexpr int SPG = F == 2 ? 4 : 8;   // stages per group: the level sums stay within 2^23
  constexpr bool HALF = SPG == 8;       // 256 rows: T would take 64 bits
  constexpr int BASE = OZ8_BASE - HALF;
  constexpr long R = SPG * OZH_STAGE;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = smem_align1024(smem_raw);
  __shared__ uint64_t a_full[OZH_MAXST], a_empty[OZH_MAXST], acc_full[2], acc_empty[2], done_bar;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  __shared__ int cexp[4][128];         // scales, by group modulo 4: X's columns, then from 64 Y's
  __shared__ const void* s_col[128];
  __shared__ double s_norm[2][128];    // Q and P of the columns

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ti = blockIdx.y % prm.tx, tj = blockIdx.y / prm.tx;
  const int i0 = 64 * ti, j0 = WPAD * tj;
  const int h = min(64, prm.h - i0), w = min(WPAD, prm.w - j0);
  const bool same = prm.sym && i0 == j0 && h == w;  // (sym: WPAD >= 64 or one tile)
  const int hpad = same ? WPAD : (h + 15) & ~15;
  // a stage: A [8 slices][WPAD rows][64 B], then B [7 slices][hpad rows][64 B]
  const uint32_t asz = 8u * WPAD * 64, ssz = asz + (same ? 0u : 7u * (uint32_t)hpad * 64);
  const int nst = prm.nst;
  double* acc = (double*)(smem + prm.acc_off);  // [hpad][128]
  const long ngroups = (prm.n + R - 1) / R;
  const long my_groups = (long)blockIdx.x < ngroups ? (ngroups - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  const int nsets = hpad <= 32 ? 2 : 1;

  if (tid < 128) {
    s_norm[0][tid] = s_norm[1][tid] = 0.0;
    const int c = tid & 63;
    s_col[tid] = tid < 64 ? (c < h ? prm.x[i0 + c] : nullptr) : (c < w ? prm.y[j0 + c] : nullptr);
  }
  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < OZH_MAXST; s++) {
      mbar_init(&a_full[s], OZH_PROD);
      mbar_init(&a_empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 8);
    }
    mbar_init(&done_bar, 1);
  }
  // the zero slice 7 of A and the rows of absent columns stay zero
  for (uint32_t o = 16u * tid; o < nst * ssz; o += 16u * OZH_THREADS) *(uint4*)(smem + o) = make_uint4(0, 0, 0, 0);
  for (int o = tid; o < hpad * 128; o += OZH_THREADS) acc[o] = 0.0;
  if (warp == 16) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;

  if (warp >= 8 && warp < 16) {
    // ------------------------------------------------------- digit slices
    // Units of 8 columns, X's first; lane = (column, quarter q): rows 4 e + q,
    // e = 0 .. 7, of the stage, so that a load takes 32 contiguous bytes of
    // each column.  A lane's 8 values fill the 16-byte chunk q of the column's
    // K-major row: the K order is permuted, alike in both operands.
    // A warp keeps its units' scales in registers and finds the next group's
    // while it cuts this one.
    const int pw = warp - 8, q = lane & 3;
    const int ub = (h + 7) >> 3, nu = same ? ub : ub + ((w + 7) >> 3);
    const int mine = pw < nu ? (nu - pw + OZH_PROD - 1) / OZH_PROD : 0;  // <= 2 units
    const void* col[2];
    uint32_t dst[2], rowstride[2];  // of slice 0 in a stage; bytes from slice to slice
    int slot[2];
    uint32_t emax[2] = {0, 0};      // the largest magnitude word so far of the group being scouted
    uint32_t anyb[2] = {0, 0};      // any bit set (subnormals)
    uint32_t es[2] = {0, 0};
    uint32_t top2[2] = {0, 0};      // the top digits' magnitudes of up to four stages,
    float topf[2] = {0.f, 0.f};     // and of the group so far
#pragma unroll
    for (int m = 0; m < 2; m++) {
      const int u = pw + OZH_PROD * m;
      const bool isb = u < ub;
      const int c = 8 * (isb ? u : u - ub) + (lane >> 2);  // column within X's or Y's tile
      const bool ok = m < mine && c < (isb ? h : w);
      slot[m] = isb ? c : 64 + c;
      col[m] = ok ? s_col[slot[m]] : nullptr;
      dst[m] = (isb && !same ? asz : 0u) + (uint32_t)c * 64u + ((uint32_t)(q ^ ((c >> 1) & 3)) << 4);
      rowstride[m] = (uint32_t)(isb && !same ? hpad : WPAD) * 64u;
    }
    auto load = [&](int m, long r0, uint2(&v)[8]) {
#pragma unroll
      for (int e = 0; e < 8; e++) {
        const long r = r0 + 4 * e + q;
        v[e] = make_uint2(0, 0);
        if (col[m] && r < prm.n) v[e] = ozh_ld2(col[m], r);
      }
    };
    auto scout = [&](int m, const uint2(&v)[8]) {
#pragma unroll
      for (int e = 0; e < 8; e++) {
        emax[m] = max(emax[m], v[e].y & 0x7FFFFFFFu);
        anyb[m] |= v[e].x;
      }
    };
    // the scouted group's scale: to the registers and, for the epilogue, slot g
    auto settle = [&](int m, long g) {
      uint32_t e = emax[m], a = anyb[m];
      e = max(e, __shfl_xor_sync(0xffffffffu, e, 1));
      e = max(e, __shfl_xor_sync(0xffffffffu, e, 2));
      a |= __shfl_xor_sync(0xffffffffu, a, 1);
      a |= __shfl_xor_sync(0xffffffffu, a, 2);
      int E = (int)(e >> 20);
      if (E == 0 && (e | a)) E = 1;  // nothing but subnormals: unsafe
      es[m] = oz8_scale(E);
      // slot g mod 4 was last read by the epilogue of group g - 4, which ended
      // before the MMAs of group g - 1, now well under way, began
      if (q == 0) {
        cexp[g & 3][slot[m]] = oz8_code(E);
        if (same) cexp[g & 3][64 + slot[m]] = oz8_code(E);
      }
      emax[m] = anyb[m] = 0;
    };
    // the group's part of Q and P (|x/S| <= (top digits + R / 2) / 128)
    auto measure = [&](int m) {
      float t = topf[m];
      t += __shfl_xor_sync(0xffffffffu, t, 1);
      t += __shfl_xor_sync(0xffffffffu, t, 2);
      topf[m] = 0.f;
      const int E = (int)(es[m] >> 20);  // 0xFFF: zeros
      if (q == 0 && col[m] && E < 2047 && E >= 64) {
        // (S^2 has to fit: other columns fail the check)
        const double S = E >= 542 && E <= 1502 ? __hiloint2double((E + 1) << 20, 0) : HUGE_VAL;
        const double P = S * (double)(t * 0.0078125f + (float)R * 0.00390625f);
        s_norm[0][slot[m]] += S * S;
        s_norm[1][slot[m]] += P * P;
      }
    };
    auto row_of = [&](long g) { return (blockIdx.x + g * gridDim.x) * R; };
    uint2 v[8];
    if (my_groups > 0) {
#pragma unroll
      for (int m = 0; m < 2; m++) {
        if (m < mine) {
#pragma unroll 1
          for (int s = 0; s < SPG; s++) {
            load(m, row_of(0) + s * OZH_STAGE, v);
            scout(m, v);
          }
          settle(m, 0);
        }
      }
      load(0, row_of(0), v);
    }
    int buf = 0;
    uint32_t phase = 1;  // of the slot's release; the first round finds it free
    for (long g = 0; g < my_groups; g++) {
      const bool more = g + 1 < my_groups;
#pragma unroll 1
      for (int s = 0; s < SPG; s++) {
        if (!abort_flag && !mbar_wait_n(&a_empty[buf], phase, &abort_flag, prm.polls)) {
          abort_flag = 1;
          atomicExch(prm.err, 31);
        }
        unsigned char* base = smem + (size_t)buf * ssz;
        const long rnext = s + 1 < SPG ? row_of(g) + (s + 1) * OZH_STAGE : row_of(g + 1);
#pragma unroll
        for (int m = 0; m < 2; m++) {
          if (m < mine) {
            uint2 vs[8];
            if (more) load(m, row_of(g + 1) + s * OZH_STAGE, vs);
            uint32_t pk[OZ8_S][4];
            {
              uint32_t lo[8], hi[8];
#pragma unroll
              for (int e = 0; e < 8; e++) {
                lo[e] = v[e].x;
                hi[e] = v[e].y;
              }
              oz8_digits8(lo, hi, es[m], pk);
              uint32_t mag[4];
              top2[m] = oz8_hadd2(top2[m], oz8_magnitudes(pk[0], mag));
              if ((s & 3) == 3) {
                topf[m] += oz8_both(top2[m]);
                top2[m] = 0;
              }
            }
            // the next unit's values
            if (m + 1 < mine)
              load(1, row_of(g) + s * OZH_STAGE, v);
            else
              load(0, rnext, v);
            if (col[m] && !abort_flag) {
#pragma unroll
              for (int t = 0; t < OZ8_S; t++)
                *(uint4*)(base + dst[m] + t * rowstride[m]) = make_uint4(pk[t][0], pk[t][1], pk[t][2], pk[t][3]);
            }
            if (more) scout(m, vs);
          }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0 && !abort_flag) mbar_arrive(&a_full[buf]);
        if (++buf == nst) {
          buf = 0;
          phase ^= 1;
        }
      }
#pragma unroll
      for (int m = 0; m < 2; m++) {
        if (m < mine) {
          measure(m);
          if (more) settle(m, g + 1);
        }
      }
    }
    // X's columns from the tiles of the first column, Y's from those of the first row
#pragma unroll
    for (int m = 0; m < 2; m++) {
      if (q == 0 && col[m] && (slot[m] < 64 ? tj : ti) == 0) {
        double* out = prm.norms + (size_t)blockIdx.x * 2 * (prm.h + prm.w) +
                      (slot[m] < 64 ? i0 + slot[m] : prm.h + j0 + slot[m] - 64);
        out[0] = s_norm[0][slot[m]];
        out[prm.h + prm.w] = s_norm[1][slot[m]];
      }
    }
  } else if (warp == 16) {
    if (lane == 0) {
      // ----------------------------------------------------- MMA issuer
      const uint32_t sbase = smem_u32(smem);
      int buf = 0;
      uint32_t phase = 0;
      for (long g = 0; g < my_groups && !abort_flag; g++) {
        const int set = (int)(g % nsets);
        if (g >= nsets && !mbar_wait_n(&acc_empty[set], (uint32_t)((g / nsets - 1) & 1), &abort_flag, prm.polls)) {
          abort_flag = 1;
          atomicExch(prm.err, 32);
          break;
        }
        const uint32_t d = tmem + (uint32_t)(set * 256);
        for (int s = 0; s < SPG; s++) {
          if (!mbar_wait_n(&a_full[buf], phase, &abort_flag, prm.polls)) {
            abort_flag = 1;
            atomicExch(prm.err, 33);
            break;
          }
          tc_fence_after();
          const uint32_t ab = sbase + (uint32_t)buf * ssz, bb = ab + (same ? 0u : asz);
          for (int ks = 0; ks < 2; ks++) {
            // block a of A against X slices u0 .. u1 - 1, 256 columns at most
            // at a time
            auto mma = [&](int a, int u0, int u1, bool fresh) {
              const int per = 256 / hpad;
              for (int u = u0; u < u1; u += per) {
                const int k = min(per, u1 - u);
                mma_bf16(d + (uint32_t)((F * a + u) * hpad), sw64_desc(ab + (uint32_t)a * 8192u + 32u * ks),
                         sw64_desc(bb + (uint32_t)(u * hpad) * 64u + 32u * ks), f16_idesc(128, hpad * k),
                         fresh ? 0u : 1u);
              }
            };
            const bool first = s == 0 && ks == 0;
            if (F == 8) {
              mma(0, 0, 7, first);
            } else {
              // a = 1 first: in a group's first step its column blocks F .. 7
              // start from zero, blocks 0 .. F - 1 from a = 0
              mma(1, 0, 8 - F, first);
              if (first) {
                mma(0, 0, F, true);
                mma(0, F, 7, false);
              } else {
                mma(0, 0, 7, false);
              }
              for (int a = 2; F * a < 7; a++) mma(a, 0, 8 - F * a, false);
            }
          }
          mma_commit(&a_empty[buf]);
          if (++buf == nst) {
            buf = 0;
            phase ^= 1;
          }
        }
        if (abort_flag) break;
        mma_commit(&acc_full[set]);
      }
      mma_commit(&done_bar);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------- epilogue
    const int quarter = warp & 3, chalf = warp >> 2;
    const int r = 32 * quarter + lane, q = r / WPAD, j = r % WPAD;
    const int c0 = chalf * (hpad / 2), c1 = c0 + hpad / 2;
    const bool live = j < w && (F < 8 || q < 7);
    bool ok = true;
    for (long g = 0; g < my_groups; g++) {
      const int set = (int)(g % nsets);
      const bool got = mbar_wait_n(&acc_full[set], (uint32_t)((g / nsets) & 1), &abort_flag, prm.polls);
      if (!__all_sync(0xffffffffu, got)) {  // tcgen05.ld needs the whole warp
        abort_flag = 1;
        atomicExch(prm.err, 34);
        ok = false;
        break;
      }
      tc_fence_after();
      const int ej = live ? cexp[g & 3][64 + j] : 1023;
      const uint32_t tl = tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(set * 256);
      // four columns at a time (not unrolled: the roles of a scheduler's warps
      // share its instruction cache)
#pragma unroll 1
      for (int i = c0; i < c1 && i < h; i += 4) {
        __syncwarp();  // (the branch below is taken by single lanes; tcgen05.ld needs the whole warp)
        uint32_t x[8][4];
#pragma unroll
        for (int c = 0; c < (F == 8 ? 7 : 8); c++)
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(x[c][0]), "=r"(x[c][1]), "=r"(x[c][2]), "=r"(x[c][3])
                       : "r"(tl + (uint32_t)(c * hpad + i)));
        if (F == 8) x[7][0] = x[7][1] = x[7][2] = x[7][3] = 0;
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        int ei[4];
        long long T[4];
        bool odd = false;
#pragma unroll
        for (int e = 0; e < 4; e++) {
          ei[e] = i + e < h ? cexp[g & 3][i + e] : 1023;
          T[e] = oz8_combine<HALF>(x[0][e], x[1][e], x[2][e], x[3][e], x[4][e], x[5][e], x[6][e], x[7][e]);
          // (|T| < 2^32: cancellation, a zero; absent entries do not count)
          odd |= !oz8_ordinary(ei[e] + ej) || ((uint32_t)((T[e] >> 32) + 1) <= 1u && live && i + e < h);
        }
        double v[4];
        if (odd) {
#pragma unroll
          for (int e = 0; e < 4; e++) {
            v[e] = oz8_scaled(T[e], ei[e] + ej - BASE - 8 * q);
            if (oz8_direct(ei[e], ej)) {
              const long r0 = (blockIdx.x + g * gridDim.x) * R;
              v[e] = live && q == 0 && i + e < h
                         ? ozh_direct(s_col[i + e], s_col[64 + j], r0, min(r0 + R, prm.n))
                         : 0.0;
            }
          }
        } else {
#pragma unroll
          for (int e = 0; e < 4; e++) v[e] = oz8_scaled_fast(T[e], ei[e] + ej - BASE - 8 * q);
        }
#pragma unroll
        for (int e = 0; e < 4; e++) acc[(size_t)(i + e) * 128 + r] += v[e];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[set]);
    }
    // the row blocks' sums, added in order of weight: entry (i, j)
    named_bar(1, 256);
    double* out = prm.partial + (size_t)blockIdx.x * prm.h * prm.w;
    for (int e = tid; e < h * w; e += 256) {
      const int i = e % h, jj = e / h;
      double s = 0.0;
#pragma unroll
      for (int k = (F == 8 ? 7 : F) - 1; k >= 0; k--) s += acc[(size_t)i * 128 + k * WPAD + jj];
      if (!ok || abort_flag) s = __longlong_as_double(0x7ff8000000000000LL);
      out[(size_t)(j0 + jj) * prm.h + i0 + i] = s;
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

// Lower bounds of sum |x_r y_r|: the CTAs' sums over every gridDim.z-th of the sampled
// chunks (32 rows of each OZH_SAMPLE, moving through them), 32 x 32 entries, in FP32 on
// values cut to 20 bits and scaled by a power of two near the column's rms scale
// (from Q; values 2^40 above it count as that much, far smaller ones as 0).  The
// CTAs of the first layer also leave the columns' Q and P over all groups in tot.
__global__ void __launch_bounds__(256) gram64_cover_kernel(blk_cols X, int h, blk_cols Y, int w, int sym, long n,
                                                           const double* __restrict__ norms, int parts, long groups,
                                                           double* __restrict__ tot, double* __restrict__ cover,
                                                           int* verdict)
{
  gb_pdl_entry();
  __shared__ float xs[32][33], ys[32][33];
  __shared__ double sq[64][5];
  __shared__ int eref[64];  // the columns' reference exponents (biased): X's, Y's
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
  if (t == 0 && blockIdx.x + blockIdx.y + blockIdx.z == 0) verdict[0] = 0;
  {
    const int c = t >> 2;
    const int k = c < 32 ? i0 + c : j0 + c - 32, hw = h + w;
    const bool on = k < (c < 32 ? h : w);
    const double* np = norms + (c < 32 || sym ? k : h + k);
    double s = 0.0;
    if (on)
#pragma unroll 4
      for (int p = t & 3; p < parts; p += 4) s += np[(size_t)p * 2 * hw];
    sq[c][t & 3] = s;
    if (blockIdx.z == 0 && (c < 32 ? blockIdx.y : blockIdx.x) == 0) {  // (whole warps)
      double q = 0.0;
      if (on)
        for (int p = t & 3; p < parts; p += 4) q += np[(size_t)p * 2 * hw + hw];
      for (int o = 1; o < 4; o <<= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        q += __shfl_xor_sync(0xffffffffu, q, o);
      }
      if (on && (t & 3) == 0) {
        tot[c < 32 ? k : h + k] = s;
        tot[hw + (c < 32 ? k : h + k)] = q;
      }
    }
  }
  __syncthreads();
  if (t < 64) {
    const double s = (sq[t][0] + sq[t][1] + sq[t][2] + sq[t][3]) / (double)groups;
    const int e = (int)((uint32_t)__double2hiint(s) >> 20) - 1023;  // of the mean of S^2
    eref[t] = s > 0.0 && e < 1000 ? 1022 + (e >> 1) : 1022;
  }
  __syncthreads();
  // a value's place in the tile: row t % 32 of the chunk, columns t / 32 + 8 k
  const uint32_t* col[8];
  int ref[8];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int c = (t >> 5) + 8 * k;
    const int i = i0 + c, j = j0 + c - 32;
    col[k] = (const uint32_t*)(c < 32 ? (i < h ? X.col[i] : NULL) : (j < w ? Y.col[j] : NULL));
    ref[k] = eref[c] - 127;
  }
  const long blocks = (n + OZH_SAMPLE - 1) / OZH_SAMPLE;
  float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
  uint32_t v[8];
  auto load = [&](long b) {
    long r = b * OZH_SAMPLE + 32 * ((5 * b + (b >> 3)) & (OZH_SAMPLE / 32 - 1));
    if (r >= n) r = b * OZH_SAMPLE;
    r += t & 31;
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = b < blocks && col[k] && r < n ? col[k][2 * r + 1] : 0u;  // the high word
  };
  load(blockIdx.z);
  for (long b = blockIdx.z; b < blocks; b += gridDim.z) {
#pragma unroll
    for (int k = 0; k < 8; k++) {
      // biased FP32 exponent e - ref, the leading 20 bits of the fraction
      const int d = (int)(v[k] & 0x7FFFFFFFu) - (ref[k] << 20);
      const int e = d < 0x100000 ? 0 : min(d, 167 << 20);
      const float f = __int_as_float(e << 3);
      const int c = (t >> 5) + 8 * k;
      if (c < 32)
        xs[c][t & 31] = f;
      else
        ys[c - 32][t & 31] = f;
    }
    __syncthreads();
    load(b + gridDim.z);
#pragma unroll 8
    for (int r = 0; r < 32; r++) {
      const float x0 = xs[tx][r], x1 = xs[tx + 16][r], y0 = ys[ty][r], y1 = ys[ty + 16][r];
      acc[0][0] = fmaf(x0, y0, acc[0][0]);
      acc[0][1] = fmaf(x0, y1, acc[0][1]);
      acc[1][0] = fmaf(x1, y0, acc[1][0]);
      acc[1][1] = fmaf(x1, y1, acc[1][1]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 2; a++)
#pragma unroll
    for (int b = 0; b < 2; b++) {
      const int ii = tx + 16 * a, jj = ty + 16 * b;
      if (i0 + ii < h && j0 + jj < w)
        cover[((size_t)blockIdx.z * w + j0 + jj) * h + i0 + ii] =
            (double)acc[a][b] * __hiloint2double(eref[ii] << 20, 0) * __hiloint2double(eref[32 + jj] << 20, 0);
    }
}

// G from the CTAs' sums, 32 threads an entry: strides of 32 in order, then a tree of
// the 32 (in one chain, 152 sums of growing size were the largest part of the error:
// 30,000 x 64 x 64 5.6e-16, multiply-adds 4.7e-16).  verdict[0] = 1 where the digits'
// error may exceed its share; [1]: the error word
__global__ void __launch_bounds__(256) gram64_finish_kernel(const double* __restrict__ partial, int parts,
                                                            const double* __restrict__ tot,
                                                            const double* __restrict__ cover, int covers, int h, int w,
                                                            int sym, const int* err, double* __restrict__ G, int ldg,
                                                            int* verdict)
{
  gb_pdl_entry();
  __shared__ double sm[2][32][9];
  const int x = threadIdx.x & 7, y = threadIdx.x >> 3;  // 8 entries a CTA
  if (blockIdx.x == 0 && threadIdx.x == 0) verdict[1] = *err;
  const long E = (long)h * w, e0 = blockIdx.x * 8L + x, e = min(e0, E - 1);
  const int i = (int)(e % h), j = (int)(e / h), hw = h + w;
  const long src = sym && i < j ? (long)i * h + j : e;
  double g = 0.0, s = 0.0;
#pragma unroll 4
  for (int p = y; p < parts; p += 32) g += partial[(size_t)p * E + src];
#pragma unroll 4
  for (int p = y; p < covers; p += 32) s += cover[(size_t)p * E + e];
  sm[0][y][x] = g;
  sm[1][y][x] = s;
  for (int o = 16; o > 0; o >>= 1) {
    __syncthreads();
    if (y < o) {
      sm[0][y][x] += sm[0][y + o][x];
      sm[1][y][x] += sm[1][y + o][x];
    }
  }
  if (y || e0 >= E) return;
  G[(size_t)j * ldg + i] = sm[0][0][x];
  const double qx = sqrt(tot[i]), px = sqrt(tot[hw + i]), qy = sqrt(tot[h + j]), py = sqrt(tot[hw + h + j]);
  // (0.9: the roundings of the FP32 sums)
  const bool ok =
      qx == 0.0 || qy == 0.0 || px * qy + qx * py + 4.0 * qx * qy <= 0.9 * 4.0 * OZH_ROUNDINGS * sm[1][0][x];
  if (!ok) verdict[0] = 1;
}

template <int F>
static int ozh_launch(gpu_Context* ctx, ozh_params& prm, double* G, int ldg, int* verdict)
{
  const int WPAD = 128 / F;
  const long R = (F == 2 ? 4 : 8) * OZH_STAGE;
  prm.tx = (prm.h + 63) / 64;
  const int ty = (prm.w + WPAD - 1) / WPAD;
  const int hmax = prm.h < 64 ? (prm.h + 15) & ~15 : 64;
  const int hpad = prm.sym && prm.h <= WPAD ? WPAD : hmax;
  const uint32_t ssz = 8u * WPAD * 64 + 7u * hpad * 64;
  const uint32_t accb = (uint32_t)(hpad > WPAD ? hpad : WPAD) * 128 * 8;
  int nst = (int)((OZH_SMEM_MAX - 1024 - accb) / ssz);
  if (nst > OZH_MAXST) nst = OZH_MAXST;
  if (nst > (int)(R / OZH_STAGE) - 1) nst = (int)(R / OZH_STAGE) - 1;  // the scale slots' reuse relies on it
  prm.nst = nst;
  prm.acc_off = (int)((nst * ssz + 1023) / 1024 * 1024);
  prm.smem = prm.acc_off + (int)accb + 1024;
  const long ngroups = (prm.n + R - 1) / R;
  long gx = ctx->num_sms / (prm.tx * ty);
  if (gx < 1) gx = 1;
  if (gx > ngroups) gx = ngroups;
  // CTAs of the check: four an SM, as many chunks as there are at most
  const int cx = (prm.h + 31) / 32, cy = (prm.w + 31) / 32;
  const long blocks = (prm.n + OZH_SAMPLE - 1) / OZH_SAMPLE;
  long cz = 4L * ctx->num_sms / (cx * cy);
  if (cz < 1) cz = 1;
  if (cz > blocks) cz = blocks;
  const size_t np = (size_t)gx * prm.h * prm.w, nt = (size_t)2 * (prm.h + prm.w), nn = (size_t)gx * nt;
  double* partial = (double*)gb_workspace(ctx, sizeof(double) * (np + nn + nt + (size_t)cz * prm.h * prm.w));
  if (!partial) return -1;
  prm.partial = partial;
  prm.norms = partial + np;
  double *tot = prm.norms + nn, *cover = tot + nt;
  // (prm.smem <= OZH_SMEM_MAX but for the rounding of acc_off; the limit is the
  // function's, for all threads)
  if (cudaFuncSetAttribute(oz_gram64_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, OZH_SMEM_MAX + 1024) !=
      cudaSuccess)
    return gb_fail(ctx, "oz_gram64: cannot reserve %d bytes of shared memory", prm.smem);
  oz_gram64_kernel<F><<<dim3((unsigned)gx, (unsigned)(prm.tx * ty)), OZH_THREADS, prm.smem,
                        (cudaStream_t)ctx->stream>>>(prm);
  blk_cols X, Y;
  for (int c = 0; c < prm.h; c++) X.col[c] = prm.x[c];
  for (int c = 0; c < prm.w; c++) Y.col[c] = prm.y[c];
  cudaStream_t st = (cudaStream_t)ctx->stream;
  gb_pdl(gram64_cover_kernel, dim3(cx, cy, (unsigned)cz), 256, 0, st, X, prm.h, Y, prm.w, prm.sym, prm.n, prm.norms,
         (int)gx, ngroups, tot, cover, verdict);
  gb_pdl(gram64_finish_kernel, (prm.h * prm.w + 7) / 8, 256, 0, st, partial, (int)gx, tot, cover, (int)cz, prm.h, prm.w,
         prm.sym, prm.err, G, ldg, verdict);
  gb_count_launch(3);
  return gb_cuda_check(ctx, (int)cudaGetLastError(), "oz_gram64");
}

// G = X' Y (ldg, device).  sym: X and Y are the same columns.  verdict[0] (device): 1
// when an entry may be further off than FP64 multiply-adds; [1]: the device error
// word (a wait that gave up; the CTA's sums are NaN).
extern "C" int gb_oz_gram64(gpu_Context* ctx, long n, const blk_cols* X, int h, const blk_cols* Y, int w, int sym,
                            double* G, int ldg, int* verdict)
{
  ozh_params prm;
  memset(&prm, 0, sizeof(prm));
  for (int c = 0; c < h; c++) prm.x[c] = X->col[c];
  for (int c = 0; c < w; c++) prm.y[c] = Y->col[c];
  prm.h = h;
  prm.w = w;
  prm.sym = sym;
  prm.n = n;
  prm.polls = ctx->opt.wait_polls > 0 ? (long)ctx->opt.wait_polls : TC_WAIT_LIMIT;
  prm.err = ctx->dcount + 5;
  if (w > 32) return ozh_launch<2>(ctx, prm, G, ldg, verdict);
  if (w > 16) return ozh_launch<4>(ctx, prm, G, ldg, verdict);
  return ozh_launch<8>(ctx, prm, G, ldg, verdict);
}
