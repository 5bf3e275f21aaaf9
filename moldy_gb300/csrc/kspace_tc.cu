// Force pass of the mixed form's reciprocal space on the tensor cores
// (tcgen05; src/ewald.c:557-566).  The structure factor and the per-site
// tables it shares are in kspace_q.cu.
#include <atomic>
#include <cmath>

#include "mdgpu_internal.h"
#include "tc.cuh"

namespace mdgpu {

__device__ __forceinline__ void tc_abort(int *flag, int *err, int bit)
{
   *(volatile int *)flag = 1;
   atomicOr(err, bit);
}

__device__ __forceinline__ bool tc_aborted(const int *flag)
{
   return *(const volatile int *)flag != 0;
}

// ------------------------------------------------------------- forces
// The force pass of ewald() (src/ewald.c:557-566): for a charged site j,
//     F_j = q_j sum_k k (sin(k.r_j) A_k - cos(k.r_j) B_k) = q_j sum_k k Im(e_jk U_k),
// U_k = A_k - i B_k.  An item i is a column (h, k) of the k-list, its
// k-vectors (h, k, +-t) taken together: with seed_ij = exp(2 pi i (h u_x +
// k u_y)), z_j(t) = C_t + i S_t and U+-_t the coefficients at l = +-t,
//     W1_ij = sum_t C_t (U+ + U-) + i S_t (U+ - U-),
//     W2_ij = sum_t t (C_t (U+ - U-) + i S_t (U+ + U-)),
//     F_j += q_j (kx f1, ky f1, kz0 f1 + dkz f2),  f1,2 = Im(seed_ij W1,2_ij).
// W is a product of the sites x t z tables (per 8 t: 8 cosines, 8 sines,
// one K-step of 16) and four coefficient rows per item, real and imaginary
// parts of W1 and W2, each pair of rows scaled by a power of two to |v| <= 1
// (the scale is folded into the item's force coefficients).  Taking l = +-t
// together halves K against a running l from the column's first k-vector
// (131,072-site water: 0.50 -> 0.42 ms, then bound by the
// epilogue's latency).  Operands are three bf16 terms on
// fixed grids (tc.cuh), six term products (hh into one accumulator, where
// sums are exact, the rest into another): the k-space force on a site is a
// near-cancelling sum over k, and two fp16 terms (2^-22 per operand, three
// products) raised the force error of the fixtures to 1.1e-5.  A CTA holds
// one 128-site tile's z tables (up to 96 KB) at a time and streams the
// coefficient rows of 32 items (N = 128) per tile of items, two K-steps per
// stage (only the K-steps an item tile's longest item needs); tensor memory
// holds two accumulator pairs, so the epilogue of one item tile (16 warps,
// four per tensor-memory lane quarter, 8 items -- one unit of four quads --
// each: the seeds by products of the site's x and y tables, the k-vector
// weights, Kahan-compensated FP32 force sums) overlaps the MMAs of the next.
// Systems with more than 64 t values run once per 64-wide t-block.
constexpr int FTC_NI = 32;                         // items per item tile (4 rows each: N = 128)
constexpr int FTC_NSB = 2;                         // coefficient stages in flight per ring (two rings)
constexpr int FTC_KSMAX = 512;                     // item tiles whose K-step counts are kept in shared memory
constexpr int FTC_ATERM = 128 * 128 * 2;           // one term of a site tile's z tables: 32 KB
constexpr int FTC_BTERM = 128 * 16 * 2;            // one term of a coefficient stage: 4 KB
constexpr int FTC_BBYTES = 3 * FTC_BTERM;          // 12 KB
constexpr int FTC_SBYTES = 2 * FTC_BBYTES;         // a stage: two K-steps (24 KB), one wait and commit per 12 MMAs
constexpr int FTC_EG = 4;                          // epilogue warps per tensor-memory lane quarter
constexpr int FTC_IPW = FTC_NI / FTC_EG;           // items of a tile per epilogue warp
constexpr int FTC_EW = 4 * FTC_EG;                 // epilogue warps
constexpr int FTC_XBYTES = 2 * FTC_EG * 128 * 3 * 4 + FTC_EW * FTC_IPW * 16;   // force sums, coefficients
// Shared memory for z tables of aterm bytes a term: no more than needed, the
// rest of the SM's 256 KB caches the x and y tables (131,072-site water:
// 0.346 ms at 208 KB, 0.377 ms with a third coefficient stage, 226 KB).
__host__ __device__ constexpr int ftc_smem(int aterm) { return 3 * aterm + 2 * FTC_NSB * FTC_SBYTES + FTC_XBYTES; }
constexpr int FTC_THREADS = 32 * (FTC_EW + 3);     // epilogue warps, a bulk-copy warp, two MMA warps
__host__ __device__ constexpr size_t ftc_utab_len(int nitems) { return (size_t)(nitems / FTC_NI) * 8 * (FTC_BBYTES / 16); }
static_assert(FTC_IPW % 4 == 0, "an epilogue warp reads its items' columns 16 at a time");
constexpr int FTC_SPLITS = 2;                      // force slots per site (two CTAs at most per site tile)
constexpr int FTC_ERR = 16;                        // error-word bit: a force-pass wait expired

// A launch takes one or two groups of sites (grid y): all, or with a framework
// molecule the others and the framework's charged sites, each with its own
// coefficients.  On a small system a launch of its own costs each kernel as
// much as its work (water on a charged wall, 1044 sites: an evaluation 144 us
// with launches for each, 125 us so).
struct FtcRanges {          // a group's work ranges
   int tiles, G;            // site tiles, ranges
   int *ustart;
};
struct FtcSecond {          // the second group: sites, ranges, and its data from the first's on
   int n, G;
   const int *ustart;
   size_t x, y, z, fpart;
};

// K-steps (8 t each) of an item tile in the t-block from t0: its first unit's
// t range is the longest (units in order of falling range)
__device__ __forceinline__ int ftc_ksteps(int4 un, int t0)
{
   return un.w < 0 ? 0 : min(max(un.z - t0 + 7, 0) >> 3, 8);
}

// Work ranges of the persistent force pass.  Unit u is (site tile u / ntl,
// item tile u % ntl); CTA c takes units ustart[c] .. ustart[c + 1] - 1, a
// contiguous run over the site tiles.  The runs split the units' weights
// (an item tile's K-steps plus one for its epilogue) evenly over G CTAs,
// with G <= the number of site tiles (or G = twice that, each CTA then half
// a tile), so no run lies strictly inside a site tile and a tile is shared
// by two CTAs at most.  One block of 256; pre holds the prefix weights of the
// item tiles, in shared memory (sh, FTC_PRE entries; with the search's reads, one
// after the other, from global memory an evaluation of 1044 sites took 127
// us in place of 125.5) or, for more tiles, after ustart[G].  Made by every evaluation: ranges kept for
// the next one would be another call's (the gradient runs over all sites) by
// the time a captured evaluation is replayed.
constexpr int FTC_PRE = 2048;
__device__ __forceinline__ void ftc_ranges(const int4 *__restrict__ fu, int t0, int ntl, int nsite_tiles, int G, int *ustart,
                                           int *sh)
{
   int *pre = ntl < FTC_PRE ? sh : ustart + G + 1;
   __shared__ int wsum[8];
   const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
   const int run = (ntl + 255) / 256, ta = min(ntl, tid * run), tb = min(ntl, ta + run);   // this thread's tiles
   int sum = 0;
   for (int t = ta; t < tb; t++) sum += ftc_ksteps(fu[t * (FTC_NI / 8)], t0) + 1;
   int inc = sum;   // inclusive over the threads
#pragma unroll
   for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
   }
   if (lane == 31) wsum[w] = inc;
   __syncthreads();
   int at = inc - sum;
   for (int k = 0; k < w; k++) at += wsum[k];
   if (tid == 0) pre[0] = 0;
   for (int t = ta; t < tb; t++) {
      at += ftc_ksteps(fu[t * (FTC_NI / 8)], t0) + 1;
      pre[t + 1] = at;
   }
   __syncthreads();
   const long long wt = pre[ntl], wall = wt * nsite_tiles;
   for (int c = threadIdx.x; c <= G; c += blockDim.x) {
      const long long target = (long long)c * wall / G;
      const long long tile = target / wt, rem = target - tile * wt;
      int lo = 0, hi = ntl;   // the first item tile whose prefix weight reaches rem
      while (lo < hi) {
         const int mid = (lo + hi) >> 1;
         if (pre[mid] >= rem)
            hi = mid;
         else
            lo = mid + 1;
      }
      ustart[c] = (int)(tile * ntl + lo);
   }
}

// Coefficient rows of each item from the dense per-(quad, t) A and B
// (k_qreduce): one warp per item, 64 t from t0.  Item 8 j + 2 q + s is quad
// q of unit fu[j] with k = +-m.  Layout per (item tile, K-step of 16): [term]
// [cosines, sines][row group 16][8 rows][8 t] bf16, row 8 q + 2 c + s for
// the items (q, s) of the tile: the two signs of k side by side, as the
// epilogue takes them in paired FP32 instructions; the force coefficients
// likewise, per q (x+ x- y+ y-), (z0+ z0- dz+ dz-).  The block after the last
// makes the group's work ranges (a cell that changes every step needs them
// every step: a launch of their own took 3-4 us).
__global__ void __launch_bounds__(256)
k_utab_tc(int nitems, QGeom g, int t0, int scalar, const int4 *__restrict__ fu, const float4 *__restrict__ ab,
          const float4 *__restrict__ ab2, uint4 *__restrict__ utab, float *__restrict__ coef, FtcRanges ra, FtcRanges rb)
{
   __shared__ float4 sv[8][64];
   static_assert(sizeof sv >= FTC_PRE * sizeof(int), "the ranges' prefix weights");
   if (blockIdx.x == gridDim.x - 1) {   // (uniform)
      const FtcRanges r = blockIdx.y ? rb : ra;
      ftc_ranges(fu, t0, nitems / FTC_NI, r.tiles, r.G, r.ustart, reinterpret_cast<int *>(sv));
      return;
   }
   if (blockIdx.y) {
      ab = ab2;
      utab += ftc_utab_len(nitems);
      coef += (size_t)nitems * 4;
   }
   const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const int i = blockIdx.x * 8 + wl;
   if (i >= nitems) return;   // (warp-uniform)
   const int4 un = fu[i >> 3];
   const int q = (i >> 1) & 3, neg = i & 1;
   float m1 = 0.f, m2 = 0.f;
#pragma unroll
   for (int h = 0; h < 2; h++) {
      const int t = t0 + lane + 32 * h;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);   // A+, B+, A-, B-
      if (un.w >= 0 && t < g.TP) v = ab[((size_t)(4 * un.w + q) * g.TP + t) * 2 + neg];
      sv[wl][lane + 32 * h] = v;
      const float a = fmaxf(fabsf(v.x + v.z), fabsf(v.x - v.z)), b = fmaxf(fabsf(v.y + v.w), fabsf(v.y - v.w));
      m1 = fmaxf(m1, fmaxf(a, b));
      m2 = fmaxf(m2, (float)t * fmaxf(a, b));
   }
#pragma unroll
   for (int o = 16; o > 0; o >>= 1) {
      m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
      m2 = fmaxf(m2, __shfl_xor_sync(0xffffffffu, m2, o));
   }
   // powers of two at or above the rows' largest magnitude
   int e1 = 0, e2 = 0;
   // (their reciprocals stay finite: rows below 2^-100 are zeros in effect)
   if (m1 > 0.f) frexpf(m1, &e1);
   if (m2 > 0.f) frexpf(m2, &e2);
   e1 = max(e1, -100);
   e2 = max(e2, -100);
   const float s1 = ldexpf(1.f, e1), s2 = ldexpf(1.f, e2), i1 = ldexpf(1.f, -e1), i2 = ldexpf(1.f, -e2);
   __syncwarp();
   const int tile = i / FTC_NI, il = i % FTC_NI, c = lane & 3, ks = lane >> 2;
#pragma unroll
   for (int kg = 0; kg < 2; kg++) {
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; e++) {
         const float4 x = sv[wl][8 * ks + e];
         const float As = x.x + x.z, Ad = x.x - x.z, Bs = x.y + x.w, Bd = x.y - x.w;
         // rows W1re, W1im, W2re, W2im: cosine and sine coefficients
         const float r = kg == 0 ? (c == 0 ? As : c == 1 ? -Bs : c == 2 ? Ad : -Bd)
                                 : (c == 0 ? Bd : c == 1 ? Ad : c == 2 ? Bs : As);
         v[e] = c < 2 ? r * i1 : (float)(t0 + 8 * ks + e) * r * i2;
      }
      unsigned int hh[4], mm[4], ll[4];
#pragma unroll
      for (int j = 0; j < 4; j++) tc::split3(v[2 * j], v[2 * j + 1], hh[j], mm[j], ll[j]);
      const int n = 8 * (il >> 1) + 2 * c + (il & 1);
      const size_t base = ((size_t)tile * 8 + ks) * (FTC_BBYTES / 16) + kg * 128 + (n >> 3) * 8 + (n & 7);
      utab[base] = make_uint4(hh[0], hh[1], hh[2], hh[3]);
      utab[base + FTC_BTERM / 16] = make_uint4(mm[0], mm[1], mm[2], mm[3]);
      utab[base + 2 * FTC_BTERM / 16] = make_uint4(ll[0], ll[1], ll[2], ll[3]);
   }
   if (lane == 0) {
      // the seeds' table scale (units of 2^-24 and 2^-31, times Q_KAPPA each) folded in
      const double f2 = 1.0 / (16777216.0 * 2147483648.0 * Q_KAPPA * Q_KAPPA);
      const double hh = un.x, kk = neg ? -(double)(un.y + q) : (double)(un.y + q);
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (un.w >= 0) {
         if (scalar) {   // f1 alone
            v[0] = (float)(f2 * s1);
         } else {
            v[0] = (float)((hh * g.b[0] + kk * g.b[3]) * f2 * s1);
            v[1] = (float)((hh * g.b[1] + kk * g.b[4]) * f2 * s1);
            v[2] = (float)((hh * g.b[2] + kk * g.b[5]) * f2 * s1);
            v[3] = (float)(g.b[8] * f2 * s2);
         }
      }
#pragma unroll
      for (int k = 0; k < 4; k++) coef[(i >> 1) * 8 + 2 * k + (i & 1)] = v[k];
   }
}

__device__ __forceinline__ void kahan_add_tc(float &s, float &c, float x)
{
   const float y = x - c;
   const float t = s + y;
   c = (t - s) - y;
   s = t;
}

// Persistent: one CTA per work range (ftc_ranges).  Per site tile of the
// range the CTA loads its z tables once (after the MMAs of the previous tile
// have completed) and runs its item tiles as before; the epilogue writes the
// tile's forces into slot 0 of fpart, or slot 1 when the range starts inside
// the tile (and zeros into slot 1 when the range covers the whole tile).
__global__ void __launch_bounds__(FTC_THREADS, 1)
k_force_tc(QGeom g, const int4 *__restrict__ fu, const float4 *__restrict__ coef, int nitems, int t0,
           const int *__restrict__ X, const int *__restrict__ Y, const uint4 *__restrict__ zsite,
           const uint4 *__restrict__ utab, int n, int G, const int *__restrict__ ustart, double *__restrict__ fpart,
           FtcSecond s2, int *__restrict__ err)
{
   using namespace tc;
   extern __shared__ __align__(1024) unsigned char sm[];
   __shared__ __align__(8) uint64_t full_a, a_free, full_b[2][FTC_NSB], empty_b[2][FTC_NSB], acc_full[2],
       acc_empty[2], done[2];
   __shared__ unsigned char s_ks[FTC_KSMAX];
   __shared__ unsigned int tmem_s;
   __shared__ int abort_s;
   const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
   const int ntl = nitems / FTC_NI;   // item tiles per site tile
   if (blockIdx.y) {
      n = s2.n;
      G = s2.G;
      ustart = s2.ustart;
      X += s2.x;
      Y += s2.y;
      zsite += s2.z;
      fpart += s2.fpart;
      utab += ftc_utab_len(nitems);
      coef += nitems;
   }
   if ((int)blockIdx.x >= G) return;   // (uniform)
   const int u0 = ustart[blockIdx.x], u1 = ustart[blockIdx.x + 1];
   if (u1 <= u0) return;              // an empty range (uniform)
   const int T0 = u0 / ntl, T1 = (u1 - 1) / ntl;
   // the range's units of site tile T: ua(T) .. ue(T) - 1; local index u - u0
   auto ua = [&](int T) { return max(u0, T * ntl); };
   auto ue = [&](int T) { return min(u1, (T + 1) * ntl); };
   // the t-block's z tables of a site tile: columns, bytes of a term
   const int fcols = min(128, 2 * (g.TP - t0));
   const unsigned int aterm = (unsigned int)fcols * 256u;
   constexpr int nsb = FTC_NSB;
   unsigned char *A = sm, *Bs = sm + 3 * aterm;
   // [2][FTC_EG][128][3]: per epilogue group, a site tile's force sums (by tile parity)
   float *red = reinterpret_cast<float *>(Bs + 2 * nsb * FTC_SBYTES);
   // per epilogue warp: its items' force coefficients
   float4 *scoef = reinterpret_cast<float4 *>(Bs + 2 * nsb * FTC_SBYTES + 2 * FTC_EG * 128 * 3 * 4);
   if (tid == 0) {
      bar_init(&full_a, 1);
      bar_init(&a_free, 2);
      for (int p = 0; p < 2; p++)
         for (int s = 0; s < FTC_NSB; s++) {
            bar_init(&full_b[p][s], 1);
            bar_init(&empty_b[p][s], 1);
         }
      for (int b = 0; b < 2; b++) {
         bar_init(&acc_full[b], 1);
         bar_init(&acc_empty[b], FTC_EW);
      }
      for (int k = 0; k < 2; k++) bar_init(&done[k], 1);
      abort_s = 0;
      bar_init_fence();
   }
   for (int t = tid; t < ntl && t < FTC_KSMAX; t += FTC_THREADS) s_ks[t] = (unsigned char)ftc_ksteps(fu[t * (FTC_NI / 8)], t0);
   __syncwarp();
   if (w == FTC_EW + 1) tmem_alloc(&tmem_s, 512);   // two buffers x (hh sums, smaller terms) x 128 columns
   fence_before_sync();
   __syncthreads();
   fence_after_sync();
   const unsigned int tmem = tmem_s;
   // K-steps of a unit's item tile
   auto ksteps = [&](int nt) { return nt < FTC_KSMAX ? (int)s_ks[nt] : ftc_ksteps(fu[nt * (FTC_NI / 8)], t0); };

   if (w == FTC_EW) {
      // ---- bulk copies: each site tile's z tables, and the coefficient rows
      // of the range's units, those of local parity p into ring p
      if (lane == 0) {
         int gi[2] = {0, 0}, na = 0;
         bool stop = false;
         for (int T = T0; T <= T1 && !stop; T++) {
            if (T > T0 && !bar_wait(&a_free, (unsigned int)(T - T0 - 1) & 1u)) {
               tc_abort(&abort_s, err, FTC_ERR);
               break;
            }
            bar_expect_tx(&full_a, 3 * aterm);
            bulk_load(A, zsite + ((size_t)T * 2 * g.TP + 2 * t0) * 48, 3 * aterm, &full_a);
            na++;
            int nt = ua(T) - T * ntl;
            for (int u = ua(T); u < ue(T) && !stop; u++, nt++) {
               const int p = (u - u0) & 1, kq = ksteps(nt);
               // stage sq: K-steps 2 sq and, within the unit's, 2 sq + 1
               for (int sq = 0; 2 * sq < kq; sq++) {
                  const int k = gi[p], s = k % nsb;
                  if ((k >= nsb && !bar_wait(&empty_b[p][s], (unsigned int)(k / nsb - 1) & 1u)) ||
                      tc_aborted(&abort_s)) {
                     tc_abort(&abort_s, err, FTC_ERR);
                     stop = true;
                     break;
                  }
                  const unsigned int bytes = 2 * sq + 1 < kq ? FTC_SBYTES : FTC_BBYTES;
                  bar_expect_tx(&full_b[p][s], bytes);
                  bulk_load(Bs + (p * nsb + s) * FTC_SBYTES, utab + ((size_t)nt * 8 + 2 * sq) * (FTC_BBYTES / 16),
                            bytes, &full_b[p][s]);
                  gi[p]++;
               }
            }
         }
         // copies still in flight complete before the CTA's shared memory goes
         if (na > 0) bar_wait(&full_a, (unsigned int)(na - 1) & 1u);
         for (int p = 0; p < 2; p++)
            for (int q = gi[p] > nsb ? gi[p] - nsb : 0; q < gi[p]; q++)
               bar_wait(&full_b[p][q % nsb], (unsigned int)(q / nsb) & 1u);
      }
   } else if (w > FTC_EW) {
      // ---- MMA issue: warp FTC_EW + 1 + p takes the units of local parity p
      // into tensor-memory buffer p (a thread issues one MMA per 150 cycles
      // whatever its N; the tensor pipe needs two at N = 128)
      const int p = w - FTC_EW - 1;
      const unsigned int idn = idesc_bf16(128, 128, false);
      const int ta[6] = {0, 0, 1, 0, 2, 1}, tb[6] = {0, 1, 0, 2, 0, 1};
      const unsigned int a0 = saddr(A), b0 = saddr(Bs + p * nsb * FTC_SBYTES);
      bool ok = true;
      int gi = 0, jj = 0;
      for (int T = T0; T <= T1; T++) {
         if (T > T0) {
            // both issuers are past the previous site tile: its z tables go
            // once their MMAs complete
            __syncwarp();
            asm volatile("bar.sync 1, 64;" : : : "memory");
            if (lane == 0) mma_commit(&a_free);
         }
         if (lane != 0) continue;
         if (ok && !bar_wait(&full_a, (unsigned int)(T - T0) & 1u)) {
            tc_abort(&abort_s, err, FTC_ERR);
            ok = false;
         }
         fence_after_sync();
         int nt = ua(T) - T * ntl;
         for (int u = ua(T); u < ue(T); u++, nt++) {
            if (((u - u0) & 1) != p) continue;
            if (ok && (tc_aborted(&abort_s) ||
                       (jj >= 1 && !bar_wait(&acc_empty[p], (unsigned int)(jj - 1) & 1u)))) {
               tc_abort(&abort_s, err, FTC_ERR);
               ok = false;
            }
            fence_after_sync();
            const int kq = ok ? ksteps(nt) : 0;
            for (int sq = 0; 2 * sq < kq; sq++) {
               const int s = gi % nsb;
               if (!bar_wait(&full_b[p][s], (unsigned int)(gi / nsb) & 1u)) {
                  tc_abort(&abort_s, err, FTC_ERR);
                  ok = false;
                  break;
               }
               fence_after_sync();
#pragma unroll
               for (int h = 0; h < 2; h++) {
                  const int ks = 2 * sq + h;
                  if (ks >= kq) break;
                  const unsigned int bs = b0 + s * FTC_SBYTES + h * FTC_BBYTES;
#pragma unroll
                  for (int t = 0; t < 6; t++) {
                     const uint64_t ad = sdesc(a0 + ta[t] * aterm + ks * 4096, 2048, 128);
                     const uint64_t bd = sdesc(bs + tb[t] * FTC_BTERM, 2048, 128);
                     mma_f16(tmem + p * 256 + (t == 0 ? 0 : 128), ad, bd, idn, ks > 0 || t > 1);
                  }
               }
               mma_commit(&empty_b[p][s]);
               gi++;
            }
            mma_commit(&acc_full[p]);
            jj++;
         }
      }
      if (lane == 0) {
         mma_commit(&done[p]);
         bar_wait(&done[p], 0);   // every MMA complete before the tensor memory is released
      }
   } else {
      // ---- epilogue: site row r of each site tile, items ig * FTC_IPW .. of
      // each item tile
      const int r = 32 * (w & 3) + lane, ig = w >> 2;
      const unsigned int trow = tmem + ((unsigned int)(32 * (w & 3)) << 16);
      float4 *wc = scoef + w * FTC_IPW;
      bool live = true;
      for (int T = T0; T <= T1; T++) {
         const int i = T * 128 + r;
         // the site's x and y tables (a stage of 32 sites, rows of 36)
         const size_t sg = (size_t)T * 4 + (r >> 5);
         const int *xb = X + sg * 2 * g.hrows * 36 + lane, *yb = Y + sg * 2 * g.mrows * 36 + lane;
         float Fx = 0.f, Fy = 0.f, Fz = 0.f, Cx = 0.f, Cy = 0.f, Cz = 0.f;
         // a unit's tables: the site's x and y values, loaded one unit ahead
         int tx[2], ty[8];
         int4 un = make_int4(0, 0, 0, -1);
         float4 cnext = make_float4(0.f, 0.f, 0.f, 0.f);
         auto fetch = [&](int nt) {
            const int pos = nt * (FTC_NI / 8) + ig;   // the warp's eight items
            un = __ldg(&fu[pos]);
            if (lane < FTC_IPW) cnext = __ldg(&coef[pos * FTC_IPW + lane]);
            const int *xp = xb + (size_t)2 * un.x * 36, *yp = yb + (size_t)2 * un.y * 36;
            tx[0] = __ldg(xp);
            tx[1] = __ldg(xp + 36);
#pragma unroll
            for (int q = 0; q < 8; q++) ty[q] = __ldg(yp + q * 36);
         };
         int nt = ua(T) - T * ntl;
         fetch(nt);
         for (int u = ua(T); u < ue(T) && live; u++, nt++) {
            const int j = u - u0, b = j & 1;
            // padding units come last; a tile whose units have no t in this
            // block issues no MMAs, so its buffer holds an earlier unit's sums
            const bool real = un.w >= 0 && un.z > t0;
            // the seeds' factors, per quad (P1, P2) and (P3, P4)
            const float ch = (float)tx[0], sh = (float)tx[1];
            float2 sd[4], sn[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
               const float cm = (float)ty[2 * q], sm4 = (float)ty[2 * q + 1];
               const float a = ch * cm, d = sh * sm4, c = sh * cm, e = ch * sm4;
               sd[q] = make_float2(a - d, a + d);   // cosine of the seed, k = +-m
               sn[q] = make_float2(c + e, c - e);   // sine
            }
            __syncwarp();
            if (lane < FTC_IPW) wc[lane] = cnext;
            __syncwarp();
            if (u + 1 < ue(T)) fetch(nt + 1);
            const bool got = !tc_aborted(&abort_s) && bar_wait(&acc_full[b], (unsigned int)(j >> 1) & 1u);
            if (!__all_sync(0xffffffffu, got && !tc_aborted(&abort_s))) {
               if (lane == 0) tc_abort(&abort_s, err, FTC_ERR);
               live = false;
               break;
            }
            fence_after_sync();
            // the warp's accumulator columns (hh sums plus the rest) into
            // registers, then the buffer goes back to its MMA warp at once:
            // the next unit's MMAs into it overlap this unit's arithmetic
            f2x wv[FTC_IPW / 4][8];
#pragma unroll
            for (int grp = 0; grp < FTC_IPW / 4; grp++) {
               float mv[16], cv[16];
               const unsigned int col = (unsigned int)(b * 256 + 4 * FTC_IPW * ig + 16 * grp);
               tmem_ld16(trow + col, mv);
               tmem_ld16(trow + col + 128, cv);
               tmem_wait2(mv, cv);
#pragma unroll
               for (int c = 0; c < 8; c++) wv[grp][c] = add2(pk2(mv[2 * c], mv[2 * c + 1]), pk2(cv[2 * c], cv[2 * c + 1]));
            }
            fence_before_sync();
            __syncwarp();
            if (lane == 0) bar_arrive(&acc_empty[b]);
            if (real) {
               f2x fx = 0ull, fy = 0ull, fz = 0ull;
#pragma unroll
               for (int q = 0; q < 4; q++) {
                  const f2x *W = &wv[q >> 1][4 * (q & 1)];
                  const f2x cs = pk2(sd[q].x, sd[q].y), sv = pk2(sn[q].x, sn[q].y);
                  const f2x f1 = fma2(cs, W[1], mul2(sv, W[0])), f2 = fma2(cs, W[3], mul2(sv, W[2]));
                  const float4 c0 = wc[2 * q], c1 = wc[2 * q + 1];
                  fx = fma2(pk2(c0.x, c0.y), f1, fx);
                  fy = fma2(pk2(c0.z, c0.w), f1, fy);
                  fz = fma2(pk2(c1.x, c1.y), f1, fma2(pk2(c1.z, c1.w), f2, fz));
               }
               float a, d;
               upk2(fx, a, d);
               kahan_add_tc(Fx, Cx, a + d);
               upk2(fy, a, d);
               kahan_add_tc(Fy, Cy, a + d);
               upk2(fz, a, d);
               kahan_add_tc(Fz, Cz, a + d);
            }
         }
         float *rt = red + (size_t)(T & 1) * FTC_EG * 128 * 3;
         float *rr = rt + ((size_t)ig * 128 + r) * 3;
         rr[0] = Fx - Cx;
         rr[1] = Fy - Cy;
         rr[2] = Fz - Cz;
         // the four groups' sums of this site tile, then its output slot
         __syncwarp();
         asm volatile("bar.sync 2, %0;" : : "n"(FTC_EW * 32) : "memory");
         if (w < 4 && i < n && !tc_aborted(&abort_s)) {
            double sx = 0.0, sy = 0.0, sz = 0.0;
            for (int k = 0; k < FTC_EG; k++) {
               const float *rg = rt + ((size_t)k * 128 + r) * 3;
               sx += (double)rg[0];
               sy += (double)rg[1];
               sz += (double)rg[2];
            }
            double *dst = fpart + (u0 > T * ntl ? 3 * (size_t)n : 0);
            dst[i] = sx;
            dst[n + i] = sy;
            dst[2 * (size_t)n + i] = sz;
            if (u0 <= T * ntl && u1 >= (T + 1) * ntl) {
               double *z = fpart + 3 * (size_t)n;
               z[i] = 0.0;
               z[n + i] = 0.0;
               z[2 * (size_t)n + i] = 0.0;
            }
         }
      }
   }
   fence_before_sync();
   __syncthreads();
   if (w == FTC_EW + 1) {
      __syncwarp();
      fence_after_sync();
      tmem_dealloc(tmem, 512);
   }
}

// The force pass of one t-block (its units fu0 .. fu0 + npos - 1 of the
// list, a multiple of four) into slots 0 and 1 of each group's fpart (one
// buffer, the second group's after the first's); returns
// the launches, -1 if out of memory.
static int force_tc_block(cudaStream_t st, const KsForceSites *grp, int ngrp, const QGeom &g, KsDev &d, bool scalar, int blk,
                          int fu0, int npos, int nsm, int *err)
{
   const int ntl = npos * 8 / FTC_NI, t0 = 64 * blk;
   const int4 *fu = d.q_fu.p + fu0;
   FtcRanges r[2] = {};
   for (int k = 0; k < ngrp; k++) {
      const int f = grp[k].f0 > 0, T = (grp[k].n + 127) / 128, G = 2 * T <= nsm ? 2 * T : std::min(nsm, T);
      if (d.tc_ustart[f].ensure((size_t)G + ntl + 2) != cudaSuccess) return -1;
      r[k].tiles = T;
      r[k].G = G;
      r[k].ustart = d.tc_ustart[f].p;
   }
   auto xat = [&](int k) { return (size_t)grp[k].f0 / 32 * 2 * g.hrows * 36; };
   auto yat = [&](int k) { return (size_t)grp[k].f0 / 32 * 2 * g.mrows * 36; };
   auto zat = [&](int k) { return (size_t)grp[k].f0 / 128 * 2 * g.TP * 48; };
   auto fat = [&](int k) { return grp[k].fpart + (size_t)blk * FTC_SPLITS * 3 * grp[k].n; };
   FtcSecond s2 = {};
   if (ngrp > 1) s2 = FtcSecond{grp[1].n, r[1].G, r[1].ustart, xat(1) - xat(0), yat(1) - yat(0), zat(1) - zat(0), (size_t)(fat(1) - fat(0))};
   k_utab_tc<<<dim3(npos + 1, ngrp), 256, 0, st>>>(
      npos * 8, g, t0, scalar ? 1 : 0, fu, reinterpret_cast<const float4 *>(grp[0].ab),
      reinterpret_cast<const float4 *>(ngrp > 1 ? grp[1].ab : nullptr), d.utab.p, reinterpret_cast<float *>(d.tc_coef.p), r[0], r[1]);
   k_force_tc<<<dim3(std::max(r[0].G, r[1].G), ngrp), FTC_THREADS, ftc_smem(256 * std::min(128, 2 * (g.TP - t0))), st>>>(
      g, fu, d.tc_coef.p, npos * 8, t0, d.q_x32.p + xat(0), d.q_y32.p + yat(0), d.zsite.p + zat(0), d.utab.p, grp[0].n, r[0].G,
      r[0].ustart, fat(0), s2, err);
   return 2;
}

int ks_force_tc(cudaStream_t st, const KsForceSites *grp, int ngrp, const QGeom &g, KsDev &d, bool scalar, int nsm, int *err)
{
   int launches = 0;
   for (int b = 0; b < d.q_nfblk; b++) {
      const int nl = force_tc_block(st, grp, ngrp, g, d, scalar, b, d.q_fblk[b], d.q_fblk[b + 1] - d.q_fblk[b], nsm, err);
      if (nl < 0) return -1;
      launches += nl;
   }
   return launches;
}

int ks_force_tc_splits(const KsDev &d) { return FTC_SPLITS * d.q_nfblk; }
size_t ks_tc_utab_len(int npos) { return ftc_utab_len((npos + 3) / 4 * FTC_NI); }

cudaError_t ks_force_tc_init()
{
   return cudaFuncSetAttribute(k_force_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, ftc_smem(FTC_ATERM));
}

}  // namespace mdgpu
