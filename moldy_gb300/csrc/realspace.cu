// Real-space link-cell forces on the GPU (the work of force_calc,
// src/force.c:1108-1320, and kernel(), src/kernel.c:157-463).
//
// Pipeline, all on one stream:
//   1. k_bin        FP64 binning of every site (or molecule centre of mass in
//                   molecular-cutoff mode) with the reference's arithmetic and
//                   edge fix-ups (cellbin, src/force.c:119-137);
//   2. scan         cell counts -> cell starts (in k_bin's last block on small
//                   grids, else two kernels);
//   3. k_scatter    sites placed cell by cell (in k_bin's last block on small
//                   systems);
//   4. k_place      each cell's members in ascending site order (deterministic
//                   layout) and per-slot records: FP64 (x,y,z,q), or FP32
//                   co-ordinates relative to the cell origin plus q, and (site
//                   id, molecule);
//   5. k_pairs_col  one warp per home site walks the stencil by columns over
//      k_pairs_col64  one interaction class at a time, accumulating the force
//                   on its own site only; energy and virial take half of each
//                   evaluation, summed in a fixed order by the last block.  No
//                   atomics on forces.  k_pairs and k_reduce_rs walk it cell
//                   by cell with frameworks, molecular cut-offs, the pair-key
//                   listing and stencils that wrap the cell more than once;
//   6. k_tooclose_x pairs across the classes below the too-close distance.
//
// The pair set is the reference's exactly: every site pair of a cell and of
// each stencil cell, with no per-pair cutoff in lazy mode and r^2 clamped to
// 1e4 rc^2 in strict mode (src/force.c:951-954).  In FP64 form r and r^2 are
// formed with the reference's operation order and no fused multiply-adds, so
// the clamp and the too-close test decide exactly as the reference does.  In
// mixed form r is formed in FP32 from cell-relative co-ordinates and an
// (hi, lo) pair of the exact cell-offset vector; decisions within a narrow
// band of the threshold are re-made in FP64 from the original co-ordinates.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "mdgpu_internal.h"

namespace mdgpu {

struct RsParams {
   int nsites, nent, nx, ny, nz, ncells, nfull, max_id, molpbc, strict, ptype, pot_in_smem;
   // the framework molecule (-1: none), its first site, and the number of
   // molecule entities binned by centre of mass in molecular-cutoff mode
   // (the framework's sites are binned one by one, src/force.c:458-470)
   int fw_mol, fw_site0, nmol_ent;
   int ncols;             // stencil columns (k_pairs_col)
   int chunk;             // home slots a block takes at a time (ColHome)
   int one_class;         // the slots are in link-cell order, one interaction class
   int ex, ey, z0, z1;    // the stencil's extents: |dx|, |dy|, dz from z0 to z1
   int cls_pot, cls_chg;  // bit k: sites of class k have a potential among them, charges
   double hinv[9];
   double h[9];
   double rn[3];          // 1/nx, 1/ny, 1/nz
   double reloc[27][3];
   double cut2, cut100, alpha, norm;
   float cut2f, bandf, alphaf, normf;
};

// Launch parameters of the real-space adjoint.
struct AdjParams {
   int loss;              // nonzero: residual weights given, loss terms wanted
   unsigned type_mask;    // bit b set: some site has identifier b
   int nslot;             // 2 max_id^2 NP + 2 gradient slots
   int ntype;             // identifiers present, and each one's index among them
   unsigned char type_index[MDGPU_ADJ_MAX_ID];
};

// ---------------------------------------------------------------- binning
__device__ __forceinline__ int cellbin_dev(double s, int n, double fn, int *bad)
{
   const double eps = 8.0 * 2.220446049250313e-16;   // 8 * precision(), force.c:437
   if (s < -0.5 + eps || s >= 0.5 - eps) {
      if (s < -0.5 + eps && s >= -0.5 - eps)
         s = -0.5;
      else if (s >= 0.5 - eps && s <= 0.5 + eps)
         s = 0.5 - eps;
      else
         *bad = 1;
   }
   int ib = (int)floor(__dmul_rn(__dadd_rn(s, 0.5), fn));
   if (ib >= n || ib < 0) {
      *bad = 1;
      ib = ib < 0 ? 0 : n - 1;
   }
   return ib;
}

// s = hinv . x with mat_vec_mul's order (src/matrix.c:54-56), no FMA.
__device__ __forceinline__ double hrow(const double *m, double a0, double a1, double a2)
{
   return __dadd_rn(__dadd_rn(__dmul_rn(m[0], a0), __dmul_rn(m[1], a1)), __dmul_rn(m[2], a2));
}

// Also the set-up of the evaluation's result record, by the last block, and
// on small grids (SCAN_ONE cells) the scan of the cell counts and on small
// systems (SCATTER_ONE sites) the placement: launches are the cost there, and
// in the last block the latency of its loads, so every thread has all of its
// own in flight (2048 sites: 14.8 us in rounds of 1024 counts and 256 sites,
// 9.5 us so; the three separate kernels 11.8 us and two more launches).
constexpr int SCAN_ONE = 8192, SCATTER_ONE = 2048;

__device__ __forceinline__ int warp_incl_scan(int v);
__device__ void block_excl_scan(int v, int *out_excl);

__global__ void __launch_bounds__(256)
k_bin(RsParams P, const double *__restrict__ site, const double *__restrict__ cofm,
      const int *__restrict__ mol_first, const int *__restrict__ mol_n, const int *__restrict__ site_cls,
      int *__restrict__ cell_of, int *__restrict__ rank, int *__restrict__ cell_count, int *__restrict__ cell_start,
      int ncount, int *__restrict__ unsorted, unsigned int *__restrict__ sync, DevOut *out)
{
   const int e = blockIdx.x * blockDim.x + threadIdx.x;
   if (e < P.nent) {
      int bad = 0;
      double s0, s1, s2;
      const bool by_site = !P.molpbc || e >= P.nmol_ent;
      const int si = !P.molpbc ? e : P.fw_site0 + (e - P.nmol_ent);   // site of a site entity
      if (by_site) {
         const int N = P.nsites;
         double x = site[si], y = site[N + si], z = site[2 * N + si];
         s0 = hrow(P.hinv, x, y, z);
         s1 = hrow(P.hinv + 3, x, y, z);
         s2 = hrow(P.hinv + 6, x, y, z);
      } else {
         s0 = cofm[3 * e];
         s1 = cofm[3 * e + 1];
         s2 = cofm[3 * e + 2];
      }
      int cx = cellbin_dev(s0, P.nx, (double)P.nx, &bad);
      int cy = cellbin_dev(s1, P.ny, (double)P.ny, &bad);
      int cz = cellbin_dev(s2, P.nz, (double)P.nz, &bad);
      int c = cz + P.nz * (cy + P.ny * cx);
      if (bad) atomicOr(&sync[SYNC_BINERR], 1u);
      if (by_site) {
         if (site_cls) c += site_cls[si] * P.ncells;   // class by class
         cell_of[si] = c;
         rank[si] = atomicAdd(&cell_count[c], 1);
      } else {
         int f = mol_first[e], n = mol_n[e];
         const int r = atomicAdd(&cell_count[c], n);
         for (int s = 0; s < n; s++) {
            cell_of[f + s] = c;
            rank[f + s] = r + s;
         }
      }
   }
   if (!last_block(&sync[SYNC_BIN])) return;
   const int t = threadIdx.x;
   unsigned int *o = reinterpret_cast<unsigned int *>(out);
   for (int q = t; q < (int)(sizeof(DevOut) / 4); q += blockDim.x) o[q] = 0u;
   __syncthreads();
   if (t == 0) {
      out->err = (int)__ldcg(&sync[SYNC_BINERR]);
      sync[SYNC_BINERR] = 0u;
   }
   if (ncount > SCAN_ONE) return;
   // one round: a run of consecutive counts per thread (a multiple of four,
   // all its loads in flight), then the sites, eight per thread in flight
   static_assert(SCAN_ONE <= 8192, "36 counts a thread");
   __shared__ int wsum[8];
   const int lane = t & 31, w = t >> 5, run = (ncount / 256 + 4) & ~3, i0 = t * run;   // 256 run > ncount
   int4 v[9];
   int sum = 0;
#pragma unroll
   for (int k = 0; k < 9; k++) {
      v[k] = make_int4(0, 0, 0, 0);
      const int i = i0 + 4 * k;
      if (4 * k < run) {
         if (i + 3 < ncount) {
            v[k] = __ldcg(reinterpret_cast<const int4 *>(cell_count + i));
         } else {
            if (i < ncount) v[k].x = __ldcg(&cell_count[i]);
            if (i + 1 < ncount) v[k].y = __ldcg(&cell_count[i + 1]);
            if (i + 2 < ncount) v[k].z = __ldcg(&cell_count[i + 2]);
         }
         sum += (v[k].x + v[k].y) + (v[k].z + v[k].w);
      }
   }
   const int inc = warp_incl_scan(sum);
   if (lane == 31) wsum[w] = inc;
   __syncthreads();
   int ex = inc - sum;
   for (int k = 0; k < w; k++) ex += wsum[k];
#pragma unroll
   for (int k = 0; k < 9; k++) {
      const int i = i0 + 4 * k;
      if (4 * k < run) {
         int4 o4;
         o4.x = ex;
         o4.y = ex + v[k].x;
         o4.z = o4.y + v[k].y;
         o4.w = o4.z + v[k].z;
         ex = o4.w + v[k].w;
         if (i + 3 <= ncount) {
            *reinterpret_cast<int4 *>(cell_start + i) = o4;
         } else {
            if (i <= ncount) cell_start[i] = o4.x;
            if (i + 1 <= ncount) cell_start[i + 1] = o4.y;
            if (i + 2 <= ncount) cell_start[i + 2] = o4.z;
         }
      }
   }
   if (P.nsites > SCATTER_ONE) return;
   __syncthreads();
   for (int b0 = t; b0 < P.nsites; b0 += 8 * 256) {
      int c[8], r[8];
#pragma unroll
      for (int k = 0; k < 8; k++) {
         const int i = b0 + 256 * k;
         c[k] = i < P.nsites ? __ldcg(&cell_of[i]) : -1;
         r[k] = i < P.nsites ? __ldcg(&rank[i]) : 0;
      }
#pragma unroll
      for (int k = 0; k < 8; k++)
         if (c[k] >= 0) r[k] += cell_start[c[k]];
#pragma unroll
      for (int k = 0; k < 8; k++)
         if (c[k] >= 0) unsorted[r[k]] = b0 + 256 * k;
   }
}

// ---------------------------------------------------------- exclusive scan
__device__ __forceinline__ int warp_incl_scan(int v)
{
   const int lane = threadIdx.x & 31;
#pragma unroll
   for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += t;
   }
   return v;
}

// Block-wide exclusive scan of 1024 values.
__device__ void block_excl_scan(int v, int *out_excl)
{
   __shared__ int wsum[32];
   const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
   int inc = warp_incl_scan(v);
   if (lane == 31) wsum[w] = inc;
   __syncthreads();
   if (w == 0) {
      int s = wsum[lane];
      int si = warp_incl_scan(s);
      wsum[lane] = si - s;
   }
   __syncthreads();
   *out_excl = inc - v + wsum[w];
   __syncthreads();
}

// (nin values in, n out: entry nin receives the total)
__global__ void __launch_bounds__(1024) k_scan_blocks(const int *__restrict__ in, int *__restrict__ out,
                                                      int *__restrict__ bsum, int nin, int n)
{
   int i = blockIdx.x * 1024 + threadIdx.x;
   int v = i < nin ? in[i] : 0, ex;
   __shared__ int last;
   block_excl_scan(v, &ex);
   if (threadIdx.x == 1023) last = ex + v;
   __syncthreads();
   if (i < n) out[i] = ex;
   if (threadIdx.x == 0) bsum[blockIdx.x] = last;
}

// The block sums before each block added to its scanned values (entry n,
// the total, among them).
__global__ void __launch_bounds__(1024) k_scan_add(int *__restrict__ out, const int *__restrict__ bsum, int n)
{
   __shared__ int sh[32];
   int s = 0;
   for (int k = threadIdx.x; k < (int)blockIdx.x; k += 1024) s += bsum[k];
   s = __reduce_add_sync(0xffffffffu, s);
   if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
   __syncthreads();
   s = __reduce_add_sync(0xffffffffu, sh[threadIdx.x & 31]);
   const int i = blockIdx.x * 1024 + threadIdx.x;
   if (i < n) out[i] += s;
}

// ------------------------------------------------------ placement by cell
__global__ void k_scatter(int n, const int *__restrict__ cell_of, const int *__restrict__ cell_start,
                          const int *__restrict__ rank, int *__restrict__ unsorted)
{
   int i = blockIdx.x * blockDim.x + threadIdx.x;
   if (i < n) unsorted[cell_start[cell_of[i]] + rank[i]] = i;
}

// Each cell's sites in ascending order (a site's place: the count of its
// cell's sites before it) and the per-slot records; leaves the cell counts
// zero for the next binning.  Null pointers: records not wanted.
__global__ void k_place(RsParams P, const double *__restrict__ site, const double *__restrict__ chg,
                        const int *__restrict__ siteid, const int *__restrict__ molmap,
                        const int *__restrict__ unsorted, const int *__restrict__ cell_of,
                        const int *__restrict__ cell_start, int *__restrict__ cell_count, int ncount,
                        int *__restrict__ sorted, double4 *__restrict__ pos64, float4 *__restrict__ pos32,
                        int2 *__restrict__ tag, int2 *__restrict__ tagz, int *__restrict__ slot_cell)
{
   const int t = blockIdx.x * blockDim.x + threadIdx.x;
   for (int q = t; q < ncount; q += gridDim.x * blockDim.x) cell_count[q] = 0;
   const int N = P.nsites;
   if (t >= N) return;
   const int i = unsorted[t], cc = cell_of[i], a = cell_start[cc], b = cell_start[cc + 1];
   int p = a;
   for (int q = a; q < b; q++) p += unsorted[q] < i;
   sorted[p] = i;
   const int c = cc >= P.ncells ? cc - P.ncells : cc;
   const int id = siteid[i], mol = molmap[i];
   double x = site[i], y = site[N + i], z = site[2 * N + i], q = chg[i];
   if (tag) tag[p] = make_int2(id, mol);
   if (tagz) tagz[p] = make_int2(id | ((c % P.nz) << 16), mol);   // with the cell's z index
   slot_cell[p] = c;
   if (pos64) pos64[p] = make_double4(x, y, z, q);
   if (pos32) {
      int cx = c / (P.ny * P.nz), cy = (c / P.nz) % P.ny, cz = c % P.nz;
      // the cell's corner in fractional co-ordinates (reciprocals: the FP64
      // pipe is the cost of this kernel; FP32 cell-relative co-ordinates
      // need the corner only to FP64 rounding)
      double s0 = (double)cx * P.rn[0] - 0.5, s1 = (double)cy * P.rn[1] - 0.5, s2 = (double)cz * P.rn[2] - 0.5;
      double ox = P.h[0] * s0 + P.h[1] * s1 + P.h[2] * s2;
      double oy = P.h[3] * s0 + P.h[4] * s1 + P.h[5] * s2;
      double oz = P.h[6] * s0 + P.h[7] * s1 + P.h[8] * s2;
      pos32[p] = make_float4((float)(x - ox), (float)(y - oy), (float)(z - oz), (float)q);
   }
}

// ---------------------------------------------------------- pair potential
#define AS1 0.254829592
#define AS2 -0.284496736
#define AS3 1.421413741
#define AS4 -1.453152027
#define AS5 1.061405429
#define ASP 0.3275911

template <typename R> __device__ __forceinline__ R dsqrt(R x);
template <> __device__ __forceinline__ double dsqrt<double>(double x) { return sqrt(x); }
template <> __device__ __forceinline__ float dsqrt<float>(float x) { return sqrtf(x); }
template <typename R> __device__ __forceinline__ R dexp(R x);
template <> __device__ __forceinline__ double dexp<double>(double x) { return exp(x); }
template <> __device__ __forceinline__ float dexp<float>(float x) { return expf(x); }

template <int PT> struct NPar { static constexpr int v = 8; };
template <> struct NPar<0> { static constexpr int v = 2; };
template <> struct NPar<1> { static constexpr int v = 3; };
template <> struct NPar<2> { static constexpr int v = 4; };
template <> struct NPar<3> { static constexpr int v = 6; };
template <> struct NPar<4> { static constexpr int v = 3; };
template <> struct NPar<6> { static constexpr int v = 7; };

// The potential holds an exponential of r (not of r^2): 6-exp, MCY, generic, Morse.
// Its argument multiplies r's rounding by up to ten, and rock salt's forces are a
// thousandth of the terms they are sums of: for these forms r is rounded correctly
// and the erfc arguments are alpha r as the cell-by-cell kernel has them.  Force of
// 1728 ions against extended precision: cell by cell 4.83-5.02e-15, r from the
// reciprocal root alone 5.8-6.0e-15, corrected 4.96-5.2e-15, with alpha r
// 4.88-5.07e-15 (32,768 ions: pairs 1.023, 1.050, 1.062 ms); water and MCY, without
// either, are below the cell-by-cell kernel's error.
template <int PT> struct ExpOfR { static constexpr bool v = PT != 0 && PT != 4; };

// Square root and its reciprocal, reciprocal and exponential: correctly rounded
// (FAST false), or the FP32 hardware approximations (FAST true: rsqrt and
// reciprocal within 2 ulp, exp within a few ulp over the arguments of the
// potentials here), which the column-walk pair kernel of the mixed form
// uses.
template <typename R, bool FAST> struct PairMath {
   // r = sqrt(x), r_r = 1 / r; XR: r is an argument of an exponential
   template <bool XR> static __device__ __forceinline__ void root(R x, R &r, R &r_r)
   {
      r = dsqrt<R>(x);
      r_r = R(1) / r;
   }
   static __device__ __forceinline__ R rcp(R x) { return R(1) / x; }
   static __device__ __forceinline__ R ex(R x) { return dexp<R>(x); }
};
template <> struct PairMath<float, true> {
   template <bool XR> static __device__ __forceinline__ void root(float x, float &r, float &r_r)
   {
      r_r = rsqrtf(x);
      r = x * r_r;
   }
   static __device__ __forceinline__ float rcp(float x) { return __fdividef(1.0f, x); }
   static __device__ __forceinline__ float ex(float x) { return __expf(x); }
};

// FP64 form of the same: the FP64 pipe (two lanes per clock and SM) bounds
// the pair loops, so the correctly rounded square root, divisions and exp
// (about 55 of 110 FP64 instructions per pair) are replaced by
//   rsqrt, rcp: the hardware's 20-bit approximation and one third-order
//     Newton (Householder) step, e -> e^3: 5 and 3 FP64 instructions, 0.507
//     ulp at most (measured, 4 million arguments, as the figures below);
//   sqrt: x rsqrt(x), 1.5 ulp at most (mean 0.35), or with a Newton step 0.5;
//   exp: Tang's table method (ACM TOMS 15, 144, 1989): x = (256 k + j)
//     ln2/256 + f, exp(x) = 2^k 2^(j/256) e^f, |f| <= ln2/512, degree 4, the
//     rounding residue of 2^(j/256) added to f: 10 instructions, 0.545 ulp (a
//     64-entry table without residues and degree 6 took 12).
//     The table is in shared memory.
// Arguments outside their range (r^2 zero or subnormal, |x| > 700) take the
// general functions.
// 2^(j/256), j = 0 .. 255, rounded from 400-bit repeated square roots, and the
// relative residue of the rounding; ln2/256 in two parts and 256/ln2
__device__ const double2 g_exp2_tab[256] = {
   {1.0, 0.000000e+00}, {1.0027112750502025, -3.626783e-17}, {1.0054299011128027, 9.447885e-17},
   {1.0081558981184175, -3.225750e-17}, {1.0108892860517005, -1.507067e-17}, {1.0136300849514894, 9.158765e-18},
   {1.016378314910953, -5.679155e-17}, {1.019133996077738, 3.534280e-17}, {1.0218971486541166, 4.999745e-17},
   {1.0246677928971357, -7.379570e-17}, {1.0274459491187637, -4.823684e-17}, {1.030231637686041, 3.222411e-17},
   {1.0330248790212284, 7.357847e-18}, {1.0358256936019572, -7.536772e-17}, {1.0386341019613787, 5.773230e-17},
   {1.041450124688316, 3.634193e-17}, {1.0442737824274138, 8.189318e-17}, {1.0471050958792898, 6.949710e-17},
   {1.0499440858006872, 5.326891e-17}, {1.0527907730046264, -9.146625e-17}, {1.0556451783605572, 1.666588e-18},
   {1.0585073227945128, -6.757300e-17}, {1.061377227289262, -1.128113e-17}, {1.0642549128844645, 4.772122e-17},
   {1.0671404006768237, -7.402825e-17}, {1.0700337118202419, -9.286775e-17}, {1.0729348675259756, -3.578660e-18},
   {1.075843889062791, -9.297554e-18}, {1.0787607977571199, -6.170655e-17}, {1.0816856149932152, -4.421455e-17},
   {1.0846183622133092, 2.919140e-17}, {1.0875590609177697, 4.973844e-18}, {1.0905077326652577, -2.793911e-17},
   {1.0934643990728858, 1.318192e-17}, {1.0964290818163769, -5.399285e-17}, {1.099401802630222, 6.522146e-17},
   {1.102382583307841, 4.776959e-17}, {1.1053714457017412, 7.453864e-17}, {1.1083684117236787, -7.927701e-17},
   {1.1113735033448175, 5.006368e-17}, {1.1143867425958924, 9.341711e-17}, {1.1174081515673693, -7.138668e-17},
   {1.1204377524096067, -5.534521e-17}, {1.12347556733302, -8.633688e-17}, {1.1265216186082418, 4.585670e-17},
   {1.129575928566288, 5.942766e-17}, {1.1326385195987192, 2.858243e-17}, {1.1357094141578055, 4.461176e-17},
   {1.1387886347566916, 7.826573e-17}, {1.1418762039695616, 4.073201e-17}, {1.1449721444318042, 4.053627e-17},
   {1.148076478840179, 6.008084e-17}, {1.1511892299529827, 2.823784e-17}, {1.154310420590216, 9.024547e-17},
   {1.1574400736337511, -7.882802e-17}, {1.1605782120274988, -2.809841e-17}, {1.1637248587775775, 3.290473e-17},
   {1.1668800369524817, -7.534519e-17}, {1.1700437696832502, -1.579209e-18}, {1.1732160801636373, -6.211612e-17},
   {1.1763969916502812, 4.721368e-17}, {1.1795865274628758, 8.555805e-17}, {1.182784710984341, 1.304528e-17},
   {1.1859915656609938, -7.765238e-18}, {1.189207115002721, 3.348462e-17}, {1.1924313825831512, 3.687886e-17},
   {1.1956643920398273, 3.861120e-17}, {1.1989061670743806, -8.181786e-17}, {1.202156731452703, 5.527550e-17},
   {1.2054161090051239, -2.785156e-17}, {1.2086843236265816, -3.927184e-17}, {1.2119613992768012, -4.035286e-17},
   {1.215247359980469, -6.346552e-17}, {1.2185422298274085, -7.391395e-17}, {1.2218460329727576, -8.684418e-17},
   {1.2251587936371455, -7.267249e-17}, {1.22848053610687, -1.545634e-17}, {1.2318112847340759, 5.998794e-17},
   {1.2351510639369334, -8.707635e-17}, {1.2384998981998165, 2.234721e-17}, {1.241857812073484, 3.750854e-17},
   {1.245224830175258, -3.756141e-17}, {1.2486009771892048, -6.616855e-17}, {1.2519862778663162, 3.861198e-17},
   {1.255380757024691, -5.346099e-18}, {1.2587844395497165, -6.690409e-17}, {1.2621973503942507, -2.443726e-17},
   {1.2656195145788063, 3.358495e-17}, {1.2690509571917332, 2.102305e-18}, {1.2724917033894028, -8.312759e-18},
   {1.275941778396392, 7.771068e-17}, {1.2794012075056693, -7.627861e-17}, {1.2828700160787783, 1.335751e-17},
   {1.2863482295460256, -2.656322e-17}, {1.2898358734066657, 6.938292e-17}, {1.2933329732290895, -2.299942e-17},
   {1.2968395546510096, 1.957259e-17}, {1.3003556433796506, 4.367058e-17}, {1.3038812651919358, 6.632257e-17},
   {1.3074164459346773, -5.611560e-17}, {1.3109612115247644, -5.478069e-17}, {1.3145155879493546, 1.725003e-17},
   {1.318079601266064, -4.140839e-17}, {1.3216532776031575, -1.876921e-17}, {1.3252366431597413, -2.157148e-17},
   {1.3288297242059544, 3.077209e-17}, {1.3324325470831615, -3.828777e-17}, {1.3360451382041458, -4.409931e-17},
   {1.339667524053303, 6.663805e-17}, {1.3432997311868353, -4.319647e-17}, {1.3469417862329458, 2.393619e-17},
   {1.3505937158920345, -6.135902e-17}, {1.3542555469368927, 5.686481e-17}, {1.3579273062129011, -7.017780e-17},
   {1.3616090206382248, 1.126452e-18}, {1.365300717204012, -7.328322e-17}, {1.3690024229745905, 7.007875e-17},
   {1.3727141650876684, -3.275234e-17}, {1.3764359707545302, -5.011921e-17}, {1.380167867260238, 7.615244e-17},
   {1.383909881963832, -4.892307e-17}, {1.387662042298529, 6.069910e-17}, {1.3914243757719262, -3.526009e-17},
   {1.3951969099662003, -6.686752e-17}, {1.3989796725383112, -6.872304e-17}, {1.4027726912202048, -3.775226e-17},
   {1.4065759938190154, 5.001447e-18}, {1.4103896082172707, 2.954183e-17}, {1.4142135623730951, -6.835809e-17},
   {1.4180478843204152, 1.603922e-17}, {1.4218926021691656, -1.130734e-17}, {1.4257477441054942, 6.930182e-17},
   {1.42961333839197, -8.416012e-18}, {1.433489413367789, -4.047783e-17}, {1.4373759974489824, -2.924798e-17},
   {1.4412731191286257, 3.887191e-18}, {1.4451808069770467, -2.092304e-17}, {1.449099089642035, -4.319515e-17},
   {1.4530279958490526, -3.977865e-17}, {1.4569675544014438, 3.877011e-17}, {1.460917794180647, -3.833465e-17},
   {1.4648787441464057, 6.506182e-17}, {1.4688504333369818, 5.763611e-17}, {1.4728328908693675, 4.543471e-17},
   {1.4768261459394993, -2.359109e-17}, {1.4808302278224719, -6.541568e-17}, {1.4848451658727524, 7.260075e-17},
   {1.488870989524397, 4.134252e-17}, {1.4929077282912648, 9.506897e-18}, {1.4969554117672355, -1.911656e-17},
   {1.5010140696264256, -4.272956e-17}, {1.5050837316234065, 4.700543e-17}, {1.5091644275934228, -6.735219e-17},
   {1.5132561874526098, 5.871113e-17}, {1.5173590411982147, -2.839604e-17}, {1.5214730189088146, -3.941173e-18},
   {1.5255981507445384, -7.226635e-17}, {1.529734466947287, 2.474803e-17}, {1.533881997840956, 5.786121e-17},
   {1.5380407738316568, 6.615346e-17}, {1.5422108254079407, 5.154830e-17}, {1.5463921831410214, 6.908959e-17},
   {1.550584877685, -9.416258e-18}, {1.5547889397770887, -5.147426e-17}, {1.559004400237837, 2.425399e-17},
   {1.5632312899713576, 4.788017e-17}, {1.567469639965553, -6.604314e-17}, {1.5717194812923414, -2.126960e-17},
   {1.5759808451078865, -6.432132e-18}, {1.5802537626528246, -3.267452e-17}, {1.5845382652524937, -1.220401e-17},
   {1.588834384317164, -3.773175e-18}, {1.593142151342267, -6.336162e-17}, {1.597461597908627, 1.556744e-17},
   {1.6017927556826934, -3.780088e-17}, {1.606135656416771, -6.446868e-17}, {1.6104903319492543, 1.534141e-17},
   {1.6148568142048607, -4.530843e-17}, {1.6192351351948637, 1.293286e-17}, {1.6236253270173289, -2.207722e-17},
   {1.6280274218573478, -4.123367e-17}, {1.632441451987275, 6.035634e-17}, {1.6368674497669644, 4.703084e-17},
   {1.6413054476440063, -5.634277e-17}, {1.645755478153965, -6.152603e-17}, {1.6502175739206177, 5.534591e-18},
   {1.6546917676561943, 5.827849e-17}, {1.6591780921616162, -4.385030e-17}, {1.6636765803267364, 3.540948e-17},
   {1.6681872651305825, 2.559172e-17}, {1.6727101796415966, -3.274157e-17}, {1.6772453570178785, 4.950945e-17},
   {1.681792830507429, 4.875161e-17}, {1.6863526334483934, -4.258577e-17}, {1.6909247992693053, -5.718570e-17},
   {1.6955093614893326, 4.269170e-17}, {1.7001063537185235, -4.719540e-18}, {1.7047158096580513, -1.600785e-17},
   {1.709337763100463, -5.773452e-17}, {1.713972247929926, 3.777176e-17}, {1.718619298122478, -1.077249e-17},
   {1.723278947746274, -5.525585e-17}, {1.7279512309618377, -6.221809e-17}, {1.732636182022311, -9.800390e-19},
   {1.7373338352737062, 1.821405e-17}, {1.7420442251551564, -8.759589e-19}, {1.746767386199169, -6.155537e-17},
   {1.7515033530318782, -2.925744e-17}, {1.7562521603732995, 1.685487e-17}, {1.761013843037584, -4.510614e-17},
   {1.7657884359332727, 5.358125e-17}, {1.7705759740635547, 3.367150e-17}, {1.7753764925265212, 3.621616e-17},
   {1.7801900265154245, -2.968575e-17}, {1.785016611318935, 8.588380e-18}, {1.789856282321401, -2.321055e-17},
   {1.7947090750031072, 1.015622e-17}, {1.7995750249405351, -1.404159e-17}, {1.804454167806624, -2.869135e-17},
   {1.809346539371032, -4.992212e-17}, {1.8142521755003989, -5.495119e-17}, {1.8191711121586085, 4.069258e-17},
   {1.8241033854070534, -5.569656e-17}, {1.8290490314048973, 3.766544e-17}, {1.8340080864093424, 1.790127e-17},
   {1.8389805867758937, 3.762394e-18}, {1.843966568958626, -3.221177e-17}, {1.8489660695104508, 4.882502e-17},
   {1.8539791250833855, 5.265371e-17}, {1.8590057724288205, -5.125700e-17}, {1.864046048397789, 3.508987e-17},
   {1.8690999899412386, -5.317268e-17}, {1.8741676341103, -3.266924e-17}, {1.8792490180565602, -8.634468e-18},
   {1.8843441790323345, -4.365759e-17}, {1.8894531543909392, -4.766018e-17}, {1.8945759815869656, 1.796393e-17},
   {1.8997126981765553, -2.031749e-17}, {1.9048633418176741, 3.430093e-17}, {1.9100279502703899, -3.094032e-17},
   {1.9152065613971474, -5.545066e-17}, {1.9203992131630474, 3.705834e-17}, {1.925605943636125, -5.149010e-17},
   {1.930826790987627, 3.194046e-17}, {1.9360617934922943, 5.336806e-17}, {1.9413109895286405, -3.419354e-17},
   {1.9465744175792332, 3.498979e-17}, {1.9518521162309783, -1.126631e-17}, {1.9571441241754002, 4.578492e-17},
   {1.9624504802089273, 5.593437e-17}, {1.9677712232331759, -5.241935e-17}, {1.9731063922552343, -3.776592e-18},
   {1.978456026387951, 2.041428e-17}, {1.9838201648502194, -1.110713e-17}, {1.9891988469672663, 4.124843e-18},
   {1.9945921121709402, 8.979134e-18},
};
constexpr double EXP_HI = 0.00270760617331689, EXP_LO = 7.453964567463233e-13, EXP_INV = 369.3299304675746;
template <bool XR> __device__ __forceinline__ void root_n(double x, double &r, double &r_r)
{
   // (range checks on the exponent bits: a compare would take the FP64 pipe)
   if ((unsigned int)__double2hiint(x) - 0x04000000u >= 0x78000000u) {
      // (zero among them: r = 0, r_r infinite, where x r_r would be NaN)
      r = sqrt(x);
      r_r = 1.0 / r;
      return;
   }
   double y;
   asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
   const double e = fma(-x, y * y, 1.0);
   r_r = fma(y * e, fma(0.375, e, 0.5), y);
   r = x * r_r;
   if (XR) r = fma(0.5 * r_r, fma(-r, r, x), r);
}
__device__ __forceinline__ double rcp_n(double x)
{
   if (((unsigned int)__double2hiint(x) & 0x7fffffffu) - 0x04000000u >= 0x78000000u) return 1.0 / x;
   double y;
   asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
   const double e = fma(-x, y, 1.0);
   return fma(y, fma(e, e, e), y);
}
__shared__ double2 exp2_tab[256];   // g_exp2_tab; filled by exp2_fill (kernels that use exp_n)
__device__ __forceinline__ void exp2_fill()
{
   for (int j = threadIdx.x; j < 256; j += blockDim.x) exp2_tab[j] = g_exp2_tab[j];
}
__device__ __forceinline__ double exp_n(double x)
{
   if (((unsigned int)__double2hiint(x) & 0x7fffffffu) >= 0x4085e000u) return exp(x);   // |x| >= 700
   const double w = fma(x, EXP_INV, 6755399441055744.0);   // x 256/ln2 + 1.5 2^52
   const int n = __double2loint(w);
   const double nf = w - 6755399441055744.0;
   // ln2/256 in two parts, the first with 21 trailing zero bits (nf exact in it)
   const double f = fma(nf, -EXP_LO, fma(nf, -EXP_HI, x));
   // (cubic coefficient: 1/6 and the best fit of f^5/120 by f^3 over the range)
   const double2 t = exp2_tab[n & 255];
   double p = fma(f, 1.0 / 24.0, 0.16666667994052387);
   p = fma(f, p, 0.5);
   p = fma(f * f, p, f + t.y);
   const double r = fma(t.x, p, t.x);
   return __hiloint2double(__double2hiint(r) + ((n >> 8) << 20), __double2loint(r));
}
template <> struct PairMath<double, true> {
   template <bool XR> static __device__ __forceinline__ void root(double x, double &r, double &r_r)
   {
      root_n<XR>(x, r, r_r);
   }
   static __device__ __forceinline__ double rcp(double x) { return rcp_n(x); }
   static __device__ __forceinline__ double ex(double x) { return exp_n(x); }
};

// One pair of kernel(): f = -U'(r)/r and U, with the erfc real-space Ewald
// term by the A&S polynomial when EW (src/kernel.c:182-353 / 355-460).
template <int PT, bool EW, typename R, bool FAST = false>
__device__ __forceinline__ void pair_fu(R r2, R qq, const R *p, R alpha, R norm, R &f, R &u, bool hp = true,
                                        bool hc = true)
{
   typedef PairMath<R, FAST> M;
   R t = R(0), ef = R(0), r = R(0), r_r = R(0), rs_r;
   if (EW || PT != 0) {
      M::template root<ExpOfR<PT>::v>(r2, r, r_r);
      rs_r = r_r * r_r;
   } else {
      rs_r = M::rcp(r2);
   }
   if (EW && hc) {
      if (FAST && sizeof(R) == 8 && !ExpOfR<PT>::v) {   // one product fewer (FP64)
         t = M::rcp(fma((R(ASP) * alpha), r, R(1)));
         ef = qq * M::ex(-(alpha * alpha) * r2);
      } else {
         R ar = alpha * r;
         t = M::rcp(R(1) + R(ASP) * ar);
         ef = qq * M::ex(-(ar * ar));
      }
      t = (t * (R(AS1) + t * (R(AS2) + t * (R(AS3) + t * (R(AS4) + t * R(AS5)))))) * ef * r_r;
      ef = t + norm * ef;
   }
   if (EW && FAST && !hp) {   // (warp-uniform: the home site's class has none)
      u = t;
      f = rs_r * ef;
      return;
   }
   if (EW && FAST && sizeof(R) == 8) {
      // FP64: a potential whose parameters are all zero adds exactly nothing
      // (rigid water's H and M: 9 of 10 pairs of their class)
      unsigned long long any = 0;
#pragma unroll
      for (int k = 0; k < NPar<PT>::v; k++) any |= (unsigned long long)__double_as_longlong((double)p[k]) << 1;
      if (any == 0) {
         u = t;
         f = rs_r * ef;
         return;
      }
   }
   if (PT == 0) {
      R r6 = (p[1] * p[1]) * rs_r;
      r6 = r6 * r6 * r6;
      R r12 = r6 * r6;
      u = t + p[0] * (r12 - r6);
      f = rs_r * (R(6) * p[0] * (R(2) * r12 - r6) + ef);
   } else if (PT == 1) {
      R e1 = p[1] * M::ex(-p[2] * r);
      R r6 = p[0] * (rs_r * rs_r * rs_r);
      u = t - r6 + e1;
      f = rs_r * (R(-6) * r6 + ef) + p[2] * e1 * r_r;
   } else if (PT == 2) {
      R e1 = p[0] * M::ex(-p[1] * r);
      R e2 = -p[2] * M::ex(-p[3] * r);
      u = t + e1 + e2;
      f = (p[1] * e1 + p[3] * e2) * r_r + ef * rs_r;
   } else if (PT == 3) {
      R e1 = p[0] * M::ex(-p[1] * r);
      R r4 = rs_r * rs_r;
      R r6 = rs_r * r4;
      R r8 = p[5] * (r4 * r4);
      R r12 = p[2] * (r6 * r6);
      r4 *= p[3];
      r6 *= p[4];
      u = t + e1 + r12 - r4 - r6 - r8;
      f = rs_r * (R(12) * r12 - R(4) * r4 - R(6) * r6 - R(8) * r8 + ef) + p[1] * e1 * r_r;
   } else if (PT == 4) {
      R r4 = rs_r * rs_r;
      R r6 = rs_r * r4;
      R r12 = p[2] * (r6 * r6);
      r6 *= p[1];
      r4 *= p[0];
      u = t + r4 + r6 + r12;
      f = rs_r * (R(4) * r4 + R(6) * r6 + R(12) * r12 + ef);
   } else {  // Morse (PT == 6)
      R e1 = p[0] * M::ex((p[1] - r) * p[2]);
      R r6 = p[3] * (rs_r * rs_r * rs_r);
      R e2 = p[4] * M::ex(R(-2) * p[5] * (r - p[6]));
      R e3 = -p[4] * R(2) * M::ex(-p[5] * (r - p[6]));
      u = t + e1 - r6 + e2 + e3;
      f = rs_r * (R(-6) * r6 + ef) + r_r * (p[2] * e1 + (R(2) * p[5]) * e2 + p[5] * e3);
   }
}

// --------------------------------------------------------------- pair loop
// s += x: plain in FP64, Kahan-compensated in FP32 (s - c is the total).
__device__ __forceinline__ void accum(double &s, double &c, double x)
{
   (void)c;
   s += x;
}
__device__ __forceinline__ void accum(float &s, float &c, float x)
{
   const float y = x - c;
   const float t = s + y;
   c = (t - s) - y;
   s = t;
}
__device__ __forceinline__ void note_too_close(DevOut *out, int a, int b)
{
   int k = atomicAdd(&out->n_too_close, 1);
   if (k < MAX_TOO_CLOSE_REC) {
      out->too_close[k][0] = a;
      out->too_close[k][1] = b;
   }
}

__device__ __forceinline__ double block_sum_d(double v, double *sh)
{
#pragma unroll
   for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
   const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
   __syncthreads();
   if (lane == 0) sh[w] = v;
   __syncthreads();
   double s = 0.0;
   if (threadIdx.x == 0)
      for (int i = 0; i < nw; i++) s += sh[i];
   return s;   // valid in thread 0
}

constexpr int PAIR_WARPS = 4;   // warps per block

// Per-warp shared rows of the stencil walk (32 WALK_E entries), and the
// stencil's cell-offset vectors (global, read by entry).
constexpr int WALK_E = 4;   // stencil entries per lane in one pass of the walk

struct WalkRows {
   int *inc, *jb, *info;
   const float4 *oh, *ol;
};

// Walks the full stencil of home slot p (in cell c) with one warp and calls
// visit(j, e, kimg) for every candidate slot j, the home site itself
// excluded: e is the stencil entry j belongs to (its cell-offset vectors are
// rows.oh[e], rows.ol[e]) and kimg the periodic image code.  A pass takes
// 32 WALK_E stencil entries (WALK_E consecutive ones per lane), lays their
// cells' slot ranges end to end by a warp prefix sum, and deals the
// candidates out 32 at a time; each lane finds its candidate's entry by
// binary search over the scanned counts.  With a few sites per cell, wider
// passes keep the lanes busier (fewer, fuller rounds).
template <bool MIXED, class Visit>
__device__ __forceinline__ void walk_stencil(const RsParams &P, int p, int c, int lane,
                                             const int *__restrict__ cell_start,
                                             const int4 *__restrict__ full,
                                             const float4 *__restrict__ off_hi,
                                             const float4 *__restrict__ off_lo, const WalkRows &rows,
                                             Visit &&visit)
{
   (void)off_hi;
   (void)off_lo;
   const int cx = c / (P.ny * P.nz), cy = (c / P.nz) % P.ny, cz = c % P.nz;
   for (int base = 0; base < P.nfull; base += 32 * WALK_E) {
      int cnt[WALK_E], jb[WALK_E], info[WALK_E], tot = 0;
#pragma unroll
      for (int u = 0; u < WALK_E; u++) {
         const int e = base + lane * WALK_E + u;
         cnt[u] = jb[u] = info[u] = 0;
         if (e < P.nfull) {
            const int4 d = __ldg(&full[e]);
            int bx = cx + d.x, by = cy + d.y, bz = cz + d.z;
            const int ix = bx < 0 ? -1 : (bx >= P.nx ? 1 : 0);
            const int iy = by < 0 ? -1 : (by >= P.ny ? 1 : 0);
            const int iz = bz < 0 ? -1 : (bz >= P.nz ? 1 : 0);
            bx -= ix * P.nx;
            by -= iy * P.ny;
            bz -= iz * P.nz;
            const int cb = bz + P.nz * (by + P.ny * bx);
            const int j0 = __ldg(&cell_start[cb]);
            cnt[u] = __ldg(&cell_start[cb + 1]) - j0;
            jb[u] = j0;
            info[u] = (9 * (ix + 1) + 3 * (iy + 1) + (iz + 1)) | (d.w << 8);
         }
         tot += cnt[u];
      }
      const int linc = warp_incl_scan(tot);
      const int T = __shfl_sync(0xffffffffu, linc, 31);
      int run = linc - tot;   // candidates before this lane's entries
#pragma unroll
      for (int u = 0; u < WALK_E; u++) {
         const int q = lane * WALK_E + u;
         rows.jb[q] = jb[u] - run;    // slot = jb[q] + candidate index
         run += cnt[u];
         rows.inc[q] = run;
         rows.info[q] = info[u];
      }
      __syncwarp();
      for (int r = 0; r < T; r += 32) {
         const int idx = r + lane;
         if (idx < T) {
            int k = 0;
#pragma unroll
            for (int s = 16 * WALK_E; s >= 1; s >>= 1)
               if (rows.inc[k + s - 1] <= idx) k += s;
            const int j = rows.jb[k] + idx;
            const int inf = rows.info[k];
            if (!((inf >> 8) && j == p)) visit(j, base + k, inf & 255);
         }
      }
      __syncwarp();
   }
}

// Separation r = x_j - x_i (+ image) from the home site to slot j, r^2 and
// q_j.  FP64 form: the reference's operation order, no fused multiply-adds.
// Mixed form: cell-relative FP32 co-ordinates plus the exact cell offset as
// an FP32 (hi, lo) pair.
template <bool MIXED, typename R>
__device__ __forceinline__ void pair_sep(const RsParams &P, int j, int k, int kimg, const WalkRows &rows,
                                         const float4 &xi32, const double4 &xi64,
                                         const double4 *__restrict__ pos64,
                                         const float4 *__restrict__ pos32, R &rx, R &ry, R &rz, R &r2,
                                         R &qj)
{
   if (MIXED) {
      const float4 xj = __ldg(&pos32[j]);
      const float4 h4 = __ldg(&rows.oh[k]), l4 = __ldg(&rows.ol[k]);
      rx = (h4.x + (xj.x - xi32.x)) + l4.x;
      ry = (h4.y + (xj.y - xi32.y)) + l4.y;
      rz = (h4.z + (xj.z - xi32.z)) + l4.z;
      r2 = rx * rx + ry * ry + rz * rz;
      qj = xj.w;
   } else {
      const double4 xj = pos64[j];
      const double *rl = P.reloc[kimg];
      rx = __dadd_rn(__dsub_rn(xj.x, xi64.x), rl[0]);
      ry = __dadd_rn(__dsub_rn(xj.y, xi64.y), rl[1]);
      rz = __dadd_rn(__dsub_rn(xj.z, xi64.z), rl[2]);
      r2 = __dadd_rn(__dadd_rn(__dmul_rn(rx, rx), __dmul_rn(ry, ry)), __dmul_rn(rz, rz));
      qj = xj.w;
   }
}

// Threshold decisions (too-close warning, strict-cutoff clamp).  FP64 form:
// exact, on the reference's r^2.  Mixed form: on the FP32 r^2, except
// within a narrow band of either threshold, where r^2 is re-formed in FP64
// from the original co-ordinates (rare).
template <bool MIXED, typename R>
__device__ __forceinline__ void pair_flags(const RsParams &P, R r2, int oi, int j, int kimg,
                                           const int *__restrict__ sorted, const double *__restrict__ site,
                                           bool &too_close, bool &clip)
{
   if (MIXED) {
      const int N = P.nsites;
      const float r2f = (float)r2;
      const bool near_clip = P.strict && !P.molpbc && fabsf(r2f - P.cut2f) < P.bandf * P.cut2f;
      const bool near_close = fabsf(r2f - (float)TOO_CLOSE) < 1e-3f;
      too_close = r2f < (float)TOO_CLOSE;
      clip = P.strict && !P.molpbc && r2f > P.cut2f;
      if (near_clip || near_close) {
         const int oj = sorted[j];
         const double *rl = P.reloc[kimg];
         double ax = __dadd_rn(__dsub_rn(site[oj], site[oi]), rl[0]);
         double ay = __dadd_rn(__dsub_rn(site[N + oj], site[N + oi]), rl[1]);
         double az = __dadd_rn(__dsub_rn(site[2 * N + oj], site[2 * N + oi]), rl[2]);
         const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(ax, ax), __dmul_rn(ay, ay)), __dmul_rn(az, az));
         too_close = d2 < TOO_CLOSE;
         clip = P.strict && !P.molpbc && d2 > P.cut2;
      }
   } else {
      too_close = (double)r2 < TOO_CLOSE;
      clip = P.strict && !P.molpbc && (double)r2 > P.cut2;
   }
}

// MODE 0: forces/energy/virial; MODE 1: emit canonical pair keys only.
//
// One warp per home site.  The warp walks the full stencil 32 entries at a
// time: lane e finds the slot range of stencil cell e (a contiguous run of
// the cell-sorted arrays), a warp prefix sum lays the ranges end to end, and
// the candidates are then dealt out 32 at a time, each lane locating its
// candidate's stencil entry by binary search over the scanned counts.  Every
// lane runs the same pair arithmetic on a different candidate, so the warp
// stays converged however unevenly the sites are spread over the cells.
template <int PT, bool EW, bool MIXED, int MODE>
__global__ void __launch_bounds__(PAIR_WARPS * 32)
k_pairs(RsParams P, const int *__restrict__ cell_start, const int *__restrict__ slot_cell,
        const int4 *__restrict__ full, const float4 *__restrict__ off_hi,
        const float4 *__restrict__ off_lo, const double4 *__restrict__ pos64,
        const float4 *__restrict__ pos32, const int2 *__restrict__ tag,
        const int *__restrict__ sorted, const double *__restrict__ site,
        const double *__restrict__ potg64, const float *__restrict__ potg32,
        const double *__restrict__ chg64,
        double *__restrict__ force, double *__restrict__ part, DevOut *out,
        unsigned long long *__restrict__ keys, long long key_cap)
{
   typedef typename std::conditional<MIXED, float, double>::type R;
   constexpr int NP = NPar<PT>::v;
   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ int s_inc[PAIR_WARPS][32 * WALK_E], s_jb[PAIR_WARPS][32 * WALK_E], s_info[PAIR_WARPS][32 * WALK_E];
   R *pot_s = reinterpret_cast<R *>(smem_raw);
   const int npot = P.max_id * P.max_id;
   const R *potg = MIXED ? (const R *)(const void *)potg32 : (const R *)(const void *)potg64;
   if (P.pot_in_smem)
      for (int q = threadIdx.x; q < npot * NPOTP; q += blockDim.x) pot_s[q] = potg[q];
   __syncthreads();
   const R *pot = P.pot_in_smem ? pot_s : potg;

   const int N = P.nsites;
   const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const int p = blockIdx.x * PAIR_WARPS + w;   // home slot of this warp
   const WalkRows rows{s_inc[w], s_jb[w], s_info[w], off_hi, off_lo};
   // per-lane partial sums: few terms each, then a warp tree reduction
   R fx = 0, fy = 0, fz = 0, pe = 0, v0 = 0, v1 = 0, v2 = 0, v3 = 0, v4 = 0, v5 = 0;
   int nev = 0;                                  // evaluations by this lane
   const R cut100 = (R)P.cut100;
   if (p < N) {
      const int c = slot_cell[p];
      const int2 ti = tag[p];
      const R *prow = pot + (size_t)ti.x * P.max_id * NPOTP;
      double4 xi64 = make_double4(0, 0, 0, 0);
      float4 xi32 = make_float4(0, 0, 0, 0);
      if (MIXED) xi32 = pos32[p]; else xi64 = pos64[p];
      const R qi = MIXED ? (R)xi32.w : (R)xi64.w;
      const R alpha = MIXED ? (R)P.alphaf : (R)P.alpha, norm = MIXED ? (R)P.normf : (R)P.norm;
      const int oi = sorted[p];
      walk_stencil<MIXED>(P, p, c, lane, cell_start, full, off_hi, off_lo, rows, [&](int j, int k, int kimg) {
         R rx, ry, rz, r2, qj;
         const int2 tj = __ldg(&tag[j]);
         if (ti.y == P.fw_mol && tj.y == P.fw_mol) return;   // no framework-framework pairs
         pair_sep<MIXED>(P, j, k, kimg, rows, xi32, xi64, pos64, pos32, rx, ry, rz, r2, qj);
         if (MODE == 1) {
            const long long a = oi, bb = sorted[j];
            if (a < bb || (a == bb && kimg < 13)) {
               unsigned long long key = ((unsigned long long)a << 37) |
                                        ((unsigned long long)bb << 5) | (unsigned long long)kimg;
               unsigned long long slot = atomicAdd((unsigned long long *)&out->npairs2, 1ull);
               if ((long long)slot < key_cap) keys[slot] = key;
            }
            return;
         }
         const bool intra = ti.y == tj.y;
         bool too_close, clip;
         pair_flags<MIXED>(P, r2, oi, j, kimg, sorted, site, too_close, clip);
         if (too_close && !intra) {
            const int oj = sorted[j];
            if (oi < oj) note_too_close(out, oi, oj);
         }
         const R r2a = r2;
         if (clip) r2 = cut100;
         R pp[NP];
         const R *pj = prow + (size_t)tj.x * NPOTP;
#pragma unroll
         for (int q = 0; q < NP; q++) pp[q] = pj[q];
         R f, u;
         pair_fu<PT, EW, R>(r2, qj * qi, pp, alpha, norm, f, u);
         if (MIXED && intra) {
            // Mixed form: an intramolecular pair's energy is exactly what
            // the intramolecular correction subtracts again, so it is left
            // out of both (FP32 roundings of identical molecules would add
            // up coherently instead of cancelling); a clamped pair keeps the
            // difference between its clamped and true energies.
            R fa, ua = R(0);
            if (clip) pair_fu<PT, EW, R>(r2a, qj * qi, pp, alpha, norm, fa, ua);
            u = clip ? u - ua : R(0);
         }
         const R hf = R(0.5) * f;
         fx -= f * rx;
         fy -= f * ry;
         fz -= f * rz;
         pe += R(0.5) * u;
         v0 += hf * rx * rx;
         v1 += hf * rx * ry;
         v2 += hf * rx * rz;
         v3 += hf * ry * ry;
         v4 += hf * ry * rz;
         v5 += hf * rz * rz;
         nev++;
      });
      if (MODE == 0) {
         // warp tree reduction of the home site's force, in the working
         // precision (each lane holds a sum of a few pairs)
         R Fx = fx, Fy = fy, Fz = fz;
#pragma unroll
         for (int o = 16; o > 0; o >>= 1) {
            Fx += __shfl_down_sync(0xffffffffu, Fx, o);
            Fy += __shfl_down_sync(0xffffffffu, Fy, o);
            Fz += __shfl_down_sync(0xffffffffu, Fz, o);
         }
         if (lane == 0) {
            force[oi] = (double)Fx;
            force[N + oi] = (double)Fy;
            force[2 * N + oi] = (double)Fz;
         }
      }
   }
   if (MODE == 1) return;
   // energy and virial: warp trees in the working precision, then the
   // block's warps summed in FP64 (FP64 is slow on this part: keep it to a
   // handful of operations per block)
   __shared__ R wred[7][PAIR_WARPS];
   R vv[7] = {pe, v0, v1, v2, v3, v4, v5};
#pragma unroll
   for (int k = 0; k < 7; k++) {
      R s = vv[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) wred[k][w] = s;
   }
   __syncthreads();
   if (threadIdx.x < 7) {
      double s = 0.0;
      for (int q = 0; q < PAIR_WARPS; q++) s += (double)wred[threadIdx.x][q];
      part[blockIdx.x * 8 + threadIdx.x] = s;
   }
   unsigned long long cnt = (unsigned long long)nev;
#pragma unroll
   for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
   if (lane == 0 && cnt) atomicAdd((unsigned long long *)&out->npairs2, cnt);
}

// Per-block energy/virial partials of the pair kernel summed in a fixed
// order, in two levels: RS_RED blocks of 256 threads each reduce a fixed
// slice of the partials into one record (k_reduce_rs), then one block sums
// those (k_reduce_rs2).  The result does not depend on timing.
constexpr int RS_RED = 64;

__device__ __forceinline__ void tree7(double (*sh)[256], int t)
{
   __syncthreads();
   for (int w = 128; w > 0; w >>= 1) {
      if (t < w)
         for (int k = 0; k < 7; k++) sh[k][t] += sh[k][t + w];
      __syncthreads();
   }
}

__global__ void __launch_bounds__(256) k_reduce_rs(const double *__restrict__ part, int nblocks,
                                                   double *__restrict__ part2)
{
   __shared__ double sh[7][256];
   const int t = threadIdx.x;
   const int per = (nblocks + gridDim.x - 1) / gridDim.x;
   const int b0 = blockIdx.x * per, b1 = min(nblocks, b0 + per);
   double s[7] = {0, 0, 0, 0, 0, 0, 0};
   for (int b = b0 + t; b < b1; b += 256)
      for (int k = 0; k < 7; k++) s[k] += part[b * 8 + k];
   for (int k = 0; k < 7; k++) sh[k][t] = s[k];
   tree7(sh, t);
   if (t < 7) part2[blockIdx.x * 8 + t] = sh[t][0];
}

// The column walks' energy and virial by their last block (few blocks):
// thread t adds up blocks t, t + 128, ..., then fixed-shape trees; the
// evaluation's result too where nothing follows.
__device__ __forceinline__ void reduce_pairs_last(const double *__restrict__ part, int nblocks, unsigned int *sync,
                                                  DevOut *out, const FinArgs &fin)
{
   if (!last_block(&sync[SYNC_PAIRS])) return;
   __shared__ double sh[7][PAIR_WARPS];
   const int t = threadIdx.x, lane = t & 31, w = t >> 5;
   double s[7] = {0, 0, 0, 0, 0, 0, 0};
   for (int b = t; b < nblocks; b += PAIR_WARPS * 32)
#pragma unroll
      for (int k = 0; k < 7; k++) s[k] += __ldcg(&part[b * 8 + k]);
#pragma unroll
   for (int k = 0; k < 7; k++) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_down_sync(0xffffffffu, s[k], o);
      if (lane == 0) sh[k][w] = s[k];
   }
   __syncthreads();
   if (t < 7) {
      double v = 0.0;
      for (int k = 0; k < PAIR_WARPS; k++) v += sh[t][k];
      if (t == 0) out->pe_rs = v;
      else out->vir_rs[t - 1] = v;
   }
   if (fin.on) {
      __threadfence();
      __syncthreads();
      if (t == 0) finalize_eval(out, fin);
   }
}

__global__ void __launch_bounds__(256) k_reduce_rs2(const double *__restrict__ part2, int n, DevOut *out)
{
   __shared__ double sh[7][256];
   const int t = threadIdx.x;
   for (int k = 0; k < 7; k++) sh[k][t] = t < n ? part2[t * 8 + k] : 0.0;
   tree7(sh, t);
   if (t == 0) {
      out->pe_rs = sh[0][0];
      for (int k = 0; k < 6; k++) out->vir_rs[k] = sh[k + 1][0];
   }
}

// ------------------------------------------------- column walk (mixed form)
// The pair kernel of the mixed form, k_pairs_col, walks the stencil by
// columns and over one interaction class at a time.
//
// Columns: for a home cell (cx, cy, cz) and a stencil column (dx, dy, dz0,
// len) the partner cells (cx+dx, cy+dy, cz+dz0 .. cz+dz0+len-1) are
// consecutive cells of the link-cell order (at most two runs where the
// column wraps the periodic cell in z), so their sites are one or two
// contiguous slot ranges: a home site needs about 75 column lookups on the
// benchmark workload instead of about 485 cell lookups.
//
// Classes: identifiers are split into class 0 (those that interact with a
// charged site, directly or through a potential with nonzero parameters)
// and class 1 (the rest).  A pair across the classes has no charge product
// and a potential with all parameters zero, so it adds exactly nothing to
// forces, energy and virial: each home site walks the sites of its own class
// only (rigid water: O meets only O, H and M only H and M -- 37.5% of the
// ordered pairs skipped).  The slots are re-laid class by class, each class
// in link-cell order, with per-class cell starts.  The reference's evaluated
// pair count (every class) is counted on demand by k_count_col, and pairs
// across the classes closer than the too-close distance are reported by
// k_tooclose_x.
constexpr int COL_E = 3;                    // stencil columns per lane in one pass
constexpr int COL_ROWS = 32 * COL_E * 2;    // slot runs per pass (two per column at most)
constexpr int COL_WIN = 384;                // candidates decoded per window (most stencils' whole list)
constexpr int COL_CHUNK = 16;               // most consecutive home slots a block takes at a time

// The home slots of a block's warp w: chunks of `chunk` consecutive slots
// (a multiple of the block's warps) dealt to the grid's blocks in turn, a
// chunk's slots to the block's warps in turn.
struct ColHome {
   int chunk, w, it, p;
   __device__ __forceinline__ ColHome(int chunk_, int w_) : chunk(chunk_), w(w_), it(0), p((int)blockIdx.x * chunk_ + w_) {}
   __device__ __forceinline__ void next()
   {
      it += PAIR_WARPS;
      p = ((it / chunk) * (int)gridDim.x + (int)blockIdx.x) * chunk + it % chunk + w;
   }
};
// Sites per chunk: of 16, 12, 8 and 4 the one with which the busiest block
// has the fewest sites, the largest of equals (neighbouring sites share
// candidates and column starts in L1): with fewer blocks than chunks of 16 a
// second round of few blocks was a tail (16,384-site water, mixed, 24 sites in
// place of 16: 63 -> 61 us, 92 -> 83 us in link order; 32,768 ions 88 -> 82
// us), and blocks without a site idle (500-site argon in FP64 57 us with 16,
// 18 us with 4).
static int col_chunk(int N, int nblk)
{
   int best = COL_CHUNK, most = 1 << 30;
   for (int ch = COL_CHUNK; ch >= PAIR_WARPS; ch -= PAIR_WARPS) {
      const int chunks = (N + ch - 1) / ch, m = (chunks + nblk - 1) / nblk * ch;
      if (m < most) {
         most = m;
         best = ch;
      }
   }
   return best;
}

// A column offset's hi and lo parts (32 bytes, 32-byte aligned) in one load.
__device__ __forceinline__ void ld_coff(const float4 *p, float4 &h, float4 &l)
{
   asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
       : "=f"(h.x), "=f"(h.y), "=f"(h.z), "=f"(h.w), "=f"(l.x), "=f"(l.y), "=f"(l.z), "=f"(l.w)
       : "l"(p));
}

// The partner cells of a home cell (cx, cy, cz) in stencil column cd =
// (dx, dy, dz0, len): cc, the link-cell index of the partner column's first
// cell; ns (1 or 2) runs of consecutive cells za[s] .. zb[s] in that column,
// with their periodic images ix, iy (-1, 0, 1) and iz[s].
struct ColRuns {
   int cc, ns, ix, iy;
   int za[2], zb[2], iz[2];
};
__device__ __forceinline__ ColRuns col_runs(const RsParams &P, int cx, int cy, int cz, int4 cd)
{
   ColRuns r;
   int bx = cx + cd.x, by = cy + cd.y;
   r.ix = bx < 0 ? -1 : (bx >= P.nx ? 1 : 0);
   r.iy = by < 0 ? -1 : (by >= P.ny ? 1 : 0);
   bx -= r.ix * P.nx;
   by -= r.iy * P.ny;
   r.cc = P.nz * (by + P.ny * bx);
   const int z0 = cz + cd.z, z1 = z0 + cd.w - 1;
   r.ns = 1;
   if (z1 < 0) { r.za[0] = z0 + P.nz; r.zb[0] = z1 + P.nz; r.iz[0] = -1; }
   else if (z0 >= P.nz) { r.za[0] = z0 - P.nz; r.zb[0] = z1 - P.nz; r.iz[0] = 1; }
   else if (z0 < 0) { r.za[0] = z0 + P.nz; r.zb[0] = P.nz - 1; r.iz[0] = -1; r.za[1] = 0; r.zb[1] = z1; r.iz[1] = 0; r.ns = 2; }
   else if (z1 >= P.nz) { r.za[0] = z0; r.zb[0] = P.nz - 1; r.iz[0] = 0; r.za[1] = 0; r.zb[1] = z1 - P.nz; r.iz[1] = 1; r.ns = 2; }
   else { r.za[0] = z0; r.zb[0] = z1; r.iz[0] = 0; }
   return r;
}

// The walk of the column kernels: calls visit(j, inf) for every slot j of the
// home cell (cx, cy, cz)'s stencil (the home slot among them), inf = index
// base << 5 | image code: the offset-table entry of slot j in cell c (its z
// alone with ZREL) is c + (inf >> 5).  csk: the cell starts of the class
// walked.  Listing the candidates costs as much as the mixed form's pair
// arithmetic (32,000-site water: 2327 instructions a home site, 10 rounds of
// about 110 of them arithmetic; 2046 so, pairs of
// 131,072-site water 356 -> 314 us), hence: the runs of a lane's
// columns stay in registers (in shared memory only where the candidates do
// not fit one window), a second run per column is looked at only where some
// column wraps the cell, and cells whose whole stencil lies inside the grid
// take a path without images.
struct ColRows {
   int *inc, *jb, *inf, *cand;
};
template <bool ZREL, class Visit>
__device__ __forceinline__ void walk_columns(const RsParams &P, const int *__restrict__ csk,
                                             const int4 *__restrict__ cols, const int *__restrict__ col_base,
                                             int cx, int cy, int cz, int lane, const ColRows &w, Visit &&visit)
{
   const bool inside = cx >= P.ex && cx + P.ex < P.nx && cy >= P.ey && cy + P.ey < P.ny && cz + P.z0 >= 0 &&
                       cz + P.z1 < P.nz;
   for (int base = 0; base < P.ncols; base += 32 * COL_E) {
      int T, nrow;   // candidates; runs per column
      {
         int cnt[2 * COL_E], jb[2 * COL_E], tot = 0, ns = 1;
#pragma unroll
         for (int u = 0; u < COL_E; u++) {
            const int q0 = lane * 2 * COL_E + 2 * u, col = base + lane * COL_E + u;
            cnt[2 * u] = cnt[2 * u + 1] = jb[2 * u] = jb[2 * u + 1] = 0;
            if (col < P.ncols) {
               const int4 cd = __ldg(&cols[col]);
               const int ob = __ldg(&col_base[col]);
               if (inside) {
                  const int cc = P.nz * (cy + cd.y + P.ny * (cx + cd.x)), z = cz + cd.z;
                  jb[2 * u] = __ldg(&csk[cc + z]);
                  cnt[2 * u] = __ldg(&csk[cc + z + cd.w]) - jb[2 * u];
                  w.inf[q0] = (ob - z - (ZREL ? 0 : cc)) * 32 | 13;
               } else {
                  const ColRuns cr = col_runs(P, cx, cy, cz, cd);
#pragma unroll
                  for (int s = 0; s < 2; s++)
                     if (s < cr.ns) {
                        jb[2 * u + s] = __ldg(&csk[cr.cc + cr.za[s]]);
                        cnt[2 * u + s] = __ldg(&csk[cr.cc + cr.zb[s] + 1]) - jb[2 * u + s];
                        const int eb = ob - cd.z - cz + cr.iz[s] * P.nz - (ZREL ? 0 : cr.cc);
                        w.inf[q0 + s] = eb * 32 | (9 * (cr.ix + 1) + 3 * (cr.iy + 1) + (cr.iz[s] + 1));
                     }
                  ns = max(ns, cr.ns);
               }
               tot += cnt[2 * u] + cnt[2 * u + 1];
            }
         }
         nrow = inside ? 1 : __reduce_max_sync(0xffffffffu, ns);
         const int linc = warp_incl_scan(tot);
         T = __shfl_sync(0xffffffffu, linc, 31);
         int run = linc - tot;
         // the runs end to end: the first window's candidates (slot | run << 24)
#pragma unroll
         for (int r = 0; r < 2 * COL_E; r++)
            if ((r & 1) == 0 || nrow == 2) {
               const int q = lane * 2 * COL_E + r, e = run + cnt[r], jq = jb[r] - run;
               if (T > COL_WIN) {   // later windows read the runs again
                  w.jb[q] = jq;
                  w.inc[q] = e;
               }
               const int b = min(e, COL_WIN);
               for (int t = run; t < b; t++) w.cand[t] = (jq + t) | (q << 24);
               run = e;
            }
      }
      __syncwarp();
      for (int w0 = 0; w0 < T; w0 += COL_WIN) {
         const int w1 = min(T, w0 + COL_WIN);
         if (w0 > 0) {
#pragma unroll
            for (int r = 0; r < 2 * COL_E; r++)
               if ((r & 1) == 0 || nrow == 2) {
                  const int q = lane * 2 * COL_E + r, q1 = q - (nrow == 2 ? 1 : 2);   // the run before
                  const int a = max(q1 >= 0 ? w.inc[q1] : 0, w0), b = min(w.inc[q], w1), jq = w.jb[q];
                  for (int t = a; t < b; t++) w.cand[t - w0] = (jq + t) | (q << 24);
               }
            __syncwarp();
         }
         for (int r0 = w0; r0 < w1; r0 += 32) {
            const int idx = r0 + lane;
            if (idx < w1) {
               const int v = w.cand[idx - w0];
               visit(v & 0xffffff, w.inf[(unsigned)v >> 24]);
            }
         }
         __syncwarp();
      }
   }
}

// Each warp takes home slots of the class-major layout in turn (eight
// blocks per SM, the grid's warps striding over the slots, so that the
// block's set-up and energy reduction are paid once per block).  Per home
// slot, a pass gives each lane
// COL_E columns (up to two slot runs each, of the home site's class); a warp
// prefix sum lays the runs end to end; windows of COL_WIN candidates are
// decoded into shared memory (slot | run << 24) and dealt out 32 at a time.
// The pair arithmetic is k_pairs's mixed form: FP32 from cell-relative
// co-ordinates and the exact cell offset as an (hi, lo) pair, decisions near
// a threshold re-made in FP64, Kahan-free per-lane sums reduced by warp
// trees.
template <int PT, bool EW>
__global__ void __launch_bounds__(PAIR_WARPS * 32, 8)
k_pairs_col(RsParams P, FinArgs fin, const int *__restrict__ cs, const int4 *__restrict__ cols, const int *__restrict__ col_base,
            const float4 *__restrict__ coff, const float4 *__restrict__ posc, const int2 *__restrict__ tagc,
            const int *__restrict__ cellc,
            const int *__restrict__ sortc, const double *__restrict__ site, const float *__restrict__ potg,
            double *__restrict__ force, double *__restrict__ part, unsigned int *__restrict__ sync, DevOut *out)
{
   typedef float R;
   constexpr int NP = NPar<PT>::v;
   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ int s_inc[PAIR_WARPS][COL_ROWS], s_jb[PAIR_WARPS][COL_ROWS], s_inf[PAIR_WARPS][COL_ROWS];
   __shared__ int s_cand[PAIR_WARPS][COL_WIN];
   R *pot_s = reinterpret_cast<R *>(smem_raw);
   const int npot = P.max_id * P.max_id;
   if (P.pot_in_smem)
      for (int q = threadIdx.x; q < npot * NPOTP; q += blockDim.x) pot_s[q] = potg[q];
   __syncthreads();
   const R *pot = P.pot_in_smem ? pot_s : potg;

   const int N = P.nsites, n0 = P.one_class ? N : cs[P.ncells];
   const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const ColRows rows{s_inc[w], s_jb[w], s_inf[w], s_cand[w]};
   // the lane's energy and virial over all its home sites (per-site sums
   // added in: two levels of FP32), kept in shared memory, which the
   // candidate loop's registers leave no room for
   __shared__ R s_tot[7][PAIR_WARPS * 32];
#pragma unroll
   for (int k = 0; k < 7; k++) s_tot[k][threadIdx.x] = R(0);
   // home slots (class-major) in chunks of COL_CHUNK consecutive slots, the
   // grid's blocks taking the chunks in turn and the block's warps the
   // chunk's slots in turn: a few resident blocks per SM take every site,
   // neighbouring sites (shared candidates and column starts in L1) at
   // about the same time
   for (ColHome hm(P.chunk, w); hm.p < N; hm.next()) {
      const int p = hm.p;
      R fx = 0, fy = 0, fz = 0, pe = 0, v0 = 0, v1 = 0, v2 = 0, v3 = 0, v4 = 0, v5 = 0;
      const int *csk = cs + (p < n0 ? 0 : P.ncells);
      const int c = cellc[p];
      const int cx = c / (P.ny * P.nz), cy = (c / P.nz) % P.ny, cz = c % P.nz;
      const int2 ti = tagc[p];
      const R *prow = pot + (size_t)(ti.x & 0xffff) * P.max_id * NPOTP;
      const float4 xi = posc[p];
      const R qi = xi.w;
      const R alpha = P.alphaf, norm = P.normf;
      const int oi = sortc[p];
      const R cut100 = (R)P.cut100;
      const bool hp = P.cls_pot >> (p >= n0) & 1, hc = P.cls_chg >> (p >= n0) & 1;
      walk_columns<true>(P, csk, cols, col_base, cx, cy, cz, lane, rows, [&](int j, int inf_q) {
         const int kimg = inf_q & 31;
         if (j == p && kimg == 13) return;
         const int2 tj = __ldg(&tagc[j]);
         const int e = (tj.x >> 16) + (inf_q >> 5);
         const float4 xj = __ldg(&posc[j]);
         float4 h4, l4;
         ld_coff(coff + 2 * e, h4, l4);
         const R rx = (h4.x + (xj.x - xi.x)) + l4.x;
         const R ry = (h4.y + (xj.y - xi.y)) + l4.y;
         const R rz = (h4.z + (xj.z - xi.z)) + l4.z;
         R r2 = rx * rx + ry * ry + rz * rz;
         const bool intra = ti.y == tj.y;
         bool too_close, clip;
         pair_flags<true>(P, r2, oi, j, kimg, sortc, site, too_close, clip);
         if (too_close && !intra) {
            const int oj = sortc[j];
            if (oi < oj) note_too_close(out, oi, oj);
         }
         const R r2a = r2;
         if (clip) r2 = cut100;
         R pp[NP];
         const R *pj = prow + (size_t)(tj.x & 0xffff) * NPOTP;
#pragma unroll
         for (int k = 0; k < NP; k++) pp[k] = pj[k];
         R f, u;
         pair_fu<PT, EW, R, true>(r2, xj.w * qi, pp, alpha, norm, f, u, hp, hc);
         if (intra) {
            // as in k_pairs: an intramolecular pair's energy is
            // what the intramolecular correction subtracts again
            R fa, ua = R(0);
            if (clip) pair_fu<PT, EW, R, true>(r2a, xj.w * qi, pp, alpha, norm, fa, ua, hp, hc);
            u = clip ? u - ua : R(0);
         }
         const R wx = f * rx, wy = f * ry, wz = f * rz;
         fx -= wx;
         fy -= wy;
         fz -= wz;
         pe += u;
         v0 += wx * rx;
         v1 += wx * ry;
         v2 += wx * rz;
         v3 += wy * ry;
         v4 += wy * rz;
         v5 += wz * rz;
      });
      R Fx = fx, Fy = fy, Fz = fz;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
         Fx += __shfl_down_sync(0xffffffffu, Fx, o);
         Fy += __shfl_down_sync(0xffffffffu, Fy, o);
         Fz += __shfl_down_sync(0xffffffffu, Fz, o);
      }
      if (lane == 0) {
         force[oi] = (double)Fx;
         force[N + oi] = (double)Fy;
         force[2 * N + oi] = (double)Fz;
      }
      // (half of each evaluation)
      s_tot[0][threadIdx.x] += R(0.5) * pe;
      s_tot[1][threadIdx.x] += R(0.5) * v0;
      s_tot[2][threadIdx.x] += R(0.5) * v1;
      s_tot[3][threadIdx.x] += R(0.5) * v2;
      s_tot[4][threadIdx.x] += R(0.5) * v3;
      s_tot[5][threadIdx.x] += R(0.5) * v4;
      s_tot[6][threadIdx.x] += R(0.5) * v5;
   }
   __shared__ R wred[7][PAIR_WARPS];
   R vv[7];
#pragma unroll
   for (int k = 0; k < 7; k++) vv[k] = s_tot[k][threadIdx.x];
#pragma unroll
   for (int k = 0; k < 7; k++) {
      R s = vv[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) wred[k][w] = s;
   }
   __syncthreads();
   if (threadIdx.x < 7) {
      double s = 0.0;
      for (int q = 0; q < PAIR_WARPS; q++) s += (double)wred[threadIdx.x][q];
      part[blockIdx.x * 8 + threadIdx.x] = s;
   }
   reduce_pairs_last(part, gridDim.x, sync, out, fin);
}

// r2 < b and r2 > b by their bits (a compare would take the FP64 pipe), for
// r2 a sum of squares and b positive and finite; both false when r2 is NaN, of
// either sign, as the compares are.
__device__ __forceinline__ bool r2_below(double r2, double b)
{
   return (unsigned long long)__double_as_longlong(r2) < (unsigned long long)__double_as_longlong(b);
}
__device__ __forceinline__ bool r2_above(double r2, double b)
{
   const unsigned long long i = (unsigned long long)__double_as_longlong(b);
   return (unsigned long long)__double_as_longlong(r2) - i - 1 < 0x7ff0000000000000ull - i;
}

// The FP64 form by columns over one interaction class at a time: k_pairs'
// FP64 arithmetic for r and r^2 (the reference's operation order), with the
// cheaper square root, reciprocal and exponential of PairMath<double, true>.
// The FP64 pipe bounds it (79 % busy at 32,000 sites): 131,072-site water
// (real-space phase) 9.75 ms with k_pairs (every class, 110 FP64 instructions
// per pair), 4.61 ms with 81 of them, 3.79 ms without those of a potential of
// zero parameters and with the shorter exponential, 3.62 ms without the
// charges' part in a class that has none; 2048-site water 0.220 -> 0.099 ms.
template <int PT, bool EW>
__global__ void __launch_bounds__(PAIR_WARPS * 32, 5)
k_pairs_col64(RsParams P, FinArgs fin, const int *__restrict__ cs, const int4 *__restrict__ cols,
              const int *__restrict__ col_base, const double4 *__restrict__ posc, const int2 *__restrict__ tagc,
              const int *__restrict__ cellc, const int *__restrict__ sortc, const double *__restrict__ potg,
              double *__restrict__ force, double *__restrict__ part, unsigned int *__restrict__ sync, DevOut *out)
{
   constexpr int NP = NPar<PT>::v;
   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ int s_inc[PAIR_WARPS][COL_ROWS], s_jb[PAIR_WARPS][COL_ROWS], s_inf[PAIR_WARPS][COL_ROWS];
   __shared__ int s_cand[PAIR_WARPS][COL_WIN];
   __shared__ double s_tot[7][PAIR_WARPS * 32];
   __shared__ double s_reloc[27][3];
   double *pot_s = reinterpret_cast<double *>(smem_raw);
   if (P.pot_in_smem)
      for (int q = threadIdx.x; q < P.max_id * P.max_id * NPOTP; q += blockDim.x) pot_s[q] = potg[q];
   for (int q = threadIdx.x; q < 81; q += blockDim.x) s_reloc[q / 3][q % 3] = P.reloc[q / 3][q % 3];
   if (EW || PT != 0) exp2_fill();
#pragma unroll
   for (int k = 0; k < 7; k++) s_tot[k][threadIdx.x] = 0.0;
   __syncthreads();
   const double *pot = P.pot_in_smem ? pot_s : potg;
   const int N = P.nsites, n0 = P.one_class ? N : cs[P.ncells];
   const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const ColRows rows{s_inc[w], s_jb[w], s_inf[w], s_cand[w]};
   const bool strict = P.strict && !P.molpbc;
   for (ColHome hm(P.chunk, w); hm.p < N; hm.next()) {
      const int p = hm.p;
      double fx = 0, fy = 0, fz = 0, pe = 0, v0 = 0, v1 = 0, v2 = 0, v3 = 0, v4 = 0, v5 = 0;
      const int *csk = cs + (p < n0 ? 0 : P.ncells);
      const int c = cellc[p];
      const int cx = c / (P.ny * P.nz), cy = (c / P.nz) % P.ny, cz = c % P.nz;
      const int2 ti = tagc[p];
      const double *prow = pot + (size_t)(ti.x & 0xffff) * P.max_id * NPOTP;
      const double4 xi = posc[p];
      const int oi = sortc[p];
      const bool hp = P.cls_pot >> (p >= n0) & 1, hc = P.cls_chg >> (p >= n0) & 1;
      walk_columns<false>(P, csk, cols, col_base, cx, cy, cz, lane, rows, [&](int j, int inf) {
         const int kimg = inf & 31;
         if (j == p && kimg == 13) return;
         const double4 xj = posc[j];
         const double *rl = s_reloc[kimg];
         const double rx = __dadd_rn(__dsub_rn(xj.x, xi.x), rl[0]);
         const double ry = __dadd_rn(__dsub_rn(xj.y, xi.y), rl[1]);
         const double rz = __dadd_rn(__dsub_rn(xj.z, xi.z), rl[2]);
         double r2 = __dadd_rn(__dadd_rn(__dmul_rn(rx, rx), __dmul_rn(ry, ry)), __dmul_rn(rz, rz));
         const int2 tj = __ldg(&tagc[j]);
         if (r2_below(r2, TOO_CLOSE) && ti.y != tj.y) {
            const int oj = sortc[j];
            if (oi < oj) note_too_close(out, oi, oj);
         }
         if (strict && r2_above(r2, P.cut2)) r2 = P.cut100;
         double pp[NP];
         const double *pj = prow + (size_t)(tj.x & 0xffff) * NPOTP;
#pragma unroll
         for (int k = 0; k < NP; k++) pp[k] = pj[k];
         double f, u;
         pair_fu<PT, EW, double, true>(r2, xj.w * xi.w, pp, P.alpha, P.norm, f, u, hp, hc);
         const double wx = f * rx, wy = f * ry, wz = f * rz;
         fx = fma(-f, rx, fx);   // (not w: one rounding fewer at the same cost)
         fy = fma(-f, ry, fy);
         fz = fma(-f, rz, fz);
         pe += u;
         v0 = fma(wx, rx, v0);
         v1 = fma(wx, ry, v1);
         v2 = fma(wx, rz, v2);
         v3 = fma(wy, ry, v3);
         v4 = fma(wy, rz, v4);
         v5 = fma(wz, rz, v5);
      });
      // the home site's force: warp trees; energy and virial (half of each
      // evaluation) into the lane's totals
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
         fx += __shfl_down_sync(0xffffffffu, fx, o);
         fy += __shfl_down_sync(0xffffffffu, fy, o);
         fz += __shfl_down_sync(0xffffffffu, fz, o);
      }
      if (lane == 0) {
         force[oi] = fx;
         force[N + oi] = fy;
         force[2 * N + oi] = fz;
      }
      s_tot[0][threadIdx.x] += pe;
      s_tot[1][threadIdx.x] += v0;
      s_tot[2][threadIdx.x] += v1;
      s_tot[3][threadIdx.x] += v2;
      s_tot[4][threadIdx.x] += v3;
      s_tot[5][threadIdx.x] += v4;
      s_tot[6][threadIdx.x] += v5;
   }
   __shared__ double wred[7][PAIR_WARPS];
#pragma unroll
   for (int k = 0; k < 7; k++) {
      double s = s_tot[k][threadIdx.x];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) wred[k][w] = s;
   }
   __syncthreads();
   if (threadIdx.x < 7) {
      double s = 0.0;
      for (int q = 0; q < PAIR_WARPS; q++) s += wred[threadIdx.x][q];
      part[blockIdx.x * 8 + threadIdx.x] = 0.5 * s;
   }
   reduce_pairs_last(part, gridDim.x, sync, out, fin);
}

// The reference's evaluated pair count after a column-walk pass (which
// leaves it out of the hot loop): per home slot the sites of every class in
// the stencil's column runs, less the site itself, summed into
// out->npairs2.  One thread per slot; run on demand (mdgpu_get_info).
__global__ void __launch_bounds__(256)
k_count_col(RsParams P, const int *__restrict__ cell_start, const int4 *__restrict__ cols,
            const int *__restrict__ cellc, DevOut *out)
{
   __shared__ unsigned long long sh[8];
   const int p = blockIdx.x * blockDim.x + threadIdx.x;
   unsigned long long n = 0;
   if (p < P.nsites) {
      const int c = cellc[p];
      const int cx = c / (P.ny * P.nz), cy = (c / P.nz) % P.ny, cz = c % P.nz;
      for (int col = 0; col < P.ncols; col++) {
         const ColRuns cr = col_runs(P, cx, cy, cz, __ldg(&cols[col]));
         for (int s = 0; s < cr.ns; s++) {
            const int *cs = cell_start + cr.cc;
            n += (unsigned long long)(__ldg(&cs[cr.zb[s] + 1]) - __ldg(&cs[cr.za[s]]));
            if (!P.one_class)   // class 1's cells
               n += (unsigned long long)(__ldg(&cs[P.ncells + cr.zb[s] + 1]) - __ldg(&cs[P.ncells + cr.za[s]]));
         }
      }
      n -= 1;   // the home site itself
   }
#pragma unroll
   for (int o = 16; o > 0; o >>= 1) n += __shfl_down_sync(0xffffffffu, n, o);
   if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = n;
   __syncthreads();
   if (threadIdx.x == 0) {
      unsigned long long t = 0;
      for (int w = 0; w < 8; w++) t += sh[w];
      if (t) atomicAdd((unsigned long long *)&out->npairs2, t);
   }
}

// Pairs across the interaction classes that come closer than the too-close
// distance (the reference warns of every evaluated pair with r^2 < 0.25,
// src/force.c:943-948, whatever its potential): such a pair lies in the
// 27-cell neighbourhood (cells at least 0.5 A thick).  For each class-0
// slot (class-major layout) nine threads take the class-1 sites of the
// neighbourhood, one column run of 3 cells each, and form r^2 in FP32 from the
// cell-relative co-ordinates and the exact cell offset (hi + lo), re-made
// in FP64 from the original co-ordinates with the reference's operation
// order within 1e-3 A^2 of the threshold, as k_pairs decides.  Reported
// once per pair, as (lower site index, higher), intramolecular pairs
// excepted.  nbcol[9]: the stencil column of each (dx, dy) in [-1, 1]^2.
struct NbCols {
   int col[9];
};

__global__ void __launch_bounds__(256)
k_tooclose_x(RsParams P, NbCols nb, const int *__restrict__ cs, const int4 *__restrict__ cols, const int *__restrict__ col_base,
             const float4 *__restrict__ coff, const float4 *__restrict__ posc, const int2 *__restrict__ tagc,
             const int *__restrict__ cellc,
             const int *__restrict__ sortc, const double *__restrict__ site, DevOut *out)
{
   const int t = blockIdx.x * blockDim.x + threadIdx.x;
   const int p = t / 9, d = t - 9 * p;   // one column of the neighbourhood per thread
   const int N = P.nsites, n0 = cs[P.ncells];
   if (p >= n0) return;
   const int *cs1 = cs + P.ncells;
   const int c = cellc[p];
   const int cx = c / (P.ny * P.nz), cy = (c / P.nz) % P.ny, cz = c % P.nz;
   const float4 xi = posc[p];
   const int moli = tagc[p].y, oi = sortc[p];
   {
      const int dx = d / 3 - 1, dy = d % 3 - 1;
      int bx = cx + dx, by = cy + dy;
      const int ix = bx < 0 ? -1 : (bx >= P.nx ? 1 : 0);
      const int iy = by < 0 ? -1 : (by >= P.ny ? 1 : 0);
      bx -= ix * P.nx;
      by -= iy * P.ny;
      const int cc = P.nz * (by + P.ny * bx);
      const int ci = nb.col[d];
      const int eb = __ldg(&col_base[ci]) - __ldg(&cols[ci]).z - cz;   // offset index of cell z: z + eb
      // cells cz-1 .. cz+1 of the column, split where they wrap in z (the
      // scan runs only with nz >= 3, so one side at most)
      const int z0 = cz - 1, z1 = cz + 1;
      int za[2], zb[2], iz[2], ns = 1;
      if (z0 < 0) { za[0] = z0 + P.nz; zb[0] = P.nz - 1; iz[0] = -1; za[1] = 0; zb[1] = z1; iz[1] = 0; ns = 2; }
      else if (z1 >= P.nz) { za[0] = z0; zb[0] = P.nz - 1; iz[0] = 0; za[1] = 0; zb[1] = z1 - P.nz; iz[1] = 1; ns = 2; }
      else { za[0] = z0; zb[0] = z1; iz[0] = 0; }
      for (int s = 0; s < ns; s++) {
         const int kimg = 9 * (ix + 1) + 3 * (iy + 1) + (iz[s] + 1);
         for (int j = cs1[cc + za[s]]; j < cs1[cc + zb[s] + 1]; j++) {
            const int2 tj = tagc[j];
            if (tj.y == moli) continue;
            const int e = (tj.x >> 16) + iz[s] * P.nz + eb;
            const float4 xj = posc[j];
            float4 h4, l4;
            ld_coff(coff + 2 * e, h4, l4);
            const float rx = (h4.x + (xj.x - xi.x)) + l4.x;
            const float ry = (h4.y + (xj.y - xi.y)) + l4.y;
            const float rz = (h4.z + (xj.z - xi.z)) + l4.z;
            const float r2 = rx * rx + ry * ry + rz * rz;
            if (r2 >= (float)TOO_CLOSE + 1e-3f) continue;
            bool close = r2 < (float)TOO_CLOSE;
            const int oj = sortc[j];
            if (fabsf(r2 - (float)TOO_CLOSE) < 1e-3f) {
               const double *rl = P.reloc[kimg];
               const double ax = __dadd_rn(__dsub_rn(site[oj], site[oi]), rl[0]);
               const double ay = __dadd_rn(__dsub_rn(site[N + oj], site[N + oi]), rl[1]);
               const double az = __dadd_rn(__dsub_rn(site[2 * (size_t)N + oj], site[2 * (size_t)N + oi]), rl[2]);
               close = __dadd_rn(__dadd_rn(__dmul_rn(ax, ax), __dmul_rn(ay, ay)), __dmul_rn(az, az)) < TOO_CLOSE;
            }
            if (close) note_too_close(out, min(oi, oj), max(oi, oj));
         }
      }
   }
}

// ----------------------------------------------------------------- adjoint
// Derivatives of one pair evaluation of pair_fu (f = -U'(r)/r, U) with
// respect to the potential parameters and the Ewald terms:
//   du[k] = dU/dp_k, df[k] = df/dp_k               (short-range part)
//   uc = erfc(alpha r)/r, fc = (uc + norm exp(-alpha^2 r^2))/r^2
//                                                   (per unit q_i q_j)
//   duc = d uc/d alpha, dfc = d fc/d alpha          (per unit q_i q_j)
// erfc is pair_fu's A&S polynomial t P(t) exp(-x^2), t = 1/(1 + p x), and
// is differentiated as such: these are the derivatives of the energy and
// force the forward kernel computes.
template <int NP, typename R>
struct PairGrad {
   R du[NP], df[NP];
   R uc, fc, duc, dfc;
};

template <int PT, bool EW, typename R, bool FAST = false>
__device__ __forceinline__ void pair_grad(R r2, const R *p, R alpha, R norm, PairGrad<NPar<PT>::v, R> &g)
{
   typedef PairMath<R, FAST> M;
   R r, r_r;
   M::template root<ExpOfR<PT>::v>(r2, r, r_r);
   const R rs_r = r_r * r_r;
   g.uc = g.fc = g.duc = g.dfc = R(0);
   if (EW) {
      const R x = alpha * r;
      const R t = M::rcp(R(1) + R(ASP) * x);
      const R pt = R(AS1) + t * (R(AS2) + t * (R(AS3) + t * (R(AS4) + t * R(AS5))));
      const R dpt = R(AS2) + t * (R(2.0 * AS3) + t * (R(3.0 * AS4) + t * R(4.0 * AS5)));
      const R ex = M::ex(-(x * x));
      // d/dx [t P(t) e^{-x^2}] with dt/dx = -p t^2
      const R derfc = ex * (-R(ASP) * t * t * (pt + t * dpt) - R(2) * x * t * pt);
      g.uc = t * pt * ex * r_r;
      g.fc = rs_r * (g.uc + norm * ex);
      g.duc = derfc;
      g.dfc = rs_r * (derfc + R(1.1283791670955126) * ex * (R(1) - R(2) * x * x));   // 2/sqrt(pi)
   }
   if (PT == 0) {   // p0 ((p1/r)^12 - (p1/r)^6)
      const R p1s = p[1] * p[1];
      R s6 = p1s * rs_r;
      s6 = s6 * s6 * s6;
      const R s12 = s6 * s6;
      const R t5 = p1s * p1s * p[1] * (rs_r * rs_r * rs_r);   // d s6 / d p1 / 6
      g.du[0] = s12 - s6;
      g.du[1] = R(6) * p[0] * t5 * (R(2) * s6 - R(1));
      g.df[0] = rs_r * R(6) * (R(2) * s12 - s6);
      g.df[1] = rs_r * R(36) * p[0] * t5 * (R(4) * s6 - R(1));
   } else if (PT == 1) {   // -p0/r^6 + p1 exp(-p2 r)
      const R E = M::ex(-p[2] * r);
      const R r6 = rs_r * rs_r * rs_r;
      g.du[0] = -r6;
      g.du[1] = E;
      g.du[2] = -r * p[1] * E;
      g.df[0] = R(-6) * rs_r * r6;
      g.df[1] = p[2] * E * r_r;
      g.df[2] = p[1] * E * (r_r - p[2]);
   } else if (PT == 2) {   // p0 exp(-p1 r) - p2 exp(-p3 r)
      const R E1 = M::ex(-p[1] * r), E3 = M::ex(-p[3] * r);
      const R e1 = p[0] * E1, e2 = -p[2] * E3;
      g.du[0] = E1;
      g.du[1] = -r * e1;
      g.du[2] = -E3;
      g.du[3] = -r * e2;
      g.df[0] = p[1] * E1 * r_r;
      g.df[1] = e1 * (r_r - p[1]);
      g.df[2] = -p[3] * E3 * r_r;
      g.df[3] = e2 * (r_r - p[3]);
   } else if (PT == 3) {   // p0 exp(-p1 r) + p2/r^12 - p3/r^4 - p4/r^6 - p5/r^8
      const R E1 = M::ex(-p[1] * r), e1 = p[0] * E1;
      const R r4 = rs_r * rs_r, r6 = r4 * rs_r, r8 = r4 * r4, r12 = r6 * r6;
      g.du[0] = E1;
      g.du[1] = -r * e1;
      g.du[2] = r12;
      g.du[3] = -r4;
      g.du[4] = -r6;
      g.du[5] = -r8;
      g.df[0] = p[1] * E1 * r_r;
      g.df[1] = e1 * (r_r - p[1]);
      g.df[2] = R(12) * rs_r * r12;
      g.df[3] = R(-4) * rs_r * r4;
      g.df[4] = R(-6) * rs_r * r6;
      g.df[5] = R(-8) * rs_r * r8;
   } else if (PT == 4) {   // p0/r^4 + p1/r^6 + p2/r^12
      const R r4 = rs_r * rs_r, r6 = r4 * rs_r, r12 = r6 * r6;
      g.du[0] = r4;
      g.du[1] = r6;
      g.du[2] = r12;
      g.df[0] = R(4) * rs_r * r4;
      g.df[1] = R(6) * rs_r * r6;
      g.df[2] = R(12) * rs_r * r12;
   } else {   // Morse: p0 e^{(p1-r)p2} - p3/r^6 + p4 (e^{-2 p5 (r-p6)} - 2 e^{-p5 (r-p6)})
      const R E1 = M::ex((p[1] - r) * p[2]), e1 = p[0] * E1;
      const R r6 = rs_r * rs_r * rs_r;
      const R d6 = r - p[6];
      const R E2 = M::ex(R(-2) * p[5] * d6), E3 = M::ex(-p[5] * d6);
      const R e2 = p[4] * E2, e3 = R(-2) * p[4] * E3;
      g.du[0] = E1;
      g.du[1] = p[2] * e1;
      g.du[2] = (p[1] - r) * e1;
      g.du[3] = -r6;
      g.du[4] = E2 - R(2) * E3;
      g.du[5] = -d6 * (R(2) * e2 + e3);
      g.du[6] = p[5] * (R(2) * e2 + e3);
      g.df[0] = r_r * p[2] * E1;
      g.df[1] = r_r * p[2] * p[2] * e1;
      g.df[2] = r_r * e1 * (R(1) + p[2] * (p[1] - r));
      g.df[3] = R(-6) * rs_r * r6;
      g.df[4] = R(2) * p[5] * r_r * (E2 - E3);
      g.df[5] = r_r * (R(2) * e2 + e3 - d6 * p[5] * (R(4) * e2 + e3));
      g.df[6] = r_r * p[5] * p[5] * (R(4) * e2 + e3);
   }
}

template <typename R>
__device__ __forceinline__ R warp_sum(R v)
{
#pragma unroll
   for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
   return v;   // valid in lane 0
}

// Gradients of the real-space energy and of G = sum_i v_i . F_i (the
// force-matching loss for residual weights v, the Hessian-vector product of
// the loss) with respect to the potential table, the site charges and
// alpha.  The same stencil walk as k_pairs, recomputed (no stored pair
// list), with the walk repeated once per partner site identifier b so that
// every lane accumulates the table entries (id_i, b, k) in registers.
//   slots [0, T)      dE/dp(a,b,k) at (a*max_id + b)*NP + k, T = max_id^2 NP
//   slots [T, 2T)     dG/dp(a,b,k)
//   slots 2T, 2T+1    dE/dalpha, dG/dalpha
//   gq[oi], gq[N+oi]  dE/dq, dG/dq of the home site (written, not added)
// The table entry (a, b) is the one the force on a site of id a from a site
// of id b reads; each ordered evaluation carries half the pair energy.
// Intramolecular pairs are left out of the energy terms (the
// intramolecular correction removes them again); the forces keep them.
// Persistent blocks: each warp takes home slots blockIdx.x*PAIR_WARPS + w,
// stepping by the grid; per-block slot sums are written to gpart.
template <int PT, bool EW, bool MIXED>
__global__ void __launch_bounds__(PAIR_WARPS * 32)
k_pairs_adj(RsParams P, AdjParams A, const int *__restrict__ cell_start,
            const int *__restrict__ slot_cell, const int4 *__restrict__ full,
            const float4 *__restrict__ off_hi, const float4 *__restrict__ off_lo,
            const double4 *__restrict__ pos64, const float4 *__restrict__ pos32,
            const int2 *__restrict__ tag, const int *__restrict__ sorted,
            const double *__restrict__ site, const double *__restrict__ potg64,
            const float *__restrict__ potg32, const double4 *__restrict__ res64,
            const float4 *__restrict__ res32, double *__restrict__ gq, double *__restrict__ gpart)
{
   typedef typename std::conditional<MIXED, float, double>::type R;
   constexpr int NP = NPar<PT>::v;
   extern __shared__ double s_acc[];
   __shared__ int s_inc[PAIR_WARPS][32 * WALK_E], s_jb[PAIR_WARPS][32 * WALK_E], s_info[PAIR_WARPS][32 * WALK_E];
   for (int q = threadIdx.x; q < A.nslot; q += blockDim.x) s_acc[q] = 0.0;
   __syncthreads();
   const R *pot = MIXED ? (const R *)(const void *)potg32 : (const R *)(const void *)potg64;
   const int N = P.nsites, T = P.max_id * P.max_id * NP;
   const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const WalkRows rows{s_inc[w], s_jb[w], s_info[w], off_hi, off_lo};
   const R alpha = MIXED ? (R)P.alphaf : (R)P.alpha, norm = MIXED ? (R)P.normf : (R)P.norm;
   const R cut100 = (R)P.cut100;
   for (int p0 = blockIdx.x * PAIR_WARPS; p0 < N; p0 += gridDim.x * PAIR_WARPS) {
      const int p = p0 + w;
      if (p >= N) break;
      const int c = slot_cell[p];
      const int2 ti = tag[p];
      double4 xi64 = make_double4(0, 0, 0, 0);
      float4 xi32 = make_float4(0, 0, 0, 0);
      if (MIXED) xi32 = pos32[p]; else xi64 = pos64[p];
      const R qi = MIXED ? (R)xi32.w : (R)xi64.w;
      R vix = 0, viy = 0, viz = 0;
      if (A.loss) {
         if (MIXED) {
            const float4 v = res32[p];
            vix = v.x; viy = v.y; viz = v.z;
         } else {
            const double4 v = res64[p];
            vix = v.x; viy = v.y; viz = v.z;
         }
      }
      const int oi = sorted[p];
      R gqe = 0, gql = 0, gae = 0, gal = 0;
      for (int b = 0; b < P.max_id; b++) {
         if (!((A.type_mask >> b) & 1u)) continue;
         R pp[NP], ge[NP], gl[NP];
         const R *pj = pot + ((size_t)ti.x * P.max_id + b) * NPOTP;
#pragma unroll
         for (int q = 0; q < NP; q++) {
            pp[q] = pj[q];
            ge[q] = gl[q] = R(0);
         }
         walk_stencil<MIXED>(P, p, c, lane, cell_start, full, off_hi, off_lo, rows, [&](int j, int k, int kimg) {
            const int2 tj = __ldg(&tag[j]);
            if (tj.x != b || (ti.y == P.fw_mol && tj.y == P.fw_mol)) return;
            R rx, ry, rz, r2, qj;
            pair_sep<MIXED>(P, j, k, kimg, rows, xi32, xi64, pos64, pos32, rx, ry, rz, r2, qj);
            bool too_close, clip;
            pair_flags<MIXED>(P, r2, oi, j, kimg, sorted, site, too_close, clip);
            if (clip) r2 = cut100;
            PairGrad<NP, R> g;
            pair_grad<PT, EW, R>(r2, pp, alpha, norm, g);
            if (ti.y != tj.y) {
#pragma unroll
               for (int q = 0; q < NP; q++) ge[q] += g.du[q];
               gqe += qj * g.uc;
               gae += qj * g.duc;
            }
            if (A.loss) {
               R vjx, vjy, vjz;
               if (MIXED) {
                  const float4 v = __ldg(&res32[j]);
                  vjx = v.x; vjy = v.y; vjz = v.z;
               } else {
                  const double4 v = res64[j];
                  vjx = v.x; vjy = v.y; vjz = v.z;
               }
               const R wi = vix * rx + viy * ry + viz * rz;            // v_i . r
               const R ws = wi - (vjx * rx + vjy * ry + vjz * rz);      // (v_i - v_j) . r
#pragma unroll
               for (int q = 0; q < NP; q++) gl[q] -= g.df[q] * wi;
               gql -= qj * g.fc * ws;
               gal -= qj * g.dfc * wi;
            }
         });
         double *se = s_acc + ((size_t)ti.x * P.max_id + b) * NP;
#pragma unroll
         for (int q = 0; q < NP; q++) {
            const R s = warp_sum(ge[q]);
            if (lane == 0) atomicAdd(se + q, 0.5 * (double)s);
         }
         if (A.loss) {
#pragma unroll
            for (int q = 0; q < NP; q++) {
               const R s = warp_sum(gl[q]);
               if (lane == 0) atomicAdd(se + T + q, (double)s);
            }
         }
      }
      gqe = warp_sum(gqe);
      gql = warp_sum(gql);
      gae = warp_sum(gae);
      gal = warp_sum(gal);
      if (lane == 0) {
         gq[oi] = (double)gqe;
         gq[N + oi] = (double)gql;
         atomicAdd(s_acc + 2 * T, 0.5 * (double)qi * (double)gae);
         atomicAdd(s_acc + 2 * T + 1, (double)qi * (double)gal);
      }
   }
   __syncthreads();
   for (int q = threadIdx.x; q < A.nslot; q += blockDim.x) gpart[(size_t)blockIdx.x * A.nslot + q] = s_acc[q];
}

// The same over the columns of the link-cell order (both forms, without a
// framework molecule or molecular cut-off): one walk for all partner
// identifiers, each lane accumulating its table entries per identifier in
// shared memory (a column of its own: no conflicts), and only the gradient
// asked for (LOSS: of G, else of the energy).  FP64 form: the cheaper
// primitives of PairMath<double, true>.  One walk instead of one per
// identifier: 16,384-site water, mixed, 458 -> 137 us (92 with eight blocks per
// SM); 2048 sites, FP64, 735 -> 190 us.  Dynamic shared memory: slot sums
// [nslot] FP64, lane sums [types NP][threads], the potential table.
template <int PT, bool EW, bool MIXED, bool LOSS>
__global__ void __launch_bounds__(PAIR_WARPS * 32, MIXED ? 8 : 4)
k_pairs_adj_col(RsParams P, AdjParams A, const int *__restrict__ cell_start, const int *__restrict__ slot_cell,
                const int4 *__restrict__ cols, const int *__restrict__ col_base, const float4 *__restrict__ coff,
                const double4 *__restrict__ pos64, const float4 *__restrict__ pos32, const int2 *__restrict__ tag,
                const int *__restrict__ sorted, const double *__restrict__ site, const double *__restrict__ potg64,
                const float *__restrict__ potg32, const double4 *__restrict__ res64, const float4 *__restrict__ res32,
                double *__restrict__ gq, double *__restrict__ gpart)
{
   typedef typename std::conditional<MIXED, float, double>::type R;
   constexpr int NP = NPar<PT>::v, NT = PAIR_WARPS * 32;
   extern __shared__ double s_acc[];
   __shared__ int s_inc[PAIR_WARPS][COL_ROWS], s_jb[PAIR_WARPS][COL_ROWS], s_inf[PAIR_WARPS][COL_ROWS];
   __shared__ int s_cand[PAIR_WARPS][COL_WIN];
   R *s_lane = reinterpret_cast<R *>(s_acc + A.nslot), *pot = s_lane + A.ntype * NP * NT;
   const int npot = P.max_id * P.max_id;
   for (int q = threadIdx.x; q < A.nslot; q += NT) s_acc[q] = 0.0;
   for (int q = threadIdx.x; q < npot * NPOTP; q += NT) pot[q] = MIXED ? (R)potg32[q] : (R)potg64[q];
   if (!MIXED) exp2_fill();
   __syncthreads();
   const int N = P.nsites, T = npot * NP;
   const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const ColRows rows{s_inc[w], s_jb[w], s_inf[w], s_cand[w]};
   R *acc = s_lane + threadIdx.x;
   const R alpha = MIXED ? (R)P.alphaf : (R)P.alpha, norm = MIXED ? (R)P.normf : (R)P.norm;
   const R cut100 = (R)P.cut100;
   for (ColHome hm(P.chunk, w); hm.p < N; hm.next()) {
      const int p = hm.p;
      for (int q = 0; q < A.ntype * NP; q++) acc[q * NT] = R(0);
      const int c = slot_cell[p];
      const int cx = c / (P.ny * P.nz), cy = (c / P.nz) % P.ny, cz = c % P.nz;
      const int2 ti = tag[p];
      const R *prow = pot + (size_t)ti.x * P.max_id * NPOTP;
      double4 xi64 = make_double4(0, 0, 0, 0);
      float4 xi32 = make_float4(0, 0, 0, 0);
      if (MIXED) xi32 = pos32[p]; else xi64 = pos64[p];
      const R qi = MIXED ? (R)xi32.w : (R)xi64.w;
      R vix = 0, viy = 0, viz = 0;
      if (LOSS) {
         if (MIXED) {
            const float4 v = res32[p];
            vix = v.x; viy = v.y; viz = v.z;
         } else {
            const double4 v = res64[p];
            vix = v.x; viy = v.y; viz = v.z;
         }
      }
      const int oi = sorted[p];
      R gqs = 0, gas = 0;
      walk_columns<false>(P, cell_start, cols, col_base, cx, cy, cz, lane, rows, [&](int j, int inf) {
         const int kimg = inf & 31;
         if (j == p && kimg == 13) return;
         const int2 tj = __ldg(&tag[j]);
         if (!LOSS && ti.y == tj.y) return;
         R rx, ry, rz, r2, qj;
         if (MIXED) {
            const float4 xj = __ldg(&pos32[j]);
            float4 h4, l4;
            ld_coff(coff + 2 * (__ldg(&slot_cell[j]) + (inf >> 5)), h4, l4);
            rx = (h4.x + (xj.x - xi32.x)) + l4.x;
            ry = (h4.y + (xj.y - xi32.y)) + l4.y;
            rz = (h4.z + (xj.z - xi32.z)) + l4.z;
            r2 = rx * rx + ry * ry + rz * rz;
            qj = xj.w;
         } else {
            const double4 xj = pos64[j];
            const double *rl = P.reloc[kimg];
            rx = __dadd_rn(__dsub_rn(xj.x, xi64.x), rl[0]);
            ry = __dadd_rn(__dsub_rn(xj.y, xi64.y), rl[1]);
            rz = __dadd_rn(__dsub_rn(xj.z, xi64.z), rl[2]);
            r2 = __dadd_rn(__dadd_rn(__dmul_rn(rx, rx), __dmul_rn(ry, ry)), __dmul_rn(rz, rz));
            qj = xj.w;
         }
         if (P.strict) {
            bool too_close, clip;
            pair_flags<MIXED>(P, r2, oi, j, kimg, sorted, site, too_close, clip);
            if (clip) r2 = cut100;
         }
         R pp[NP];
         const R *pj = prow + (size_t)tj.x * NPOTP;
#pragma unroll
         for (int q = 0; q < NP; q++) pp[q] = pj[q];
         PairGrad<NP, R> g;
         pair_grad<PT, EW, R, !MIXED>(r2, pp, alpha, norm, g);
         R *aj = acc + (int)A.type_index[tj.x] * NP * NT;
         if (LOSS) {
            R vjx, vjy, vjz;
            if (MIXED) {
               const float4 v = __ldg(&res32[j]);
               vjx = v.x; vjy = v.y; vjz = v.z;
            } else {
               const double4 v = res64[j];
               vjx = v.x; vjy = v.y; vjz = v.z;
            }
            const R wi = vix * rx + viy * ry + viz * rz;            // v_i . r
            const R ws = wi - (vjx * rx + vjy * ry + vjz * rz);      // (v_i - v_j) . r
#pragma unroll
            for (int q = 0; q < NP; q++) aj[q * NT] -= g.df[q] * wi;
            gqs -= qj * g.fc * ws;
            gas -= qj * g.dfc * wi;
         } else {
#pragma unroll
            for (int q = 0; q < NP; q++) aj[q * NT] += g.du[q];
            gqs += qj * g.uc;
            gas += qj * g.duc;
         }
      });
      double *se = s_acc + (LOSS ? T : 0) + (size_t)ti.x * P.max_id * NP;
      for (int b = 0; b < P.max_id; b++) {
         if (!((A.type_mask >> b) & 1u)) continue;
#pragma unroll
         for (int q = 0; q < NP; q++) {
            const R s = warp_sum(acc[((int)A.type_index[b] * NP + q) * NT]);
            if (lane == 0) atomicAdd(se + b * NP + q, LOSS ? (double)s : 0.5 * (double)s);
         }
      }
      gqs = warp_sum(gqs);
      gas = warp_sum(gas);
      if (lane == 0) {
         gq[(LOSS ? N : 0) + oi] = (double)gqs;
         atomicAdd(s_acc + 2 * T + (LOSS ? 1 : 0), (LOSS ? 1.0 : 0.5) * (double)qi * (double)gas);
      }
   }
   __syncthreads();
   for (int q = threadIdx.x; q < A.nslot; q += NT) gpart[(size_t)blockIdx.x * A.nslot + q] = s_acc[q];
}

// Slot sums over blocks: one block per slot, in a fixed order.
__global__ void __launch_bounds__(128) k_adj_slots(const double *__restrict__ gpart, int nblocks, int nslot,
                                                   double *__restrict__ slots)
{
   __shared__ double sh[4];
   const int q = blockIdx.x;
   double s = 0.0;
   for (int b = threadIdx.x; b < nblocks; b += 128) s += gpart[(size_t)b * nslot + q];
   s = warp_sum(s);
   if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
   __syncthreads();
   if (threadIdx.x == 0) slots[q] = (sh[0] + sh[1]) + (sh[2] + sh[3]);
}

// --------------------------------------------------------------------- RDF
// Site-pair distance histogram (rdf_inner + rdf_accum, src/force.c:1010-1103,
// src/rdf.c:94-107): the same warp-per-site walk over the strict stencil at
// the RDF limit, r^2 in FP64 with the reference's operation order from the
// original co-ordinates, bin = (int)(rbin sqrt(r^2)) kept when < nbins.
// Counts per (id_i, id_j, bin) in a shared-memory histogram per block when it
// fits (HIST_SMEM), else directly in global memory.
constexpr int HIST_SMEM = 8192;

__global__ void __launch_bounds__(PAIR_WARPS * 32)
k_rdf(RsParams P, const int *__restrict__ cell_start, const int *__restrict__ slot_cell,
      const int4 *__restrict__ full, const int2 *__restrict__ tag, const int *__restrict__ sorted,
      const double *__restrict__ site, double rbin, int nbins, unsigned long long *__restrict__ counts)
{
   __shared__ unsigned int hist[HIST_SMEM];
   __shared__ int s_inc[PAIR_WARPS][32 * WALK_E], s_jb[PAIR_WARPS][32 * WALK_E], s_info[PAIR_WARPS][32 * WALK_E];
   const int nh = P.max_id * P.max_id * nbins;
   const bool in_smem = nh <= HIST_SMEM;
   if (in_smem)
      for (int q = threadIdx.x; q < nh; q += blockDim.x) hist[q] = 0u;
   __syncthreads();
   const int N = P.nsites;
   const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const int p = blockIdx.x * PAIR_WARPS + w;
   const WalkRows rows{s_inc[w], s_jb[w], s_info[w], nullptr, nullptr};
   if (p < N) {
      const int c = slot_cell[p];
      const int oi = sorted[p];
      const int2 ti = tag[p];
      const int idi = ti.x;
      const double xi = site[oi], yi = site[N + oi], zi = site[2 * N + oi];
      walk_stencil<false>(P, p, c, lane, cell_start, full, nullptr, nullptr, rows, [&](int j, int, int kimg) {
         if (ti.y == P.fw_mol && __ldg(&tag[j]).y == P.fw_mol) return;
         const int oj = sorted[j];
         const double *rl = P.reloc[kimg];
         const double rx = __dadd_rn(__dsub_rn(site[oj], xi), rl[0]);
         const double ry = __dadd_rn(__dsub_rn(site[N + oj], yi), rl[1]);
         const double rz = __dadd_rn(__dsub_rn(site[2 * N + oj], zi), rl[2]);
         const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(rx, rx), __dmul_rn(ry, ry)), __dmul_rn(rz, rz));
         const int bin = __double2int_rz(__dmul_rn(rbin, sqrt(r2)));
         if (bin < nbins) {
            const int q = (idi * P.max_id + __ldg(&tag[j]).x) * nbins + bin;
            if (in_smem)
               atomicAdd(&hist[q], 1u);
            else
               atomicAdd(&counts[q], 1ull);
         }
      });
   }
   __syncthreads();
   if (in_smem)
      for (int q = threadIdx.x; q < nh; q += blockDim.x)
         if (hist[q]) atomicAdd(&counts[q], (unsigned long long)hist[q]);
}

// -------------------------------------------------------------- host side
// The slots class by class, or one list of every class.
static void set_one_class(RsParams &P, bool one)
{
   P.one_class = one;
   if (one) {
      P.cls_pot = P.cls_pot != 0;
      P.cls_chg = P.cls_chg != 0;
   }
}
static bool col_walk_ok(const mdgpu_ctx *c);

static RsParams make_params(mdgpu_ctx *c)
{
   RsParams P;
   memset(&P, 0, sizeof P);
   const RsGeom &g = c->rs;
   P.nsites = c->nsites;
   P.fw_mol = c->fw_mol;
   P.fw_site0 = c->fw_site0;
   P.nmol_ent = c->nmols_nf;
   P.nent = c->ctl.molpbc ? c->nmols_nf + (c->nsites - c->fw_site0) : c->nsites;
   P.nx = g.nx; P.ny = g.ny; P.nz = g.nz; P.ncells = g.ncells;
   P.rn[0] = 1.0 / g.nx; P.rn[1] = 1.0 / g.ny; P.rn[2] = 1.0 / g.nz;
   P.nfull = (int)g.full.size();
   P.ncols = (int)g.cols.size();
   P.z0 = g.nz;
   P.z1 = -g.nz;
   for (const int4 &cd : g.cols) {
      P.ex = std::max(P.ex, std::abs(cd.x));
      P.ey = std::max(P.ey, std::abs(cd.y));
      P.z0 = std::min(P.z0, cd.z);
      P.z1 = std::max(P.z1, cd.z + cd.w - 1);
   }
   P.cls_pot = c->cls_pot;
   P.cls_chg = c->cls_chg;
   P.max_id = c->max_id;
   P.molpbc = c->ctl.molpbc;
   P.strict = c->ctl.strict_cutoff;
   P.ptype = c->ptype;
   for (int i = 0; i < 9; i++) P.hinv[i] = g.hinv[i];
   for (int i = 0; i < 9; i++) P.h[i] = g.h[i];
   for (int k = 0; k < 27; k++)
      for (int r = 0; r < 3; r++) P.reloc[k][r] = g.reloc[k][r];
   P.cut2 = g.cut2;
   P.cut100 = g.cut100;
   P.alpha = c->ctl.alpha;
   P.norm = 2.0 * c->ctl.alpha / sqrt(PI);
   P.cut2f = (float)g.cut2;
   P.bandf = 1e-4f;
   P.alphaf = (float)P.alpha;
   P.normf = (float)P.norm;
   return P;
}

mdgpu_status rs_prepare(mdgpu_ctx *c)
{
   RsDev &d = c->rd;
   const RsGeom &g = c->rs;
   const int N = c->nsites;
   cudaStream_t st = c->stream;
#define CK(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) return cuda_check(c, e_, #x); } while (0)
   if (c->sys_dirty) {
      CK(d.siteid.ensure(N));
      CK(d.molmap.ensure(N));
      CK(d.chg.ensure(N));
      CK(d.ent_mol.ensure(2 * (size_t)c->nmols));
      CK(cudaMemcpyAsync(d.siteid.p, c->site_id.data(), N * sizeof(int), cudaMemcpyHostToDevice, st));
      CK(cudaMemcpyAsync(d.molmap.p, c->molmap.data(), N * sizeof(int), cudaMemcpyHostToDevice, st));
      CK(cudaMemcpyAsync(d.chg.p, c->chg.data(), N * sizeof(double), cudaMemcpyHostToDevice, st));
      std::vector<int> mf(2 * (size_t)c->nmols);
      for (int m = 0; m < c->nmols; m++) {
         mf[m] = c->mol_first[m];
         mf[c->nmols + m] = c->mol_nsites[m];
      }
      CK(cudaMemcpyAsync(d.ent_mol.p, mf.data(), mf.size() * sizeof(int), cudaMemcpyHostToDevice, st));
      const size_t np = (size_t)c->max_id * c->max_id * NPOTP;
      CK(d.pot64.ensure(np));
      CK(d.pot32.ensure(np));
      std::vector<float> p32(np);
      for (size_t i = 0; i < np; i++) p32[i] = (float)c->potpar[i];
      CK(cudaMemcpyAsync(d.pot64.p, c->potpar.data(), np * sizeof(double), cudaMemcpyHostToDevice, st));
      CK(cudaMemcpyAsync(d.pot32.p, p32.data(), np * sizeof(float), cudaMemcpyHostToDevice, st));
      // interaction classes: identifiers joined when they interact (both
      // charged, or a potential with a nonzero parameter either way); the
      // group holding the charged identifiers (else the most populous) is
      // class 0, every other group class 1
      {
         const int M = c->max_id, npar = pot_nparams(c->ptype);
         std::vector<int> grp(M), pop(M, 0);
         std::vector<char> charged(M, 0);
         for (int i = 0; i < N; i++) {
            pop[c->site_id[i]]++;
            if (c->chg[i] != 0.0) charged[c->site_id[i]] = 1;
         }
         for (int a = 0; a < M; a++) grp[a] = a;
         auto root = [&](int a) { while (grp[a] != a) a = grp[a] = grp[grp[a]]; return a; };
         for (int a = 0; a < M; a++)
            for (int b = 0; b < M; b++) {
               bool link = charged[a] && charged[b];
               for (int k = 0; k < npar && !link; k++)
                  link = c->potpar[((size_t)a * M + b) * NPOTP + k] != 0.0;
               if (link) grp[root(a)] = root(b);
            }
         int g0 = -1, best = -1;
         std::vector<int> gpop(M, 0);
         for (int a = 0; a < M; a++) gpop[root(a)] += pop[a];
         for (int a = 0; a < M; a++)
            if (charged[a]) g0 = root(a);
         if (g0 < 0)
            for (int a = 0; a < M; a++)
               if (gpop[root(a)] > best) best = gpop[g0 = root(a)];
         c->cls_of_id.assign(M, 0);
         c->ncls = 1;
         for (int a = 0; a < M; a++)
            if (pop[a] > 0 && root(a) != g0) {
               c->cls_of_id[a] = 1;
               c->ncls = 2;
            }
         for (int a = 0; a < M; a++)
            if (pop[a] == 0) c->cls_of_id[a] = 0;
         // which classes have a potential, and charges, among their sites
         c->cls_pot = c->cls_chg = 0;
         for (int a = 0; a < M; a++) {
            if (pop[a] == 0) continue;
            if (charged[a]) c->cls_chg |= 1 << c->cls_of_id[a];
            for (int b = 0; b < M; b++)
               for (int k = 0; pop[b] > 0 && k < npar; k++)
                  if (c->potpar[((size_t)a * M + b) * NPOTP + k] != 0.0) c->cls_pot |= 1 << c->cls_of_id[a];
         }
         std::vector<int> sc(N);
         for (int i = 0; i < N; i++) sc[i] = c->cls_of_id[c->site_id[i]];
         CK(d.site_cls.ensure(N));
         CK(cudaMemcpyAsync(d.site_cls.p, sc.data(), N * sizeof(int), cudaMemcpyHostToDevice, st));
         CK(cudaStreamSynchronize(st));
      }
      CK(cudaStreamSynchronize(st));
      CK(d.cell_of.ensure(N));
      CK(d.sorted.ensure(N));
      CK(d.rank.ensure(N));
      CK(d.unsorted.ensure(N));
      CK(d.pos32.ensure(N));
      CK(d.tag.ensure(N));
      CK(d.tagc.ensure(N));
      CK(d.slot_cell.ensure(N));
   }
   if (c->rs_valid && !c->rs_uploaded) {
      if (2 * (size_t)g.ncells > d.cell_count.n) {
         CK(d.cell_count.ensure(2 * (size_t)g.ncells));
         c->counts_clean = false;
      }
      CK(d.cell_start.ensure(2 * (size_t)g.ncells + 1));
      CK(d.blocksum.ensure((2 * (size_t)g.ncells + 1 + 1023) / 1024 + 2));
      std::vector<float4> coff(2 * g.coff_hi.size());
      for (size_t e = 0; e < g.coff_hi.size(); e++) {
         coff[2 * e] = g.coff_hi[e];
         coff[2 * e + 1] = g.coff_lo[e];
      }
      TablePack &k = d.geom;
      CK(k.begin());
      const size_t o[6] = {k.add(g.full), k.add(g.off_hi), k.add(g.off_lo), k.add(g.cols), k.add(g.col_base), k.add(coff)};
      CK(k.send(st));
      k.at(d.full.p, o[0]);
      k.at(d.off_hi.p, o[1]);
      k.at(d.off_lo.p, o[2]);
      k.at(d.cols.p, o[3]);
      k.at(d.col_base.p, o[4]);
      k.at(d.coff.p, o[5]);
      c->rs_uploaded = true;
   }
   const int nb = (N + PAIR_WARPS - 1) / PAIR_WARPS;
   CK(d.part.ensure((size_t)nb * 8));
   if (c->prec == MDGPU_FP64) CK(d.pos64.ensure(N));
   if (!d.sync.p) {
      CK(d.sync.ensure(SYNC_N));
      CK(cudaMemsetAsync(d.sync.p, 0, SYNC_N * sizeof(unsigned int), st));
   }
   return MDGPU_OK;
}

// Opts a pair kernel in to dyn bytes of dynamic shared memory.  The 48 KB a
// block has without that cover static and dynamic memory together, and these
// kernels have 6 to 28 KB of static memory.
template <class F> static cudaError_t allow_smem(F *kfn, size_t dyn)
{
   if (dyn <= 16 * 1024) return cudaSuccess;
   return cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
}

template <int PT, bool EW, bool MIXED, int MODE>
static cudaError_t launch_pairs_t(const RsParams &P, mdgpu_ctx *c, double *force, DevOut *out,
                                  unsigned long long *keys, long long key_cap, size_t smem)
{
   RsDev &d = c->rd;
   const int nb = (P.nsites + PAIR_WARPS - 1) / PAIR_WARPS;
   auto kfn = k_pairs<PT, EW, MIXED, MODE>;
   const cudaError_t e = allow_smem(kfn, smem);
   if (e != cudaSuccess) return e;
   kfn<<<nb, PAIR_WARPS * 32, smem, c->stream>>>(P, d.cell_start.p, d.slot_cell.p, d.full.p, d.off_hi.p, d.off_lo.p,
                                     d.pos64.p, d.pos32.p, d.tag.p, d.sorted.p, c->cur_site,
                                     d.pot64.p, d.pot32.p, d.chg.p, force, d.part.p, out, keys, key_cap);
   return cudaGetLastError();
}

template <int PT>
static cudaError_t launch_pairs_pt(const RsParams &P, mdgpu_ctx *c, bool ew, bool mixed, int mode,
                                   double *force, DevOut *out, unsigned long long *keys,
                                   long long key_cap, size_t smem)
{
   if (mode == 1) return launch_pairs_t<PT, false, false, 1>(P, c, force, out, keys, key_cap, smem);
   if (mixed)
      return ew ? launch_pairs_t<PT, true, true, 0>(P, c, force, out, keys, key_cap, smem)
                : launch_pairs_t<PT, false, true, 0>(P, c, force, out, keys, key_cap, smem);
   return ew ? launch_pairs_t<PT, true, false, 0>(P, c, force, out, keys, key_cap, smem)
             : launch_pairs_t<PT, false, false, 0>(P, c, force, out, keys, key_cap, smem);
}

template <int PT, bool EW, bool MIXED, bool LOSS>
static cudaError_t launch_adj_col_t(const RsParams &P, const AdjParams &A, mdgpu_ctx *c, int nblk, size_t smem)
{
   RsDev &d = c->rd;
   AdjDev &a = c->ad;
   auto kfn = k_pairs_adj_col<PT, EW, MIXED, LOSS>;
   const cudaError_t e = allow_smem(kfn, smem);
   if (e != cudaSuccess) return e;
   kfn<<<nblk, PAIR_WARPS * 32, smem, c->stream>>>(P, A, d.cell_start.p, d.slot_cell.p, d.cols.p, d.col_base.p,
                                                   d.coff.p, d.pos64.p, d.pos32.p, d.tag.p, d.sorted.p, c->cur_site,
                                                   d.pot64.p, d.pot32.p, a.res64.p, a.res32.p, a.gq.p, a.gpart.p);
   return cudaGetLastError();
}

template <int PT, bool EW, bool MIXED>
static cudaError_t launch_adj_t(const RsParams &P, const AdjParams &A, mdgpu_ctx *c, int nblk)
{
   RsDev &d = c->rd;
   AdjDev &a = c->ad;
   // the column walk keeps lane sums and the potential table in shared
   // memory: within 160 KB (it needs 28 KB with four identifiers and two
   // parameters, the benchmark's water)
   const size_t smem = A.nslot * sizeof(double) +
                       ((size_t)A.ntype * NPar<PT>::v * PAIR_WARPS * 32 + (size_t)P.max_id * P.max_id * NPOTP) *
                          (MIXED ? sizeof(float) : sizeof(double));
   if (col_walk_ok(c) && smem <= 160 * 1024)
      return A.loss ? launch_adj_col_t<PT, EW, MIXED, true>(P, A, c, nblk, smem)
                    : launch_adj_col_t<PT, EW, MIXED, false>(P, A, c, nblk, smem);
   k_pairs_adj<PT, EW, MIXED><<<nblk, PAIR_WARPS * 32, A.nslot * sizeof(double), c->stream>>>(
      P, A, d.cell_start.p, d.slot_cell.p, d.full.p, d.off_hi.p, d.off_lo.p, d.pos64.p, d.pos32.p, d.tag.p,
      d.sorted.p, c->cur_site, d.pot64.p, d.pot32.p, a.res64.p, a.res32.p, a.gq.p, a.gpart.p);
   return cudaGetLastError();
}

template <int PT>
static cudaError_t launch_adj_pt(const RsParams &P, const AdjParams &A, mdgpu_ctx *c, bool ew, bool mixed,
                                 int nblk)
{
   if (mixed)
      return ew ? launch_adj_t<PT, true, true>(P, A, c, nblk) : launch_adj_t<PT, false, true>(P, A, c, nblk);
   return ew ? launch_adj_t<PT, true, false>(P, A, c, nblk) : launch_adj_t<PT, false, false>(P, A, c, nblk);
}

int pot_nparams(int ptype)
{
   switch (ptype) {
   case 0: return NPar<0>::v;
   case 1: return NPar<1>::v;
   case 2: return NPar<2>::v;
   case 3: return NPar<3>::v;
   case 4: return NPar<4>::v;
   case 6: return NPar<6>::v;
   default: return 0;
   }
}

mdgpu_status rs_adjoint(mdgpu_ctx *c, bool loss)
{
   AdjDev &a = c->ad;
   cudaStream_t st = c->stream;
   RsParams P = make_params(c);
   const int N = c->nsites;
   const bool mixed = c->prec == MDGPU_MIXED;
   const int np = pot_nparams(c->ptype);
   AdjParams A;
   A.loss = loss ? 1 : 0;
   A.type_mask = 0;
   for (int id : c->site_id) A.type_mask |= 1u << id;
   A.nslot = 2 * c->max_id * c->max_id * np + 2;
   A.ntype = 0;
   for (int b = 0; b < MDGPU_ADJ_MAX_ID; b++) A.type_index[b] = (unsigned char)((A.type_mask >> b) & 1u ? A.ntype++ : 0);
   // as many blocks as are resident: the kernel's launch bounds, or what its
   // shared memory (with many identifiers) leaves room for (the walk waits for
   // its gathers: 16,384-site water, mixed, 134 us with four blocks per SM, 92
   // us with eight)
   const size_t smem = (size_t)A.nslot * sizeof(double) + 20 * 1024 +
                       ((size_t)A.ntype * np * PAIR_WARPS * 32 + (size_t)c->max_id * c->max_id * NPOTP) *
                          (mixed ? sizeof(float) : sizeof(double));
   const int per_sm = std::max(1, std::min(mixed ? 8 : 4, (int)(227 * 1024 / smem)));
   const int nblk = std::min((N + PAIR_WARPS - 1) / PAIR_WARPS, per_sm * 152);
   P.chunk = col_chunk(N, nblk);
   CK(a.gq.ensure(2 * (size_t)N));
   CK(a.gpart.ensure((size_t)nblk * A.nslot));
   CK(a.slots.ensure((size_t)A.nslot));
   const bool ew = c->ctl.alpha > 0.0;
   cudaError_t e;
   switch (c->ptype) {
   case 0: e = launch_adj_pt<0>(P, A, c, ew, mixed, nblk); break;
   case 1: e = launch_adj_pt<1>(P, A, c, ew, mixed, nblk); break;
   case 2: e = launch_adj_pt<2>(P, A, c, ew, mixed, nblk); break;
   case 3: e = launch_adj_pt<3>(P, A, c, ew, mixed, nblk); break;
   case 4: e = launch_adj_pt<4>(P, A, c, ew, mixed, nblk); break;
   case 6: e = launch_adj_pt<6>(P, A, c, ew, mixed, nblk); break;
   default: return fail(c, MDGPU_E_PTYPE, "KERNEL called with unknown potential type");
   }
   CK(e);
   k_adj_slots<<<A.nslot, 128, 0, st>>>(a.gpart.p, nblk, A.nslot, a.slots.p);
   CK(cudaGetLastError());
   c->launches += 2;
   return MDGPU_OK;
}

mdgpu_status rs_rdf(mdgpu_ctx *c, double limit, int nbins)
{
   RsDev &d = c->rd;
   const RsGeom &g = c->rs;
   cudaStream_t st = c->stream;
   if (!(limit > 0.0) || nbins <= 0) return fail(c, MDGPU_E_ARG, "RDF limit and bin count must be positive");
   if (c->class_major) {   // binned for a force call: again in link-cell order
      c->link_order = true;
      const mdgpu_status s = rs_launch(c, c->cur_site, c->cofm_in.p, c->force.p, true, nullptr, 0, nullptr);
      c->link_order = false;
      if (s != MDGPU_OK) return s;
   }
   double key[11];
   std::memcpy(key, g.h, 9 * sizeof(double));
   key[9] = limit;
   key[10] = (double)(g.nx + 1000 * (g.ny + 1000 * g.nz));
   if (d.rdf_nfull == 0 || std::memcmp(key, d.rdf_key, sizeof key) != 0) {
      std::vector<int4> full;
      mdgpu_status s = build_rdf_stencil(g.h, limit, g.nx, g.ny, g.nz, full);
      if (s == MDGPU_E_CUTOFF)
         return fail(c, s, "RDF limit > 1 * cell dimension (neighbour cells beyond one image)");
      if (s) return fail(c, s, "RDF stencil");
      CK(d.rdf_full.ensure(full.size()));
      CK(cudaMemcpyAsync(d.rdf_full.p, full.data(), full.size() * sizeof(int4), cudaMemcpyHostToDevice, st));
      CK(cudaStreamSynchronize(st));
      d.rdf_nfull = (int)full.size();
      std::memcpy(d.rdf_key, key, sizeof key);
   }
   const size_t nh = (size_t)c->max_id * c->max_id * nbins;
   CK(d.rdf_counts.ensure(nh));
   CK(cudaMemsetAsync(d.rdf_counts.p, 0, nh * sizeof(unsigned long long), st));
   RsParams P = make_params(c);
   P.nfull = d.rdf_nfull;
   const double rbin = (double)nbins / limit;   // src/rdf.c:99
   const int N = c->nsites;
   k_rdf<<<(N + PAIR_WARPS - 1) / PAIR_WARPS, PAIR_WARPS * 32, 0, st>>>(
      P, d.cell_start.p, d.slot_cell.p, d.rdf_full.p, d.tag.p, d.sorted.p, c->cur_site, rbin, nbins, d.rdf_counts.p);
   CK(cudaGetLastError());
   c->launches += 1;
   return MDGPU_OK;
}

mdgpu_status rs_launch(mdgpu_ctx *c, const double *d_site, const double *d_cofm, double *d_force,
                       bool cells_only, unsigned long long *d_keys, int64_t key_cap,
                       cudaEvent_t sorted_ready)
{
   RsDev &d = c->rd;
   const RsGeom &g = c->rs;
   cudaStream_t st = c->stream;
   RsParams P = make_params(c);
   const int N = c->nsites;
   DevOut *out = c->out.p;
   c->cur_site = d_site;
   phase_mark(c, MDGPU_PH_CELLS);
   // class by class where the column walk follows; the adjoint, the RDF and
   // the key listing read the plain link-cell order
   c->class_major = c->ncls == 2 && g.nbr27 && col_walk_ok(c) && !d_keys && !c->ks_all_sites && !c->link_order;
   const int ncount = g.ncells * (c->class_major ? 2 : 1), nent = P.nent;
   if (!c->counts_clean) CK(cudaMemsetAsync(d.cell_count.p, 0, d.cell_count.n * sizeof(int), st));
   c->counts_clean = false;
   k_bin<<<(nent + 255) / 256, 256, 0, st>>>(P, d_site, d_cofm, d.ent_mol.p, d.ent_mol.p + c->nmols,
                                             c->class_major ? d.site_cls.p : nullptr, d.cell_of.p, d.rank.p,
                                             d.cell_count.p, d.cell_start.p, ncount, d.unsorted.p, d.sync.p, out);
   c->launches += 2;
   if (ncount > SCAN_ONE) {
      const int n = ncount + 1, nbs = (n + 1023) / 1024;
      k_scan_blocks<<<nbs, 1024, 0, st>>>(d.cell_count.p, d.cell_start.p, d.blocksum.p, ncount, n);
      k_scan_add<<<nbs, 1024, 0, st>>>(d.cell_start.p, d.blocksum.p, n);
      c->launches += 2;
   }
   if (ncount > SCAN_ONE || N > SCATTER_ONE) {
      k_scatter<<<(N + 255) / 256, 256, 0, st>>>(N, d.cell_of.p, d.cell_start.p, d.rank.p, d.unsorted.p);
      c->launches += 1;
   }
   const bool mixed = c->prec == MDGPU_MIXED && d_keys == nullptr;
   if (!mixed) CK(d.pos64.ensure(N));
   k_place<<<(N + 127) / 128, 128, 0, st>>>(P, d_site, d.chg.p, d.siteid.p, d.molmap.p, d.unsorted.p, d.cell_of.p,
                                            d.cell_start.p, d.cell_count.p, ncount, d.sorted.p,
                                            mixed ? nullptr : d.pos64.p, d_keys == nullptr ? d.pos32.p : nullptr,
                                            c->class_major ? nullptr : d.tag.p, d.tagc.p, d.slot_cell.p);
   CK(cudaGetLastError());
   c->counts_clean = true;
   if (sorted_ready) CK(cudaEventRecord(sorted_ready, st));
   phase_mark(c, MDGPU_PH_PAIRS);
   if (cells_only) return MDGPU_OK;
   return rs_pairs(c, d_force, d_keys, key_cap);
#undef CK
}

// The column walk serves both forms without a framework molecule or
// molecular cut-off, where every stencil column wraps the cell at most once
// and its packed words hold the grid: 27 bits of a cell index (walk_columns'
// index base), 15 of a z index (tagc).
static bool col_walk_ok(const mdgpu_ctx *c)
{
   static const bool off = [] {
      const char *e = std::getenv("MDGPU_PAIRS_COLUMNS");
      return e && e[0] == '0';
   }();
   return !off && c->rs.cols_ok && c->fw_mol < 0 && !c->ctl.molpbc && c->nsites < (1 << 24) &&
          c->rs.ncells < (1 << 25) && c->rs.nz <= (1 << 15) &&
          c->max_id < (1 << 16) && c->rs.cols.size() > 0;
}

template <int PT, bool EW>
static cudaError_t launch_col_t(const RsParams &P, mdgpu_ctx *c, double *force, bool mixed, size_t smem, int nb)
{
   RsDev &d = c->rd;
   FinArgs fin = c->fin;   // nothing follows without Ewald
   fin.on = fin.on && !fin.has_ewald;
   if (!mixed) {
      auto kfn = k_pairs_col64<PT, EW>;
      const cudaError_t e = allow_smem(kfn, smem);
      if (e != cudaSuccess) return e;
      kfn<<<nb, PAIR_WARPS * 32, smem, c->stream>>>(P, fin, d.cell_start.p, d.cols.p, d.col_base.p, d.pos64.p, d.tagc.p,
                                                    d.slot_cell.p, d.sorted.p, d.pot64.p, force, d.part.p, d.sync.p,
                                                    c->out.p);
      return cudaGetLastError();
   }
   auto kfn = k_pairs_col<PT, EW>;
   const cudaError_t e = allow_smem(kfn, smem);
   if (e != cudaSuccess) return e;
   kfn<<<nb, PAIR_WARPS * 32, smem, c->stream>>>(P, fin, d.cell_start.p, d.cols.p, d.col_base.p, d.coff.p, d.pos32.p,
                                                 d.tagc.p, d.slot_cell.p, d.sorted.p, c->cur_site, d.pot32.p, force,
                                                 d.part.p, d.sync.p, c->out.p);
   return cudaGetLastError();
}

// Class split of the binned slots, the column-walk pair kernel and, with
// two classes, the too-close scan across them.
static mdgpu_status rs_pairs_col(mdgpu_ctx *c, RsParams P, double *d_force, bool ew, bool mixed, size_t smem)
{
#define CK(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) return cuda_check(c, e_, #x); } while (0)
   RsDev &d = c->rd;
   cudaStream_t st = c->stream;
   const int N = c->nsites;
   const bool two = c->class_major;
   set_one_class(P, !two);
   // eight resident blocks per SM (the kernel's launch bounds), each warp
   // looping over home sites: the per-block set-up and energy reduction once
   // per block instead of once per four sites
   if (c->nsm <= 0) CK(cudaDeviceGetAttribute(&c->nsm, cudaDevAttrMultiProcessorCount, c->device));
   const int nb = std::min((N + PAIR_WARPS - 1) / PAIR_WARPS, (mixed ? 8 : 5) * c->nsm);
   c->rs_nblk = nb;
   P.chunk = col_chunk(N, nb);
   cudaError_t e;
   switch (c->ptype) {
   case 0: e = ew ? launch_col_t<0, true>(P, c, d_force, mixed, smem, nb) : launch_col_t<0, false>(P, c, d_force, mixed, smem, nb); break;
   case 1: e = ew ? launch_col_t<1, true>(P, c, d_force, mixed, smem, nb) : launch_col_t<1, false>(P, c, d_force, mixed, smem, nb); break;
   case 2: e = ew ? launch_col_t<2, true>(P, c, d_force, mixed, smem, nb) : launch_col_t<2, false>(P, c, d_force, mixed, smem, nb); break;
   case 3: e = ew ? launch_col_t<3, true>(P, c, d_force, mixed, smem, nb) : launch_col_t<3, false>(P, c, d_force, mixed, smem, nb); break;
   case 4: e = ew ? launch_col_t<4, true>(P, c, d_force, mixed, smem, nb) : launch_col_t<4, false>(P, c, d_force, mixed, smem, nb); break;
   case 6: e = ew ? launch_col_t<6, true>(P, c, d_force, mixed, smem, nb) : launch_col_t<6, false>(P, c, d_force, mixed, smem, nb); break;
   default: return fail(c, MDGPU_E_PTYPE, "KERNEL called with unknown potential type");
   }
   CK(e);
   c->launches += 1;
   if (two) {
      NbCols nb;
      for (int k = 0; k < 9; k++) nb.col[k] = c->rs.nbcol[k];
      k_tooclose_x<<<(9 * N + 255) / 256, 256, 0, st>>>(P, nb, d.cell_start.p, d.cols.p, d.col_base.p, d.coff.p,
                                                    d.pos32.p, d.tagc.p, d.slot_cell.p, d.sorted.p,
                                                    c->cur_site, c->out.p);
      CK(cudaGetLastError());
      c->launches += 1;
   }
   return MDGPU_OK;
#undef CK
}

mdgpu_status rs_count_pairs(mdgpu_ctx *c)
{
#define CK(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) return cuda_check(c, e_, #x); } while (0)
   if (!c->npairs_pending) return MDGPU_OK;
   RsParams P = make_params(c);
   set_one_class(P, !c->class_major);
   cudaStream_t st = c->stream;
   DevOut *out = c->out.p;
   CK(cudaMemsetAsync(&out->npairs2, 0, sizeof(out->npairs2), st));
   k_count_col<<<(c->nsites + 255) / 256, 256, 0, st>>>(P, c->rd.cell_start.p, c->rd.cols.p, c->rd.slot_cell.p, out);
   CK(cudaGetLastError());
   int64_t n2 = 0;
   CK(cudaMemcpyAsync(&n2, &out->npairs2, sizeof(n2), cudaMemcpyDeviceToHost, st));
   CK(cudaStreamSynchronize(st));
   c->info.npairs = n2 / 2;
   c->npairs_pending = false;
   return MDGPU_OK;
#undef CK
}

mdgpu_status rs_pairs(mdgpu_ctx *c, double *d_force, unsigned long long *d_keys, int64_t key_cap)
{
#define CK(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) return cuda_check(c, e_, #x); } while (0)
   RsDev &d = c->rd;
   cudaStream_t st = c->stream;
   RsParams P = make_params(c);
   const int N = c->nsites;
   DevOut *out = c->out.p;
   const bool mixed = c->prec == MDGPU_MIXED && d_keys == nullptr;
   const size_t potb = (size_t)c->max_id * c->max_id * NPOTP * (mixed ? sizeof(float) : sizeof(double));
   P.pot_in_smem = potb <= 96 * 1024;
   const size_t smem = P.pot_in_smem ? potb : 0;
   const bool ew = c->ctl.alpha > 0.0;
   const int mode = d_keys ? 1 : 0;
   cudaError_t e;
   c->npairs_pending = false;
   c->rs_nblk = (N + PAIR_WARPS - 1) / PAIR_WARPS;   // blocks of partial sums for the reduction
   if (mode == 0 && col_walk_ok(c)) {
      const mdgpu_status s = rs_pairs_col(c, P, d_force, ew, mixed, smem);
      if (s != MDGPU_OK) return s;
      c->npairs_pending = true;   // counted on demand (rs_count_pairs)
      if (c->fin.on && !c->fin.has_ewald) c->fin.on = 0;   // its last block has summed the evaluation up
      phase_mark(c, MDGPU_PH_KPREP);
      return MDGPU_OK;
   } else {
   switch (c->ptype) {
   case 0: e = launch_pairs_pt<0>(P, c, ew, mixed, mode, d_force, out, d_keys, key_cap, smem); break;
   case 1: e = launch_pairs_pt<1>(P, c, ew, mixed, mode, d_force, out, d_keys, key_cap, smem); break;
   case 2: e = launch_pairs_pt<2>(P, c, ew, mixed, mode, d_force, out, d_keys, key_cap, smem); break;
   case 3: e = launch_pairs_pt<3>(P, c, ew, mixed, mode, d_force, out, d_keys, key_cap, smem); break;
   case 4: e = launch_pairs_pt<4>(P, c, ew, mixed, mode, d_force, out, d_keys, key_cap, smem); break;
   case 6: e = launch_pairs_pt<6>(P, c, ew, mixed, mode, d_force, out, d_keys, key_cap, smem); break;
   default: return fail(c, MDGPU_E_PTYPE, "KERNEL called with unknown potential type");
   }
   CK(e);
   c->launches += 1;
   }
   if (mode == 0) {
      CK(d.part2.ensure(8 * RS_RED));
      k_reduce_rs<<<RS_RED, 256, 0, st>>>(d.part.p, c->rs_nblk, d.part2.p);
      k_reduce_rs2<<<1, 256, 0, st>>>(d.part2.p, RS_RED, out);
      c->launches += 2;
      CK(cudaGetLastError());
   }
   phase_mark(c, MDGPU_PH_KPREP);
   return MDGPU_OK;
#undef CK
}

}  // namespace mdgpu
