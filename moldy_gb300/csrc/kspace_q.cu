// Reciprocal space on the tensor cores by products of one-dimensional trig
// tables: the structure factor of both forms and the force pass of the FP64
// form (the S(k) and force sums of ewald(), src/ewald.c:523-579).
//
// A quad is a pair (h, m), m = |k| >= 0: the columns (h, +-m) of the k-list.
// With the per-site tables X = cos, sin(2 pi h s_x), Y = cos, sin(2 pi m s_y)
// and Z = cos, sin(2 pi t s_z), t = |l|, the four k-vectors (h, s m, r t),
// s, r = +-1, have
//     exp(i k.r) = [(P1 - s P2) + i (P3 + s P4)] (C_t + i r S_t),
//     P1 = ch cm, P2 = sh sm, P3 = sh cm, P4 = ch sm,
// so the eight real sums  Q_pc = sum_j q_j P_p {C_t, S_t}  give S(k) of all
// four (k_qreduce), and the force sums are eight real sums the other way
// round.  Against one seed per k-column and the running l this is half the
// tensor-core work per k-vector (both signs of l from one product) and one
// multiplication per operand element in place of half a sine/cosine pair.
//
// Arithmetic.  Every operand is a fixed-point integer cut into NS balanced
// base-256 digits d in [-128, 127], held as fp16 (exact), digit i of weight
// 2^(-7 - 8 i).  A product of digits i and j goes to accumulator group
// g = i + j; groups g < NS are kept.  In a group all products are integers
// below 2^14, so the FP32 accumulators are exact while fewer than
// 2^10 / (g + 1) terms are added; they are read back and added up in
// wide integers (NS = 7: 96 bits, every 128 terms) or FP32 (NS = 3, every
// 1024 terms, where only group 0 has to be exact).
//   NS = 3  mixed form: operands to 2^-24, as the FP32 path
//   NS = 7  FP64 form: operands to 2^-56, products left out below 2^-56:
//           errors below the rounding of an FP64 multiply-add per term.
// The tables themselves are integer polynomials of the exact integer phases
// (qsincos), good to 2^-60 and 2^-29.
// Digits laid end to end: operand B holds its NS digits as consecutive rows
// blocks, so one MMA of digit i of A by digits 0 .. NS - 1 - i of B adds to
// groups i .. NS - 1 at once (NS instructions per K-step in place of
// NS (NS + 1) / 2, and A is read from shared memory NS times).
//
// Measured, 131,072-site water (98,304 charged sites, 69,876 k-vectors),
// against one FP64 recurrence per k and site, or the seed-and-run bf16
// products of the mixed form: FP64 structure factor 119.4 -> 1.30 ms, forces
// 130.4 -> 4.80 ms; mixed structure factor 0.414 -> 0.262 ms.  What bounds the
// FP64 passes: each of the two A buffers goes round build (1500 cycles), MMAs
// (1800) and two barriers; the read-back of a segment (its conversions) is a
// quarter of the force pass.  Force error
// of the FP64 form against extended precision (2048-site water; rock salt,
// 5832 ions): 6.1e-15 -> 2.2e-15; 1.5e-14 -> 1.1e-14.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>

#include "mdgpu_internal.h"
#include "tc.cuh"

namespace mdgpu {

// ---------------------------------------------------------------- layout
constexpr int Q_KS = 32;                          // K per stage: sites, or K-rows (two units)
constexpr int Q_OP = 128 * Q_KS * 2;              // one digit of a 128-row operand stage: 8 KB
constexpr int Q_BW = 16;                          // operand / read-back warps
constexpr int Q_THREADS = 32 * (Q_BW + 3);        // and a bulk-copy warp, two MMA warps
constexpr int Q_ERR = 8, Q_FERR = 16;             // error-word bits: structure factor, force pass
constexpr int Q_NOT_FINITE = 8192;                // scale exponent: a value is infinite or NaN

template <int NS> struct QCfg;
template <> struct QCfg<3> {
   typedef int T;
   typedef float P;                               // structure-factor partials
   static constexpr int RS = 36;                  // table row: 32 sites, padded against bank conflicts
   static constexpr int MT = 2;                   // 128-row tiles per CTA
   static constexpr int NB = 3;                   // B operands in flight; one table buffer more
   static constexpr int NTMAX = 64;               // columns (2 t-width) of a t-block
   static constexpr int SEG = 32;                 // stages between read-backs
};
template <> struct QCfg<7> {
   typedef long long T;
   typedef double P;
   static constexpr int RS = 34;
   static constexpr int MT = 1;
   static constexpr int NB = 2;
   static constexpr int NTMAX = 64;
   static constexpr int SEG = 4;
};
// bytes: a stage's table rows, its B operand; the A operand; all
template <int NS> constexpr int Q_TAB = 2 * (Q_XMAX + Q_YMAX) * QCfg<NS>::RS * (int)sizeof(typename QCfg<NS>::T);
// (ND: digits of operand B, NS unless weights of a wide range need more)
template <int ND> constexpr int Q_B = 64 * Q_KS * 2 * ND;
template <int NS, int NA = NS> constexpr int Q_A = QCfg<NS>::MT * NA * Q_OP;
template <int NS, int ND, int NA = NS>
constexpr int Q_SMEM = 2 * Q_A<NS, NA> + QCfg<NS>::NB * Q_B<ND> + (QCfg<NS>::NB + 1) * Q_TAB<NS>;
constexpr int Q_FNB = 3, Q_FSMEM = 2 * Q_A<7> + Q_FNB * Q_B<7>;   // FP64 force pass: no table rows in shared memory
static_assert(Q_SMEM<3, 4, 4> <= 226 * 1024 && Q_SMEM<7, 7> <= 226 * 1024 && Q_FSMEM <= 220 * 1024, "one CTA's shared memory");
static_assert(Q_B<3> % 128 == 0 && Q_TAB<3> % 128 == 0 && Q_TAB<7> % 128 == 0, "stage buffers stay aligned");

// ------------------------------------------------------ fixed-point trig
// sin, cos(2 pi p / 2^64) in units of 2^-63: the phase is reduced to an
// eighth turn, p = quadrant + w (1/8), |w| <= 1, and the Taylor series of
// sin and cos (pi w / 4) are summed in v = w^2 / 4 by 64-bit integer Horner
// steps (coefficients (pi/4)^n 4^k / n! in units of 2^-64; terms left out
// below 2^-62).
__device__ __forceinline__ void qsincos(unsigned long long p, long long &s, long long &c)
{
   const unsigned int qd = (unsigned int)((p + (1ull << 61)) >> 62);
   const long long r = (long long)(p - ((unsigned long long)qd << 62));
   const unsigned long long w = (unsigned long long)(r < 0 ? -r : r) << 2;    // |w| 2^63
   const unsigned long long v = __umul64hi(w, w);                             // w^2 / 4 in 2^-64
   unsigned long long a = 0x355d865ull;
   a = 0x16fadb9f1ull - __umul64hi(v, a);
   a = 0x7a3d0d3406ull - __umul64hi(v, a);
   a = 0x1e3074fde887ull - __umul64hi(v, a);
   a = 0x541e0d21fb9e0ull - __umul64hi(v, a);
   a = 0x9969667315ec2eull - __umul64hi(v, a);
   a = 0xa335e33bad570e9ull - __umul64hi(v, a);
   a = 0x52aef39896f94afbull - __umul64hi(v, a);
   a = 0xc90fdaa22168c235ull - __umul64hi(v, a);
   unsigned long long b = 0x4a8316ull;
   b = 0x2418c586ull - __umul64hi(v, b);
   b = 0xdb7127a26ull - __umul64hi(v, b);
   b = 0x3f3a7146ec8ull - __umul64hi(v, b);
   b = 0xd368f9510254ull - __umul64hi(v, b);
   b = 0x1e1f506891babbull - __umul64hi(v, b);
   b = 0x2aba78fc797ff40ull - __umul64hi(v, b);
   b = 0x20783e1036b58767ull - __umul64hi(v, b);
   b = 0x9de9e64df22ef2d2ull - __umul64hi(v, b);
   unsigned long long sn = __umul64hi(w, a);
   unsigned long long cs = (1ull << 63) - __umul64hi(v, b);
   sn -= sn >> 8;                                                             // times Q_KAPPA
   cs -= cs >> 8;
   const long long S = r < 0 ? -(long long)sn : (long long)sn, C = (long long)cs;
   const bool sw = qd & 1u, ng = qd & 2u;
   s = sw ? C : S;
   c = sw ? -S : C;
   if (ng) {
      s = -s;
      c = -c;
   }
}
// The same for a 32-bit phase, in units of 2^-31 (terms left out below 2^-32).
__device__ __forceinline__ void qsincos(unsigned int p, int &s, int &c)
{
   const unsigned int qd = (p + (1u << 29)) >> 30;
   const int r = (int)(p - (qd << 30));
   const unsigned int w = (unsigned int)(r < 0 ? -r : r) << 2;
   const unsigned int v = __umulhi(w, w);
   unsigned int a = 0x1e30u;
   a = 0x541e1u - __umulhi(v, a);
   a = 0x996966u - __umulhi(v, a);
   a = 0xa335e34u - __umulhi(v, a);
   a = 0x52aef399u - __umulhi(v, a);
   a = 0xc90fdaa2u - __umulhi(v, a);
   unsigned int b = 0x3f4u;
   b = 0xd369u - __umulhi(v, b);
   b = 0x1e1f50u - __umulhi(v, b);
   b = 0x2aba790u - __umulhi(v, b);
   b = 0x20783e10u - __umulhi(v, b);
   b = 0x9de9e64eu - __umulhi(v, b);
   unsigned int sn = __umulhi(w, a), cs = (1u << 31) - __umulhi(v, b);
   sn -= (sn + 128) >> 8;   // (rounded: truncation biases the energy by 1e-9 of the self-energy)
   cs -= (cs + 128) >> 8;
   const int S = r < 0 ? -(int)sn : (int)sn, C = (int)cs;
   const bool sw = qd & 1u, ng = qd & 2u;
   s = sw ? C : S;
   c = sw ? -S : C;
   if (ng) {
      s = -s;
      c = -c;
   }
}
// phase n u (n a table index) in the form's width; 32-bit phases are
// rounded from the 64-bit product, so their error does not grow with n
__device__ __forceinline__ void qtrig(int n, unsigned long long u, long long &s, long long &c)
{
   qsincos((unsigned long long)n * u, s, c);
}
__device__ __forceinline__ void qtrig(int n, unsigned long long u, int &s, int &c)
{
   qsincos((unsigned int)(((unsigned long long)n * u + 0x80000000ull) >> 32), s, c);
}

// A 64-bit table value as (signed low word, high word): ah 2^32 + al.
__device__ __forceinline__ long long qbalance(long long v)
{
   const int lo = (int)v;
   return (long long)((unsigned long long)((v - lo) & ~0xffffffffll) | (unsigned int)lo);
}
__device__ __forceinline__ int qbalance(int v) { return v; }

// Biased product of two table values (units of 2^-31 / 2^-63 again): every
// byte but the lowest is a digit plus 128, the lowest rounds.
__device__ __forceinline__ unsigned int qmul(int a, int b)
{
   const unsigned int t = (unsigned int)__mulhi(a, b);
   return t + t + 0x80808080u;
}
__device__ __forceinline__ unsigned long long qmul(long long a, long long b)   // balanced values
{
   const int ah = (int)(a >> 32), al = (int)a, bh = (int)(b >> 32), bl = (int)b;
   int m;
   long long t;
   asm("mad.hi.s32 %0, %1, %2, %3;" : "=r"(m) : "r"(al), "r"(bh), "r"(__mulhi(ah, bl)));
   asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(t) : "r"(ah), "r"(bh), "l"((long long)m));
   return (unsigned long long)(t + t) + 0x8080808080808080ull;
}

// Digit i of two biased values as an fp16 pair (first value in the low half).
__device__ __forceinline__ unsigned int qpair(unsigned int bytes)   // 0x??B?A: values plus 128 in bytes 0 and 2
{
   unsigned int r;
   const unsigned int v = (bytes & 0x00ff00ffu) | 0x64006400u;       // fp16 1024 + byte
   asm("add.f16x2 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(0xe480e480u));   // - 1152
   return r;
}
template <int I> __device__ __forceinline__ unsigned int qdigit(unsigned int a, unsigned int b)
{
   return qpair(__byte_perm(a, b, (3 - I) | ((7 - I) << 8)));
}
template <int I> __device__ __forceinline__ unsigned int qdigit(unsigned long long a, unsigned long long b)
{
   if (I < 4)
      return qdigit<(I < 4 ? I : 0)>((unsigned int)(a >> 32), (unsigned int)(b >> 32));
   return qdigit<(I >= 4 ? I - 4 : 0)>((unsigned int)a, (unsigned int)b);
}
// NS = 3, operand A: x in units of 2^-24 (24 bits), y of 2^-31, the product
// rounded to 2^-23, its digits plus 128 in bytes 3, 2, 1 and the high byte
// of fp16 1024 in byte 0, so that one byte permutation gives an fp16 pair
// without a mask.  The ALU pipe (permutations, masks, adds; half the rate of
// the FMA pipe) bounds the operand build: the multiplications are written so
// that they run on the FMA pipe (c256 = 256 is not a constant to the
// compiler, or it would shift and add on the ALU).
struct QA {
   unsigned int v;
};
__device__ __forceinline__ QA qmul_a(int x, int y, unsigned int c256)
{
   const long long t = (long long)x * y + 0x80000000ll;
   QA r;
   asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r.v) : "r"((unsigned int)(t >> 32)), "r"(c256), "r"(0x80808064u));
   return r;
}
__device__ __forceinline__ unsigned long long qmul_a(long long x, long long y, unsigned int) { return qmul(x, y); }
template <int I> __device__ __forceinline__ unsigned int qdigit(QA a, QA b)
{
   unsigned int r;
   const unsigned int v = __byte_perm(a.v, b.v, (3 - I) | ((7 - I) << 8) | (4 << 12));
   asm("add.f16x2 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(0xe480e480u));   // - 1152
   return r;
}
// The NS digits of eight values (K order) to dst + i stride.
template <int NS, int I, typename U> struct QStore {
   static __device__ __forceinline__ void run(unsigned char *dst, int stride, const U (&v)[8])
   {
      *reinterpret_cast<uint4 *>(dst) =
         make_uint4(qdigit<I>(v[0], v[1]), qdigit<I>(v[2], v[3]), qdigit<I>(v[4], v[5]), qdigit<I>(v[6], v[7]));
      QStore<NS, I + 1, U>::run(dst + stride, stride, v);
   }
};
template <int NS, typename U> struct QStore<NS, NS, U> {
   static __device__ __forceinline__ void run(unsigned char *, int, const U (&)[8]) {}
};
template <int NS, typename U> __device__ __forceinline__ void qstore(unsigned char *dst, int stride, const U (&v)[8])
{
   QStore<NS, 0, U>::run(dst, stride, v);
}

__device__ __forceinline__ unsigned long long q_fixed64(double s)
{
   // frac(s) 2^64 for |s| < 2 (as k_prep)
   return (unsigned long long)__double2ll_rn(s * 4611686018427387904.0) << 2;
}

__device__ __forceinline__ int q_blkcols(const QGeom &g, int b) { return 2 * min(g.TW, g.TP - b * g.TW); }

// ------------------------------------------------------------- per site
// One block per 32-site stage of the charged list (slots; sites past n get
// phase and charge zero): the X and Y tables, the structure factor's B
// operand (digits of q z, the charge scaled by a power of two to |q| < 1),
// and per form: NS = 3 the force pass's A operand (zsite: three bf16 terms
// of z per 128-site tile and 64-wide t-block, [term][per 8 t: cosines,
// sines][row group][8 sites][8 t]); NS = 7 the z values in FP64 (zd).
template <int NS, int ND>
__global__ void __launch_bounds__(256)
k_qtab(int n, int ns, QGeom g, const int *__restrict__ slots, const double *__restrict__ site,
       const double *__restrict__ chg, double hi0, double hi1, double hi2, double hi3, double hi4, double hi5,
       double hi6, double hi7, double hi8, double qinv, typename QCfg<NS>::T *__restrict__ X,
       typename QCfg<NS>::T *__restrict__ Y, unsigned char *__restrict__ ztab, uint4 *__restrict__ zsite,
       double *__restrict__ zd, int *__restrict__ XW)
{
   typedef typename QCfg<NS>::T T;
   constexpr int RS = QCfg<NS>::RS;
   __shared__ unsigned long long su[3][32];
   __shared__ T sq[32];
   __shared__ T sz[64][33];   // [per 8 t: 8 cosines, 8 sines][site] of a 32-wide run of t
   const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, stage = blockIdx.x;
   if (w == 0) {
      const int i = stage * 32 + lane;
      unsigned long long ux = 0, uy = 0, uz = 0;
      double q = 0.0;
      const int si = i < n ? slots[i] : -1;   // (-1: filler before a framework's sites)
      if (si >= 0) {
         const double x = site[si], y = site[ns + si], z = site[2 * (size_t)ns + si];
         ux = q_fixed64(hi0 * x + hi1 * y + hi2 * z);
         uy = q_fixed64(hi3 * x + hi4 * y + hi5 * z);
         uz = q_fixed64(hi6 * x + hi7 * y + hi8 * z);
         q = chg[si] * qinv * Q_KAPPA;
      }
      su[0][lane] = ux;
      su[1][lane] = uy;
      su[2][lane] = uz;
      sq[lane] = NS == 3 ? (T)__double2int_rn(q * 2147483648.0)
                         : (T)qbalance((T)__double2ll_rn(q * 9223372036854775808.0));
   }
   __syncthreads();
   {
      const unsigned long long ux = su[0][lane], uy = su[1][lane];
      T *xb = X + (size_t)stage * 2 * g.hrows * RS + lane, *yb = Y + (size_t)stage * 2 * g.mrows * RS + lane;
      for (int r = w; r < g.hrows + g.mrows; r += 8) {
         const bool y = r >= g.hrows;
         const int k = y ? r - g.hrows : r;
         T s, c;
         qtrig(k, y ? uy : ux, s, c);
         if (ND == 4 && !y) {   // and in full for the four-digit structure factor
            int *d = XW + ((size_t)stage * 2 * g.hrows + 2 * k) * RS + lane;
            d[0] = c;
            d[RS] = s;
         }
         if (NS == 3 && !y) {   // X in units of 2^-24
            c = (c + 64) >> 7;
            s = (s + 64) >> 7;
         }
         T *d = (y ? yb : xb) + (size_t)2 * k * RS;
         d[0] = qbalance(c);
         d[RS] = qbalance(s);
      }
   }
   const unsigned long long uz = su[2][lane];
   for (int t0 = 0; t0 < g.TP; t0 += 32) {
      const int nt = min(32, g.TP - t0);   // a multiple of 8
      __syncthreads();
      for (int t = w; t < nt; t += 8) {
         T s, c;
         qtrig(t0 + t, uz, s, c);
         const int col = 16 * (t >> 3) + (t & 7);
         sz[col][lane] = qbalance(c);
         sz[col + 8][lane] = qbalance(s);
         if (NS == 7) {
            double *d = zd + ((size_t)stage * 2 * g.TP + 2 * t0 + col) * 32 + lane;
            d[0] = (double)c * (1.0 / (9223372036854775808.0 * Q_KAPPA));
            d[8 * 32] = (double)s * (1.0 / (9223372036854775808.0 * Q_KAPPA));
         }
      }
      __syncthreads();
      {
         // digits of q z: 8 sites (kg) of one column per thread
         const int kg = tid & 3, c8 = (tid >> 2) & 7, cg = tid >> 5;
         if (8 * cg < 2 * nt) {
            auto qz = [&](int e) { return qmul(sq[8 * kg + e], sz[8 * cg + c8][8 * kg + e]); };
            decltype(qz(0)) v[8];
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = qz(e);
            const int tcol = 2 * t0 + 8 * cg, b = tcol / (2 * g.TW), lc = tcol - 2 * b * g.TW;
            const int nT = q_blkcols(g, b);
            unsigned char *d = ztab + (size_t)stage * 2 * g.TP * Q_KS * 2 * ND + (size_t)2 * b * g.TW * Q_KS * 2 * ND +
                               (size_t)lc * Q_KS * 2 + kg * 128 + c8 * 16;
            qstore<ND>(d, nT * Q_KS * 2, v);
         }
      }
      if (NS == 3) {
         // force pass: 8 t of one site per thread, cosines or sines
         const int sl = tid & 31, cg = tid >> 5;
         if (8 * cg < 2 * nt) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = (float)sz[8 * cg + e][sl] * (float)(1.0 / (2147483648.0 * Q_KAPPA));
            unsigned int h[4], m[4], l[4];
#pragma unroll
            for (int j = 0; j < 4; j++) tc::split3(v[2 * j], v[2 * j + 1], h[j], m[j], l[j]);
            const int i = stage * 32 + sl, tile = i >> 7, r = i & 127;
            const int tcol = 2 * t0 + 8 * cg, fb = tcol / 128, fc = tcol - 128 * fb;   // 64-wide t-block of the force pass
            const int fcols = min(128, 2 * g.TP - 128 * fb);
            uint4 *d = zsite + ((size_t)tile * 2 * g.TP + 128 * fb) * 3 * 16 + (size_t)(fc >> 3) * 128 + (r >> 3) * 8 + (r & 7);
            const size_t ts = (size_t)fcols * 16;   // uint4 per term
            d[0] = make_uint4(h[0], h[1], h[2], h[3]);
            d[ts] = make_uint4(m[0], m[1], m[2], m[3]);
            d[2 * ts] = make_uint4(l[0], l[1], l[2], l[3]);
         }
      }
   }
}

// ------------------------------------------------------ shared CTA parts
__device__ __forceinline__ void q_abort(int *flag, int *err, int bit)
{
   *(volatile int *)flag = 1;
   atomicOr(err, bit);
}
__device__ __forceinline__ bool q_aborted(const int *flag) { return *(const volatile int *)flag != 0; }

struct QBars {
   uint64_t full_b[3], empty_b[3], full_t[4], full_a[2], empty_a[2], accf, acce, done[2];
};
__device__ __forceinline__ void q_init(QBars &B)
{
   for (int s = 0; s < 3; s++) {
      tc::bar_init(&B.full_b[s], 1);
      tc::bar_init(&B.empty_b[s], 2);   // released by both MMA issuers
   }
   for (int s = 0; s < 4; s++) tc::bar_init(&B.full_t[s], 1);
   for (int s = 0; s < 2; s++) {
      tc::bar_init(&B.full_a[s], Q_BW);
      tc::bar_init(&B.empty_a[s], 2);
   }
   tc::bar_init(&B.accf, 2);
   tc::bar_init(&B.acce, Q_BW);
   tc::bar_init(&B.done[0], 1);
   tc::bar_init(&B.done[1], 1);
   tc::bar_init_fence();
}

// MMA issue of one thread (issuer p of two) over nst stages in segments of
// SEG.  NS = 3: issuer p takes 128-row tile p, its groups in columns 256 p
// on.  NS = 7: issuer 0 adds to groups 0 .. 3, issuer 1 to groups 4 .. 6 (a
// thread issues an MMA about every 150 cycles whatever its width: 11 wide
// ones per K-step, 4 and 7, where halves of the columns took 14 narrow ones).
// Operand stages: A [tile][digit][row group 16][kg 4][8 rows][16 B], B
// [digit][col group][kg 4][8][16 B].
template <int NS, int ND, int NA, int NB>
__device__ __forceinline__ void q_issue(QBars &B, unsigned char *Abuf, unsigned char *Bbuf, unsigned int tmem, int p,
                                        int nst, int nT, int *abort_s, int *err, int errbit)
{
   using namespace tc;
   constexpr int SEG = QCfg<NS>::SEG;
   const unsigned int a0 = saddr(Abuf) + (QCfg<NS>::MT == 2 ? p * NA * Q_OP : 0), b0 = saddr(Bbuf);
   const unsigned int d0 = tmem + (QCfg<NS>::MT == 2 ? 256u * p : 0u);
   const int g0 = NS == 7 && p == 1 ? 4 : 0, g1 = NS == 7 && p == 0 ? 4 : ND;   // this issuer's groups
   for (int st = 0; st < nst; st++) {
      const int sa = st & 1, sb = st % NB, seg = st / SEG;
      if (!bar_wait(&B.full_a[sa], (unsigned int)(st >> 1) & 1u) ||
          !bar_wait(&B.full_b[sb], (unsigned int)(st / NB) & 1u) ||
          (st % SEG == 0 && seg > 0 && !bar_wait(&B.acce, (unsigned int)(seg - 1) & 1u)) || q_aborted(abort_s)) {
         q_abort(abort_s, err, errbit);
         break;
      }
      fence_after_sync();
#pragma unroll
      for (int ks = 0; ks < 2; ks++)
#pragma unroll
         for (int i = 0; i < NA; i++) {
            const int ga = max(i, g0);   // first group of digit i of A
            if (ga < g1)
               mma_f16(d0 + ga * nT, sdesc(a0 + sa * Q_A<NS, NA> + i * Q_OP + ks * 256, 128, 512),
                       sdesc(b0 + sb * Q_B<ND> + (ga - i) * nT * Q_KS * 2 + ks * 256, 128, 512),
                       idesc_f16(128, (g1 - ga) * nT, false), st % SEG != 0 || ks > 0 || i > 0);
         }
      mma_commit(&B.empty_a[sa]);
      mma_commit(&B.empty_b[sb]);
      if (st % SEG == SEG - 1 || st == nst - 1) mma_commit(&B.accf);
   }
   mma_commit(&B.done[p]);
   bar_wait(&B.done[p], 0);   // every MMA complete before the tensor memory is released
}

// 4 consecutive FP32 columns of this thread's lane of tensor memory
__device__ __forceinline__ void q_ld4(unsigned int taddr, float (&v)[4])
{
   asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                : "r"(taddr)
                : "memory");
}
template <int N> __device__ __forceinline__ void q_ldwait(float (&v)[N][4])
{
   asm volatile("tcgen05.wait::ld.sync.aligned;" : : : "memory");
#pragma unroll
   for (int i = 0; i < N; i++) asm volatile("" : "+f"(v[i][0]), "+f"(v[i][1]), "+f"(v[i][2]), "+f"(v[i][3]));
}

// 96-bit signed sums (three words)
struct Q96 {
   unsigned int w0, w1, w2;
};
// the seven groups of one output as an integer, group 6 of weight 1: low
// part (groups 3..6) and high part (groups 0..2, weight 2^32)
__device__ __forceinline__ Q96 q_combine(float d0, float d1, float d2, float d3, float d4, float d5, float d6)
{
   const long long lo = (long long)__float2int_rn(d6) + (long long)__float2int_rn(d5) * 256 +
                        (long long)__float2int_rn(d4) * 65536 + (long long)__float2int_rn(d3) * 16777216;
   const long long hi = (long long)__float2int_rn(d2) + (long long)__float2int_rn(d1) * 256 +
                        (long long)__float2int_rn(d0) * 65536;
   Q96 r;
   const unsigned int sx = (unsigned int)(lo >> 63);
   asm("add.cc.u32 %0, %3, %4;\n\taddc.u32 %1, %5, %6;\n\tmov.u32 %2, %7;"
       : "=&r"(r.w1), "=&r"(r.w2), "=&r"(r.w0)
       : "r"((unsigned int)(lo >> 32)), "r"((unsigned int)hi), "r"(sx), "r"((unsigned int)(hi >> 32)),
         "r"((unsigned int)lo));
   return r;
}
__device__ __forceinline__ void q_add(Q96 &a, const Q96 &b)
{
   asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
       : "+r"(a.w0), "+r"(a.w1), "+r"(a.w2)
       : "r"(b.w0), "r"(b.w1), "r"(b.w2));
}
__device__ __forceinline__ Q96 q_shift(Q96 v, int s)   // arithmetic shift right, 0 <= s < 96
{
   while (s >= 32) {
      v.w0 = v.w1;
      v.w1 = v.w2;
      v.w2 = (unsigned int)((int)v.w2 >> 31);
      s -= 32;
   }
   v.w0 = __funnelshift_r(v.w0, v.w1, s);
   v.w1 = __funnelshift_r(v.w1, v.w2, s);
   v.w2 = (unsigned int)((int)v.w2 >> s);
   return v;
}
__device__ __forceinline__ double q_value(const Q96 &v)
{
   return (double)(long long)(((unsigned long long)v.w2 << 32) | v.w1) * 4294967296.0 + (double)v.w0;
}

// ----------------------------------------------------- structure factor
// Grid: (row tiles, site ranges, channels).  The first r0 ranges share stages
// 0 .. n0 - 1, the others those from s1 to nstages - 1 (a framework's).  part[channel][range][quad row 4
// quad + p][2 TP]; channel c reads its own digits, zstride further on each.
// NA = 4 (mixed form with a framework molecule, or charges of very different
// size): 32-bit operands.  The energy
// and stress there are differences of the framework's large and the other
// sites' small sums, and charges of any ratio share the digits' grid: with
// three digits the stress of a clay (500 sites) was 1.5e-5 off, with FP32
// sums over the sites 2.1e-6.
template <int NS, int ND, int NA>
__global__ void __launch_bounds__(Q_THREADS, 1)
k_sfac_q(QGeom g, unsigned int c256, const QTile *__restrict__ tiles, const int4 *__restrict__ units, const unsigned char *__restrict__ X,
         const unsigned char *__restrict__ Y, const unsigned char *__restrict__ ztab, size_t zstride, int r0, int n0, int s1, int nstages, int per,
         typename QCfg<NS>::P *__restrict__ part, int *__restrict__ err)
{
   using namespace tc;
   typedef typename QCfg<NS>::T T;
   constexpr int RS = QCfg<NS>::RS, MT = QCfg<NS>::MT, NB = QCfg<NS>::NB, NTB = NB + 1, SEG = QCfg<NS>::SEG;
   extern __shared__ __align__(1024) unsigned char sm[];
   __shared__ __align__(8) QBars B;
   __shared__ unsigned int tmem_s;
   __shared__ int abort_s;
   unsigned char *Abuf = sm, *Sbuf = sm + 2 * Q_A<NS, NA>, *Tbuf = Sbuf + NB * Q_B<ND>;
   const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
   const QTile &ti = tiles[blockIdx.x];
   const bool fw = (int)blockIdx.y >= r0;
   const int nT = ti.nT, st0 = fw ? s1 + ((int)blockIdx.y - r0) * per : blockIdx.y * per;
   const int nst = min(fw ? nstages : n0, st0 + per) - st0;
   if (nst <= 0) return;   // (uniform)
   if (tid == 0) {
      q_init(B);
      abort_s = 0;
   }
   __syncwarp();
   if (w == Q_BW + 1) tmem_alloc(&tmem_s, 512);
   fence_before_sync();
   __syncthreads();
   fence_after_sync();
   const unsigned int tmem = tmem_s;

   if (w == Q_BW) {
      // ---- bulk copies: a stage's digits of q z, and the tile's table rows
      // a stage ahead of them (the operand is built from them before its
      // MMAs; the rows of stage st - NB were read before its MMAs, so the
      // wait for those frees them too)
      if (lane == 0) {
         const unsigned int bb = (unsigned int)(nT * Q_KS * 2 * ND);
         const unsigned int xb = (unsigned int)(2 * ti.nx * RS * sizeof(T)), yb = (unsigned int)(2 * ti.ny * RS * sizeof(T));
         auto table = [&](int st) {
            unsigned char *d = Tbuf + (st % NTB) * Q_TAB<NS>;
            const size_t sg = (size_t)(st0 + st);
            bar_expect_tx(&B.full_t[st % NTB], xb + yb);
            bulk_load(d, X + (sg * g.hrows + ti.xlo) * 2 * RS * sizeof(T), xb, &B.full_t[st % NTB]);
            bulk_load(d + 2 * Q_XMAX * RS * sizeof(T), Y + (sg * g.mrows + ti.ylo) * 2 * RS * sizeof(T), yb,
                      &B.full_t[st % NTB]);
         };
         int issued = 0, tabs = 1;
         table(0);
         for (int st = 0; st < nst; st++) {
            const int s = st % NB;
            if ((st >= NB && !bar_wait(&B.empty_b[s], (unsigned int)(st / NB - 1) & 1u)) || q_aborted(&abort_s)) {
               q_abort(&abort_s, err, Q_ERR);
               break;
            }
            bar_expect_tx(&B.full_b[s], bb);
            bulk_load(Sbuf + s * Q_B<ND>, ztab + blockIdx.z * zstride + ((size_t)(st0 + st) * 2 * g.TP + ti.col0) * Q_KS * 2 * ND,
                      bb, &B.full_b[s]);
            issued = st + 1;
            if (tabs < nst) table(tabs++);
         }
         // copies still in flight complete before the CTA's shared memory goes
         for (int st = issued > NB ? issued - NB : 0; st < issued; st++)
            bar_wait(&B.full_b[st % NB], (unsigned int)(st / NB) & 1u);
         for (int st = tabs > NTB ? tabs - NTB : 0; st < tabs; st++)
            bar_wait(&B.full_t[st % NTB], (unsigned int)(st / NTB) & 1u);
      }
   } else if (w > Q_BW) {
      if (lane == 0)
         q_issue<NS, ND, NA, NB>(B, Abuf, Sbuf, tmem, w - Q_BW - 1, nst, nT, &abort_s, err, Q_ERR);
   } else {
      // ---- A operand: row 8 w + (lane & 7) of each 128-row tile (product
      // p of a quad), sites 8 kg .. 8 kg + 7 of the stage
      const int r = 8 * w + (lane & 7), kg = lane >> 3, p = r & 3;
      int xo[MT], yo[MT];   // this row's table offsets
#pragma unroll
      for (int mt = 0; mt < MT; mt++) {
         const int u = ti.unit[8 * mt + (r >> 4)];
         const int4 un = u >= 0 ? units[u] : make_int4(ti.xlo, ti.ylo, 0, 0);
         const int hx = un.x - ti.xlo, my = un.y + (u >= 0 ? (r >> 2) & 3 : 0) - ti.ylo;
         xo[mt] = (2 * hx + (p == 1 || p == 2)) * RS + 8 * kg;
         yo[mt] = (2 * my + (p & 1)) * RS + 8 * kg;
      }
      // read-back: lane quarter w % 4 (row 32 (w % 4) + lane), a quarter of
      // the columns of each tile / part
      const int cq = w >> 2;
      const int ncw = nT >> 2;                    // columns per warp
      constexpr int MAXC = QCfg<NS>::NTMAX / 16;  // chunks of four columns
      constexpr int NACC = MT * MAXC * 4;
      float af[NS == 3 ? NACC : 1];
      Q96 ai[NS == 7 ? NACC : 1];
#pragma unroll
      for (int i = 0; i < NACC; i++) {
         if (NS == 3) af[NS == 3 ? i : 0] = 0.f;
         else ai[NS == 7 ? i : 0] = Q96{0u, 0u, 0u};
      }
      const unsigned int trow = tmem + ((unsigned int)(32 * (w & 3)) << 16);
      // first column of this warp in tensor memory and the group stride
      const int pl = cq * ncw;
      auto flush = [&](int seg) -> bool {
         const bool got = bar_wait(&B.accf, (unsigned int)seg & 1u);
         if (!__all_sync(0xffffffffu, got && !q_aborted(&abort_s))) {
            if (lane == 0) q_abort(&abort_s, err, Q_ERR);
            return false;
         }
         fence_after_sync();
#pragma unroll
         for (int mt = 0; mt < MT; mt++)
#pragma unroll
            for (int ch = 0; ch < MAXC; ch++)
               if (4 * ch < ncw) {
                  const int lc = pl + 4 * ch;   // column of the block
                  const unsigned int col = 256u * mt + lc;
                  float d[ND][4];
#pragma unroll
                  for (int k = 0; k < ND; k++) q_ld4(trow + col + k * nT, d[k]);
                  q_ldwait(d);
#pragma unroll
                  for (int e = 0; e < 4; e++) {
                     const int i = (mt * MAXC + ch) * 4 + e;
                     if (NS == 3) {
                        const float lo = ND == 3 ? d[2][e] : fmaf(d[2][e], 256.f, d[ND - 1][e]);
                        af[NS == 3 ? i : 0] += fmaf(d[0][e], ND == 3 ? 65536.f : 16777216.f, fmaf(d[1][e], ND == 3 ? 256.f : 65536.f, lo));
                     } else
                        q_add(ai[NS == 7 ? i : 0], q_combine(d[0][e], d[1][e], d[2][e], d[ND > 4 ? 3 : 0][e], d[ND > 4 ? 4 : 0][e],
                                                            d[ND > 4 ? 5 : 0][e], d[ND > 4 ? 6 : 0][e]));
                  }
               }
         fence_before_sync();
         __syncwarp();
         if (lane == 0) bar_arrive(&B.acce);
         return true;
      };
      bool live = true;
      for (int st = 0; st < nst && live; st++) {
         const int sa = st & 1, sb = st % NTB;
         const bool got = (st < 2 || bar_wait(&B.empty_a[sa], (unsigned int)((st >> 1) - 1) & 1u)) &&
                          bar_wait(&B.full_t[sb], (unsigned int)(st / NTB) & 1u);
         if (!__all_sync(0xffffffffu, got && !q_aborted(&abort_s))) {
            if (lane == 0) q_abort(&abort_s, err, Q_ERR);
            live = false;
            break;
         }
         const T *xs = reinterpret_cast<const T *>(Tbuf + sb * Q_TAB<NS>);
         const T *ys = xs + 2 * Q_XMAX * RS;
         unsigned char *A = Abuf + sa * Q_A<NS, NA> + (r >> 3) * 512 + kg * 128 + (r & 7) * 16;
#pragma unroll
         for (int mt = 0; mt < MT; mt++) {
            constexpr int PV = 16 / (int)sizeof(T);   // values per 16-byte load
            T xv[8], yv[8];
#pragma unroll
            for (int e = 0; e < 8 / PV; e++) {
               *reinterpret_cast<uint4 *>(xv + e * PV) = *reinterpret_cast<const uint4 *>(xs + xo[mt] + e * PV);
               *reinterpret_cast<uint4 *>(yv + e * PV) = *reinterpret_cast<const uint4 *>(ys + yo[mt] + e * PV);
            }
            auto mul = [&](int e) {
               if constexpr (NA == 4) return qmul(xv[e], yv[e]);
               else return qmul_a(xv[e], yv[e], c256);
            };
            decltype(mul(0)) v[8];
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = mul(e);
            qstore<NA>(A + mt * NA * Q_OP, Q_OP, v);
         }
         fence_async_smem();
         __syncwarp();
         if (lane == 0) bar_arrive(&B.full_a[sa]);
         // the previous segment is read back once the first stage of this
         // one is built (its build overlaps the segment's last MMAs)
         if (st > 0 && st % SEG == 0) live = flush(st / SEG - 1);
      }
      if (live) live = flush((nst - 1) / SEG);
      if (live) {
#pragma unroll
         for (int mt = 0; mt < MT; mt++) {
            const int row = 32 * (w & 3) + lane;
            const int u = ti.unit[8 * mt + (row >> 4)];
            if (u >= 0) {
               typename QCfg<NS>::P *dst =
                  part + (((size_t)blockIdx.z * gridDim.y + blockIdx.y) * 4 * g.nquads + (size_t)u * 16 + (row & 15)) * 2 * g.TP +
                  ti.col0 + pl;
#pragma unroll
               for (int ch = 0; ch < MAXC; ch++)
                  if (4 * ch < ncw) {
                     const int i = (mt * MAXC + ch) * 4;
                     if constexpr (NS == 3) {
                        *reinterpret_cast<float4 *>(dst + 4 * ch) = make_float4(af[i], af[i + 1], af[i + 2], af[i + 3]);
                     } else {
                        reinterpret_cast<double2 *>(dst + 4 * ch)[0] = make_double2(q_value(ai[i]), q_value(ai[i + 1]));
                        reinterpret_cast<double2 *>(dst + 4 * ch)[1] = make_double2(q_value(ai[i + 2]), q_value(ai[i + 3]));
                     }
                  }
            }
         }
      }
   }
   fence_before_sync();
   __syncthreads();
   if (w == Q_BW + 1) {
      __syncwarp();
      fence_after_sync();
      tmem_dealloc(tmem, 512);
   }
}

// ------------------------------------------------- per-k energy and stress
// Sum of nr values a plane apart: FP32 partials compensated (an FP64 add or
// conversion per partial would bound the per-k pass), FP64 ones plainly.
// Sixteen loads in flight: the latency of the loads is what a small system's
// sum takes (48 ranges at 2048 sites).
template <typename R, typename F> __device__ __forceinline__ void q_ranges(const R *p, size_t plane, int nr, F &&add)
{
   int k = 0;
   for (; k + 16 <= nr; k += 16) {
      R v[16];
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] = __ldg(p + (k + j) * plane);
#pragma unroll
      for (int j = 0; j < 16; j++) add(v[j]);
   }
   R v[15];
#pragma unroll
   for (int j = 0; j < 15; j++) v[j] = k + j < nr ? __ldg(p + (k + j) * plane) : R(0);
#pragma unroll
   for (int j = 0; j < 15; j++)
      if (k + j < nr) add(v[j]);
}
__device__ __forceinline__ double q_rangesum(const float *p, size_t plane, int nr)
{
   float s = 0.f, c = 0.f;
   q_ranges(p, plane, nr, [&](float v) {
      const float y = v - c, t = s + y;
      c = (t - s) - y;
      s = t;
   });
   return (double)s - (double)c;
}
__device__ __forceinline__ double q_rangesum(const double *p, size_t plane, int nr)
{
   double s = 0.0;
   q_ranges(p, plane, nr, [&](double v) { s += v; });
   return s;
}

// Energy and stress come from seven sums over the k-vectors, of the energy e
// and of e c2 times the products of the integers (h, k, l) (the last block
// brings those to Cartesian axes): FP64 instructions, 16 cycles each for a
// warp, and their latency bound this kernel.
// A block takes 32 consecutive (quad, t) at a time (all its groups in one
// reduction, a warp per sum; 2048-site water 23 us with shuffles of seven
// sums in four warps and four loads in flight, 10.7 us so): warp
// k adds up sum k of each over the site ranges, then one thread per
// (quad, t) and (s, r) forms its k-vector's S(k), energy and stress
// (src/ewald.c:525-553) and A = coeff Re S, B = coeff Im S, laid out
// [quad][t][s][r] (zero where there is no such k-vector).
// FW: with a framework molecule, whose sums are in the nrf ranges after the
// others, framework-framework terms are left out (src/ewald.c:528-579): the
// energy is 1/2 coeff (Cn (Cn + 2 Cf) + Sn (Sn + 2 Sf)), the framework sites
// feel the others' sums alone (abf).
template <typename R, bool FW>
__global__ void __launch_bounds__(256)
k_qreduce(QGeom g, const int4 *__restrict__ units, const double2 *__restrict__ coeff, int nranges, double scale,
          const R *__restrict__ part, int nrf, R *__restrict__ ab, R *__restrict__ abf, double *__restrict__ blk,
          unsigned int *__restrict__ sync, DevOut *__restrict__ out)
{
   __shared__ double sq[FW ? 16 : 8][32];
   __shared__ double se[7][128], sl[8];
   const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
   double e[7] = {0, 0, 0, 0, 0, 0, 0};
   for (int grp = blockIdx.x; grp * 32 < g.nquads * g.TP; grp += gridDim.x) {
   const int i = grp * 32 + lane, quad = i / g.TP, t = i - quad * g.TP;
   const int4 un = quad < g.nquads ? units[quad >> 2] : make_int4(0, 0, 0, 0);
   const bool live = t < un.z;   // the unit's t range: its columns were computed
   {
      const size_t row = 2 * (size_t)g.TP;
      const size_t plane = 4 * (size_t)g.nquads * row;
      const R *src = part + ((size_t)quad * 4 + (w >> 1)) * row + 16 * (t >> 3) + 8 * (w & 1) + (t & 7);
      sq[w][lane] = live ? scale * q_rangesum(src, plane, nranges) : 0.0;
      if (FW) sq[(FW ? 8 : 0) + w][lane] = live ? scale * q_rangesum(src + nranges * plane, plane, nrf) : 0.0;
   }
   __syncthreads();
   // (s, r) = warp w of the first four
   if (w < 4 && quad < g.nquads) {
      double A = 0.0, Bc = 0.0, An = 0.0, Bn = 0.0;
      const double2 cf = live ? coeff[(size_t)i * 4 + w] : make_double2(0.0, 0.0);
      if (cf.x != 0.0) {
         double q[8];
#pragma unroll
         for (int k = 0; k < 8; k++) q[k] = sq[k][lane];
         const double s = w & 2 ? -1.0 : 1.0, r = w & 1 ? -1.0 : 1.0;
         const double C = (q[0] - s * q[2]) - r * (q[5] + s * q[7]);
         const double S = (q[4] + s * q[6]) + r * (q[1] - s * q[3]);
         const double hh = un.x, kk = s * (un.y + (quad & 3)), l = r * t;
         double Cf = 0.0, Sf = 0.0;
         if (FW) {
#pragma unroll
            for (int k = 0; k < 8; k++) q[k] = sq[(FW ? 8 : 0) + k][lane];
            Cf = (q[0] - s * q[2]) - r * (q[5] + s * q[7]);
            Sf = (q[4] + s * q[6]) + r * (q[1] - s * q[3]);
         }
         const double pek = 0.5 * cf.x * (FW ? C * (C + Cf + Cf) + S * (S + Sf + Sf) : C * C + S * S), pc = pek * cf.y;
         const double ph = pc * hh, pk = pc * kk, pl = pc * l;
         e[0] += pek;
         e[1] = fma(ph, hh, e[1]);
         e[2] = fma(ph, kk, e[2]);
         e[3] = fma(ph, l, e[3]);
         e[4] = fma(pk, kk, e[4]);
         e[5] = fma(pk, l, e[5]);
         e[6] = fma(pl, l, e[6]);
         An = cf.x * C;
         Bn = cf.x * S;
         A = FW ? cf.x * (C + Cf) : An;
         Bc = FW ? cf.x * (S + Sf) : Bn;
      }
      ab[(size_t)i * 8 + 2 * w] = (R)A;
      ab[(size_t)i * 8 + 2 * w + 1] = (R)Bc;
      if (FW) {
         abf[(size_t)i * 8 + 2 * w] = (R)An;
         abf[(size_t)i * 8 + 2 * w + 1] = (R)Bn;
      }
   }
   __syncthreads();
   }
   if (w < 4)
#pragma unroll
      for (int k = 0; k < 7; k++) se[k][threadIdx.x] = e[k];
   __syncthreads();
   if (w < 7) {
      double v = (se[w][lane] + se[w][lane + 32]) + (se[w][lane + 64] + se[w][lane + 96]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) blk[blockIdx.x * 8 + w] = v;
   }
   // the blocks' sums by the last block, a warp per sum
   if (!last_block(&sync[SYNC_KRED])) return;
   if (w < 7) {
      double v = 0.0;
      for (int b = lane; b < (int)gridDim.x; b += 32) v += __ldcg(&blk[b * 8 + w]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) sl[w] = v;
   }
   __syncthreads();
   if (threadIdx.x < 7) {
      // stress (x, y) = delta e - sum over axes of b[axis][x] b[axis'][y] times the products' sums
      const int k = threadIdx.x, x = k < 4 ? 0 : k < 6 ? 1 : 2, y = k < 4 ? k - 1 : k < 6 ? k - 3 : 2;
      if (k == 0) {
         out->pe_k = sl[0];
      } else {
         const double m[9] = {sl[1], sl[2], sl[3], sl[2], sl[4], sl[5], sl[3], sl[5], sl[6]};
         double v = x == y ? sl[0] : 0.0;
         for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) v -= g.b[3 * i + x] * g.b[3 * j + y] * m[3 * i + j];
         out->st_k[k - 1] = v;
      }
   }
}

// ------------------------------------------------- force pass, FP64 form
// F_j = q_j sum_k k (A sin k.r_j - B cos k.r_j) as three sums over the quad
// rows with the integer weights h, k, l:
//     H_a(j) = sum_col z_col(j) sum_rows P_row(j) U_a(row, col),
// the inner sum a matrix product (sites x quad rows, built per stage from
// the tables, times quad rows x columns), F = q b^T (H_h, H_k, H_l).
// A segment is 8 units (128 quad rows) of one t-block, units in order of
// rising |(h, m)| so that the coefficients of a segment, which share a
// power-of-two scale, are of similar size.
// Coefficients of quad (h, m) at t for one weight set (h, k, l, or 1): v[p] of P_p C_t and
// v[4 + p] of P_p S_t.
__device__ __forceinline__ void q_coefs(const double *ab, int set, int h, int m, int t, double (&v)[8])
{
#pragma unroll
   for (int k = 0; k < 8; k++) v[k] = 0.0;
#pragma unroll
   for (int x = 0; x < 4; x++) {
      const double s = x & 2 ? -1.0 : 1.0, r = x & 1 ? -1.0 : 1.0;
      const double wt = set == 0 ? (double)h : set == 1 ? s * m : set == 2 ? r * t : 1.0;
      const double A = wt * ab[2 * x], Bc = wt * ab[2 * x + 1];
      v[0] -= Bc;
      v[1] += s * Bc;
      v[2] += A;
      v[3] += s * A;
      v[4] += r * A;
      v[5] -= r * s * A;
      v[6] += r * Bc;
      v[7] += r * s * Bc;
   }
}

// Grid: (segments, sets from set0).  The segment's B operand, [stage 4][digit]
// [col group][kg 4][8 cols][8 K], and its scale exponent.  Digits hold no NaN
// or infinity: where a coefficient is one, the exponent says so, and the force
// pass hands NaN on.
__global__ void __launch_bounds__(256)
k_qcoef(QGeom g, int set0, const QSeg *__restrict__ segs, int nseg, const int4 *__restrict__ units,
        const double *__restrict__ ab, unsigned char *__restrict__ bq, int *__restrict__ bexp)
{
   constexpr int NS = 7;
   __shared__ long long smax[8];
   const int seg = blockIdx.x, set = blockIdx.y, tid = threadIdx.x;
   const QSeg &sg = segs[seg];
   const int nT = q_blkcols(g, sg.blk), tw = nT / 2, t0 = sg.blk * g.TW;
   long long mb = 0;   // the largest magnitude's bits (infinity and NaN are the largest)
   for (int i = tid; i < 32 * tw; i += 256) {
      const int ql = i / tw, t = t0 + i % tw, u = sg.unit[ql >> 2];
      if (u < 0) continue;
      const int4 un = units[u];
      if (t >= un.z) continue;
      double v[8];
      q_coefs(ab + ((size_t)(4 * u + (ql & 3)) * g.TP + t) * 8, set0 + set, un.x, un.y + (ql & 3), t, v);
#pragma unroll
      for (int k = 0; k < 8; k++) mb = max(mb, __double_as_longlong(fabs(v[k])));
   }
#pragma unroll
   for (int o = 16; o > 0; o >>= 1) mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, o));
   if ((tid & 31) == 0) smax[tid >> 5] = mb;
   __syncthreads();
   mb = smax[0];
   for (int k = 1; k < 8; k++) mb = max(mb, smax[k]);
   double mx = __longlong_as_double(mb);
   int e = -4096;
   if (mb >= 0x7ff0000000000000ll) {
      e = Q_NOT_FINITE;
      mx = 0.0;
   }
   if (mx > 0.0) frexp(mx, &e);
   if (tid == 0) bexp[set * nseg + seg] = e;
   const double sc = mx > 0.0 ? ldexp(Q_KAPPA * Q_KAPPA, 63 - e) : 0.0;
   unsigned char *base = bq + ((size_t)set * nseg + seg) * 4 * (QCfg<NS>::NTMAX * Q_KS * 2 * NS);
   // two quads (8 K values) at one t per thread
   for (int i = tid; i < 16 * tw; i += 256) {
      const int pr = i & 15, tl = i >> 4, t = t0 + tl;
      unsigned long long vc[8], vs[8];
#pragma unroll
      for (int x = 0; x < 2; x++) {
         const int ql = 2 * pr + x, u = sg.unit[ql >> 2];
         double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
         if (u >= 0) {
            const int4 un = units[u];
            if (t < un.z) q_coefs(ab + ((size_t)(4 * u + (ql & 3)) * g.TP + t) * 8, set0 + set, un.x, un.y + (ql & 3), t, v);
         }
#pragma unroll
         for (int k = 0; k < 4; k++) {
            vc[4 * x + k] = (unsigned long long)__double2ll_rn(v[k] * sc) + 0x8080808080808080ull;
            vs[4 * x + k] = (unsigned long long)__double2ll_rn(v[4 + k] * sc) + 0x8080808080808080ull;
         }
      }
      const int stage = pr >> 2, kg = pr & 3, lc = 16 * (tl >> 3) + (tl & 7);
#pragma unroll
      for (int cs = 0; cs < 2; cs++) {
         const int col = lc + 8 * cs;
         unsigned char *d = base + (size_t)stage * (QCfg<NS>::NTMAX * Q_KS * 2 * NS) +
                            (size_t)(col & ~7) * Q_KS * 2 + kg * 128 + (col & 7) * 16;
         if (cs == 0) qstore<NS>(d, nT * Q_KS * 2, vc);
         else qstore<NS>(d, nT * Q_KS * 2, vs);
      }
   }
}

// Grid: (site tiles of 128, sets, runs of up to per segments of one t-block).
// hpart[run][set][n].  The run is found from the t-blocks' first segments
// (seg0) here: a list of runs kept on the device would be another call's by
// the time a captured evaluation is replayed.
__global__ void __launch_bounds__(Q_THREADS, 1)
k_force_q(QGeom g, const QSeg *__restrict__ segs, int nseg, const int *__restrict__ seg0, int per,
          const int4 *__restrict__ units, const long long *__restrict__ X, const long long *__restrict__ Y,
          const double *__restrict__ zd, const unsigned char *__restrict__ bq, const int *__restrict__ bexp, int n,
          double *__restrict__ hpart, int *__restrict__ err)
{
   using namespace tc;
   constexpr int NS = 7, RS = QCfg<NS>::RS, NB = Q_FNB, SEG = QCfg<NS>::SEG;
   constexpr int BST = QCfg<NS>::NTMAX * Q_KS * 2 * NS;   // a stage's B operand
   extern __shared__ __align__(1024) unsigned char sm[];
   __shared__ __align__(8) QBars B;
   __shared__ unsigned int tmem_s;
   __shared__ int abort_s;
   __shared__ double red[4][128];
   unsigned char *Abuf = sm, *Sbuf = sm + 2 * Q_A<NS>;
   const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
   const int tile = blockIdx.x, set = blockIdx.y;
   __shared__ int s_run[3];   // first segment, segments, t-block
   if (tid == 0) {
      int b = 0, run = blockIdx.z;
      for (; b < g.nblk - 1; b++) {
         const int nr = (seg0[b + 1] - seg0[b] + per - 1) / per;
         if (run < nr) break;
         run -= nr;
      }
      s_run[0] = seg0[b] + run * per;
      s_run[1] = min(per, seg0[b + 1] - s_run[0]);
      s_run[2] = b;
      q_init(B);
      abort_s = 0;
   }
   __syncwarp();
   if (w == Q_BW + 1) tmem_alloc(&tmem_s, 512);
   fence_before_sync();
   __syncthreads();
   fence_after_sync();
   const unsigned int tmem = tmem_s;
   const int sg0 = s_run[0], nst = s_run[1] * SEG, blk = s_run[2], nT = q_blkcols(g, blk);

   if (w == Q_BW) {
      if (lane == 0) {
         const unsigned int bb = (unsigned int)(nT * Q_KS * 2 * NS);
         const unsigned char *src = bq + ((size_t)set * nseg + sg0) * SEG * BST;
         int issued = 0;
         for (int st = 0; st < nst; st++) {
            const int s = st % NB;
            if ((st >= NB && !bar_wait(&B.empty_b[s], (unsigned int)(st / NB - 1) & 1u)) || q_aborted(&abort_s)) {
               q_abort(&abort_s, err, Q_FERR);
               break;
            }
            bar_expect_tx(&B.full_b[s], bb);
            bulk_load(Sbuf + s * Q_B<NS>, src + (size_t)st * BST, bb, &B.full_b[s]);
            issued = st + 1;
         }
         for (int st = issued > NB ? issued - NB : 0; st < issued; st++)
            bar_wait(&B.full_b[st % NB], (unsigned int)(st / NB) & 1u);
      }
   } else if (w > Q_BW) {
      if (lane == 0)
         q_issue<NS, NS, NS, NB>(B, Abuf, Sbuf, tmem, w - Q_BW - 1, nst, nT, &abort_s, err, Q_FERR);
   } else {
      // ---- A operand: site j of the tile, two quads (8 K) per stage
      const int j = tid & 127, kg = tid >> 7;
      const size_t sg = (size_t)tile * 4 + (j >> 5);
      const long long *xb = X + sg * 2 * g.hrows * RS + (j & 31), *yb = Y + sg * 2 * g.mrows * RS + (j & 31);
      unsigned char *Aw = Abuf + (j >> 3) * 512 + kg * 128 + (j & 7) * 16;
      int emax = -4096;
      for (int k = lane; k < nseg; k += 32) emax = max(emax, bexp[set * nseg + k]);
      emax = __reduce_max_sync(0xffffffffu, emax);
      constexpr int MAXC = QCfg<NS>::NTMAX / 16;
      Q96 ai[MAXC * 4];
#pragma unroll
      for (int i = 0; i < MAXC * 4; i++) ai[i] = Q96{0u, 0u, 0u};
      const unsigned int trow = tmem + ((unsigned int)(32 * (w & 3)) << 16);
      const int cq = w >> 2, ncw = nT >> 2, pl = cq * ncw;
      auto flush = [&](int seg) -> bool {
         const bool got = bar_wait(&B.accf, (unsigned int)seg & 1u);
         if (!__all_sync(0xffffffffu, got && !q_aborted(&abort_s))) {
            if (lane == 0) q_abort(&abort_s, err, Q_FERR);
            return false;
         }
         fence_after_sync();
         const int sh = emax - bexp[set * nseg + sg0 + seg];
#pragma unroll
         for (int ch = 0; ch < MAXC; ch++)
            if (4 * ch < ncw) {
               const unsigned int col = pl + 4 * ch;
               float d[NS][4];
#pragma unroll
               for (int k = 0; k < NS; k++) q_ld4(trow + col + k * nT, d[k]);
               q_ldwait(d);
               if (sh < 96)
#pragma unroll
                  for (int e = 0; e < 4; e++)
                     q_add(ai[4 * ch + e],
                           q_shift(q_combine(d[0][e], d[1][e], d[2][e], d[3][e], d[4][e], d[5][e], d[6][e]), sh));
            }
         fence_before_sync();
         __syncwarp();
         if (lane == 0) bar_arrive(&B.acce);
         return true;
      };
      // a stage's table values are fetched a stage ahead, its unit two stages
      long long xv[2], yv[4];
      auto unit = [&](int st) {
         const int u = segs[sg0 + st / SEG].unit[2 * (st % SEG) + (kg >> 1)];
         return u >= 0 ? *reinterpret_cast<const int2 *>(units + u) : make_int2(0, 0);
      };
      auto fetch = [&](int2 un) {
         const long long *x = xb + (size_t)2 * un.x * RS, *y = yb + (size_t)2 * (un.y + 2 * (kg & 1)) * RS;
         xv[0] = __ldg(x);
         xv[1] = __ldg(x + RS);
#pragma unroll
         for (int k = 0; k < 4; k++) yv[k] = __ldg(y + k * RS);
      };
      fetch(unit(0));
      int2 next = unit(min(1, nst - 1));
      bool live = true;
      for (int st = 0; st < nst && live; st++) {
         const int sa = st & 1;
         unsigned long long v[8];
#pragma unroll
         for (int x = 0; x < 2; x++) {
            v[4 * x] = qmul(xv[0], yv[2 * x]);
            v[4 * x + 1] = qmul(xv[1], yv[2 * x + 1]);
            v[4 * x + 2] = qmul(xv[1], yv[2 * x]);
            v[4 * x + 3] = qmul(xv[0], yv[2 * x + 1]);
         }
         if (st + 1 < nst) {
            fetch(next);
            next = unit(min(st + 2, nst - 1));
         }
         const bool got = st < 2 || bar_wait(&B.empty_a[sa], (unsigned int)((st >> 1) - 1) & 1u);
         if (!__all_sync(0xffffffffu, got && !q_aborted(&abort_s))) {
            if (lane == 0) q_abort(&abort_s, err, Q_FERR);
            live = false;
            break;
         }
         qstore<NS>(Aw + sa * Q_A<NS>, Q_OP, v);
         fence_async_smem();
         __syncwarp();
         if (lane == 0) bar_arrive(&B.full_a[sa]);
         if (st > 0 && st % SEG == 0) live = flush(st / SEG - 1);
      }
      if (live) live = flush((nst - 1) / SEG);
      // the columns contracted with the site's z values
      double f = 0.0;
      if (live) {
         const int row = 32 * (w & 3) + lane;
         const double *z = zd + (((size_t)tile * 4 + (row >> 5)) * 2 * g.TP + 2 * blk * g.TW + pl) * 32 + (row & 31);
#pragma unroll
         for (int i = 0; i < MAXC * 4; i++)
            if (i < ncw) f = fma(q_value(ai[i]), z[(size_t)i * 32], f);
      }
      red[cq][32 * (w & 3) + lane] = f;
      asm volatile("bar.sync 2, %0;" : : "n"(Q_BW * 32) : "memory");
      if (tid < 128) {
         const int i = tile * 128 + tid;
         if (i < n && !q_aborted(&abort_s)) {
            const double s = (red[0][tid] + red[1][tid]) + (red[2][tid] + red[3][tid]);
            // units of the product: 2^-62 over the four table scales, times the coefficients' scale
            const double sc = emax >= Q_NOT_FINITE ? __longlong_as_double(0x7ff8000000000000ll)
                              : emax > -4096       ? ldexp(1.0 / (Q_KAPPA * Q_KAPPA * Q_KAPPA * Q_KAPPA), emax - 62)
                                                   : 0.0;
            hpart[((size_t)blockIdx.z * gridDim.y + set) * n + i] = s * sc;
         }
      }
   }
   fence_before_sync();
   __syncthreads();
   if (w == Q_BW + 1) {
      __syncwarp();
      fence_after_sync();
      tmem_dealloc(tmem, 512);
   }
}

// force[site of slot i] += q b^T (H_h, H_k, H_l), the items' sums in order
__global__ void __launch_bounds__(256)
k_fsum_q(int n, int N, int nitems, QGeom g, const double *__restrict__ hpart, const int *__restrict__ slots,
         const double *__restrict__ chg, double *__restrict__ force, FinArgs fin, DevOut *out)
{
   if (fin.on && blockIdx.x == 0 && threadIdx.x == 255) finalize_eval(out, fin);   // every sum is complete
   const int i = blockIdx.x * blockDim.x + threadIdx.x;
   if (i >= n) return;
   double H[3] = {0, 0, 0};
   for (int k = 0; k < nitems; k++)
#pragma unroll
      for (int s = 0; s < 3; s++) H[s] += hpart[((size_t)k * 3 + s) * n + i];
   const int si = slots[i];
   const double q = chg[si];
   force[si] += q * (g.b[0] * H[0] + g.b[3] * H[1]);
   force[N + si] += q * (g.b[1] * H[0] + g.b[4] * H[1]);
   force[2 * (size_t)N + si] += q * (g.b[2] * H[0] + g.b[5] * H[1] + g.b[8] * H[2]);
}

// ----------------------------------------------------------------- adjoint
// Weighted structure factors V_a = sum_j q_j v_ja exp(i k.r_j) (a = x, y, z)
// and the per-site sums of the adjoint's reciprocal space (adjoint.cu): the
// weights take the charges' place in operand B, one more digit than the
// charges in the mixed form (residual weights spread over decades: a few
// close contacts dominate them, and the digits' grid is that of the largest).

// wmax[a]: high word of max |q v_a| (zeroed before): its FP64 exponent, so that
// no weight of the FP64 form is out of range, and above every finite one where
// a weight is infinite or NaN
template <typename V4>
__global__ void __launch_bounds__(256)
k_qwmax(int n, const int *__restrict__ slots, const double *__restrict__ chg, const V4 *__restrict__ res,
        unsigned int *__restrict__ wmax)
{
   const int i = blockIdx.x * blockDim.x + threadIdx.x;
   unsigned int m[3] = {0u, 0u, 0u};
   if (i < n) {
      const double q = chg[slots[i]];
      const V4 v = res[i];
      m[0] = (unsigned int)__double2hiint(fabs(q * (double)v.x));
      m[1] = (unsigned int)__double2hiint(fabs(q * (double)v.y));
      m[2] = (unsigned int)__double2hiint(fabs(q * (double)v.z));
   }
#pragma unroll
   for (int a = 0; a < 3; a++) {
      const unsigned int x = __reduce_max_sync(0xffffffffu, m[a]);
      if ((threadIdx.x & 31) == 0 && x) atomicMax(&wmax[a], x);
   }
}
__device__ __forceinline__ int q_wexp(unsigned int hi)   // a power of two above (subnormal ones too)
{
   return (int)(hi >> 20) - 1022;
}
// the channel's scale, NaN where a weight is not finite (its digits are not
// either then)
__device__ __forceinline__ double q_wscale(double scale, unsigned int hi)
{
   return hi >= 0x7ff00000u ? __longlong_as_double(0x7ff8000000000000ll) : ldexp(scale, q_wexp(hi));
}

// Operand B of the three weighted channels, per 32-site stage as in k_qtab.
template <int NS, int ND, typename V4>
__global__ void __launch_bounds__(256)
k_qwtab(int n, int ns, QGeom g, const int *__restrict__ slots, const double *__restrict__ site,
        const double *__restrict__ chg, double hi6, double hi7, double hi8, const V4 *__restrict__ res,
        const unsigned int *__restrict__ wmax, unsigned char *__restrict__ ztab, size_t zstride)
{
   typedef typename QCfg<NS>::T T;
   __shared__ unsigned long long su[32];
   __shared__ T sw[3][32];
   __shared__ T sz[64][33];
   const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, stage = blockIdx.x;
   if (w < 4) {
      const int i = stage * 32 + lane;
      const int si = i < n ? slots[i] : 0;
      if (w == 3) {
         su[lane] = i < n ? q_fixed64(hi6 * site[si] + hi7 * site[ns + si] + hi8 * site[2 * (size_t)ns + si]) : 0ull;
      } else {
         double x = 0.0;
         if (i < n) {
            const V4 v = res[i];
            x = chg[si] * (double)(w == 0 ? v.x : w == 1 ? v.y : v.z);
         }
         x = ldexp(x * Q_KAPPA, (NS == 3 ? 31 : 63) - q_wexp(wmax[w]));
         sw[w][lane] = NS == 3 ? (T)__double2int_rn(x) : (T)qbalance((T)__double2ll_rn(x));
      }
   }
   __syncthreads();
   const unsigned long long uz = su[lane];
   for (int t0 = 0; t0 < g.TP; t0 += 32) {
      const int nt = min(32, g.TP - t0);
      __syncthreads();
      for (int t = w; t < nt; t += 8) {
         T s, c;
         qtrig(t0 + t, uz, s, c);
         const int col = 16 * (t >> 3) + (t & 7);
         sz[col][lane] = qbalance(c);
         sz[col + 8][lane] = qbalance(s);
      }
      __syncthreads();
      const int kg = tid & 3, c8 = (tid >> 2) & 7, cg = tid >> 5;
      if (8 * cg < 2 * nt) {
         const int tcol = 2 * t0 + 8 * cg, b = tcol / (2 * g.TW), lc = tcol - 2 * b * g.TW;
         const int nT = q_blkcols(g, b);
         unsigned char *d = ztab + (size_t)stage * 2 * g.TP * Q_KS * 2 * ND + (size_t)2 * b * g.TW * Q_KS * 2 * ND +
                            (size_t)lc * Q_KS * 2 + kg * 128 + c8 * 16;
#pragma unroll
         for (int a = 0; a < 3; a++) {
            auto wz = [&](int e) { return qmul(sw[a][8 * kg + e], sz[8 * cg + c8][8 * kg + e]); };
            decltype(wz(0)) v[8];
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = wz(e);
            qstore<ND>(d + a * zstride, nT * Q_KS * 2, v);
         }
      }
   }
}

// Per (quad, t) and (s, r): the alpha derivatives (blk: dE/dalpha, dG/dalpha
// per block) and the coefficients of the per-site sum, laid out as A, B in
// k_qreduce.  With T = sum_a k_a V_a, P + i Q = coeff T: (-P, -Q) for the
// loss (sum_k cos Q - sin P = Im(e U), U = -P + i Q), (B, -A) for the energy
// (A cos + B sin).  Channel sums over nr0 (charges) and nrv (weights) ranges.
template <typename R>
__global__ void __launch_bounds__(256)
k_qadj(QGeom g, const int4 *__restrict__ units, const double2 *__restrict__ coeff, double alpha, int loss, int nr0,
       double scale0, const R *__restrict__ part, int nrv, double scalev, const unsigned int *__restrict__ wmax,
       const R *__restrict__ partv, R *__restrict__ ab, double *__restrict__ blk)
{
   __shared__ double sq[4][8][32];
   __shared__ double sh[4][2];
   const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
   const int i = blockIdx.x * 32 + lane, quad = i / g.TP, t = i - quad * g.TP;
   const int4 un = quad < g.nquads ? units[quad >> 2] : make_int4(0, 0, 0, 0);
   const bool live = t < un.z;
   {
      // warp w: sum w of every channel
      const size_t row = 2 * (size_t)g.TP, plane = 4 * (size_t)g.nquads * row;
      const size_t at = ((size_t)quad * 4 + (w >> 1)) * row + 16 * (t >> 3) + 8 * (w & 1) + (t & 7);
      sq[0][w][lane] = live ? scale0 * q_rangesum(part + at, plane, nr0) : 0.0;
      for (int ch = 1; ch < 4; ch++)
         sq[ch][w][lane] = live && loss ? q_wscale(scalev, wmax[ch - 1]) *
                                             q_rangesum(partv + (size_t)(ch - 1) * nrv * plane + at, plane, nrv)
                                        : 0.0;
   }
   __syncthreads();
   if (w >= 4) return;
   double ea = 0.0, la = 0.0;
   if (quad < g.nquads) {
      double o0 = 0.0, o1 = 0.0;
      const double2 cf = live ? coeff[(size_t)i * 4 + w] : make_double2(0.0, 0.0);
      if (cf.x != 0.0) {
         const double s = w & 2 ? -1.0 : 1.0, r = w & 1 ? -1.0 : 1.0;
         double C[4], S[4];
#pragma unroll
         for (int ch = 0; ch < 4; ch++) {
            double q[8];
#pragma unroll
            for (int k = 0; k < 8; k++) q[k] = sq[ch][k][lane];
            C[ch] = (q[0] - s * q[2]) - r * (q[5] + s * q[7]);
            S[ch] = (q[4] + s * q[6]) + r * (q[1] - s * q[3]);
         }
         const double hh = un.x, kk = s * (un.y + (quad & 3)), l = r * t;
         const double kx = hh * g.b[0] + kk * g.b[3], ky = hh * g.b[1] + kk * g.b[4];
         const double kz = hh * g.b[2] + kk * g.b[5] + l * g.b[8];
         const double dcf = cf.x * (kx * kx + ky * ky + kz * kz) / (2.0 * alpha * alpha * alpha);
         ea = 0.5 * dcf * (C[0] * C[0] + S[0] * S[0]);
         if (loss) {
            const double Tc = kx * C[1] + ky * C[2] + kz * C[3], Ts = kx * S[1] + ky * S[2] + kz * S[3];
            la = dcf * (C[0] * Ts - S[0] * Tc);
            o0 = -cf.x * Tc;
            o1 = -cf.x * Ts;
         } else {
            o0 = cf.x * S[0];
            o1 = -cf.x * C[0];
         }
      }
      ab[(size_t)i * 8 + 2 * w] = (R)o0;
      ab[(size_t)i * 8 + 2 * w + 1] = (R)o1;
   }
#pragma unroll
   for (int o = 16; o > 0; o >>= 1) {
      ea += __shfl_down_sync(0xffffffffu, ea, o);
      la += __shfl_down_sync(0xffffffffu, la, o);
   }
   if (lane == 0) {
      sh[w][0] = ea;
      sh[w][1] = la;
   }
   asm volatile("bar.sync 1, 128;" : : : "memory");
   if (threadIdx.x < 2)
      blk[blockIdx.x * 2 + threadIdx.x] = (sh[0][threadIdx.x] + sh[1][threadIdx.x]) + (sh[2][threadIdx.x] + sh[3][threadIdx.x]);
}

// gq[site] += the per-site sum (items' / splits' partials s1 in order) and,
// for the loss, v . H with H = sum_k k (A sin - B cos) of the forward's
// force pass: FP64 items of (h, k, l) sums, or FP32-form Cartesian splits.
template <bool MIXED, typename V4>
__global__ void __launch_bounds__(256)
k_qadj_site(int n, int np, QGeom g, const double *__restrict__ hpart, const double *__restrict__ s1,
            const V4 *__restrict__ res, int loss, const int *__restrict__ slots, double *__restrict__ gq)
{
   const int i = blockIdx.x * blockDim.x + threadIdx.x;
   if (i >= n) return;
   double v = 0.0;
   for (int k = 0; k < np; k++) v += s1[(size_t)k * (MIXED ? 3 : 1) * n + i];
   if (loss) {
      double H[3] = {0, 0, 0};
      for (int k = 0; k < np; k++)
#pragma unroll
         for (int a = 0; a < 3; a++) H[a] += hpart[((size_t)k * 3 + a) * n + i];
      const V4 r = res[i];
      const double x = r.x, y = r.y, z = r.z;
      if (MIXED)
         v += x * H[0] + y * H[1] + z * H[2];
      else
         v += x * (g.b[0] * H[0] + g.b[3] * H[1]) + y * (g.b[1] * H[0] + g.b[4] * H[1]) +
              z * (g.b[2] * H[0] + g.b[5] * H[1] + g.b[8] * H[2]);
   }
   gq[slots[i]] += v;
}

// ------------------------------------------------------------- host side
#define CK(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) return cuda_check(c, e_, #x); } while (0)

// Shared-memory sizes, set once per device outside any stream capture
// (contexts may be created from several host threads: the per-device flags
// are atomic, and setting the attribute twice is harmless).
static cudaError_t q_init_device(int device)
{
   static std::atomic<unsigned long long> done{0};
   const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0ull;
   if (bit && (done.load() & bit)) return cudaSuccess;
   cudaError_t e = cudaFuncSetAttribute(k_sfac_q<3, 3, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, Q_SMEM<3, 3>);
   if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sfac_q<3, 4, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, Q_SMEM<3, 4, 4>);
   if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sfac_q<3, 4, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, Q_SMEM<3, 4>);
   if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sfac_q<7, 7, 7>, cudaFuncAttributeMaxDynamicSharedMemorySize, Q_SMEM<7, 7>);
   if (e == cudaSuccess) e = cudaFuncSetAttribute(k_force_q, cudaFuncAttributeMaxDynamicSharedMemorySize, Q_FSMEM);
   if (e == cudaSuccess) e = ks_force_tc_init();
   if (e == cudaSuccess && bit) done.fetch_or(bit);
   return e;
}

// Stages of 32 sites, padded to the force passes' 128-site tiles.
static size_t q_stages(int n) { return (size_t)((n + 127) / 128) * 4; }

// The quad list of the current k-list and its device copy.
mdgpu_status ks_q_prepare(mdgpu_ctx *c, int ns)
{
   KsDev &d = c->kd;
   QList &q = c->kl.q;
   CK(q_init_device(c->device));
   if (c->nsm <= 0) CK(cudaDeviceGetAttribute(&c->nsm, cudaDevAttrMultiProcessorCount, c->device));
   if (q.ns == ns || c->kl.nk == 0) return MDGPU_OK;
   build_qlist(c->kl, ns);
   q.ns = 0;   // not there until the copy is on its way: it may be refused
   TablePack &k = d.q_lists;
   CK(k.begin());
   const size_t o[6] = {k.add(q.units), k.add(q.coeff), k.add(q.tiles), k.add(q.segs), k.add(q.fu), k.add(q.seg0)};
   CK(k.send(c->stream));
   k.at(d.q_units.p, o[0]);
   k.at(d.q_coeff.p, o[1]);
   k.at(d.q_tiles.p, o[2]);
   k.at(d.q_segs.p, o[3]);
   k.at(d.q_fu.p, o[4]);
   k.at(d.q_seg0.p, o[5]);
   d.q_fblk = q.fblk;
   d.q_nfblk = q.fblk.empty() ? 0 : (int)q.fblk.size() - 1;
   q.ns = ns;
   return MDGPU_OK;
}

// The scale of the charges: FP64, a power of two above the largest; mixed,
// the largest itself (its 31-bit fixed point then holds charges in simple
// ratios, rigid water's 1 : -2, exactly: their rounding is the same at every
// site of a kind and does not average out).  NaN where a charge is not finite,
// which the digits cannot hold: the sums' scale then makes every result NaN.
static double q_charge_scale(const mdgpu_ctx *c, int ns)
{
   if (std::isnan(c->qmax)) return c->qmax;
   int e = 0;
   const double q = c->qmax > 0 ? c->qmax : 1.0;
   std::frexp(q, &e);
   return ns == 3 ? q : std::ldexp(1.0, e);
}

mdgpu_status ks_q_tables(mdgpu_ctx *c, int ns, int n, bool wide, const int *slots, const double *d_site)
{
   KsDev &d = c->kd;
   const QGeom &g = c->kl.q.g;
   const size_t S = q_stages(n);
   const double *hi = c->kl.hinv;
   const double qinv = 1.0 / q_charge_scale(c, ns);
   CK(d.q_ztab.ensure(S * 2 * g.TP * Q_KS * 2 * (ns == 3 && wide ? 4 : ns)));
   if (ns == 3) {
      CK(d.q_x32.ensure(S * 2 * g.hrows * QCfg<3>::RS));
      CK(d.q_y32.ensure(S * 2 * g.mrows * QCfg<3>::RS));
      CK(d.zsite.ensure(S / 4 * 2 * g.TP * 48));
      if (wide) {
         CK(d.q_xw32.ensure(S * 2 * g.hrows * QCfg<3>::RS));
         k_qtab<3, 4><<<(unsigned int)S, 256, 0, c->stream>>>(n, c->nsites, g, slots, d_site, c->rd.chg.p, hi[0], hi[1], hi[2],
                                                           hi[3], hi[4], hi[5], hi[6], hi[7], hi[8], qinv, d.q_x32.p,
                                                           d.q_y32.p, d.q_ztab.p, d.zsite.p, nullptr, d.q_xw32.p);
      } else {
         k_qtab<3, 3><<<(unsigned int)S, 256, 0, c->stream>>>(n, c->nsites, g, slots, d_site, c->rd.chg.p, hi[0], hi[1], hi[2],
                                                           hi[3], hi[4], hi[5], hi[6], hi[7], hi[8], qinv, d.q_x32.p,
                                                           d.q_y32.p, d.q_ztab.p, d.zsite.p, nullptr, nullptr);
      }
   } else {
      CK(d.q_x64.ensure(S * 2 * g.hrows * QCfg<7>::RS));
      CK(d.q_y64.ensure(S * 2 * g.mrows * QCfg<7>::RS));
      CK(d.q_zd.ensure(S * 2 * g.TP * 32));
      k_qtab<7, 7><<<(unsigned int)S, 256, 0, c->stream>>>(n, c->nsites, g, slots, d_site, c->rd.chg.p, hi[0], hi[1], hi[2],
                                                        hi[3], hi[4], hi[5], hi[6], hi[7], hi[8], qinv, d.q_x64.p,
                                                        d.q_y64.p, d.q_ztab.p, nullptr, d.q_zd.p, nullptr);
   }
   CK(cudaGetLastError());
   return MDGPU_OK;
}

// Site ranges: the count for which the waves of (tile, range) CTAs, each its
// stages plus a start-up of about six, come out shortest.  A framework's
// sites (slots f0 on) have ranges of their own.
mdgpu_status ks_q_sfac(mdgpu_ctx *c, int ns, int n, bool wide, int f0, int nf)
{
   KsDev &d = c->kd;
   const QList &q = c->kl.q;
   const int n0 = (n + 31) / 32, s1 = f0 / 32, nstf = (nf + 31) / 32, nst = n0 + nstf, nt = (int)q.tiles.size();
   const size_t plane = 4 * (size_t)q.g.nquads * 2 * q.g.TP, psz = ns == 3 ? sizeof(float) : sizeof(double);
   long long best = -1;
   int per = nst;
   for (int r = 1; r <= 64 && r <= nst; r++) {
      if (r > 1 && (r + 1) * plane * psz > (256u << 20)) break;
      const int p = (nst + r - 1) / r, nr = (n0 + p - 1) / p + (nstf + p - 1) / p;
      const long long cost = (long long)((nt * nr + c->nsm - 1) / c->nsm) * (p + 6);
      if (best < 0 || cost < best) {
         best = cost;
         per = p;
      }
   }
   const int R0 = (n0 + per - 1) / per, R = R0 + (nstf + per - 1) / per;
   CK(d.q_part.ensure(R * plane * psz));
   const dim3 grid(nt, R);
   if (ns == 3 && wide)
      k_sfac_q<3, 4, 4><<<grid, Q_THREADS, Q_SMEM<3, 4, 4>, c->stream>>>(q.g, 256u, d.q_tiles.p, d.q_units.p,
         (const unsigned char *)d.q_xw32.p, (const unsigned char *)d.q_y32.p, d.q_ztab.p, 0, R0, n0, s1, s1 + nstf, per,
         (float *)d.q_part.p, &c->out.p->err);
   else if (ns == 3)
      k_sfac_q<3, 3, 3><<<grid, Q_THREADS, Q_SMEM<3, 3>, c->stream>>>(q.g, 256u, d.q_tiles.p, d.q_units.p,
         (const unsigned char *)d.q_x32.p, (const unsigned char *)d.q_y32.p, d.q_ztab.p, 0, R0, n0, s1, s1 + nstf, per,
         (float *)d.q_part.p, &c->out.p->err);
   else
      k_sfac_q<7, 7, 7><<<grid, Q_THREADS, Q_SMEM<7, 7>, c->stream>>>(q.g, 256u, d.q_tiles.p, d.q_units.p,
         (const unsigned char *)d.q_x64.p, (const unsigned char *)d.q_y64.p, d.q_ztab.p, 0, R0, n0, s1, s1 + nstf, per,
         (double *)d.q_part.p, &c->out.p->err);
   CK(cudaGetLastError());
   d.q_nranges = R0;
   d.q_nrangesf = R - R0;
   return MDGPU_OK;
}

template <typename R, bool FW>
static void q_reduce(mdgpu_ctx *c, int nb, double scale, DBuf<R> &ab, DBuf<R> &abf)
{
   KsDev &d = c->kd;
   k_qreduce<R, FW><<<nb, 256, 0, c->stream>>>(c->kl.q.g, d.q_units.p, d.q_coeff.p, d.q_nranges, scale,
                                               (const R *)d.q_part.p, d.q_nrangesf, ab.p, abf.p, d.blk.p,
                                               c->rd.sync.p, c->out.p);
}
mdgpu_status ks_q_reduce(mdgpu_ctx *c, int ns, bool fw, bool wide)
{
   KsDev &d = c->kd;
   const QGeom &g = c->kl.q.g;
   const size_t nqt = (size_t)g.nquads * g.TP;
   const int nb = (int)std::min<size_t>((nqt + 31) / 32, 4 * (size_t)c->nsm);
   const double k4 = Q_KAPPA * Q_KAPPA * Q_KAPPA * Q_KAPPA;
   const double scale = q_charge_scale(c, ns) * std::ldexp(1.0 / k4, ns == 7 ? -62 : wide ? -38 : -30);
   CK(d.blk.ensure((size_t)nb * 8));
   if (ns == 3) {
      CK(d.q_ab32.ensure(nqt * 8));
      if (fw) CK(d.q_abf32.ensure(nqt * 8));
      if (fw) q_reduce<float, true>(c, nb, scale, d.q_ab32, d.q_abf32);
      else q_reduce<float, false>(c, nb, scale, d.q_ab32, d.q_abf32);
   } else {
      CK(d.q_ab64.ensure(nqt * 8));
      if (fw) CK(d.q_abf64.ensure(nqt * 8));
      if (fw) q_reduce<double, true>(c, nb, scale, d.q_ab64, d.q_abf64);
      else q_reduce<double, false>(c, nb, scale, d.q_ab64, d.q_abf64);
   }
   CK(cudaGetLastError());
   return MDGPU_OK;
}

// Runs of segments of the FP64 force pass over T site tiles: the length for
// which the waves of (site tile, set, run) CTAs come out shortest.
static void q_runs(mdgpu_ctx *c, int T)
{
   KsDev &d = c->kd;
   const QList &q = c->kl.q;
   long long best = -1;
   int mx = 1;
   for (size_t b = 0; b + 1 < q.seg0.size(); b++) mx = std::max(mx, q.seg0[b + 1] - q.seg0[b]);
   for (int p = 1; p <= mx; p++) {
      int k = 0;
      for (size_t b = 0; b + 1 < q.seg0.size(); b++) k += (q.seg0[b + 1] - q.seg0[b] + p - 1) / p;
      if (k > 16 && p < mx) continue;
      const long long cost = (3LL * T * k + c->nsm - 1) / c->nsm * (4LL * p + 7);
      if (best < 0 || cost < best) {
         best = cost;
         d.q_per = p;
         d.q_nitems = k;
      }
   }
}

// (a framework's sites take the runs chosen for the others', if there are any)
mdgpu_status ks_q_force64(mdgpu_ctx *c, int n, int f0)
{
   KsDev &d = c->kd;
   const QList &q = c->kl.q;
   const int nseg = (int)q.segs.size(), T = (n + 127) / 128;
   if (f0 == 0 || c->ncharged == c->ncharged_fw) q_runs(c, T);
   CK(d.q_bq.ensure((size_t)3 * nseg * 4 * QCfg<7>::NTMAX * Q_KS * 2 * 7));
   CK(d.q_bexp.ensure((size_t)3 * nseg));
   DBuf<double> &hpart = f0 > 0 ? d.fpartf : d.fpart;
   CK(hpart.ensure((size_t)d.q_nitems * 3 * n));
   k_qcoef<<<dim3(nseg, 3), 256, 0, c->stream>>>(q.g, 0, d.q_segs.p, nseg, d.q_units.p,
                                                 f0 > 0 ? d.q_abf64.p : d.q_ab64.p, d.q_bq.p, d.q_bexp.p);
   k_force_q<<<dim3(T, 3, d.q_nitems), Q_THREADS, Q_FSMEM, c->stream>>>(
      q.g, d.q_segs.p, nseg, d.q_seg0.p, d.q_per, d.q_units.p, d.q_x64.p + (size_t)f0 / 32 * 2 * q.g.hrows * QCfg<7>::RS,
      d.q_y64.p + (size_t)f0 / 32 * 2 * q.g.mrows * QCfg<7>::RS, d.q_zd.p + (size_t)f0 / 32 * 2 * q.g.TP * 32, d.q_bq.p,
      d.q_bexp.p, n, hpart.p, &c->out.p->err);
   CK(cudaGetLastError());
   c->launches += 1;
   return MDGPU_OK;
}

mdgpu_status ks_q_fsum64(mdgpu_ctx *c, int n, int f0, const int *slots, double *d_force, const FinArgs &fin)
{
   const double *hpart = f0 > 0 ? c->kd.fpartf.p : c->kd.fpart.p;
   k_fsum_q<<<(n + 255) / 256, 256, 0, c->stream>>>(n, c->nsites, c->kd.q_nitems, c->kl.q.g, hpart, slots + f0,
                                                    c->rd.chg.p, d_force, fin, c->out.p);
   CK(cudaGetLastError());
   return MDGPU_OK;
}

// Reciprocal-space adjoint over all sites (slots: every site in link-cell
// order, as the forward pass before it ran): adds into gq and writes the
// alpha derivatives' block records into a.blk (two each; their number in
// *nblocks).
mdgpu_status ks_q_adjoint(mdgpu_ctx *c, bool loss, const int *slots, double *gq, int *nblocks)
{
   KsDev &d = c->kd;
   AdjDev &a = c->ad;
   const QList &q = c->kl.q;
   const QGeom &g = q.g;
   cudaStream_t st = c->stream;
   const int ns = q.ns, nd = ns == 3 ? 4 : 7, N = c->nsites, nst = (N + 31) / 32, nt = (int)q.tiles.size();
   const size_t nqt = (size_t)g.nquads * g.TP, plane = 4 * (size_t)g.nquads * 2 * g.TP;
   const double k4 = Q_KAPPA * Q_KAPPA * Q_KAPPA * Q_KAPPA;
   const double *hi = c->kl.hinv;
   const size_t psz = ns == 3 ? sizeof(float) : sizeof(double);
   int R = 1;
   CK(a.wmax.ensure(3));
   if (loss) {
      const size_t S = q_stages(N), zstride = S * 2 * g.TP * Q_KS * 2 * nd;
      CK(a.zw.ensure(3 * zstride));
      CK(cudaMemsetAsync(a.wmax.p, 0, 3 * sizeof(unsigned int), st));
      long long best = -1;
      for (int r = 1; r <= 64 && r <= nst; r++) {
         if (r > 1 && 3 * r * plane * psz > (256u << 20)) break;
         const long long cost = (long long)((3 * nt * r + c->nsm - 1) / c->nsm) * ((nst + r - 1) / r + 6);
         if (best < 0 || cost < best) {
            best = cost;
            R = r;
         }
      }
      const int per = (nst + R - 1) / R;
      R = (nst + per - 1) / per;
      CK(a.partv.ensure(3 * (size_t)R * plane * psz));
      const dim3 grid(nt, R, 3);
      const int nb = (N + 255) / 256;
      if (ns == 3) {
         k_qwmax<float4><<<nb, 256, 0, st>>>(N, slots, c->rd.chg.p, a.res32.p, a.wmax.p);
         k_qwtab<3, 4, float4><<<nst, 256, 0, st>>>(N, N, g, slots, c->cur_site, c->rd.chg.p, hi[6], hi[7], hi[8],
                                                    a.res32.p, a.wmax.p, a.zw.p, zstride);
         k_sfac_q<3, 4, 3><<<grid, Q_THREADS, Q_SMEM<3, 4>, st>>>(g, 256u, d.q_tiles.p, d.q_units.p,
            (const unsigned char *)d.q_x32.p, (const unsigned char *)d.q_y32.p, a.zw.p, zstride, R, nst, 0, nst, per,
            (float *)a.partv.p, &c->out.p->err);
      } else {
         k_qwmax<double4><<<nb, 256, 0, st>>>(N, slots, c->rd.chg.p, a.res64.p, a.wmax.p);
         k_qwtab<7, 7, double4><<<nst, 256, 0, st>>>(N, N, g, slots, c->cur_site, c->rd.chg.p, hi[6], hi[7], hi[8],
                                                     a.res64.p, a.wmax.p, a.zw.p, zstride);
         k_sfac_q<7, 7, 7><<<grid, Q_THREADS, Q_SMEM<7, 7>, st>>>(g, 256u, d.q_tiles.p, d.q_units.p,
            (const unsigned char *)d.q_x64.p, (const unsigned char *)d.q_y64.p, a.zw.p, zstride, R, nst, 0, nst, per,
            (double *)a.partv.p, &c->out.p->err);
      }
      CK(cudaGetLastError());
      c->launches += 3;
   }
   const int nb = (int)((nqt + 31) / 32);
   *nblocks = nb;
   CK(a.blk.ensure(2 * (size_t)nb));
   const double qs = q_charge_scale(c, ns);
   if (ns == 3) {
      CK(a.ab32.ensure(nqt * 8));
      k_qadj<float><<<nb, 256, 0, st>>>(g, d.q_units.p, d.q_coeff.p, c->ctl.alpha, loss ? 1 : 0, d.q_nranges,
         qs * std::ldexp(1.0 / k4, c->q_spread ? -38 : -30), (const float *)d.q_part.p, R, std::ldexp(1.0 / k4, -38), a.wmax.p, (const float *)a.partv.p, a.ab32.p, a.blk.p);
      const int sp = ks_force_tc_splits(d);
      CK(a.gkpart.ensure((size_t)sp * 3 * N));
      const KsForceSites grp{N, 0, a.ab32.p, a.gkpart.p};
      const int nl = ks_force_tc(st, &grp, 1, g, d, true, c->nsm, &c->out.p->err);
      if (nl < 0) return fail(c, MDGPU_E_NOMEM, "device allocation failed (force-pass work ranges)");
      c->launches += nl;
      k_qadj_site<true, float4><<<(N + 255) / 256, 256, 0, st>>>(N, sp, g, d.fpart.p, a.gkpart.p, a.res32.p,
                                                                 loss ? 1 : 0, slots, gq);
   } else {
      CK(a.ab64.ensure(nqt * 8));
      k_qadj<double><<<nb, 256, 0, st>>>(g, d.q_units.p, d.q_coeff.p, c->ctl.alpha, loss ? 1 : 0, d.q_nranges,
         qs * std::ldexp(1.0 / k4, -62), (const double *)d.q_part.p, R, std::ldexp(1.0 / k4, -62), a.wmax.p, (const double *)a.partv.p, a.ab64.p, a.blk.p);
      const int nseg = (int)q.segs.size(), T = (N + 127) / 128;
      CK(a.gkpart.ensure((size_t)d.q_nitems * N));
      k_qcoef<<<dim3(nseg, 1), 256, 0, st>>>(g, 3, d.q_segs.p, nseg, d.q_units.p, a.ab64.p, d.q_bq.p, d.q_bexp.p);
      k_force_q<<<dim3(T, 1, d.q_nitems), Q_THREADS, Q_FSMEM, st>>>(
         g, d.q_segs.p, nseg, d.q_seg0.p, d.q_per, d.q_units.p, d.q_x64.p, d.q_y64.p, d.q_zd.p, d.q_bq.p, d.q_bexp.p, N,
         a.gkpart.p, &c->out.p->err);
      c->launches += 2;
      k_qadj_site<false, double4><<<(N + 255) / 256, 256, 0, st>>>(N, d.q_nitems, g, d.fpart.p, a.gkpart.p, a.res64.p,
                                                                   loss ? 1 : 0, slots, gq);
   }
   CK(cudaGetLastError());
   c->launches += 2;
   return MDGPU_OK;
}
#undef CK

}  // namespace mdgpu
