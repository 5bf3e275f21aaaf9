// Internal declarations of libmoldy_gb300: the context, the host-side
// geometry (link-cell stencil, k-vector list) and the launch functions of
// the real-space (realspace.cu) and reciprocal-space (kspace.cu) kernels.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <cstring>
#include <vector>

#include "../../include/moldy_gb300.h"

namespace mdgpu {

constexpr int NPOTP = 8;          // parameters per potential (src/defs.h:144)
constexpr int KI = 16;            // k-vectors per k-space work item
constexpr int KT = 64;            // k-vectors per item of mdgpu_tc_items (4 KI runs)
constexpr int FT_THREADS = 128;   // k_force32: threads per block, two sites each
constexpr double PI = 3.14159265358979323846;
constexpr double ALPHAMIN = 1e-7; // src/defs.h:181
constexpr double TOO_CLOSE = 0.25;// r^2 warning threshold, src/force.c:89
constexpr int MAX_TOO_CLOSE_REC = 16;

// ---- host-side geometry of one real-space call -------------------------
struct RsGeom {
   int nx = 0, ny = 0, nz = 0, ncells = 0;
   int n_half = 0;                 // half-space stencil (reference list)
   std::vector<int> half;          // 3 ints per offset, reference order
   std::vector<int4> full;         // (dx,dy,dz,is_zero) both half-spaces
   std::vector<float4> off_hi, off_lo;  // h.(d/n) as float hi + lo parts
   double h[9];
   double hinv[9];                 // src/matrix.c invert() of h
   double reloc[27][3];            // image translations, src/force.c:1282-1293
   double origin_step[9];          // h / n (column j scaled by 1/n_j)
   double cut2 = 0, cut100 = 0;
   double key[12];                 // h, cutoff, subcell, strict: cache key
   // The full stencil as columns: offsets of one (dx, dy) with consecutive
   // dz form one column (dx, dy, dz_min, length); col_base[i] indexes the
   // column's first entry in coff_hi/coff_lo, which hold the cell-offset
   // vectors of its dz values in order (FP32 hi + lo parts).  cols_ok: every
   // column is at most nz long (so it wraps the periodic cell at most once).
   std::vector<int4> cols;
   std::vector<int> col_base;
   std::vector<float4> coff_hi, coff_lo;
   bool cols_ok = false;
   // every offset of the 27-cell neighbourhood is in the stencil and each
   // cell is at least 0.5 A thick (any pair closer than the too-close
   // distance lies in neighbouring cells)
   bool nbr27 = false;
   int nbcol[9] = {0};             // column of each (dx, dy) in [-1, 1]^2 (when nbr27)
};

// Builds the stencil and cell geometry; returns MDGPU_E_CUTOFF as the
// reference's FATAL CUTOFF would fire.
mdgpu_status build_rs_geom(const double *h, const mdgpu_control &ctl, RsGeom &g);
mdgpu_status build_rdf_stencil(const double *h, double limit, int nx, int ny, int nz, std::vector<int4> &full);

// ---- tensor-core reciprocal space: quads (kspace_q.cu) --------------------
constexpr double Q_KAPPA = 255.0 / 256.0;   // scale of every table value: no top digit overflows
// Geometry of one k-list's tables.
struct QGeom {
   int hrows, mrows;       // X and Y values per site: h = 0 .. hrows - 1, m = 0 .. mrows - 1 (a multiple of 4)
   int TP;                 // t values (columns 2 TP: per 8 t, 8 cosines and 8 sines)
   int TW, nblk;           // t-blocks: width, count (the last one may be narrower)
   int nquads;             // 4 x units
   double b[9];            // 2 pi h^-1, row-major
};
// Row tile of a t-block: its units (four quads (h, m0 .. m0 + 3) each, -1
// padding) and the table ranges it reads.
constexpr int Q_XMAX = 8, Q_YMAX = 24;   // h and m values a row tile may span
struct QTile {
   int col0, nT;                 // first column of its t-block, columns
   int xlo, nx, ylo, ny;         // h and m values spanned
   int unit[16];
};
// Eight units of one t-block (the K-rows between two read-backs of the FP64
// force pass).
struct QSeg {
   int blk;
   int unit[8];
};
struct QList {
   int ns = 0;                     // digits it was built for (3 mixed, 7 FP64)
   QGeom g{};
   std::vector<int4> units;        // (h, m0, t range, 0)
   std::vector<double2> coeff;     // [quad][TP][s][r]: src/ewald.c:510-511 (0: no such k-vector)
   std::vector<QTile> tiles;       // structure factor
   std::vector<QSeg> segs;         // FP64 force pass
   std::vector<int> seg0;          // first segment of each t-block, and the end
   std::vector<int4> fu;           // mixed force pass: (h, m0, t range, unit), per 64-wide t-block
   std::vector<int> fblk;          // first entry of each of its t-blocks, and the end
};

// ---- host-side k-vector list ---------------------------------------------
struct KList {
   int hmax = 0, kmax = 0, lmax = 0, nk = 0, nitems = 0;
   std::vector<int4> item;         // (h, k, l0, count)
   std::vector<int> item_k0;       // index of the item's first k-vector
   std::vector<double2> item_kxy;  // (kx, ky) of the item's (h,k) column
   std::vector<double> kz;         // per k-vector
   double dkz = 0;                 // kz step from l to l + 1 (2 pi hinv[2][2])
   std::vector<double> coeff, coeff2;  // src/ewald.c:510-511
   double key[12];                 // h, k_cutoff, alpha
   double vol = 0;
   double hinv[9];
   QList q;
};

mdgpu_status build_klist(const double *h, const mdgpu_control &ctl, KList &kl);
// Quads of the list for ns digits (kl.q).
void build_qlist(KList &kl, int ns);
// Runs of up to KT l values of one (h, k) column (mdgpu_tc_items).
void build_tc_items(const KList &kl, std::vector<int4> &item, std::vector<int4> &k0);

// ---- first-call constants (host, FP64, reference arithmetic) -------------
double host_poteval(const double *potpar, double r, int ptype, double chgsq, double alpha);
double intramolecular_energy(const std::vector<mdgpu_species> &spec,
                             const std::vector<int> &spec_ids, const std::vector<double> &spec_pf,
                             const double *potpar, int max_id, int ptype,
                             const std::vector<double> &chg, double alpha);
void ewald_self_sheet(const std::vector<mdgpu_species> &spec, const std::vector<double> &spec_pf,
                      const std::vector<double> &chg, double alpha, double *self,
                      double *sheet, int *nsitesxf);
void ewald_self_sheet_grad(const std::vector<mdgpu_species> &spec, const std::vector<double> &spec_pf,
                           const std::vector<double> &chg, double alpha, double vol, double *g_chg,
                           double *g_alpha);
// Constant of the distant-potential correction (distant_const,
// src/accel.c:293-328 with dist_pot, src/kernel.c:103-150): energy x volume.
double distant_const(const mdgpu_ctx *c);
// The pressure form (iflag 1 of the same function, src/accel.c:316-320).
double distant_pconst(const mdgpu_ctx *c);
double det3(const double *a);
void inv3(const double *a, double *b);

// ---- device buffers ----------------------------------------------------------
// How often a buffer of a context has been freed for a larger one: a captured
// step holds the pointers of its time and is good for the count of its time
// only.  The buffers find their context's count while it is being constructed
// (it is the context's first member; the context's constructor ends that).
struct BufferMoves {
   uint64_t n = 0;
   static inline thread_local uint64_t *of_new = nullptr;
   BufferMoves() { of_new = &n; }
};

// Owned by the context: freed by release() or when the context is deleted
// (on its device: mdgpu_destroy selects it first).
template <typename T>
struct DBuf {
   T *p = nullptr;
   size_t n = 0;
   uint64_t *moves = BufferMoves::of_new;
   DBuf() = default;
   DBuf(const DBuf &) = delete;
   DBuf &operator=(const DBuf &) = delete;
   ~DBuf() { release(); }
   cudaError_t ensure(size_t want) {
      if (want <= n && p) return cudaSuccess;
      if (p) {
         cudaFree(p);
         if (moves) ++*moves;
      }
      p = nullptr;
      n = 0;
      cudaError_t e = cudaMalloc(&p, (want ? want : 1) * sizeof(T));
      if (e == cudaSuccess) n = want;
      return e;
   }
   void release() {
      if (p) cudaFree(p);
      p = nullptr;
      n = 0;
   }
};

// Host tables that change together (with the cell shape, every step of a
// constant-pressure run), gathered here and sent in one copy: a copy costs the
// host 3 to 5 us to issue whatever its size, and waiting for it a round trip.
// The source may be read after send() returns (a GPU that reads pageable
// memory in place need not stage it), so begin() waits for the copy before it
// is rewritten: done long before, where an evaluation lies between.
struct TablePack {
   std::vector<unsigned char> h;
   DBuf<unsigned char> d;
   cudaEvent_t sent = nullptr;
   TablePack() = default;
   TablePack(const TablePack &) = delete;
   TablePack &operator=(const TablePack &) = delete;
   ~TablePack()
   {
      if (sent) {
         cudaEventSynchronize(sent);
         cudaEventDestroy(sent);
      }
   }
   cudaError_t begin()
   {
      const cudaError_t e = sent ? cudaEventSynchronize(sent) : cudaEventCreateWithFlags(&sent, cudaEventDisableTiming);
      if (e == cudaSuccess) h.clear();
      return e;
   }
   template <typename T> size_t add(const std::vector<T> &v)   // its offset
   {
      const size_t o = (h.size() + 255) & ~(size_t)255;
      h.resize(o + v.size() * sizeof(T));
      if (!v.empty()) std::memcpy(h.data() + o, v.data(), v.size() * sizeof(T));
      return o;
   }
   cudaError_t send(cudaStream_t st)
   {
      // a capture would keep reading h when replayed: refused, as a wait would be
      cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
      cudaError_t e = cudaStreamIsCapturing(st, &cap);
      if (e == cudaSuccess && cap != cudaStreamCaptureStatusNone) e = cudaErrorStreamCaptureUnsupported;
      if (e == cudaSuccess) e = d.ensure(h.size());
      if (e == cudaSuccess && !h.empty()) e = cudaMemcpyAsync(d.p, h.data(), h.size(), cudaMemcpyHostToDevice, st);
      return e == cudaSuccess ? cudaEventRecord(sent, st) : e;
   }
   template <typename T> void at(T *&p, size_t o) const { p = reinterpret_cast<T *>(d.p + o); }
};
template <typename T> struct DView {   // a table of a pack
   T *p = nullptr;
};

// Device-resident outputs of one evaluation (all FP64).
struct DevOut {
   double pe_rs;          // sum of pair energies (before eintra)
   double vir_rs[6];      // xx xy xz yy yz zz
   double pe_k;           // sum of k-space energies (before self/sheet)
   double st_k[6];
   double vir_in[6];      // sum x_i (x) f_in_i, reference-semantics calls only
   int err;               // bit 0: co-ordinate out of range; bit 2: a
                          // structure-factor tile copy timed out
   int n_too_close;
   int64_t npairs2;       // full-list pair evaluations (2x reference count)
   int too_close[MAX_TOO_CLOSE_REC][2];
   double fin[11];        // energies [2] and stress [9] of mdgpu_forces
};

// DevOut::err as a status and its message (null: no error).
inline const char *eval_error(int err, mdgpu_status &s)
{
   s = err & 1 ? MDGPU_E_RANGE : err ? MDGPU_E_CUDA : MDGPU_OK;
   if (err & 1) return "Co-ordinate out of range in BIN (fill_cells)";
   if (err & 4) return "a structure-factor tile copy did not complete (bounded wait expired)";
   if (err & 8) return "a tensor-core structure-factor stage did not complete (bounded wait expired)";
   if (err & 16) return "a tensor-core force-pass stage did not complete (bounded wait expired)";
   return err ? "unknown device error" : nullptr;
}
// The error word of a dynamics run: bit 1 its own (quaternions), from bit 8 on
// the errors of every step's evaluation (the next one clears DevOut).
constexpr int MD_ERR_QNORM = 2, MD_ERR_EVAL = 8;
__host__ __device__ inline int md_err_add(int run, int eval) { return run | eval << MD_ERR_EVAL; }

// What the last kernel of an evaluation adds up (finalize_eval): the
// first-call constants and where the energies and the stress go besides
// DevOut::fin (pe null: nowhere).  on: the kernel's last block does it.
struct FinArgs {
   int on = 0, has_ewald = 0;
   double eintra = 0, self = 0, sheet_v = 0;
   double *pe = nullptr, *st = nullptr;
};

// Device counters of kernels whose last block to finish has a task of its
// own; each is zero between evaluations (that block resets it).
enum { SYNC_BIN = 0, SYNC_BINERR, SYNC_PAIRS, SYNC_KRED, SYNC_FSUM, SYNC_N };

struct RsDev {
   DBuf<int> cell_of, cell_count, cell_start, slot_cell, sorted, blocksum;
   DBuf<double4> pos64;    // sorted: x, y, z, q
   DBuf<float4> pos32;     // sorted: x - cell origin (x, y, z), q
   DBuf<int2> tag;         // sorted: site id, molecule
   DBuf<int> molmap, siteid, ent_mol;
   DBuf<double> chg, cofm;
   TablePack geom;         // the link-cell tables: full .. off_lo, cols .. coff
   DView<int4> full;
   DView<float4> off_hi, off_lo;
   DBuf<double> pot64;
   DBuf<float> pot32;
   DBuf<double> part;      // per-block partial energies/virials
   DBuf<double> part2;     // their first-level sums
   DBuf<unsigned long long> keys;
   DBuf<int4> rdf_full;    // RDF stencil (strict, at the RDF limit)
   // column walk of the mixed pair kernel (k_pairs_col): the stencil's
   // columns and their offsets (where it runs with two interaction classes
   // the slots are laid class by class: cell_start then holds class 0's
   // cells, class 1's, and the end)
   DView<int4> cols;
   DView<int> col_base;
   DView<float4> coff;     // [e][2]: the column offsets' hi and lo parts side by side (32 B per entry)
   DBuf<int2> tagc;        // per slot: site id with the cell's z index above 16 bits, molecule
   DBuf<int> site_cls;     // interaction class of every site
   DBuf<int> rank, unsorted;   // place of a site among its cell's, slots before the sort within cells
   DBuf<unsigned int> sync;    // counters (SYNC_*)
   DBuf<unsigned long long> rdf_counts;
   double rdf_key[11] = {0};
   int rdf_nfull = 0;
};

struct KsDev {
   DBuf<int4> item;
   DBuf<int> item_k0;
   DBuf<double2> item_kxy64;
   DBuf<float2> item_kxy32;
   DBuf<double> kz64, coeff, coeff2;
   DBuf<float4> kdat32;    // per k: (A_k, B_k, kz, 0)
   DBuf<double4> kdat64;
   DBuf<int4> ph32;        // per site: fixed-point phases (32-bit) + q bits
   DBuf<float2> z32;       // per site: exp(2 pi i s_z)
   DBuf<float2> zp32;      // per site: exp(2 pi i t s_z), t = 0..KI-1
   DBuf<ulonglong2> ph64a; // per site: (ux, uy) 64-bit phases
   DBuf<ulonglong2> ph64b; // per site: (uz, q bits)
   DBuf<double2> z64;
   DBuf<float2> part32;    // [chunks][nk] structure-factor partials
   DBuf<double2> part64;
   DBuf<double> fpart;     // [splits][3][N] force partials
   DBuf<double> blk;       // per-block energy/stress partials
   DBuf<double> blk2;      // their first-level sums
   DBuf<unsigned int> kcount;   // k_kfinal_part: blocks finished (the last one sums the slices)
   // framework molecule: framework-charge channel, its structure factor,
   // negated framework coefficients, its sites' records held compactly
   DBuf<int> fslot, sortedc;
   DBuf<int4> phf32, phc32;
   DBuf<ulonglong2> phf64b, pac64, pbc64;
   DBuf<float2> partf32, zpc32;
   DBuf<double2> partf64, zc64;
   DBuf<float4> kdatf32;
   DBuf<double4> kdatf64;
   DBuf<double> fpartf;
   // charged sites only (a site without charge adds nothing to S(k) and
   // gets no k-space force): their slots in link-cell order
   DBuf<int> kslots, kscan, kbsum;
   // tensor-core passes (kspace_q.cu, kspace_tc.cu): the quad list; the
   // per-site tables (X, Y fixed point; z digits as the structure factor's B
   // operand; z as the mixed force pass's A operand or in FP64); the
   // structure-factor partials; per (quad, t) A and B; the force passes'
   // coefficient operands
   TablePack q_lists;      // q_units .. q_segs
   DView<int4> q_units, q_fu;
   DView<double2> q_coeff;
   DView<QTile> q_tiles;
   DView<QSeg> q_segs;
   DView<int> q_seg0;
   DBuf<int> q_x32, q_y32, q_bexp;
   DBuf<long long> q_x64, q_y64;
   DBuf<unsigned char> q_ztab, q_bq, q_part;
   DBuf<double> q_zd, q_ab64;
   DBuf<float> q_ab32;
   int q_nfblk = 0;                 // mixed force pass: t-blocks and their entries of q_fu
   std::vector<int> q_fblk;
   int q_per = 1, q_nitems = 0;     // FP64 force pass of this evaluation: segments per run, runs
   int q_nranges = 0, q_nrangesf = 0;   // site ranges of q_part, the framework's after them
   DBuf<double> q_abf64;   // the framework sites' coefficients (whole S(k) without the framework's)
   DBuf<float> q_abf32;
   DBuf<int> q_xw32;       // X in full width (mixed form, framework)
   uint64_t kslots_gen = 0;   // configuration the framework part of kslots is for
   DBuf<uint4> zsite;      // force pass: z tables as the A operand, per 128 sites
   DBuf<uint4> utab;       // force pass: per-item coefficient rows (B operand)
   DBuf<float4> tc_coef;   // per item: kx s1, ky s1, kz0 s1, dkz s2 (row scales s)
   DBuf<int> tc_ustart[2]; // force pass: the CTAs' work ranges (ftc_ranges), of the framework's sites
};

// Buffers of the adjoint (parameter-gradient) passes.
struct AdjDev {
   DBuf<double4> res64;    // per slot: residual weight v of the site (FP64 form)
   DBuf<float4> res32;     // per slot: the same in FP32 (mixed form)
   DBuf<double> fref;      // [3][N] reference forces
   DBuf<double> gq;        // [2][N] dE/dq, dG/dq per site
   DBuf<double> gpart;     // per-block real-space gradient slots
   DBuf<double> slots;     // summed real-space slots
   DBuf<double> scal;      // loss, k-space dE/dalpha, dG/dalpha
   DBuf<double> lpart;     // per-block loss partials
   DBuf<int4> phv32;       // [3][N] mixed-form phases with weight q v_a
                           // ([6][N] with a framework: its sites' weights after)
   DBuf<ulonglong2> phv64; // [3][N] (u_z, weight q v_a) for the FP64 form
   DBuf<float2> partv32;   // [3][chunks][nk] weighted structure-factor partials
                           // ([6][chunks][nk] with a framework)
   DBuf<double2> partv64;
   DBuf<float4> kadj32;    // per k: A, B, P, Q
   DBuf<double4> kadj64;
   DBuf<float4> kadjf32;   // per k: the framework sites' A, B, P, Q, negated
   DBuf<double4> kadjf64;
   DBuf<float4> resc32;    // the framework sites' residual weights, compacted
   DBuf<double4> resc64;
   DBuf<double> gkpartf;   // [splits][2][nf] framework correction partials
   DBuf<float> kz32;       // per k: k_z
   DBuf<double> gkpart;    // [splits][2][N] k-space charge-gradient partials
   DBuf<double> blk;       // per-block k-space dE/dalpha, dG/dalpha
   // tensor-core passes: largest weights, the weights' digits, their
   // structure factors, the per-site pass's coefficients
   DBuf<unsigned int> wmax;
   DBuf<unsigned char> zw, partv;
   DBuf<double> ab64;
   DBuf<float> ab32;
};

// Rigid-molecule dynamics (integrate.cu): one species' constants.
struct MdSpec {
   double mass;
   double inertia[3], rinertia[3];   // principal moments and their inverses
   int nsites, pf0;                  // sites per molecule, first principal-frame site
   int framework;                    // fixed framework: momentum zeroed after the kicks
};

struct MdHost {
   bool ready = false;
   std::vector<MdSpec> spec;
   double h[9];
   double half = 0;                  // dt / 2
   double dist = 0;                  // distant-potential constant (energy x volume)
   double distp = 0;                 // distant-pressure constant (stress x volume)
   int nosym = 0, saxis = 0, nmols_r = 0;
   // one captured step (CUDA graph), replayed by mdgpu_md_run
   cudaGraphExec_t graph = nullptr;
   uint64_t graph_gen = 0, graph_moves = 0;   // configuration and buffers it was captured with
   int64_t graph_launches = 0;       // kernels one replay launches
   bool graph_class_major = false, graph_npairs_pending = false;   // how it leaves the slots, the pair count
   int graph_cap = 0;                // record capacity it was captured with
   uint64_t warm_gen = 0;            // configuration of the last direct step
   // constant temperature (mdgpu_md_set_thermostat)
   int d_of_f = 0;                   // degrees of freedom as start_up counts them
   bool therm = false;
   double temp = 0, ttmass = 0, gkt = 0, ahalf = 0;
   // constant pressure (mdgpu_md_set_barostat): mode 1 anisotropic, 2
   // uniform dilation; h (above) and its momentum advance on the host
   int baro = 0, strain_mask = 0;
   double pressure = 0, pmass = 0;
   double hmom[9] = {0};
   std::vector<double> kpart_h;      // host copies of block sums
};

struct MdDev {
   DBuf<double> cofm, mom, quat, amom;   // [nmols][3], [nmols][3], [nmols_r][4] x2
   DBuf<int> counter;                    // index of the next energy record
   DBuf<int> mol_spec, mol_q, mol_site0, site_mol, site_pf;
   DBuf<double> pf;                      // principal-frame sites of every species
   DBuf<MdSpec> spec;
   DBuf<double> kpart, energies;
   DBuf<int> err;
   DBuf<double> molf, molt;              // molecular forces, principal torques
   DBuf<double> vpart, virc;             // virial correction (dump records)
   DBuf<float> rec;                      // batch of dump records
   DBuf<double> therm;                   // s, its momentum, H_0, H_0 evaluated
   DBuf<double> tpart;                   // block sums of the thermostat momentum's increments
   DBuf<double> kdpart;                  // block sums of the kinetic stress (constant pressure)
};

}  // namespace mdgpu

struct mdgpu_ctx {
   mdgpu::BufferMoves moves;   // (first: the buffers below count in it)
   mdgpu_ctx() { mdgpu::BufferMoves::of_new = nullptr; }
   int device = 0;
   int nsm = 0;        // multiprocessors of the device (read when first needed)
   cudaStream_t own_stream = nullptr, stream = nullptr;
   mdgpu_precision prec = MDGPU_MIXED;
   std::string err;

   // system
   bool have_system = false, have_control = false;
   int nsites = 0, nmols = 0, max_id = 0, ptype = 0;
   // the framework molecule (species flagged framework come last; the
   // reference supports one framework molecule, src/force.c:1218-1220):
   // its index, its first site and the count of molecules before it
   int fw_mol = -1, fw_site0 = 0, nmols_nf = 0;
   std::vector<mdgpu_species> spec;
   std::vector<int> spec_ids;       // concatenated per-species site ids
   std::vector<double> spec_pf;     // concatenated principal-frame sites
   std::vector<int> site_id, molmap, mol_first, mol_nsites;
   std::vector<double> chg, potpar;
   mdgpu_control ctl{};
   bool sys_dirty = true;           // device copies out of date

   // first-call constants (recomputed after set_system)
   bool have_eintra = false, have_self = false;
   double eintra = 0, self_energy = 0, sheet_energy = 0;
   int nsitesxf = 0;

   // cached geometry
   mdgpu::RsGeom rs;
   bool rs_valid = false, rs_uploaded = false;
   mdgpu::KList kl;
   bool kl_valid = false, kl_uploaded = false;
   bool class_major = false;      // the slots of the last binning are laid class by class
   bool link_order = false;       // binning in plain link-cell order wanted (RDF)
   bool counts_clean = false;     // cell_count is all zero (k_place leaves it so)
   mdgpu::FinArgs fin;            // of the evaluation in progress
   cudaStream_t pairs_after_tables = nullptr;   // ks_launch starts the pair kernel on this stream
   bool npairs_pending = false;   // the last real-space pass left the pair count to rs_count_pairs
   int rs_nblk = 0;               // blocks (energy/virial partials) of the last real-space pass

   mdgpu::RsDev rd;
   mdgpu::KsDev kd;
   mdgpu::AdjDev ad;
   mdgpu::MdHost mdh;
   mdgpu::MdDev md;
   mdgpu::DBuf<double> site, force, force_in, cofm_in, small;
   const double *cur_site = nullptr;   // site array of the launch in progress
   std::vector<double> h_stage;        // small host arrays of the reference-style calls, gathered
   std::vector<double> last_cofm;      // centres of mass of the last force_calc
   mdgpu::DBuf<mdgpu::DevOut> out;
   mdgpu::DevOut *h_out = nullptr;  // pinned mirror

   mdgpu_info info{};
   int64_t launches = 0;
   bool timing = false;
   // the k-space passes run over every site, not only the charged ones
   // (the adjoint's backward passes read every site's phases)
   bool ks_all_sites = false;
   // reciprocal space on the tensor cores (MDGPU_KSPACE_TC=0 at context
   // creation selects the CUDA-core passes)
   bool tc_sfac = true;
   uint64_t ncharged_gen = 0;       // configuration the count below is for
   int ncharged = 0;                // sites with a nonzero charge
   int ncharged_fw = 0;             // of them, of the framework molecule
   int n_class0 = 0;                // sites of interaction class 0
   double qmax = 0;                 // and their largest |q| (NaN if one is not finite)
   bool q_spread = false;           // largest far above the root mean square (see ks_on_tc)
   cudaEvent_t ev[MDGPU_NPHASES + 1] = {};
   // second (high-priority) stream: the k-space passes run on it beside
   // the pair kernel
   cudaStream_t side_stream = nullptr;
   cudaEvent_t ev_fork = nullptr, ev_pairs = nullptr, ev_join = nullptr;
   bool ev_marked[MDGPU_NPHASES + 1] = {};
   bool have_nabor_note = false;
   // interaction classes of the site identifiers (realspace.cu): class 0
   // holds the identifiers that interact with charged sites, class 1 the
   // rest; pairs across the classes add exactly nothing.  ncls 1 when
   // every identifier is in class 0.
   std::vector<int> cls_of_id;
   int ncls = 1;
   int cls_pot = 0, cls_chg = 0;    // bit k: class k has a potential, charges among its sites
   // bumped by every call that changes what a captured step would launch
   // (system, control, parameters, precision, stream, dynamics state)
   uint64_t gen = 1;
   int note_nx = 0, note_ny = 0, note_nz = 0, note_nabors = 0;
};

namespace mdgpu {
// realspace.cu
mdgpu_status rs_prepare(mdgpu_ctx *c);   // upload geometry/system tables
// cells_only: bin and order the sites (the k-space passes stream them in
// link-cell order) without the pair kernel.
// sorted_ready (or null): recorded on the stream once the link-cell order
// (c->rd.sorted) is complete, before the per-slot records.
mdgpu_status rs_launch(mdgpu_ctx *c, const double *d_site, const double *d_cofm,
                       double *d_force, bool cells_only, unsigned long long *d_keys,
                       int64_t key_cap, cudaEvent_t sorted_ready = nullptr);
// Real-space adjoint over the slots binned by the last rs_launch: gradients
// into c->ad.gq ([2][N], written) and c->ad.slots; residual weights from
// c->ad.res64/res32 when loss.
mdgpu_status rs_adjoint(mdgpu_ctx *c, bool loss);
// The pair kernel and its energy/virial reduction over the sites binned by
// the last rs_launch, on c->stream (rs_launch without cells_only runs both).
mdgpu_status rs_pairs(mdgpu_ctx *c, double *d_force, unsigned long long *d_keys, int64_t key_cap);
// The reference's evaluated pair count of the last real-space pass into
// c->info.npairs, when that pass left it out (the column walk); waits for
// the context's stream.
mdgpu_status rs_count_pairs(mdgpu_ctx *c);
int pot_nparams(int ptype);     // parameters the potential type reads
// Site-pair distance histogram of the sites binned by the last rs_launch:
// full-list counts [max_id][max_id][nbins] into c->rd.rdf_counts (zeroed
// first); each unordered pair appears once from each side.
mdgpu_status rs_rdf(mdgpu_ctx *c, double limit, int nbins);
// kspace.cu
mdgpu_status ks_prepare(mdgpu_ctx *c);
// The passes of the current system and form are those on the tensor cores.
bool ks_on_tc(mdgpu_ctx *c);
// join: an event the final force sum waits for (the pair kernel running on
// another stream writes d_force first), or null.
mdgpu_status ks_launch(mdgpu_ctx *c, const double *d_site, double *d_force, bool accumulate,
                       cudaEvent_t join = nullptr);
struct KsShape {
   int chunks, chunk, splits, per_split;
};
// Chunks of the structure-factor pass and k-splits of a per-site pass
// (ipt items per thread, spt sites per thread).
KsShape ks_shape(int N, int nitems, int ipt, int spt);
// Reciprocal-space passes on the tensor cores.  kspace_q.cu: both forms'
// tables, structure factor and per-k sums (A and B per (quad, t), energy
// and stress into DevOut), and the FP64 form's force pass.  kspace_tc.cu: the mixed form's force pass, F_slot / q into
// fpart[split][3][nsites], or with scalar the sum over k of A sin - B cos
// into its first component (returns the launches, -1 if out of memory).
mdgpu_status ks_q_prepare(mdgpu_ctx *c, int ns);
// (wide: the mixed form's structure factor in four digits)
mdgpu_status ks_q_tables(mdgpu_ctx *c, int ns, int n, bool wide, const int *slots, const double *d_site);
// n sites and, from slot f0 (a multiple of 128) on, nf of a framework molecule
mdgpu_status ks_q_sfac(mdgpu_ctx *c, int ns, int n, bool wide, int f0, int nf);
mdgpu_status ks_q_reduce(mdgpu_ctx *c, int ns, bool fw, bool wide);
// sites from slot f0 (zero or the framework's first) on
mdgpu_status ks_q_force64(mdgpu_ctx *c, int n, int f0);
mdgpu_status ks_q_fsum64(mdgpu_ctx *c, int n, int f0, const int *slots, double *d_force, const FinArgs &fin);
// a group of sites of the mixed force pass: n from slot f0 on, their A and B
// per (quad, t), their force sums
struct KsForceSites {
   int n, f0;
   const float *ab;
   double *fpart;
};
int ks_force_tc(cudaStream_t st, const KsForceSites *grp, int ngrp, const QGeom &g, KsDev &d, bool scalar, int nsm, int *err);
mdgpu_status ks_q_adjoint(mdgpu_ctx *c, bool loss, const int *slots, double *gq, int *nblocks);
int ks_force_tc_splits(const KsDev &d);
size_t ks_tc_utab_len(int npos);
cudaError_t ks_force_tc_init();
// api.cu
mdgpu_status fail(mdgpu_ctx *c, mdgpu_status s, const std::string &msg);
mdgpu_status cuda_check(mdgpu_ctx *c, cudaError_t e, const char *what);
// Cell geometry, k-list and first-call constants current for h and the
// control record, device tables uploaded.
mdgpu_status ensure_ready(mdgpu_ctx *c, const double *h, bool need_rs, bool need_ks);
// Copies the device result record back, waits, reports device-side errors.
mdgpu_status sync_out(mdgpu_ctx *c);

// Marks the boundary before phase `i` (MDGPU_NPHASES marks the end).
inline void phase_mark(mdgpu_ctx *c, int i)
{
   if (!c->timing) return;
   if (!c->ev[i]) cudaEventCreate(&c->ev[i]);
   cudaEventRecord(c->ev[i], c->stream);
   c->ev_marked[i] = true;
}

#ifdef __CUDACC__
// True in every thread of the grid's last block to get here (all its threads
// call it, once); count (zero before) is reset.  What the other blocks wrote
// before their call is visible to the last one through L2 (__ldcg).
__device__ __forceinline__ bool last_block(unsigned int *count)
{
   __shared__ bool last;
   __threadfence();
   __syncthreads();
   if (threadIdx.x == 0) {
      last = atomicAdd(count, 1u) == gridDim.x * gridDim.y * gridDim.z - 1;
      if (last) *count = 0u;
   }
   __syncthreads();
   if (last) __threadfence();
   return last;
}

// Energies and stress of an evaluation from its sums (one thread).
__device__ __forceinline__ void finalize_eval(DevOut *out, const FinArgs &f)
{
   double r[11];
   const double e = f.has_ewald ? 1.0 : 0.0, d = f.has_ewald ? f.sheet_v : 0.0;
   r[0] = -f.eintra + __ldcg(&out->pe_rs);
   r[1] = f.has_ewald ? (-f.self + f.sheet_v) + __ldcg(&out->pe_k) : 0.0;
   double v[6];
   for (int k = 0; k < 6; k++) v[k] = __ldcg(&out->vir_rs[k]) + (f.has_ewald ? e * __ldcg(&out->st_k[k]) : 0.0);
   r[2] = v[0] + d;
   r[3] = v[1];
   r[4] = v[2];
   r[5] = 0.0;
   r[6] = v[3] + d;
   r[7] = v[4];
   r[8] = 0.0;
   r[9] = 0.0;
   r[10] = v[5] + d;
   for (int k = 0; k < 11; k++) out->fin[k] = r[k];
   if (f.pe) {
      f.pe[0] = r[0];
      f.pe[1] = r[1];
      for (int k = 0; k < 9; k++) f.st[k] = r[2 + k];
   }
}
#endif
}  // namespace mdgpu
