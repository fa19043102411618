// internal.cuh -- the handle types behind the C ABI and the helpers the
// translation units share.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

// Device CSR matrix.  The CSR arrays are the master copy (OFELI's SpMatrix
// layout, 0-based int32 columns on the device); a SELL-32 copy of the values
// (slices of 32 consecutive rows stored column-major, rows kept in natural
// order) is rebuilt lazily when the values change and feeds the SpMV inside
// the Krylov loops.
struct ofg_matrix {
   int64_t n = 0, nnz = 0;
   ofg::DBuf<int32_t> row_ptr, col;
   ofg::DBuf<double> val;
   uint64_t version = 1;  // bumped whenever values change
   // the value array was handed out (ofg_matrix_device_arrays): the caller may
   // write through the pointer at any time, without a new version
   bool exposed = false;

   // diagonal position of every row (OFELI's id[i]-1); -1 if absent
   ofg::DBuf<int32_t> dpos;
   bool dpos_ready = false;
   bool dpos_complete = false;

   // SELL-32 layout
   int64_t nslices = 0;
   ofg::DBuf<int32_t> sell_ptr;  // nslices+1, offsets in entries
   ofg::DBuf<int32_t> sell_col;  // padded entries point at a valid row, value 0
   ofg::DBuf<int32_t> sell_src;  // CSR index of every SELL entry, -1 for padding
   ofg::DBuf<double> sell_val;
   ofg::DBuf<float> sell_val32;
   ofg::DBuf<uint16_t> sell_valbf;  // BF16 bit patterns of the values
   // column - row of every SELL entry (0 for padding) when every offset fits
   // in 16 bits (idx16 = 1; 0 = does not fit; -1 = not built yet)
   ofg::DBuf<int16_t> sell_d16;
   int idx16 = -1;
   // slices whose 32 rows have the same 16-bit offset at every position k
   // (structured meshes in natural order): sell_uni[s] = start of the
   // slice's w offsets in sell_utab, -1 for a slice that keeps per-entry
   // offsets; uni_nnz = nonzeros in the uniform slices (built once, with the
   // 16-bit offsets)
   ofg::DBuf<int32_t> sell_uni;
   ofg::DBuf<int16_t> sell_utab;
   int64_t uni_nnz = 0, utab_len = 0;
   bool uni_ready = false;
   bool sell_ready = false;
   uint64_t sell_version = 0, sell32_version = 0, sellbf_version = 0;
   int max_row = 0;
   double avg_row = 0;

   // column-major copy of the pattern for the transposed product (built on
   // first use): column c's entries t_ptr[c] .. t_ptr[c+1], their rows in
   // ascending order and their CSR positions
   ofg::DBuf<int64_t> t_ptr;
   ofg::DBuf<int32_t> t_row, t_pos;
   bool t_ready = false;

   // element-to-CSR map of the mesh this pattern came from
   ofg_mesh* mesh = nullptr;
   // (built on first use: the batched solver, rows longer than kRowAcc)
   ofg::DBuf<int32_t> emap;  // ne * nen * nen, -1 where a DOF is imposed
   // the assembly's incidence records (see assembly.cu): node slices of 32,
   // record p of lane l of slice s at (inc_ptr[s] + p) * 32 + l
   bool inc_on = false;
   ofg::DBuf<int32_t> inc_ptr;   // slices + 1
   ofg::DBuf<int4> inc;          // element (-1: none), its other nodes (3-D: three)
   ofg::DBuf<int32_t> inc_meta;  // own place in the element, row offsets of its columns
};

struct ofg_mesh {
   int dim = 2, nen = 3;
   int64_t nn = 0, ne = 0, neq = 0;
   ofg::DBuf<double> coords;  // nn * dim
   ofg::DBuf<int32_t> elem;   // ne * nen, 0-based
   ofg::DBuf<int32_t> code;   // nn
   ofg::DBuf<int32_t> dof;    // nn, 1-based equation number or 0
   // node -> element adjacency (elements in ascending order)
   ofg::DBuf<int32_t> n2e_ptr, n2e;
   // the structured rectangle's cells and line codes (rect_nx < 0 otherwise),
   // kept for the sides Mesh::put writes
   int64_t rect_nx = -1, rect_ny = -1;
   int rect_code[4] = {0, 0, 0, 0};   // cx0, cxN, cy0, cyN
};

namespace ofg {
// Strand plan of one sweep direction (see prec.cu).
struct SweepPlan {
   int64_t nstrands = 0;
   DBuf<int32_t> start;       // logical row where each strand starts, nstrands+1
   DBuf<double> strand_dot;   // per-strand partial dot products
   DBuf<int> ticket;          // [0] next strand, [1] finished strands
   // per-segment slot layout of the dependency entries: segment s of strand
   // t (t's rows in 32-row groups) owns slots seg_off[s] .. seg_off[s+1],
   // stored column-major (slot k of lane l at seg_off[s] + 32 k + l), in
   // the CSR's column order
   int64_t nseg = 0;
   int wmax = 0;              // slots of the widest segment
   DBuf<int32_t> tseg;        // first segment of each strand, nstrands+1
   DBuf<int32_t> seg_off;     // nseg+1
   DBuf<int32_t> sl_col;      // physical column, -1 for padding
   DBuf<int32_t> sl_src;      // CSR index of the value, -1 for padding
   DBuf<double> sl_val;
   // per segment: the lowest row of the previous strand that this or a
   // later segment of its strand reads from the band's shared-memory ring
   // (INT32_MAX: none); the solve sweeps publish it so that the previous
   // strand's warp never overwrites a ring slot still to be read
   DBuf<int32_t> seg_keep;
};

// Wavefront plan of one sweep direction (see wave.cu): lines in groups of up
// to 32, the coefficients in the order the steps read them.
constexpr int kWaveExt = 4;        // entries a row may have in earlier groups
// The wavefront is taken when a line has at least kWaveMinLine rows on
// average and a step at least kWaveMinLanes active lanes.  On 2-D grids it is
// the faster form wherever these hold, long and thin ones included (us per CG
// iteration with ILU, strands of prec.cu / wavefront: 8 lines of 8 rows
// 65 / 37, 5 of 16 78 / 38, 5 of 1024 134 / 112, 8 of 2048 235 / 191, 32 of
// 8192 977 / 680, 1000 of 9 4380 / 171).
constexpr int64_t kWaveMinLine = 8;
constexpr int64_t kWaveMinLanes = 4;
// With entries in earlier groups (3-D) a row along a line costs the wavefront
// more (its right-hand side waits for the plane before, then the chunk), a
// line in a plane the strands; both pay per plane.  It is taken where
//    (rows a line)^2 planes <= kWaveLongLine (lines a plane)^2,
// a plane being a run of lines each coupled to the one before.  Measured on
// 316 boxes of 16 to 1500 rows, 8 to 128 lines, 3 to 128 planes (CG with ILU
// and SSOR, strands / wavefront, us per iteration with ILU): 63^3 1.30 times
// as fast, 127^3 1.45, 256 x 32 x 16 182 / 177; refused: 1024 x 16 x 64
// 540 / 671, 1024 x 128 x 16 589 / 634, 512 x 64 x 64 601 / 677.  Near the
// line one form or the other is up to 14 % faster; worst on the wavefront's
// side are deep boxes whose lines fill the strands' segments of 32 rows
// (32 x 32 x 128: 492 / 531).
constexpr double kWaveLongLine = 800.0;
struct WavePlan {
   bool on = false, fwd = true;
   bool ext = false;          // some row has entries in earlier groups
   bool clean = false;        // equal lines, one step apart
   int ngroups = 0;
   int64_t tiles = 0;         // 32-step layout tiles
   DBuf<int32_t> line, shift, dshift, eoff;
   DBuf<int32_t> g_line, g_tile, g_nch, g_edge, g_sm1, tile_g;
   DBuf<int32_t> stpos;       // forward, D-ILU: transposed positions in SELL order
   DBuf<double> coef, ecoef;  // step order; ecoef: natural order
   DBuf<double> edge;         // last lines of the groups on their way to the next group
   DBuf<double> gdot;
   DBuf<int> ticket;
};
}  // namespace ofg

namespace ofg {
// learned.cu: frees the network buffers kept for a learned preconditioner
void learned_release(const ofg_prec* P);
}  // namespace ofg

struct ofg_prec {
   ofg_matrix* A = nullptr;
   int type = OFG_DIAG;
   ofg::DBuf<double> pivot;  // DIAG/DILU/ILU: inverse pivots; SSOR: diagonal
   uint64_t version = 0;     // matrix version the factorisation belongs to
   // forward-sweep result, kept at the "not ready" sentinel between sweeps
   ofg::DBuf<double> t;
   ofg::DBuf<int> status;    // bounded-wait failures (bit 0: timeout, bit 1: wave)
   ofg::SweepPlan fwd, bwd;
   ofg::WavePlan wfwd, wbwd;  // both on and of the same `ext`, or both off
   ofg::DBuf<int32_t> tpos;  // D-ILU: transposed position of each lower entry
   ofg::DBuf<double> dot;    // (r, z) of the last backward sweep that was asked for it
   int grid = 0;             // blocks of the persistent factorisation sweep launch
   int solve_grid = 0;       // blocks of the persistent solve sweep launch
   // frozen: the solvers keep the preconditioner as it was set up even after
   // the matrix values changed (ofg_prec_freeze; refreshed by ofg_prec_update)
   bool frozen = false;
   // LEARNED: the network that predicts the factor G, and G (lower rows) and
   // G^T (upper rows) as matrices of their own; M = G^T G
   ofg_learned* net = nullptr;
   ofg_matrix* gl = nullptr;
   ofg_matrix* gu = nullptr;
   ofg::DBuf<double> partials;
   ofg::DBuf<unsigned> counter;
   ~ofg_prec()
   {
      if (type == OFG_LEARNED) ofg::learned_release(this);
      delete gl;
      delete gu;
   }
};

namespace ofg {

// matrix.cu
void ensure_dpos(ofg_matrix* A);
void ensure_sell(ofg_matrix* A);
// the same from the values as they are now, also where they were written
// through the pointer that ofg_matrix_device_arrays gave out
void refresh_sell(ofg_matrix* A);
void ensure_sell32(ofg_matrix* A);
void ensure_sell_bf16(ofg_matrix* A);
// new values into the FP64, FP32 and BF16 SELL copies in one pass, *inexact
// set when one is not exact in BF16; the BF16 copy, or null, with nothing
// done, when the copies are not stale or not laid out yet
const __nv_bfloat16* refresh_sell_all(ofg_matrix* A, int* inexact);
// builds the 16-bit column offsets once per pattern; true when they fit
bool ensure_sell_d16(ofg_matrix* A);
// after ensure_sell_d16 returned true
void ensure_sell_uniform(ofg_matrix* A);
void spmv_csr(const ofg_matrix* A, const double* x, double* y, bool add);
void spmv_sell(const ofg_matrix* A, const double* x, double* y, const int* skip = nullptr);
void matrix_touch(ofg_matrix* A);
void matrix_finish_pattern(ofg_matrix* A);
// a mesh with its coordinate, connectivity and code buffers allocated, and
// the rest (equation numbers from the codes, node-to-element lists) built
// once those hold the mesh (mesh.cu)
ofg_mesh* new_mesh(int dim, int64_t nn, int64_t ne);
void finish_mesh(ofg_mesh* m);
// the element-to-CSR map of a matrix made from a mesh
void ensure_emap(ofg_matrix* A);
// longest row the assembly sums in shared memory
constexpr int kRowAcc = 16;
// an incidence record's meta word: bits 0-1 the node's place in the element,
// then 5 bits per element node: its column's offset in the row, or kIncNone
constexpr int kIncNone = 31;
__host__ __device__ inline int inc_offset(int32_t meta, int j) { return (meta >> (2 + 5 * j)) & 31; }
void scan_exclusive_i64(const int64_t* d_in, int64_t* d_out, int64_t n);

// prec.cu
void prec_setup(ofg_prec* P);
// true when the solvers must set the preconditioner up again before use: the
// matrix values changed since, and the preconditioner is not frozen
inline bool prec_stale(const ofg_prec* P) { return !P->frozen && P->version != P->A->version; }
// z = M^{-1} r on device buffers (r and z may alias).  With rz != nullptr
// the sweep preconditioners also leave (r, z) in *rz (device scalar).  With
// skip != nullptr every launch is a no-op while *skip != 0.
void prec_apply_device(ofg_prec* P, const double* r, double* z, double* rz = nullptr,
                       const int* skip = nullptr);
void check_status(ofg_prec* P);

// The "value not ready yet" marker of the triangular sweeps: a NaN payload
// that IEEE arithmetic never produces (results are the canonical NaN).
constexpr unsigned long long kSentinelBits = 0x7FF4DEADBEEF0001ULL;
void fill_sentinel(double* p, int64_t n);

// wave.cu: the wavefront plan of a direction (chain: row rho depends on
// row rho - 1, logical order; tpos: transposed positions when a
// factorisation is wanted); false when the matrix has no such lines
bool wave_build(ofg_matrix* A, bool fwd, const int8_t* chain, const int32_t* tpos, WavePlan& p);
void wave_diagonal(ofg_prec* P, int invert, int* bad);  // P->pivot from the current diagonal
void wave_factor(ofg_prec* P);                // D-ILU pivots of the current values
void wave_values(ofg_prec* P, WavePlan& p);   // the plan's copy of values and pivots
void wave_solve(ofg_prec* P, bool fwd, const double* in, double* out, double* reset,
                const double* dot_with, double* dot_out, const int* skip);
void wave_repair(WavePlan& p);                // after a wait ran out

// learned.cu: run the network on the matrix's current values and rebuild
// G / G^T; z = G^T G r in FP64 (r and z may alias; rz as above when they
// do not)
void learned_setup(ofg_prec* P);
void learned_apply(ofg_prec* P, const double* r, double* z, double* rz, const int* skip);

}  // namespace ofg
