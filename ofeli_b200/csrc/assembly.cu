// assembly.cu -- Equation::build() for P1 elements on the device.
//
// One thread per mesh node gathers the CSR row of the node's equation and its
// RHS entry: it zeroes the row, then walks the node's elements in ascending
// element number (the node-to-element lists are sorted), computes each
// element's matrix and RHS in registers (FP64, the same formulas as
// Triang3/Tetra4 and the element classes, imposed values lifted as
// Equation::updateBC does) and adds the element row into its own CSR row and
// RHS entry.  Every matrix entry and RHS entry therefore receives its element
// contributions in OFELI's element-loop order, starting from zero, so the
// assembled values are the reference's bit for bit on any mesh; a thread
// writes only its own row, so there are no atomics and no element colouring.
// Each node computes only its own row of an element (geometry is recomputed
// by each of the element's 3 or 4 nodes; the FP64 arithmetic is cheap beside
// the gathers).  An element's Jacobian is checked by
// the thread of its first node, equation or not, and the lowest bad element
// is reported as OFELI's element loop would meet it first.
//
// Algorithmic bytes per launch: node-to-element lists 4*(nn+1) + 4*nen*ne,
// connectivity 4*nen*ne, coordinates 8*dim*nn, code and equation number
// 8*nn, the element-to-CSR map 4*nen^2*ne, the node fields read
// (f, or u_old and v) 8*nn each, k 8*ne when given, CSR row pointers
// 4*(n+1), A written 8*nnz,
// b written 8*n.
#include "element.cuh"

namespace ofg {
namespace {

using namespace elem;

// One thread per node: the node's CSR row and RHS entry, gathered over its
// elements in ascending order (see the file comment).
template <class Elem>
__global__ void __launch_bounds__(256) assemble_rows(int64_t nn, const int32_t* __restrict__ n2e_ptr,
                                                     const int32_t* __restrict__ n2e,
                                                     const int32_t* __restrict__ elem,
                                                     const int32_t* __restrict__ dof,
                                                     const int32_t* __restrict__ emap,
                                                     const int32_t* __restrict__ row_ptr, Elem el,
                                                     double* __restrict__ a, double* __restrict__ b,
                                                     unsigned* bad)
{
   // each thread sums its row in shared memory (a column per thread)
   __shared__ double racc[kRowAcc * 256];
   int64_t stride = (int64_t)gridDim.x * blockDim.x;
   for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += stride) {
      const int32_t r = dof[i];   // 1-based equation, 0 for an imposed node
      const double bi =
         gather_node_rows(i, r, n2e_ptr[i], n2e_ptr[i + 1], n2e, elem, emap, row_ptr, el, a,
                          [&](int64_t e) { atomicMin(bad, (unsigned)e); }, racc + threadIdx.x, 256);
      if (r) b[r - 1] = bi;
   }
}

// The same over the incidence records of the matrix: what a node needs of an
// element (number, other nodes, the columns' places in its row) as one
// 16-byte record (3-D: and a word), the records of 32 nodes side by side, so
// that a warp streams them in whole lines.  The lists, the connectivity and
// the element-to-CSR map above are three dependent gathers of 4-byte words
// (L1 at 50 to 92 % of its rate); here only the other nodes' coordinates and
// fields are gathered.
template <class Elem>
__global__ void __launch_bounds__(256) assemble_incidences(
   int64_t nn, const int32_t* __restrict__ inc_ptr, const int4* __restrict__ inc,
   const int32_t* __restrict__ inc_meta, const int32_t* __restrict__ dof,
   const int32_t* __restrict__ row_ptr, Elem el, double* __restrict__ a, double* __restrict__ b,
   unsigned* bad)
{
   constexpr int NEN = Elem::NEN;
   __shared__ double racc_all[kRowAcc * 256];
   double* racc = racc_all + threadIdx.x;  // entry j at racc[256 j]
   const int64_t stride = (int64_t)gridDim.x * blockDim.x;
   for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += stride) {
      const int64_t s = i >> 5;
      const int32_t beg = inc_ptr[s], w = inc_ptr[s + 1] - beg;
      const int64_t at = (int64_t)beg * 32 + (i & 31);
      const int32_t r = dof[i];   // 1-based equation, 0 for an imposed node
      int32_t rs = 0, rl = 0;
      if (r) {
         rs = row_ptr[r - 1];
         rl = row_ptr[r] - rs;
         for (int32_t j = 0; j < rl; ++j) racc[j * 256] = 0.0;
      }
      Corners<NEN, Elem::DIM> own;
      own.load(0, el.coords(), i);
      double bi = 0.0;
      int4 next = w > 0 ? inc[at] : make_int4(-1, 0, 0, 0);
      int32_t next_meta = NEN == 4 && w > 0 ? inc_meta[at] : 0;
      for (int32_t p = 0; p < w; ++p) {
         const int4 rec = next;
         const int32_t meta = NEN == 3 ? rec.w : next_meta;
         if (p + 1 < w) {
            next = inc[at + (int64_t)(p + 1) * 32];
            if (NEN == 4) next_meta = inc_meta[at + (int64_t)(p + 1) * 32];
         }
         if (rec.x < 0) break;   // the node's last element was the one before
         const int li = meta & 3;
         // the element's nodes in its own order: the node itself at place li
         const int32_t other[3] = {rec.y, rec.z, rec.w};
         int32_t en[NEN];
         Corners<NEN, Elem::DIM> X, O;
#pragma unroll
         for (int k = 0; k < NEN - 1; ++k) O.load(k, el.coords(), other[k]);
#pragma unroll
         for (int j = 0; j < NEN; ++j) {
            const int hi = j < NEN - 1 ? j : NEN - 2, lo = j > 0 ? j - 1 : 0;
            en[j] = j == li ? (int32_t)i : j < li ? other[hi] : other[lo];
#pragma unroll
            for (int d = 0; d < Elem::DIM; ++d)
               X.x[j][d] = j == li ? own.x[0][d] : j < li ? O.x[hi][d] : O.x[lo][d];
         }
         if (!r) {   // no row here: only the Jacobian check of the elements it leads
            if (li == 0 && !el.geometry_ok(X)) atomicMin(bad, (unsigned)rec.x);
            continue;
         }
         int32_t off[NEN];
#pragma unroll
         for (int j = 0; j < NEN; ++j) {
            off[j] = inc_offset(meta, j);
            if (off[j] == kIncNone) off[j] = -1;
         }
         double krow[NEN], frow;
         if (!el.row(rec.x, X, en, li, i, off, krow, frow)) {
            if (li == 0) atomicMin(bad, (unsigned)rec.x);
            continue;
         }
#pragma unroll
         for (int j = 0; j < NEN; ++j)
            if (off[j] >= 0) racc[off[j] * 256] += krow[j];
         bi += frow;
      }
      if (r) {
         for (int32_t j = 0; j < rl; ++j) a[rs + j] = racc[j * 256];
         b[r - 1] = bi;
      }
   }
}

void check_jacobian(const DBuf<unsigned>& bad)
{
   unsigned h = 0;
   bad.download(&h, 1);
   if (h != 0xffffffffu)
      throw Error(OFG_ERR_JACOBIAN,
                  "non-positive Jacobian determinant in element " + std::to_string((int64_t)h + 1));
}

// Launches the row-gather kernel for one element kind and checks Jacobians.
template <class Elem>
void assemble(ofg_mesh* m, ofg_matrix* A, const Elem& el, double* db, int node_fields,
              int elem_fields)
{
   OFG_REQUIRE(A->mesh == m, OFG_ERR_ARG, "matrix pattern was not built from this mesh");
   DBuf<unsigned> bad(1);   // lowest bad element; all ones: none
   OFG_CUDA(cudaMemsetAsync(bad.p, 0xFF, sizeof(unsigned), stream()));
   if (m->nn) {
      const int nen = m->nen;
      // records, or node-to-element lists, connectivity and element-to-CSR map
      const double lists = A->inc_on ? (nen == 3 ? 16.0 : 20.0) * nen * m->ne
                                     : 4.0 * (m->nn + 1) + 8.0 * nen * m->ne + 4.0 * nen * nen * m->ne;
      double bytes = lists + 8.0 * m->dim * m->nn + 8.0 * m->nn + 8.0 * node_fields * m->nn +
                     8.0 * elem_fields * m->ne + 4.0 * (A->n + 1) +
                     8.0 * A->nnz + 8.0 * A->n;
      int* worked = prof_begin();
      if (worked) OFG_CUDA(cudaMemsetAsync(worked, 1, sizeof(int), stream()));
      const unsigned grid = grid_for(m->nn, 256, 16);
      if (A->inc_on)
         assemble_incidences<Elem><<<grid, 256, 0, stream()>>>(
            m->nn, A->inc_ptr.p, A->inc.p, A->inc_meta.p, m->dof.p, A->row_ptr.p, el, A->val.p, db,
            bad.p);
      else
         assemble_rows<Elem><<<grid, 256, 0, stream()>>>(
            m->nn, m->n2e_ptr.p, m->n2e.p, m->elem.p, m->dof.p, A->emap.p, A->row_ptr.p, el,
            A->val.p, db, bad.p);
      prof_end(PROF_ASSEMBLY, bytes);
      count_launch();
      OFG_LAUNCH_CHECK();
   }
   matrix_touch(A);
   check_jacobian(bad);
}

__global__ void insert_bc_kernel(int64_t nn, const int32_t* code, const int32_t* dof,
                                 const double* x, const double* bc, double* u)
{
   int64_t stride = (int64_t)gridDim.x * blockDim.x;
   for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += stride)
      u[i] = code[i] == 0 ? x[dof[i] - 1] : (bc ? bc[i] : 0.0);
}

}  // namespace

}  // namespace ofg

using namespace ofg;

extern "C" {

int ofg_assemble_p1(ofg_mesh* m, ofg_matrix* A, const double* kel, const double* f,
                    const double* bc, double* b)
{
   return guarded("ofg_assemble_p1", [&] {
      OFG_REQUIRE(m && A && b, OFG_ERR_ARG, "null argument");
      In<double> dk(kel, m->ne), df(f, m->nn), dbc(bc, m->nn);
      InOut<double> db(b, A->n, false);
      if (m->dim == 2)
         assemble(m, A, LaplaceT3{m->coords.p, m->code.p, dk.d, df.d, dbc.d}, db.d, f ? 1 : 0,
                  kel ? 1 : 0);
      else
         assemble(m, A, DiffusionT4{m->coords.p, m->code.p, dk.d, df.d, dbc.d}, db.d, f ? 1 : 0,
                  kel ? 1 : 0);
      db.finish();
   });
}

int ofg_assemble_cd2d_scheme(ofg_mesh* m, ofg_matrix* A, double eps, const double* v, double dt,
                             int scheme, const double* u_old, const double* bc, double* b)
{
   return guarded("ofg_assemble_cd2d_scheme", [&] {
      OFG_REQUIRE(m && A && b && v && u_old, OFG_ERR_ARG, "null argument");
      OFG_REQUIRE(m->dim == 2, OFG_ERR_ARG, "DC2DT3 needs a 2-D mesh");
      OFG_REQUIRE(dt > 0, OFG_ERR_ARG, "time step must be positive");
      OFG_REQUIRE(scheme == 1 || scheme == 2 || scheme == 3, OFG_ERR_ARG,
                  "scheme must be FORWARD_EULER (1), BACKWARD_EULER (2) or CRANK_NICOLSON (3)");
      In<double> dv(v, 2 * m->nn), du(u_old, m->nn), dbc(bc, m->nn);
      InOut<double> db(b, A->n, false);
      assemble(m, A, ConvDiffT3{m->coords.p, m->code.p, eps, 1. / dt, dv.d, du.d, dbc.d, scheme},
               db.d, 3, 0);
      db.finish();
   });
}

int ofg_assemble_cd2d(ofg_mesh* m, ofg_matrix* A, double eps, const double* v, double dt,
                      const double* u_old, const double* bc, double* b)
{
   return ofg_assemble_cd2d_scheme(m, A, eps, v, dt, 2, u_old, bc, b);
}

int ofg_insert_bc(const ofg_mesh* m, const double* x, const double* bc, double* u)
{
   return guarded("ofg_insert_bc", [&] {
      OFG_REQUIRE(m && x && u, OFG_ERR_ARG, "null argument");
      In<double> dx(x, m->neq), dbc(bc, m->nn);
      InOut<double> du(u, m->nn, false);
      insert_bc_kernel<<<grid_for(m->nn, 256), 256, 0, stream()>>>(m->nn, m->code.p, m->dof.p, dx.d,
                                                                    dbc.d, du.d);
      count_launch();
      OFG_LAUNCH_CHECK();
      du.finish();
   });
}

}  // extern "C"
