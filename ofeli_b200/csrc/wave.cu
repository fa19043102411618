// wave.cu -- triangular sweeps and the D-ILU factorisation on matrices whose
// rows form grid lines (structured meshes in natural order): a wavefront in
// one warp instead of a scan per 32 rows.
//
// A line is a maximal run of rows that each depend on the row just before.
// Up to 32 consecutive lines form a group, one lane a line; where the group's
// first line depends on the line before, lane 0 carries that one and 31 lines
// follow.  Lane l starts its line `shift` steps after
// lane l - 1, so that at every step the value a row needs from the previous
// line was computed one (slot A) or two (slot B) steps earlier by the
// neighbouring lane, and the value of the row before (slot L) one step
// earlier by the lane itself: a step is one shuffle and three multiply-adds,
// in the plain order of a serial substitution.  Entries of rows in earlier
// groups (slots E: the previous plane of a 3-D grid) are folded into the
// right-hand side by loader warps.
//
// What bounds it: the dependency chain, (columns + lines) steps and one
// hand-off per group.  A step's chain is a shuffle (24 cycles, measured) and
// three dependent FP64 operations (8 each); with the shared-memory traffic
// around it a step takes about 90 cycles (the sweep's time less the
// hand-offs).  A hand-off between SMs takes about 3000 (one-way latency 530
// to 1070, measured, plus the chunk it travels in).  At 2049^2 a solve sweep
// takes 294 us where the sweeps of prec.cu, which resolve 32 rows of a line
// by a scan, took 1040; the factorisation 0.56 instead of 13.4 ms.  On the
// 129^3 cube a sweep takes 365 instead of 530 us, the factorisation 0.44
// instead of 4.6 ms: there the chain is 127 planes of about 2.6 us, a chunk
// of steps and a trip through L2 each.
//
// One block works on a group at a time, its warps in roles:
//   * warp 0 computes, kWaveF steps (a chunk) at a time, from shared memory;
//   * warp 1 feeds: one bulk copy per tile of 32 steps brings the
//     coefficients, stored in the order the steps read them; without E slots
//     it also copies the right-hand side (cp.async, 8 bytes a row);
//   * warp 2 polls the line before the group (the previous group's last lane
//     stores it to `edge` as it goes) and hands it on as lane 0's right-hand
//     side;
//   * the next ones store the results and accumulate the dot product;
//   * with E slots, the last eight warps form the right-hand side: they wait
//     for the earlier groups' results (readiness travels with the data, as in
//     prec.cu), four lines each.
// Within the block, too, readiness travels with the data wherever the compute
// warp is involved: places in shared memory hold a sentinel until written.
// Groups are taken in order from a ticket counter, so whatever a block waits
// for belongs to a block that is already running.  Every wait is bounded.
#include <algorithm>
#include <climits>
#include <cstring>
#include <type_traits>

#include "internal.cuh"
#include "mbar.cuh"

namespace ofg {
namespace {

constexpr int kWaveF = 8;        // steps per chunk
constexpr int kWaveTile = 32;    // steps per tile, the unit of the bulk copies
constexpr int kTileChunks = kWaveTile / kWaveF;
constexpr int kWavePitch = 34;   // row pitch of the [step][lane] tiles: 8 steps x 2 lanes hit 16 banks once
constexpr int kWaveCPitch = 68;  // the same for the pairs of the right-hand side
constexpr int kExt = kWaveExt;
constexpr int kExtWarps = 8;
constexpr int kAuxAhead = 8;     // chunks the storing warps prefetch to L2
constexpr int kExtAhead = 8;     // chunks the loader warps prefetch to L2
constexpr unsigned long long kWaveLimitNs = 4000000000ull;

enum { W_FWD_DILU = 0, W_FWD_SSOR = 1, W_BWD_DILU = 2, W_BWD_SSOR = 3, W_FACTOR = 4 };

// tiles in shared memory (a power of two)
constexpr int wave_tiles(int mode) { return mode == W_FACTOR ? 2 : 4; }
constexpr bool wave_fwd(int mode) { return mode == W_FWD_DILU || mode == W_FWD_SSOR || mode == W_FACTOR; }
// doubles per step and lane of the coefficient stream
constexpr int wave_slots(int mode) { return mode == W_FACTOR ? 6 : 3; }
// warps that store the results: one beside the loader warps (12 warps in all:
// three per scheduler, 168 registers a thread), else four, one chunk of
// every tile each (with two, the divisions of SSOR's forward sweep held up
// the chain: 475 instead of 255 us at 2049^2)
constexpr int wave_stores(bool ext) { return ext ? 1 : 4; }
constexpr int wave_threads(bool ext) { return 32 * (ext ? 3 + wave_stores(ext) + kExtWarps : 8); }

struct WaveArgs {
   int64_t n;
   int ngroups;
   const int32_t* line;     // first logical row of every line, nlines + 1
   const int32_t* g_line;   // first line of every group, ngroups + 1
   const int32_t* shift;    // per line: its first step within the group
   const int32_t* g_tile;   // first layout tile of every group
   const int32_t* g_nch;    // chunks of kWaveF steps of every group
   const int32_t* g_edge;   // offset of the line before the group in `edge`, -1: none
   const int32_t* g_sm1;    // that line's shift (>= 0)
   const int32_t* eoff;     // per line: column - row (logical) of the E slots
   bool clean;              // see wave_build
   const double* coef;
   const double* ecoef;     // kExt arrays of n values, the sentinel where absent
   const double* ecoef_t;   // FACTOR: the transposed entries
   double* edge;
   const double* in;
   const double* piv;
   double* out;
   double* reset;
   const double* dot_with;
   double* gdot;
   double* dot_out;
   int* ticket;             // [0] next group, [1] finished partials, [2] finished blocks
   int* status;
   const int* skip;
   int* worked;
};

__device__ __forceinline__ bool wave_empty(double v)
{
   return (unsigned long long)__double_as_longlong(v) == kSentinelBits;
}
__device__ __forceinline__ double wave_sentinel() { return __longlong_as_double((long long)kSentinelBits); }
// a value that came in from outside: the sentinel's own bits become another NaN
__device__ __forceinline__ double wave_plain(double v)
{
   return wave_empty(v) ? __longlong_as_double(0x7FF8000000000000ll) : v;
}

__device__ __forceinline__ unsigned long long global_ns()
{
   unsigned long long t;
   asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
   return t;
}

__device__ __forceinline__ bool mbar_test(uint32_t addr, uint32_t phase)
{
   uint32_t done;
   asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}\n"
      : "=r"(done)
      : "r"(addr), "r"(phase)
      : "memory");
   return done;
}

// the same, suspending the thread for a while when the phase is not complete
// (a spinning warp would take load/store slots from the compute warp)
__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t phase)
{
   uint32_t done;
   asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}\n"
      : "=r"(done)
      : "r"(addr), "r"(phase)
      : "memory");
   return done;
}

__device__ __forceinline__ void mbar_arrive(uint32_t addr)
{
   asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(addr) : "memory");
}

// A wait gives up when another wait of the block gave up, or after
// kWaveLimitNs: it then sets the status and makes the block stop.
__device__ __forceinline__ bool wave_give_up(unsigned long long t0, volatile int* stop, int* status)
{
   if (*stop) return true;
   if (global_ns() - t0 <= kWaveLimitNs) return false;
   *stop = 1;
   atomicOr(status, 1);
   return true;
}

// (no function calls: they would constrain the compute warp's registers)
__device__ __forceinline__ bool wave_bar(uint32_t bar, uint32_t phase, volatile int* stop,
                                         int* status)
{
   if (mbar_test(bar, phase)) return true;
   const unsigned long long t0 = global_ns();
   for (;;) {
#pragma unroll 1
      for (int q = 0; q < 64; ++q)
         if (mbar_try(bar, phase)) return true;
      if (wave_give_up(t0, stop, status)) return false;
   }
}

__device__ __forceinline__ void prefetch_l2(const void* p)
{
   asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar)
{
   asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

// 8 bytes to shared memory, zeros when !valid
__device__ __forceinline__ void copy8(uint32_t dst, const double* src, bool valid)
{
   asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src),
                "r"(valid ? 8 : 0)
                : "memory");
}

template <int MODE>
struct WaveShared {
   static constexpr int NS = wave_slots(MODE), NT = wave_tiles(MODE);
   double coef[NT * kTileChunks][kWaveF * NS * 32];
   double c[NT * kTileChunks][kWaveF / 2 * kWaveCPitch];
   double z[NT * kTileChunks][kWaveF * kWavePitch];
   unsigned long long full[NT], empty[NT];
   int group, stop, unfed;  // unfed: tiles that a block that gave up left out
};

// Where chunk `ch` of a group lies in shared memory; tiles: those of the
// block's earlier groups
template <int MODE>
struct ChunkAt {
   int tile, slot;
   unsigned phase;
   __device__ __forceinline__ ChunkAt(unsigned tiles, int ch)
   {
      constexpr unsigned NT = wave_tiles(MODE);
      const unsigned t = tiles + (unsigned)ch / kTileChunks;
      tile = (int)(t % NT);
      phase = (t / NT) & 1u;
      slot = tile * kTileChunks + ch % kTileChunks;
   }
};

// The coefficients of a chunk of kWaveF steps, in the order and pairing the
// compute warp reads them with 16-byte loads.  Solve: (A, B) of every step,
// then L of two steps at a time.  Factorisation: (a, transposed a) of slots
// A, B and L of every step.
template <int MODE>
__host__ __device__ constexpr int coef_pos(int slot, int step, int lane)
{
   if (MODE == W_FACTOR) return ((step * 3 + slot % 3) * 32 + lane) * 2 + slot / 3;
   if (slot < 2) return (step * 32 + lane) * 2 + slot;
   return kWaveF * 64 + ((step >> 1) * 32 + lane) * 2 + (step & 1);
}
// the right-hand side, two steps a pair
__device__ __forceinline__ int c_pos(int step, int lane)
{
   return (step >> 1) * kWaveCPitch + lane * 2 + (step & 1);
}

// Operands in registers: the coefficients of the next kAhead steps, the
// right-hand sides of the chunk
constexpr int kAhead = 4;
template <int NS>
struct WaveOps {
   double a[kAhead][NS], c[kWaveF];
};

// One step of a line, in OFELI's order (columns ascending: B, A, then the row
// before).  The factorisation has its roundings, too.
template <int MODE>
__device__ __forceinline__ double wave_step(const double (&a)[wave_slots(MODE)], double c, double u1,
                                            double u2, double zl, bool act)
{
   if constexpr (MODE == W_FACTOR) {
      double s = __dsub_rn(c, __dmul_rn(__dmul_rn(a[1], u2), a[4]));
      s = __dsub_rn(s, __dmul_rn(__dmul_rn(a[0], u1), a[3]));
      s = __dsub_rn(s, __dmul_rn(__dmul_rn(a[2], zl), a[5]));
      // (the value hidden from the compiler, which else branches around the
      // division lane by lane: 190 instead of 360 cycles a step)
      double x = act ? s : 1.0;
      asm volatile("" : "+d"(x));
      return __drcp_rn(x);
   }
   else {
      (void)act;
      // (the sum in OFELI's order, columns ascending, then the difference:
      // c - B u2 - L z - A u1 in that order would be 10 % faster, but moved
      // BiCGStab + ILU on the 65^2 system from OFELI's 53 iterations to 58;
      // this form takes 54)
      double t = a[1] * u2;
      t = fma(a[0], u1, t);
      t = fma(a[2], zl, t);
      return c - t;
   }
}

// the coefficients of steps q and q + 1 (q even) of a chunk
template <int MODE>
__device__ __forceinline__ void load_coefs(const WaveShared<MODE>& sh, int slot, int q, int lane,
                                           WaveOps<wave_slots(MODE)>& o)
{
   auto pair = [&](int pos) { return *reinterpret_cast<const double2*>(&sh.coef[slot][pos]); };
   if constexpr (MODE == W_FACTOR) {
#pragma unroll
      for (int r = q; r < q + 2; ++r)
#pragma unroll
         for (int k = 0; k < 3; ++k) {
            const double2 v = pair(coef_pos<MODE>(k, r, lane));
            o.a[r % kAhead][k] = v.x;
            o.a[r % kAhead][k + 3] = v.y;
         }
   }
   else {
#pragma unroll
      for (int r = q; r < q + 2; ++r) {
         const double2 v = pair(coef_pos<MODE>(0, r, lane));
         o.a[r % kAhead][0] = v.x;
         o.a[r % kAhead][1] = v.y;
      }
      const double2 l = pair(coef_pos<MODE>(2, q, lane));
      o.a[q % kAhead][2] = l.x;
      o.a[(q + 1) % kAhead][2] = l.y;
   }
}

// the right-hand sides of steps q and q + 1 (q even); ordered by the waits
// around it only
template <int MODE>
__device__ __forceinline__ void load_rhs(const WaveShared<MODE>& sh, int slot, int q, int lane,
                                         double (&c)[kWaveF])
{
   asm volatile("ld.relaxed.cta.shared.v2.f64 {%0, %1}, [%2];"
                : "=d"(c[q]), "=d"(c[q + 1])
                : "r"(smem_u32(&sh.c[slot][c_pos(q, lane)])));
}

// What one lane (or the mapped line of a helper lane) needs to know of a line
struct LineInfo {
   int32_t start, len, shift;
};

__device__ __forceinline__ LineInfo wave_line(const WaveArgs& g, int l, int l0, int l1)
{
   LineInfo i{0, 0, 0};
   if (l >= l0 && l < l1) {
      i.start = g.line[l];
      i.len = g.line[l + 1] - i.start;
      i.shift = g.shift[l];
   }
   return i;
}

// (ordered among themselves only: the waits around them order the rest)
__device__ __forceinline__ void st_shared(double* p, double v)
{
   asm volatile("st.relaxed.cta.shared.f64 [%0], %1;" ::"r"(smem_u32(p)), "d"(v));
}
__device__ __forceinline__ double ld_shared(const double* p)
{
   double v;
   asm volatile("ld.relaxed.cta.shared.f64 %0, [%1];" : "=d"(v) : "r"(smem_u32(p)));
   return v;
}
__device__ __forceinline__ void st_edge(double* p, double v)
{
   asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v));
}

// the largest exponent word of four values
__device__ __forceinline__ int max4(double a, double b, double c, double d)
{
   auto hi = [](double v) { return __double2hiint(v) & 0x7fffffff; };
   return max(max(hi(a), hi(b)), max(hi(c), hi(d)));
}

// some right-hand side of the chunk is not finite (the sentinel is a NaN)
__device__ __forceinline__ bool any_special(const double (&c)[kWaveF])
{
   const int m = max(max4(c[0], c[1], c[2], c[3]), max4(c[4], c[5], c[6], c[7]));
   return __any_sync(0xffffffffu, m >= 0x7ff00000);
}

// The compute warp's state across steps
template <int NS>
struct WaveRun {
   WaveOps<NS> op;
   double z, u1, u2;  // own last result; the neighbour's last two
   bool go;   // the next chunk's operands are loaded and finite
};

// The steps of one chunk (`slot`; `nx`: the next one).  FAST: no right-hand
// side is special, and a lane whose line is not active, has no line, or (lane
// 0) carries the line before the group as its right-hand side computes like
// any other: its coefficients are 0, so the result is the right-hand side, as
// long as the values it sees are finite (wave_build says where that holds).
// The coefficients are read kAhead steps ahead and the next chunk's
// right-hand sides and readiness early in this one, so that the chunks follow
// each other without a wait.
template <int MODE, bool EXT, bool FAST>
__device__ __forceinline__ void wave_steps(WaveShared<MODE>& sh, int slot, int next, bool same_tile,
                                           uint32_t next_bar, unsigned next_phase, bool next_ok,
                                           int j0, int len, int lane, bool carry,
                                           double* edge_out,
                                           WaveRun<wave_slots(MODE)>& R)
{
   double cn[kWaveF];
   bool have = same_tile, special = false;
   int m = 0;
#pragma unroll
   for (int s = 0; s < kWaveF; ++s) {
      const bool act = (unsigned)(j0 + s) < (unsigned)len;
      double zn = wave_step<MODE>(R.op.a[s % kAhead], R.op.c[s], R.u1, R.u2, R.z, act);
      if (!FAST && !act) zn = 0.0;
      if ((!FAST || MODE == W_FACTOR) && carry) zn = R.op.c[s];
      R.z = zn;
      R.u2 = R.u1;
      // (first of the step's shared-memory operations: the next step waits for it)
      R.u1 = __shfl_up_sync(0xffffffffu, zn, 1);
      st_shared(&sh.z[slot][s * kWavePitch + lane], zn);
      if (edge_out && act) st_edge(edge_out + s, zn);
      if (s & 1) {
         const int q = s - 1 + kAhead;
         load_coefs<MODE>(sh, q < kWaveF ? slot : next, q % kWaveF, lane, R.op);
      }
      if (s == 0 && !same_tile) have = mbar_test(next_bar, next_phase);
      if (s < 4) load_rhs<MODE>(sh, next, 2 * s, lane, cn);
      // spread over the steps, so that no step waits for it
      if (s == 4) m = max4(cn[0], cn[1], cn[2], cn[3]);
      if (s == 5) m = max(m, max4(cn[4], cn[5], cn[6], cn[7]));
      if (s == 6) special = __any_sync(0xffffffffu, m >= 0x7ff00000);
      // (one answer for the warp, of the lanes' own tests of the barrier; its
      // place measured, us per CG + ILU iteration at 512^2 and 63^3: without a
      // vote 166.0 and 328.2, after step 1 167.6 and 330, 2 167.8 and 331, 3
      // 167.6 and 331, 5 166.4 and 330, 7 170.0 and 328.4, within the vote on
      // special values 168.5 and 330; set-up with the factorisation at 2047^2:
      // without 1042, after step 1 to 5 1078, 1058, 1075, 1051, 1076, 6 1050,
      // 7 1053)
      if (s == (EXT ? 7 : MODE == W_FACTOR ? 6 : 5)) have = __all_sync(0xffffffffu, have);
   }
   R.go = next_ok && have && !special;
#pragma unroll
   for (int q = 0; q < kWaveF; ++q) R.op.c[q] = cn[q];
}

// All chunks of a group.  The operands of the next chunk are read whether or
// not they have arrived, since a branch per step costs more: when they had
// not, they are waited for and read again.  The warp signals nothing: the
// storing warps see its results arrive (the z tile holds the sentinel
// before), which also tells that the operands of those steps are free; a
// barrier arrival with its fence costs 100 to 200 cycles a chunk.
// lo, hi: the steps in which the fast form may be used.  The right-hand sides
// of lane 0 where it carries a line, with E slots those of all lanes, arrive
// on their own, the sentinel in their places until then; the others come with
// the tile, whatever bits they hold.
template <int MODE, bool EXT>
__device__ __forceinline__ void wave_compute(WaveShared<MODE>& sh, int* status, unsigned tiles,
                                             int nch, int lane, bool carry, const LineInfo& li,
                                             double* edge_out, int lo, int hi)
{
   WaveRun<wave_slots(MODE)> R;
   R.z = R.u1 = R.u2 = 0.0;
   R.go = false;
   bool special = false;  // the chunk before had a right-hand side that is not finite
   // one chunk's steps
   auto steps = [&](auto fast, int ch) {
      const ChunkAt<MODE> at(tiles, ch), nx(tiles, ch + 1);
      const int t0 = ch * kWaveF;
      wave_steps<MODE, EXT, decltype(fast)::value>(
         sh, at.slot, nx.slot, nx.tile == at.tile, smem_u32(&sh.full[nx.tile]), nx.phase,
         ch + 1 < nch && t0 + kWaveF >= lo && t0 + 2 * kWaveF <= hi && !special, t0 - li.shift,
         li.len, lane, carry, edge_out ? edge_out + t0 : nullptr, R);
   };
   int ch = 0;
#pragma unroll 1
   while (ch < nch) {
      const ChunkAt<MODE> at(tiles, ch);
      wave_bar(smem_u32(&sh.full[at.tile]), at.phase, &sh.stop, status);
#pragma unroll
      for (int q = 0; q < kAhead; q += 2) load_coefs<MODE>(sh, at.slot, q, lane, R.op);
      const unsigned long long w0 = global_ns();
      for (unsigned spins = 1;; ++spins) {
#pragma unroll
         for (int q = 0; q < kWaveF; q += 2) load_rhs<MODE>(sh, at.slot, q, lane, R.op.c);
         bool missing = false;
#pragma unroll
         for (int q = 0; q < kWaveF; ++q) missing = missing || wave_empty(R.op.c[q]);
         if (!__any_sync(0xffffffffu, (EXT || carry) && missing)) break;
         if ((spins & 255u) == 0 && __any_sync(0xffffffffu, wave_give_up(w0, &sh.stop, status)))
            break;
      }
      const bool was = special;
      special = any_special(R.op.c);
      const int t0 = ch * kWaveF;
      if (special || was || t0 < lo || t0 + kWaveF > hi) {
         steps(std::false_type(), ch++);
         R.go = false;
         continue;
      }
      // the common case, a loop of its own (its instructions stay together)
#pragma unroll 1
      do steps(std::true_type(), ch++);
      while (R.go);
   }
}

template <int MODE, bool EXT>
__global__ void __launch_bounds__(wave_threads(EXT), 1) wave_sweep(WaveArgs g)
{
   constexpr bool FWD = wave_fwd(MODE);
   constexpr int NS = wave_slots(MODE), NST = wave_stores(EXT);
   using Sh = WaveShared<MODE>;
   extern __shared__ __align__(128) unsigned char wave_raw[];
   Sh& sh = *reinterpret_cast<Sh*>(wave_raw);
   const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
   const int n = (int)g.n;
   if (threadIdx.x == 0) {
      for (int s = 0; s < Sh::NT; ++s) {
         // full: the bulk copy's announcing arrival and, without loader
         // warps, the right-hand side (every lane of warp 1)
         asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&sh.full[s])),
                      "r"(1 + (EXT ? 0 : 32)));
         asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&sh.empty[s])),
                      "r"(NST));
      }
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      sh.stop = 0;
      sh.unfed = 0;
   }
   for (int i = threadIdx.x; i < Sh::NT * kTileChunks * kWaveF * kWavePitch; i += blockDim.x)
      (&sh.z[0][0])[i] = wave_sentinel();
   for (int i = threadIdx.x; i < Sh::NT * kTileChunks * kWaveF / 2 * kWaveCPitch; i += blockDim.x)
      (&sh.c[0][0])[i] = wave_sentinel();
   // the kernel before may still be running up to here (programmatic dependent
   // launch); the next one may set itself up from here on, when every block
   // of this grid has started
   pdl_wait();
   pdl_release();
   if (g.skip && *g.skip) return;
   prof_mark(g.worked);
   unsigned tiles = 0;  // of the groups before this one: place and phase of every role
   for (;;) {
      __syncthreads();
      if (threadIdx.x == 0) {
         int t = g.ngroups;
         if (!sh.stop && !*(volatile int*)g.status) t = atomicAdd(&g.ticket[0], 1);
         sh.group = t;
      }
      __syncthreads();
      const int grp = sh.group;
      if (grp >= g.ngroups) break;
      const int l0 = g.g_line[grp], l1 = g.g_line[grp + 1];
      const int tile0 = g.g_tile[grp];
      const int nch = g.g_nch[grp];
      const int ein = g.g_edge[grp];
      const int plen = ein >= 0 ? g.line[l0] - g.line[l0 - 1] : 0;
      const int sm1 = g.g_sm1[grp];
      const int first = ein >= 0 ? 1 : 0;  // lane of the group's first line
      const int ntile = (nch + kTileChunks - 1) / kTileChunks;

      if (w == 0) {
         // ------------------------------------------------------- compute
         const LineInfo li = wave_line(g, l0 + lane - first, l0, l1);
         // the group's last line goes on to the next group, entry j at step j + shift
         const int eo = grp + 1 < g.ngroups ? g.g_edge[grp + 1] : -1;
         double* edge_out = eo >= 0 && lane == l1 - l0 - 1 + first ? g.edge + eo - li.shift : nullptr;
         // fast steps: all, or those in which every line is active
         const int lo = g.clean ? 0 : __reduce_max_sync(0xffffffffu, li.shift);
         const int hi = g.clean ? INT_MAX
                                : __reduce_min_sync(0xffffffffu, li.len ? li.shift + li.len : INT_MAX);
         wave_compute<MODE, EXT>(sh, g.status, tiles, nch, lane, first && lane == 0, li, edge_out, lo,
                                 hi);
      }
      else if (w == 1) {
         // ---------------------------------------------------------- feed
         LineInfo li[8];
         if (!EXT) {
#pragma unroll
            for (int q = 0; q < 8; ++q) li[q] = wave_line(g, l0 + 4 * q + (lane >> 3) - first, l0, l1);
         }
         for (int tl = 0; tl < ntile; ++tl) {
            const ChunkAt<MODE> at(tiles, tl * kTileChunks);
            // (one answer for the warp: a tile's copies are issued by all
            // lanes or none)
            if (tiles + tl >= Sh::NT &&
                !__all_sync(0xffffffffu, wave_bar(smem_u32(&sh.empty[at.tile]), at.phase ^ 1u,
                                                  &sh.stop, g.status))) {
               if (lane == 0) sh.unfed = ntile - tl;
               break;
            }
            const uint32_t bar = smem_u32(&sh.full[at.tile]);
            if (lane == 0) {
               constexpr uint32_t bytes = kWaveTile * NS * 32 * sizeof(double);
               mbar_expect_tx(bar, bytes);
               bulk_load(smem_u32(&sh.coef[at.slot][0]),
                         g.coef + (size_t)(tile0 + tl) * kWaveTile * NS * 32, bytes, bar);
            }
            if (!EXT) {
               const int tt = lane & 7;
#pragma unroll 1
               // (no chunk past the group's: nothing would clear lane 0's
               // places there, and where the block's next group hands a line
               // to lane 0 they must read as not written yet)
               for (int cc = 0; cc < kTileChunks && tl * kTileChunks + cc < nch; ++cc) {
                  const int t = (tl * kTileChunks + cc) * kWaveF + tt;
#pragma unroll
                  for (int q = 0; q < 8; ++q) {
                     const int j = t - li[q].shift;
                     const bool valid = (unsigned)j < (unsigned)li[q].len;
                     const int rho = li[q].start + (valid ? j : 0);
                     if (4 * q + (lane >> 3) >= first)
                        copy8(smem_u32(&sh.c[at.slot + cc][c_pos(tt, 4 * q + (lane >> 3))]),
                              g.in + (FWD ? rho : n - 1 - rho), valid);
                  }
               }
               asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar)
                            : "memory");
            }
         }
      }
      else if (w == 2) {
         // ---------------------------------------- the line before the group
         // lane 0's right-hand side at step t: entry t - sm1 of that line,
         // zero outside it
         double* src = g.edge + (first ? ein : 0);
         for (int tl = 0; first && tl < ntile; ++tl) {
            const ChunkAt<MODE> at(tiles, tl * kTileChunks);
            // (one answer for the warp: the polls below are votes)
            if (tiles + tl >= Sh::NT &&
                !__all_sync(0xffffffffu, wave_bar(smem_u32(&sh.empty[at.tile]), at.phase ^ 1u,
                                                  &sh.stop, g.status)))
               break;
            const int i = tl * kWaveTile + lane - sm1;
            // (past the group's chunks nothing clears the place again)
            const bool there = tl * kWaveTile + lane < nch * kWaveF;
            double* dst = &sh.c[at.slot + (lane >> 3)][c_pos(lane & 7, 0)];
            bool todo = there && (unsigned)i < (unsigned)plen;
            if (there && !todo) st_shared(dst, 0.0);
            const unsigned long long w0 = global_ns();
            for (unsigned spins = 1; __any_sync(0xffffffffu, todo); ++spins) {
               if (todo) {
                  const double v = ld_relaxed(src + i);
                  if (!wave_empty(v)) {
                     st_shared(dst, v);
                     src[i] = wave_sentinel();  // for the next sweep
                     todo = false;
                  }
               }
               if ((spins & 255u) == 0 &&
                   __any_sync(0xffffffffu, wave_give_up(w0, &sh.stop, g.status)))
                  break;
            }
         }
      }
      else if (EXT ? w < 3 + NST : w != 4) {
         // --------------------------------------------------------- results
         // (without E slots warp 4 stays idle: it would share warp 0's scheduler)
         const int f = w == 3 ? 0 : w - 4, tt = lane & 7;
         LineInfo li[8];
#pragma unroll
         for (int q = 0; q < 8; ++q) li[q] = wave_line(g, l0 + 4 * q + (lane >> 3) - first, l0, l1);
         // per row: the pivot that scales the result (forward: see wave_fill),
         // or the row's entry of dot_with
         const double* aux = FWD ? (MODE == W_FACTOR || EXT ? nullptr : g.piv) : g.dot_with;
         double dot = 0.0, dw[8];
         auto fetch = [&](int ch) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
               const int j = ch * kWaveF + tt - li[q].shift;
               dw[q] = FWD ? 1.0 : 0.0;
               if (ch < nch && (unsigned)j < (unsigned)li[q].len) {
                  const int rho = li[q].start + j;
                  dw[q] = aux[FWD ? rho : n - 1 - rho];
               }
            }
         };
         // the rows of a chunk some way ahead, into L2 (one lane a sector)
         auto prefetch = [&](int ch) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
               const int j = ch * kWaveF + tt - li[q].shift;
               if ((tt & 3) == 0 && (unsigned)j < (unsigned)li[q].len) {
                  const int rho = li[q].start + j;
                  prefetch_l2(aux + (FWD ? rho : n - 1 - rho));
               }
            }
         };
         if (aux) {
            for (int ch = f + NST; ch < f + kAuxAhead; ch += NST) prefetch(ch);
            fetch(f);
         }
         // (every warp walks whole tiles, so that each arrives on `empty`)
         for (int ch = f; ch < ntile * kTileChunks; ch += NST) {
            const ChunkAt<MODE> at(tiles, ch);
            if (ch < nch) {
               if (aux) prefetch(ch + kAuxAhead);
               const int t = ch * kWaveF + tt;
               double* zt = &sh.z[at.slot][tt * kWavePitch + (lane >> 3)];
               double zv[8];
               const unsigned long long w0 = global_ns();
               for (unsigned spins = 1;; ++spins) {
                  // the last step first: one load a poll
                  bool ok = !wave_empty(ld_shared(&sh.z[at.slot][(kWaveF - 1) * kWavePitch + lane]));
                  ok = __all_sync(0xffffffffu, ok);
                  if (ok) {
#pragma unroll
                     for (int q = 0; q < 8; ++q) {
                        zv[q] = ld_shared(zt + 4 * q);
                        ok = ok && !wave_empty(zv[q]);
                     }
                     if (__all_sync(0xffffffffu, ok)) break;
                  }
                  else if (!EXT) __nanosleep(64);
                  if ((spins & 63u) == 0 &&
                      __any_sync(0xffffffffu, wave_give_up(w0, &sh.stop, g.status)))
                     break;
               }
#pragma unroll
               for (int q = 0; q < 8; ++q) {
                  const int j = t - li[q].shift;
                  if ((unsigned)j < (unsigned)li[q].len) {
                     const int rho = li[q].start + j;
                     const int row = FWD ? rho : n - 1 - rho;
                     double v = zv[q];
                     if (MODE == W_FWD_DILU && !EXT) v *= dw[q];
                     if (MODE == W_FWD_SSOR && !EXT) v /= dw[q];
                     if (EXT) st_relaxed(g.out + row, v);
                     else g.out[row] = v;
                     if (g.reset) g.reset[row] = wave_sentinel();
                  }
               }
               // the chunk's places are free again
#pragma unroll
               for (int q = 0; q < 8; ++q) st_shared(zt + 4 * q, wave_sentinel());
               if (EXT) {
#pragma unroll
                  for (int q = 0; q < 8; ++q)
                     st_shared(&sh.c[at.slot][c_pos(tt, 4 * q + (lane >> 3))], wave_sentinel());
               }
               else if (lane < kWaveF) {
                  st_shared(&sh.c[at.slot][c_pos(lane, 0)], wave_sentinel());
               }
               if (!FWD && aux) {
                  // (inactive rows: 0 * 0)
#pragma unroll
                  for (int q = 0; q < 8; ++q) dot += dw[q] * zv[q];
               }
               if (aux) fetch(ch + NST);
            }
            if (ch % kTileChunks >= kTileChunks - NST) {
               __syncwarp();
               if (lane == 0) mbar_arrive(smem_u32(&sh.empty[at.tile]));
            }
         }
         if (!FWD && aux) {
            dot = warp_sum(dot);
            int fin = 0;
            if (lane == 0) {
               g.gdot[NST * grp + f] = dot;
               __threadfence();
               fin = atomicAdd(&g.ticket[1], 1) == NST * g.ngroups - 1;
            }
            fin = __shfl_sync(0xffffffffu, fin, 0);
            if (fin) {
               __threadfence();
               double acc = 0.0;
               for (int q = lane; q < NST * g.ngroups; q += 32) acc += ld_relaxed(g.gdot + q);
               acc = warp_sum(acc);
               if (lane == 0) *g.dot_out = acc;
            }
         }
      }
      else if (EXT) {
         // ------------------------------------ right-hand side with E slots
         // four lines a warp, eight steps of each
         const int tt = lane & 7, ln = 4 * (w - 3 - NST) + (lane >> 3);
         const LineInfo li = wave_line(g, l0 + ln - first, l0, l1);
         int32_t off[kExt];
#pragma unroll
         for (int k = 0; k < kExt; ++k) off[k] = li.len ? g.eoff[(l0 + ln - first) * kExt + k] : 0;
         struct {
            double a[kExt], at[kExt], b, pv;
         } r;
         auto row_of = [&](int ch, int& row) {
            const int j = ch * kWaveF + tt - li.shift;
            const int rho = li.start + j;
            row = FWD ? rho : n - 1 - rho;
            return (unsigned)j < (unsigned)li.len;
         };
         auto fetch = [&](int ch) {
            r.b = MODE == W_FACTOR ? 1.0 : 0.0;
            r.pv = 1.0;
#pragma unroll
            for (int k = 0; k < kExt; ++k) r.a[k] = wave_sentinel();
            int row;
            if (ch >= nch || !row_of(ch, row)) return;
            r.b = g.in[row];
            if (!FWD) r.pv = g.piv[row];
#pragma unroll
            for (int k = 0; k < kExt; ++k) {
               r.a[k] = g.ecoef[(size_t)k * g.n + row];
               if (MODE == W_FACTOR) r.at[k] = g.ecoef_t[(size_t)k * g.n + row];
            }
         };
         // what fetch reads kExtAhead chunks later, into L2 (one lane a sector)
         auto prefetch = [&](int ch) {
            int row;
            if ((tt & 3) || !row_of(ch, row)) return;
            prefetch_l2(g.in + row);
            if (!FWD) prefetch_l2(g.piv + row);
#pragma unroll
            for (int k = 0; k < kExt; ++k) {
               prefetch_l2(g.ecoef + (size_t)k * g.n + row);
               if (MODE == W_FACTOR) prefetch_l2(g.ecoef_t + (size_t)k * g.n + row);
            }
         };
         for (int ch = 1; ch < kExtAhead; ++ch) prefetch(ch);
         fetch(0);
         for (int ch = 0; ch < nch; ++ch) {
            prefetch(ch + kExtAhead);
            const ChunkAt<MODE> at(tiles, ch);
            if (ch % kTileChunks == 0 && tiles + ch / kTileChunks >= Sh::NT &&
                !wave_bar(smem_u32(&sh.empty[at.tile]), at.phase ^ 1u, &sh.stop, g.status))
               break;
            const int rho = li.start + ch * kWaveF + tt - li.shift;
            const double* src[kExt];
            double v[kExt];
            unsigned pend = 0;
#pragma unroll
            for (int k = 0; k < kExt; ++k) {
               const int c = rho + off[k];
               src[k] = g.out + (FWD ? c : n - 1 - c);
               v[k] = 0.0;
               if (!wave_empty(r.a[k])) pend |= 1u << k;
            }
            double c = FWD ? wave_plain(r.b) : r.b;   // (backward it is multiplied first)
            const unsigned long long w0 = global_ns();
            for (unsigned spins = 1; pend; ++spins) {
#pragma unroll
               for (int k = 0; k < kExt; ++k)
                  if ((pend >> k) & 1) v[k] = ld_relaxed(src[k]);
#pragma unroll
               for (int k = 0; k < kExt; ++k)
                  if (!wave_empty(v[k])) pend &= ~(1u << k);
               if ((spins & 255u) == 0 && wave_give_up(w0, &sh.stop, g.status)) break;
            }
            if (MODE == W_FACTOR) {
#pragma unroll
               for (int k = 0; k < kExt; ++k)
                  if (!wave_empty(r.a[k]))
                     c = __dsub_rn(c, __dmul_rn(__dmul_rn(r.a[k], v[k]), r.at[k]));
            }
            else {
               // backward, `in` is the forward sweep's y: t = p y
               if (MODE == W_BWD_DILU) c = r.pv * c;
               if (MODE == W_BWD_SSOR) c = c / r.pv;
#pragma unroll
               for (int k = 0; k < kExt; ++k)
                  if (!wave_empty(r.a[k])) c = fma(-r.a[k], v[k], c);
            }
            if (ln >= first) st_shared(&sh.c[at.slot][c_pos(tt, ln)], c);
            fetch(ch + 1);
         }
      }
      tiles += ntile;
   }
   // a block that gave up may have copies in flight into its shared memory,
   // which has to stay until they have arrived: the last tiles fed (one a
   // place of the ring) are waited for, with a limit
   if (w == 1 && sh.stop) {
      const unsigned fed = tiles - sh.unfed;
      const unsigned long long t0 = global_ns();
      for (unsigned t = fed > Sh::NT ? fed - Sh::NT : 0; t < fed; ++t)
         while (!mbar_test(smem_u32(&sh.full[t % Sh::NT]), (t / Sh::NT) & 1u) &&
                global_ns() - t0 <= kWaveLimitNs) {
         }
   }
   if (threadIdx.x == 0) {
      __threadfence();
      if (atomicAdd(&g.ticket[2], 1) == (int)gridDim.x - 1) {
         g.ticket[0] = 0;
         g.ticket[1] = 0;
         g.ticket[2] = 0;
      }
   }
}

// -------------------------------------------------------------- the plan --
// lower entries (logical order) of a row: CSR range and logical column
struct Lower {
   const int32_t *rp, *col, *dpos;
   int64_t n;
   bool fwd;
   __device__ int64_t row(int64_t rho) const { return fwd ? rho : n - 1 - rho; }
   __device__ void range(int64_t row, int32_t& kb, int32_t& ke) const
   {
      if (fwd) { kb = rp[row]; ke = dpos[row]; }
      else { kb = dpos[row] + 1; ke = rp[row + 1]; }
   }
   __device__ int32_t lcol(int32_t k) const { return fwd ? col[k] : (int32_t)n - 1 - col[k]; }
};

// One warp per line: the range of (position in the previous line) - (own
// position) over the couplings to the line before, the highest row needed
// from other lines, the distinct offsets of those (kExt at most).  *bad: a
// row depends on a row of its own line other than the one before, too many
// offsets.
__global__ void wave_line_stats(Lower a, int nlines, const int32_t* __restrict__ line,
                                int32_t* dmin, int32_t* dmax, int32_t* emax, int32_t* eoff,
                                int* bad)
{
   const int l = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
   const int lane = threadIdx.x & 31;
   if (l >= nlines) return;
   const int32_t beg = line[l], end = line[l + 1], pbeg = l > 0 ? line[l - 1] : beg;
   int32_t lo = INT_MAX, hi = INT_MIN, em = -1;
   for (int32_t rho = beg + lane; rho < end; rho += 32) {
      int32_t kb, ke;
      a.range(a.row(rho), kb, ke);
      for (int32_t k = kb; k < ke; ++k) {
         const int32_t c = a.lcol(k);
         if (c >= beg) {
            if (c != rho - 1) atomicOr(bad, 1);
         }
         else if (c >= pbeg) {
            const int32_t d = (c - pbeg) - (rho - beg);
            lo = min(lo, d);
            hi = max(hi, d);
         }
         else {
            em = max(em, c);
            const int32_t off = c - rho;
            bool found = false;
            for (int q = 0; q < kExt && !found; ++q) {
               int32_t cur = __ldcg(eoff + (size_t)l * kExt + q);
               if (cur == 0) cur = atomicCAS(eoff + (size_t)l * kExt + q, 0, off);
               found = cur == 0 || cur == off;
            }
            if (!found) atomicOr(bad, 2);
         }
      }
   }
   lo = __reduce_min_sync(0xffffffffu, lo);
   hi = __reduce_max_sync(0xffffffffu, hi);
   em = __reduce_max_sync(0xffffffffu, em);
   if (lane == 0) {
      dmin[l] = lo;
      dmax[l] = hi;
      emax[l] = em;
   }
}

// One warp per line: slot A must be present exactly where the neighbouring
// lane is active one step earlier, slot B where it is two steps earlier, so
// that a coefficient stored as 0 only ever meets a lane that holds 0.
__global__ void wave_verify(Lower a, int nlines, const int32_t* __restrict__ line,
                            const int32_t* __restrict__ dshift, int* bad)
{
   const int l = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
   const int lane = threadIdx.x & 31;
   if (l >= nlines) return;
   const int32_t beg = line[l], end = line[l + 1], pbeg = l > 0 ? line[l - 1] : beg;
   const int32_t ds = dshift[l];  // shift(l) - shift(l - 1); INT_MIN: not coupled
   if (ds == INT_MIN) return;
   for (int32_t rho = beg + lane; rho < end; rho += 32) {
      int32_t kb, ke;
      a.range(a.row(rho), kb, ke);
      int na = 0, nb = 0;
      bool wrong = false;
      for (int32_t k = kb; k < ke; ++k) {
         const int32_t c = a.lcol(k);
         if (c >= beg || c < pbeg) continue;
         const int32_t delta = (rho - beg) + ds - (c - pbeg);  // steps between the two rows
         if (delta == 1) ++na;
         else if (delta == 2) ++nb;
         else wrong = true;
      }
      const int32_t i1 = (rho - beg) + ds - 1, plen = beg - pbeg;
      if (wrong || na != (i1 >= 0 && i1 < plen) || nb != (i1 >= 1 && i1 - 1 < plen))
         atomicOr(bad, 4);
   }
}

struct FillArgs {
   Lower a;
   const int32_t *sp, *scol;  // the SELL copy: entry k of a row at sell_at(row, k)
   const double* sval;
   const int32_t* stpos;    // FACTOR: transposed positions (CSR) in SELL order
   const double* val;       // FACTOR: the CSR values
   const int32_t* tile_g;   // group of every layout tile
   const int32_t *g_line, *g_tile, *g_edge, *line, *shift, *dshift, *eoff;
   const double* piv;       // solve: inverse pivots, or (ssor) the diagonal
   bool ssor;
   double* coef;
   double* ecoef;           // null without E slots
   double* ecoef_t;
   double* diag;            // FACTOR: the diagonal, natural order
};

// entry k (in CSR order) of a row in the SELL-32 copy
__device__ __forceinline__ int64_t sell_at(const int32_t* sp, int64_t row, int k)
{
   return sp[row >> 5] + 32 * (int64_t)k + (row & 31);
}

// Forward, a sweep solves for y = D t (t_i = p_i y_i, p the inverse pivots),
//    y_i = b_i - sum a_ij p_j y_j,
// and the storing warps scale; backward, z_i = t_i - sum (p_i a_ij) z_j.  The
// products a p (SSOR: quotients a / d) are formed here, once per set of
// values, so that a step of the sweep has no multiplication or division by
// the pivot on its chain.
//
// The coefficients in step order: one block per tile of 32 steps; the rows
// are read along the lines and turned through shared memory, so that the
// writes are coalesced.  The factorisation reads its entries, the diagonal
// and the transposed positions from the SELL copy (447 -> 243 us at 129^3,
// 240 -> 190 at 2049^2 against the CSR rows); the solve's triangle is read
// from the CSR rows (at 129^3 125 us, 145 from the SELL copy).
template <bool FAC>
__global__ void __launch_bounds__(256) wave_fill(FillArgs f)
{
   constexpr int NS = FAC ? 6 : 3, H = FAC ? 3 : 0;
   extern __shared__ double fill_tile[];  // [NS][kWaveTile][33]
   auto at = [&](int k, int step, int ln) -> double& {
      return fill_tile[(k * kWaveTile + step) * 33 + ln];
   };
   const int t = blockIdx.x, g = f.tile_g[t];
   const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
   const int l0 = f.g_line[g], l1 = f.g_line[g + 1];
   const int first = f.g_edge[g] >= 0 ? 1 : 0;  // lane of the group's first line
   const int step = (t - f.g_tile[g]) * kWaveTile + lane;
   for (int ln = w; ln < 32; ln += 8) {
      double s[NS];
#pragma unroll
      for (int k = 0; k < NS; ++k) s[k] = 0.0;
      const int l = l0 + ln - first;
      if (l >= l0 && l < l1) {
         const int32_t beg = f.line[l], len = f.line[l + 1] - beg;
         const int32_t pbeg = l > 0 ? f.line[l - 1] : beg;
         const int32_t ds = f.dshift[l];
         const int j = step - f.shift[l];
         if ((unsigned)j < (unsigned)len) {
            const int32_t rho = beg + j;
            const int64_t row = f.a.row(rho);
            int32_t kb, ke;
            f.a.range(row, kb, ke);
            const int32_t r0 = FAC ? f.a.rp[row] : 0;
            if (FAC) f.diag[row] = f.sval[sell_at(f.sp, row, f.a.dpos[row] - r0)];
            const double own = FAC ? 1.0 : f.piv[row];
            double e[kExt], et[kExt];
#pragma unroll
            for (int q = 0; q < kExt; ++q) e[q] = et[q] = wave_sentinel();
            for (int32_t k = kb; k < ke; ++k) {
               const int64_t at = FAC ? sell_at(f.sp, row, k - r0) : k;
               const int32_t pc = FAC ? f.scol[at] : f.a.col[at];
               const int32_t c = f.a.fwd ? pc : (int32_t)f.a.n - 1 - pc;
               const double v = FAC ? f.sval[at] : f.val[at];
               const double vt = FAC ? f.val[f.stpos[at]] : 0.0;
               double vs = v;
               if (!FAC) {
                  const double p = f.a.fwd ? f.piv[pc] : own;
                  vs = f.ssor ? v / p : v * p;
               }
               if (c >= beg) {
                  s[2] = vs;
                  if (FAC) s[2 + H] = vt;
               }
               else if (c >= pbeg) {
                  // computed one step before this row (A) or two (B)
                  if (j + ds - (c - pbeg) == 1) {
                     s[0] = vs;
                     if (FAC) s[0 + H] = vt;
                  }
                  else {
                     s[1] = vs;
                     if (FAC) s[1 + H] = vt;
                  }
               }
               else {
#pragma unroll
                  for (int q = 0; q < kExt; ++q)
                     if (f.eoff[(size_t)l * kExt + q] == c - rho) {
                        e[q] = wave_plain(vs);
                        et[q] = vt;
                     }
               }
            }
            if (f.ecoef) {
#pragma unroll
               for (int q = 0; q < kExt; ++q) {
                  f.ecoef[(size_t)q * f.a.n + row] = e[q];
                  if (FAC) f.ecoef_t[(size_t)q * f.a.n + row] = et[q];
               }
            }
         }
      }
#pragma unroll
      for (int k = 0; k < NS; ++k) at(k, lane, ln) = s[k];
   }
   __syncthreads();
   constexpr int M = FAC ? W_FACTOR : W_FWD_DILU;  // the layout's mode
   double* dst = f.coef + (size_t)t * kWaveTile * NS * 32;
   for (int i = threadIdx.x; i < kWaveTile * NS * 32; i += 256) {
      const int chunk = i / (kWaveF * NS * 32), p = i % (kWaveF * NS * 32);
      // the inverse of coef_pos
      int k, st;
      const int ln = (p >> 1) & 31, half = p & 1, row = p >> 6;
      if (M == W_FACTOR) { k = row % 3 + 3 * half; st = row / 3; }
      else if (row < kWaveF) { k = half; st = row; }
      else { k = 2; st = (row - kWaveF) * 2 + half; }
      dst[i] = at(k, chunk * kWaveF + st, ln);
   }
}

// the transposed positions in SELL order (-1: none or padding)
__global__ void sell_transposed(int64_t total, const int32_t* ssrc, const int32_t* tpos, int32_t* out)
{
   int64_t stride = (int64_t)gridDim.x * blockDim.x;
   for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride)
      out[i] = ssrc[i] >= 0 ? tpos[ssrc[i]] : -1;
}

// The diagonal (or its inverses) from the SELL copy; the lowest row with a
// zero in *bad
__global__ void wave_diag(int64_t n, const int32_t* rp, const int32_t* dpos, const int32_t* sp,
                          const double* sval, double* piv, int invert, int* bad)
{
   int64_t stride = (int64_t)gridDim.x * blockDim.x;
   for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
      const double a = sval[sell_at(sp, i, dpos[i] - rp[i])];
      if (a == 0.0) atomicMin(bad, (int)i);
      piv[i] = invert ? 1.0 / a : a;
   }
}

// tpos of every strictly lower entry present?
__global__ void wave_transposed(int64_t n, const int32_t* rp, const int32_t* dpos,
                                const int32_t* tpos, int* bad)
{
   int64_t stride = (int64_t)gridDim.x * blockDim.x;
   for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride)
      for (int32_t k = rp[r]; k < dpos[r]; ++k)
         if (tpos[k] < 0) atomicOr(bad, 8);
}

template <int MODE, bool EXT>
void launch_wave(const WaveArgs& g)
{
   const size_t smem = sizeof(WaveShared<MODE>);
   // (cheap, and must hold on every device the caller selects)
   OFG_CUDA(cudaFuncSetAttribute(wave_sweep<MODE, EXT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
   const int blocks = std::min(g.ngroups, num_sms());
   launch_pdl_smem(wave_sweep<MODE, EXT>, (unsigned)blocks, (unsigned)wave_threads(EXT), smem, g);
}

template <int MODE>
void launch_wave(const WavePlan& p, const WaveArgs& g)
{
   if (p.ext) launch_wave<MODE, true>(g);
   else launch_wave<MODE, false>(g);
}

Lower lower_of(const ofg_matrix* A, bool fwd)
{
   return Lower{A->row_ptr.p, A->col.p, A->dpos.p, A->n, fwd};
}

FillArgs fill_args(const ofg_matrix* A, const WavePlan& p)
{
   FillArgs f{};
   f.a = lower_of(A, p.fwd);
   f.val = A->val.p;
   f.sp = A->sell_ptr.p;
   f.scol = A->sell_col.p;
   f.sval = A->sell_val.p;
   f.stpos = p.stpos.p;
   f.tile_g = p.tile_g.p;
   f.g_line = p.g_line.p;
   f.g_tile = p.g_tile.p;
   f.g_edge = p.g_edge.p;
   f.line = p.line.p;
   f.shift = p.shift.p;
   f.dshift = p.dshift.p;
   f.eoff = p.eoff.p;
   f.ecoef = p.ext ? p.ecoef.p : nullptr;
   return f;
}

template <bool FAC>
void launch_fill(const WavePlan& p, const FillArgs& f)
{
   const size_t smem = sizeof(double) * (FAC ? 6 : 3) * kWaveTile * 33;
   OFG_CUDA(cudaFuncSetAttribute(wave_fill<FAC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
   wave_fill<FAC><<<(unsigned)p.tiles, 256, smem, stream()>>>(f);
   count_launch();
   OFG_LAUNCH_CHECK();
}

WaveArgs wave_args(const ofg_prec* P, const WavePlan& p)
{
   WaveArgs g{};
   g.n = P->A->n;
   g.ngroups = p.ngroups;
   g.line = p.line.p;
   g.g_line = p.g_line.p;
   g.shift = p.shift.p;
   g.g_tile = p.g_tile.p;
   g.g_nch = p.g_nch.p;
   g.g_edge = p.g_edge.p;
   g.g_sm1 = p.g_sm1.p;
   g.eoff = p.eoff.p;
   g.clean = p.clean;
   g.coef = p.coef.p;
   g.ecoef = p.ecoef.p;
   g.edge = p.edge.p;
   g.piv = P->pivot.p;
   g.gdot = p.gdot.p;
   g.ticket = p.ticket.p;
   g.status = P->status.p;
   return g;
}

}  // namespace

bool wave_build(ofg_matrix* A, bool fwd, const int8_t* chain, const int32_t* tpos, WavePlan& p)
{
   const int64_t n = A->n;
   p.fwd = fwd;
   if (n < 1) return false;
   std::vector<int32_t> line(1, 0);
   for (const int8_t* q = chain + 1; (q = (const int8_t*)std::memchr(q, 0, chain + n - q)); ++q) {
      line.push_back((int32_t)(q - chain));
      if ((int64_t)line.size() * kWaveMinLine > n + kWaveMinLine) return false;
   }
   line.push_back((int32_t)n);
   const int nl = (int)line.size() - 1;
   p.line.alloc(line.size());
   p.line.upload(line.data(), line.size());
   const Lower low = lower_of(A, fwd);
   DBuf<int32_t> dmin(nl), dmax(nl), emax(nl);
   DBuf<int> bad(1);
   bad.zero();
   p.eoff.alloc((size_t)nl * kExt);
   p.eoff.zero();
   const unsigned wgrid = (unsigned)(((int64_t)nl * 32 + 255) / 256);
   wave_line_stats<<<wgrid, 256, 0, stream()>>>(low, nl, p.line.p, dmin.p, dmax.p, emax.p, p.eoff.p,
                                                bad.p);
   count_launch();
   OFG_LAUNCH_CHECK();
   if (tpos && fwd) {
      wave_transposed<<<grid_for(n, 256), 256, 0, stream()>>>(n, A->row_ptr.p, A->dpos.p, tpos,
                                                              bad.p);
      count_launch();
      OFG_LAUNCH_CHECK();
   }
   if (bad.to_host(1)[0]) return false;
   std::vector<int32_t> hmin = dmin.to_host(nl), hmax = dmax.to_host(nl), hem = emax.to_host(nl),
                        heo = p.eoff.to_host((size_t)nl * kExt);
   std::vector<int32_t> g_line, g_tile, g_nch, g_edge, g_sm1, tile_g, shift(nl), dshift(nl);
   p.ext = false;
   p.clean = true;
   for (int l = 0; l < nl; ++l) {
      auto* e = &heo[(size_t)l * kExt];
      // ascending columns, unused slots (0) last
      std::sort(e, e + kExt);
      if (e[0]) p.ext = true;
   }
   int64_t edge = 0, steps = 0;
   int g0 = 0, room = 32;
   auto close = [&](int l1) {
      if (l1 == g0) return;
      int32_t m = 0;
      for (int l = g0; l < l1; ++l) m = std::min(m, shift[l]);
      int64_t T = 0;
      for (int l = g0; l < l1; ++l) {
         shift[l] -= m;
         T = std::max<int64_t>(T, (int64_t)shift[l] + (line[l + 1] - line[l]));
      }
      g_sm1.back() -= m;
      const int64_t tiles = (T + kWaveTile - 1) / kWaveTile;
      g_nch.push_back((int32_t)((T + kWaveF - 1) / kWaveF));
      for (int64_t t = 0; t < tiles; ++t) tile_g.push_back((int32_t)g_line.size() - 1);
      steps += T;
   };
   for (int l = 0; l < nl; ++l) {
      const bool coupled = hmin[l] != INT_MAX;
      if (coupled && (hmax[l] - hmin[l] > 1 || hmax[l] > (1 << 20) || hmin[l] < -(1 << 20)))
         return false;
      const int eline =
         hem[l] < 0 ? -1 : (int)(std::upper_bound(line.begin(), line.end(), hem[l]) - line.begin()) - 1;
      dshift[l] = coupled ? hmax[l] + 1 : INT_MIN;
      // clean: a lane that is not active never sees an active lane's values in
      // a way that reaches an active row (equal lines, one step apart: before
      // its start the neighbour has not started either, and after its end only
      // lanes that have ended read it), so that no value, finite or not, needs
      // masking outside the lines
      if (coupled && (dshift[l] != 1 || line[l + 1] - line[l] != line[l] - line[l - 1])) p.clean = false;
      if (l == 0 || l == g0 + room || !coupled || eline >= g0) {
         close(l);
         g0 = l;
         room = coupled ? 31 : 32;
         g_line.push_back(l);
         g_tile.push_back((int32_t)tile_g.size());
         if (coupled) {
            g_edge.push_back((int32_t)edge);
            edge += line[l] - line[l - 1];
            shift[l] = dshift[l];
         }
         else {
            g_edge.push_back(-1);
            shift[l] = 0;
         }
         g_sm1.push_back(0);
      }
      else {
         shift[l] = shift[l - 1] + dshift[l];
      }
      // (a group's padding must stay a fraction of its rows: see the mean below)
      if (std::abs(shift[l]) > (1 << 24)) return false;
   }
   close(nl);
   g_line.push_back(nl);
   const int64_t tiles = (int64_t)tile_g.size();
   if (n < kWaveMinLanes * steps || tiles * kWaveTile * 32 * 4 > INT_MAX) return false;
   if (p.ext) {
      // see kWaveLongLine
      const double planes = (double)std::count(g_edge.begin(), g_edge.end(), -1);
      const double rows = (double)n / nl, lines = nl / planes;
      if (rows * rows * planes > kWaveLongLine * lines * lines) return false;
   }
   p.ngroups = (int)g_line.size() - 1;
   p.tiles = tiles;
   auto put = [&](DBuf<int32_t>& d, const std::vector<int32_t>& h) {
      d.alloc(h.size());
      d.upload(h.data(), h.size());
   };
   put(p.g_line, g_line);
   put(p.g_tile, g_tile);
   put(p.g_nch, g_nch);
   put(p.g_edge, g_edge);
   put(p.g_sm1, g_sm1);
   put(p.tile_g, tile_g);
   put(p.shift, shift);
   put(p.dshift, dshift);
   p.eoff.upload(heo.data(), heo.size());
   wave_verify<<<wgrid, 256, 0, stream()>>>(low, nl, p.line.p, p.dshift.p, bad.p);
   count_launch();
   OFG_LAUNCH_CHECK();
   if (bad.to_host(1)[0]) return false;
   if (tpos) {
      ensure_sell(A);
      const int64_t total = (int64_t)A->sell_val.n;
      p.stpos.alloc(total);
      sell_transposed<<<grid_for(total, 256), 256, 0, stream()>>>(total, A->sell_src.p, tpos,
                                                                   p.stpos.p);
      count_launch();
      OFG_LAUNCH_CHECK();
   }
   p.edge.alloc(edge > 0 ? edge : 1);
   fill_sentinel(p.edge.p, (int64_t)p.edge.n);
   p.coef.alloc((size_t)tiles * kWaveTile * 3 * 32);
   p.ecoef.alloc(p.ext ? (size_t)kExt * n : 1);
   p.gdot.alloc(4 * (size_t)p.ngroups);
   p.ticket.alloc(4);
   p.ticket.zero();
   OFG_CUDA(cudaStreamSynchronize(stream()));
   p.on = true;
   return true;
}

void wave_diagonal(ofg_prec* P, int invert, int* bad)
{
   const ofg_matrix* A = P->A;
   wave_diag<<<grid_for(A->n, 256), 256, 0, stream()>>>(A->n, A->row_ptr.p, A->dpos.p, A->sell_ptr.p,
                                                        A->sell_val.p, P->pivot.p, invert, bad);
   count_launch();
   OFG_LAUNCH_CHECK();
}

void wave_factor(ofg_prec* P)
{
   const ofg_matrix* A = P->A;
   const WavePlan& p = P->wfwd;
   const int64_t n = A->n;
   DBuf<double> coef((size_t)p.tiles * kWaveTile * 6 * 32), et(p.ext ? (size_t)kExt * n : 1), dg(n);
   FillArgs f = fill_args(A, p);
   f.coef = coef.p;
   f.ecoef_t = et.p;
   f.diag = dg.p;
   launch_fill<true>(p, f);
   if (p.ext) fill_sentinel(P->pivot.p, n);
   WaveArgs g = wave_args(P, p);
   g.coef = coef.p;
   g.ecoef_t = et.p;
   g.in = dg.p;
   g.out = P->pivot.p;
   g.worked = prof_begin();
   launch_wave<W_FACTOR>(p, g);
   prof_end(PROF_SWEEP, 0.0);
}

void wave_values(ofg_prec* P, WavePlan& p)
{
   FillArgs f = fill_args(P->A, p);
   f.coef = p.coef.p;
   f.piv = P->pivot.p;
   f.ssor = P->type == OFG_SSOR;
   launch_fill<false>(p, f);
}

void wave_solve(ofg_prec* P, bool fwd, const double* in, double* out, double* reset,
                const double* dot_with, double* dot_out, const int* skip)
{
   const WavePlan& p = fwd ? P->wfwd : P->wbwd;
   WaveArgs g = wave_args(P, p);
   g.in = in;
   g.out = out;
   g.reset = reset;
   g.dot_with = dot_with;
   g.dot_out = dot_out;
   g.skip = skip;
   g.worked = prof_begin();
   const bool dilu = P->type != OFG_SSOR;
   if (fwd) {
      if (dilu) launch_wave<W_FWD_DILU>(p, g);
      else launch_wave<W_FWD_SSOR>(p, g);
   }
   else {
      if (dilu) launch_wave<W_BWD_DILU>(p, g);
      else launch_wave<W_BWD_SSOR>(p, g);
   }
   // one triangle (FP64 value + column in the CSR's terms), pivots, input, output
   const ofg_matrix* A = P->A;
   prof_end(PROF_SWEEP, 6.0 * (double)(A->nnz - A->n) + 32.0 * (double)A->n);
}

void wave_repair(WavePlan& p)
{
   if (!p.on) return;
   fill_sentinel(p.edge.p, (int64_t)p.edge.n);
   p.ticket.zero();
}

}  // namespace ofg
