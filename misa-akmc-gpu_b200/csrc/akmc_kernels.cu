// akmc_kernels.cu -- sm_100a kernels of the vacancy-hop path.
//
// One sector round of the synchronous sublattice (src/algorithms/sl/sublattice.inl:64-177)
// runs as three launches:
//   k_bucket   one thread per vacancy: find its domain block, keep it if it lies in
//              the block's active sector, append it to the block's list;
//   k_hop      one CTA per active block: stage the sector plus a 2-cell halo (occupancy
//              bytes and the int32 density cache) into shared memory and run the hop
//              loop there.  EAM: all warps form the terms that a vacancy's 8 jumps share, two sum
//              the jumps; pair bond: a warp evaluates a vacancy.  Every warp forms the ordered
//              total and selects for itself, and the hop's updates are spread over the warps; each
//              hop writes its two occupancy bytes and 78 densities through to global memory (one
//              pair-bond vacancy: its path's sites, when its loop ends);
//   k_finalize one thread per block: clock of blocks without vacancies, next round.
// Concurrently active sectors are at least 4 cells apart, so the staged regions of
// different blocks never overlap and no atomics are needed on the lattice.
#include <cuda_runtime.h>

#include <cfloat>
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <type_traits>
#include <utility>

#include "akmc_device.h"

namespace akmc {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kStageRows = 4;  // rows of the staged region each warp has in flight
// CTAs that look after a block at a time: a sweep visits at most nblocks * kSweepWatch / CTAs blocks (and one
// per thread).  More only makes the visits wait on one another: with every thread of every CTA visiting, a
// context of a few hundred blocks had each of its round words read hundreds of thousands of times a sweep.
// 512 rounds of 180 blocks: 23.5 ms so, 11.7 with 16, 11.8 with 8, 13.1 with 4 (then blocks wait for a visit:
// 56 and 113 ms with 2 and 1); 4096 blocks: the same from 8 on.  With cheaper visits (flow_ready) 8, 16 and 32
// are within 1%.
constexpr int kSweepWatch = 16;
// Nanoseconds a k_flow CTA sleeps after a sweep that moved no block on (0: none).
#ifndef AKMC_SWEEP_SLEEP_NS
#define AKMC_SWEEP_SLEEP_NS 256
#endif
enum : int { kPairBond = 0, kEam64 = 1, kEam32 = 2 };  // energy kinds, one kernel instance each
// CTA shape: W warps.  EAM: all of them form a vacancy's dE terms (Geometry::foot_*, 256 lanes' worth),
// two sum its 8 jumps, and the hop's other work (write-through, ordered list, clock, random draws) is spread
// over the rest.  Pair bond: one warp evaluates a vacancy.  The hop kernels are built for W = 8 and W = 4;
// a context picks one (akmc_context_config).  One 8-warp CTA per SM: a hop is a chain of dependent
// instructions, so its latency is what counts, and two CTAs per SM (128 registers a thread instead of 255,
// so spills in the loop, and the other CTA's sweeps and hops on the same issue slots) measured slower: 40.6
// against 33.5 ms for 1024 rounds of the 256^3 lattice end to end, 30.2 against 27.7 ms for 256 rounds of
// 512 boxes.  Two CTAs of W = 4 (255 registers again) are within a few per cent of that where every SM has
// rounds to run (512 boxes in 16-cell blocks: 48.5 against 47.9 M hops/s), and a third slower along a chain
// (128 rounds of one block: 13.0 against 9.6 ms), so 8 is what a context gets that does not ask.
template <int W>
struct Shape {
  static_assert(8 % W == 0, "whole jump directions per warp");
  static constexpr int kEvalWarps = W;
  static constexpr int kJumpsPerWarp = 8 / W;
  static constexpr int kThreads = 32 * W;
  static constexpr int kCtl = 32 * (W - 1);  // control thread: first lane of the last warp, which also draws ahead
  static constexpr int kClk = W == 8 ? 192 : 96;  // the thread that runs the sector's clock
  static constexpr int kOrdWarp = W == 8 ? 4 : 3;  // the warp that keeps the ordered list
  static constexpr int kCtasPerSm = W <= 4 ? 2 : 1;
};
// The shape's constants under their short names inside a kernel or device function of shape W.
#define AKMC_SHAPE(W)                                         \
  constexpr int kEvalWarps = Shape<W>::kEvalWarps;            \
  constexpr int kJumpsPerWarp = Shape<W>::kJumpsPerWarp;      \
  constexpr int kThreads = Shape<W>::kThreads;                \
  constexpr int kCtl = Shape<W>::kCtl;                        \
  (void)kEvalWarps;                                           \
  (void)kJumpsPerWarp;                                        \
  (void)kThreads;                                             \
  (void)kCtl

__device__ __forceinline__ int wrap1(int v, int m) { return v < 0 ? v + m : (v >= m ? v - m : v); }

// Reference rank split: block k of n cells over p blocks starts at k (n/p) + min(k, n%p).
__device__ __forceinline__ int block_of(int c, int n, int p) {
  const int q = n / p, r = n % p;
  const int big = r * (q + 1);
  return c < big ? c / (q + 1) : r + (c - big) / q;
}

struct Region {
  int slo[3], w[3];
  int ox, oy, oz;  // origin in sites (x doubled); may be negative (periodic wrap)
  int LX, LY, LZ, n;  // row pitch in sites and rows of the shared layout, its sites
  int LXt, xo, nt;    // region row width, its first site within the pitch, sites staged
  int ey, ez;         // rows of the region in y and z (LY, LZ: the pitch, the job's box with tma)
  int tma;            // staged by one tensor copy per array
  int hx;             // cells before the sector in x within the pitch (the 2-cell halo, plus xo / 2)
  int bulk;           // rows staged by 16-byte copies: bo occupancy bytes and br densities each
  int bo, br;
};

// The staged region of a block's sector: the sector and a 2-cell halo.  With J.bulk (shared memory sized for
// the wider rows) each row's span is rounded out to 16-site boundaries from its unwrapped origin R.ox (which may
// lie before the row or run past its end: the sector never wraps, its halo may; the row's halo entries hold the
// sites past either end), so that copies of 16 bytes start on 16-byte boundaries in both arrays.
__device__ __forceinline__ void make_region(const int32_t (&c0)[3], const int32_t (&c1)[3], const JobDev& J, int sec,
                                            Region& R) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int half = (c1[d] - c0[d]) / 2;
    if ((sec >> d) & 1) {
      R.slo[d] = c0[d] + half;
      R.w[d] = c1[d] - c0[d] - half;
    } else {
      R.slo[d] = c0[d];
      R.w[d] = half;
    }
  }
  R.ox = 2 * (R.slo[0] - 2);
  R.oy = R.slo[1] - 2;
  R.oz = R.slo[2] - 2;
  R.LX = 2 * (R.w[0] + 4);
  R.LY = R.w[1] + 4;
  R.LZ = R.w[2] + 4;
  R.LXt = R.LX;
  R.xo = 0;
  R.bulk = 0;
  R.bo = R.br = 0;
  if (J.bulk) {
    const int x0 = R.ox & ~15;  // rounds down, negative origins included
    const int xo = R.ox - x0;
    const int bo = (xo + R.LXt + 15) & ~15;
    // the span [x0, x0 + bo) lies inside the row and its halo (always, for blocks of >= 8 cells:
    // x0 >= -16 and x0 + bo <= sx + 19)
    if (x0 >= -kHaloL && x0 + bo <= J.sx + kHaloR) {
      R.xo = xo;
      R.ox = x0;
      R.LX = (R.LXt + 14 + 15) & ~15;  // one pitch for every alignment: tables stay valid
      R.bo = bo;
      R.br = (xo + R.LXt + 3) & ~3;
      R.bulk = 1;
    }
  }
  R.ey = R.LY;
  R.ez = R.LZ;
  R.tma = 0;
  if (R.bulk && J.tma) {
    // every region of the job takes the box as its pitch (the shell tables stay valid across
    // them); one that does not wrap in y or z is one box of the lattice
    R.LX = J.tbox[0];
    R.LY = J.tbox[1];
    R.LZ = J.tbox[2];
    R.tma = R.oy >= 0 && R.oy + R.ey <= J.sy && R.oz >= 0 && R.oz + R.ez <= J.sz;
  }
  R.hx = R.slo[0] - R.ox / 2;
  R.n = R.LX * R.LY * R.LZ;
  R.nt = R.tma ? R.n : R.LXt * R.ey * R.ez;
}

// Rounds with vacancies a CTA can take in one sweep (a sweep finds a few).
constexpr int kMaxTake = 16;
// A block's round handed to the CTA with what the block record holds for it: read by the thread that took the
// block (k_flow's sweep), in flight together, so that the CTA itself waits for no record.
struct alignas(16) Round {
  int64_t r, t;        // the round and the launch's target
  int64_t hops;        // the block's hops so far
  double evo;          // the active sector's clock
  uint64_t str[2][4];  // selection and residence-time streams
  int32_t gb, job, local;
  int32_t c0[3], c1[3];  // block cells
};
constexpr int kTermSets = 2;
constexpr int kZeroTerm = kTermSlots - 2;  // a term that is always 0
constexpr int kTrashTerm = kTermSlots - 1;  // written by the evaluations that belong to no term, never read
// A lane's share of the dE terms (Geometry::foot_*): its site's local offset by x parity of the vacancy, the
// terms its two F evaluations give, their shell pairs and density changes for a moving Fe atom.
struct alignas(16) Slot {
  int32_t off[2];
  int32_t tA, tB;  // kTrashTerm: none
  int32_t hA, hB;
  int32_t dA, dB;
};
// Draws of the two random streams made ahead of their use: a ring of two batches.
constexpr int kDrawBatch = 8, kDrawRing = 2 * kDrawBatch;

// Shared-memory working set of one CTA (followed by the staged region).
struct Smem {
  double e0[9];                   // migration energy prefactor by the moving atom's code
  double b1[9 * 5], b2[9 * 5];    // pair-bond energies by the neighbour's code and the source's bond index
  union {                       // phi_XY(shell s) - phi_XY(shell t), index (X*4+Y)*64 + s*8 + t,
    double dphi64[4 * 4 * 64];  // in the precision of the kernel's kind
    float dphi32[4 * 4 * 64];
  };
  int32_t dfq[4 * 64];          // f_X(shell s) - f_X(shell t) in Q.24, index X*64 + s*8 + t
  int32_t fq1[4];               // f_X at the first shell
  // 1nn b by x parity p at 8 p + b: (local offset, dX, dy, dz)
  alignas(16) int4 d1[16];
  uint8_t rf[8][kFootSlots];    // Geometry::foot_refresh
  int32_t rl[2][8][kRefreshN];  // Geometry::refresh: packed (dx, dy, dz) and shells
  alignas(16) Slot slot[kFootSlots];  // a lane's share of the dE terms
  alignas(16) int4 ix[64][2];         // a lane's share of the jump sums (jump_rates), by x parity
  // dE terms of a vacancy's jumps (Geometry::foot_out), of two vacancies at a time: FP64 a double
  // each (0.0: a vacancy's site), FP32-comp (term, 1.0f for an atom's site); then its own and its
  // targets' embedding values (FP32-comp: the F cells, in fx).  The pair-bond loop keeps its path here.
  alignas(16) double term[kTermSets][kTermSlots];
  float4 fx[kTermSets][9];
  int32_t vidx[kMaxV];          // vacancy table index of record k
  // Vacancy record k: (local site, local x, y, z) and (global x, y, z, site id), x in doubled
  // sites.  A hop's record and rates are written after its middle barrier, when every warp has
  // selected from the old ones.
  alignas(16) int4 vpk[kMaxV][2];
  alignas(16) double rates[kMaxV][8];
  alignas(8) uint8_t vX[kMaxV][8];  // code of jump b's target atom (0: the target is a vacancy)
  uint8_t vact[kMaxV];          // vacancy still inside the active sector
  int32_t ord[2][kMaxV];        // the active vacancies in z-y-x order (ascending site id), in two sets
  int32_t nord[2];
  // F-table window, two planes: FP64 (c0, c1) x kFWin then (c2, c3) x kFWin;
  // FP32 (hi, lo, c1, c2) x kFWin then c3 x kFWin
  alignas(16) unsigned char fwin[kFWin * 32];
  alignas(8) uint64_t mbar;                    // completion barrier of the window's bulk copy
  uint64_t mbar_st;                            // completion barrier of the region's bulk copies
  uint32_t mbar_phase, mbst_phase;
  int32_t win_pot;                             // potential (and precision) the window holds
  int32_t tab_key[2];                          // potential, kind and region strides the tables hold
  int32_t ctl_ok;          // the region's copies arrived
  int32_t ctl_stop;        // the sector's window is reached (or the hop cap): no more selections
  // the block's selection (0) and residence-time (1) streams: running state, the draws made
  // ahead, the state after each, and what the draws stand for (uniform, -ln uniform)
  uint64_t str[2][4];
  uint64_t raw[2][kDrawRing];
  alignas(16) uint64_t sts[kDrawRing][2][4];
  double du[kDrawRing], dl[kDrawRing];
  Round round[kMaxTake];   // rounds handed over by a sweep; [0] alone in the other kernels
  JobDev job;              // the job of the running block (job_key: its index), copied when it changes
  int32_t job_key;
  int32_t fnv;             // vacancies of the running sector
  int32_t fslot[kMaxV];    // and their slots (k_flow)
  int32_t flow_ncand, flow_stop, flow_progress, flow_more;
  // run_block's clock thread: hops, n_act sum and evaluations of the block-round, selections made, the
  // sector's clock
  int64_t c_nh, c_nact, c_evals;
  int32_t c_sel, c_path;
  double c_time;
  // device counters summed per CTA and added once when the kernel ends (per-round atomics on
  // the same addresses from every CTA queue up); hops of the current job likewise
  unsigned long long acc[6];  // counters 0 (hops), 1, 3, 4, 5, 6
  int32_t acc_job;
  unsigned long long acc_job_hops;
};

// A reloaded lattice may hold codes above 8, which no table has a row for: what is looked up for them as neighbours
// lies within the working set.
static_assert(offsetof(Smem, b2) + sizeof(double) * (255 * 5 + 9) <= sizeof(Smem) &&
                  offsetof(Smem, dphi64) + sizeof(double) * ((3 * 4 + 96 + 1) * 64) <= sizeof(Smem),
              "codes up to 255 (atom_index 96)");

// --- bulk copy global -> shared with an mbarrier (cp.async.bulk, TMA unit) -----------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Arms the barrier for `bytes` of bulk copies (then issued with bulk_copy).
__device__ __forceinline__ void bulk_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// Global -> shared bulk copy; addresses 16-byte aligned, size a multiple of 16.
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// Waits for the barrier phase with an iteration limit; false when the limit is reached.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t phase) {
  for (int it = 0; it < (1 << 22); ++it) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(phase)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// F-table access: cells inside the shared-memory window, the rest from global memory.
struct FTab {
  const unsigned char* win;
  int kw0;
  const Potential* pot;      // the full tables (far cells), read on the rare path only
  unsigned int* status;
};

// Job constants of the running block, held in registers (the job record sits in global
// memory, where every store of the hop loop would otherwise force a reload).
struct JobC {
  uint8_t* occ;
  int32_t* rho;
  int sx, sy, sz, px;
};

__device__ __forceinline__ int local_delta(int32_t w, int LX, int LY) {
  return unpack_dx(w) + LX * (unpack_dy(w) + LY * unpack_dz(w));
}
__device__ __forceinline__ int local_delta(int32_t w, const Region& R) { return local_delta(w, R.LX, R.LY); }

// Region layout after Smem: int32 densities, then occupancy bytes (16-byte aligned).
__device__ __forceinline__ uint8_t* occ_of(int32_t* rho_s, int nreg) {
  return reinterpret_cast<uint8_t*>(rho_s) + ((static_cast<size_t>(nreg) * 4 + 127) & ~static_cast<size_t>(127));
}

template <int W>
__device__ void load_tables(Smem& sm, const Potential& P, const Geometry& G, const Region& R, int kind) {
  AKMC_SHAPE(W);
  const bool eam = kind != kPairBond;
  const int tid = threadIdx.x;
  if (tid < 16) {
    const int32_t w = G.nn1[tid >> 3][tid & 7];
    sm.d1[tid] = make_int4(local_delta(w, R), unpack_dx(w), unpack_dy(w), unpack_dz(w));
  }
  if (tid < 9) sm.e0[tid] = e0_of(static_cast<uint8_t>(tid));
  if (!eam) {
    if (tid < 45) {  // codes that are no atom's (a reloaded lattice may hold some) bind as a vacancy
      const int code = tid / 5, i = tid % 5;
      sm.b1[tid] = P.b1[bond_index(static_cast<uint8_t>(code))][i];
      sm.b2[tid] = P.b2[bond_index(static_cast<uint8_t>(code))][i];
    }
    return;
  }
  if (tid < 4) sm.fq1[tid] = P.fq[tid][1];
  for (int i = tid; i < 4 * 4 * 64; i += kThreads) {
    const int xy = i >> 6, hs = (i >> 3) & 7, ht = i & 7;
    const double* ph = &P.phi64[0][0][0] + xy * 8;
    const float* pf = &P.phi32[0][0][0] + xy * 8;
    if (kind == kEam64) sm.dphi64[i] = ph[hs] - ph[ht];
    else sm.dphi32[i] = pf[hs] - pf[ht];
    if (i < 4 * 64) sm.dfq[i] = P.fq[i >> 6][hs] - P.fq[i >> 6][ht];
  }
  for (int i = tid; i < 8 * kFootSlots / 4; i += kThreads)
    reinterpret_cast<uint32_t*>(&sm.rf[0][0])[i] = __ldg(reinterpret_cast<const uint32_t*>(&G.foot_refresh[0][0]) + i);
  for (int i = tid; i < 2 * 8 * kRefreshN; i += kThreads) (&sm.rl[0][0][0])[i] = __ldg(&G.refresh[0][0][0] + i);
  for (int i = tid; i < kFootSlots; i += kThreads) {
    Slot c;
    c.off[0] = local_delta(__ldg(&G.foot_site[0][i]), R);
    c.off[1] = local_delta(__ldg(&G.foot_site[1][i]), R);
    const int out = __ldg(&G.foot_out[i]), sh = __ldg(&G.foot_shells[i]);
    const int tA = out & 1023, tB = (out >> 10) & 1023;
    c.tA = (tA == kFootNone ? kTrashTerm : tA) | (out >> 20) << 10;  // leader lane and raw in the high bits
    c.tB = tB == kFootNone ? kTrashTerm : tB;
    c.hA = sh & 63;
    c.hB = (sh >> 8) & 63;
    c.dA = P.fq[0][c.hA >> 3] - P.fq[0][c.hA & 7];
    c.dB = P.fq[0][c.hB >> 3] - P.fq[0][c.hB & 7];
    sm.slot[i] = c;
  }
  for (int i = tid; i < 128; i += kThreads) {  // lane (i / 2) of a pair of warps, parity i % 2
    const int p = i & 1, lane = (i >> 1) & 31, b = 4 * (i >> 6) + (lane >> 3), sub = lane & 7;
    auto t = [&](int k) -> int32_t { return k < kJumpN ? __ldg(&G.term[p][b][k]) : kZeroTerm; };
    sm.ix[i >> 1][p] = make_int4(t(sub) | t(sub + 32) << 10 | t(sub + 64) << 20, t(sub + 8) | t(sub + 40) << 10 | t(sub + 72) << 20,
                                 t(sub + 16) | t(sub + 48) << 10 | t(sub + 24) << 20, t(sub + 56));
  }
  if (tid < kTermSets) sm.term[tid][kZeroTerm] = 0.0;
}


// Cells outside the shared-memory window (rare): global memory, range-checked.  status null: a density off the table is
// no error (the nearest end cell stands in).
__device__ __noinline__ double F64_far(const double2* g64lo, const double2* g64hi, unsigned int* status, int32_t r,
                                       double p) {
  const int k = r >> kRhoCellShift;
  int kc = k;
  if (r < 0 || k > kTabN - 2) {
    if (status) atomicOr(status, kErrRhoRange);
    kc = r < 0 ? 0 : kTabN - 2;
  }
  const double2 lo = __ldg(g64lo + kc), hi = __ldg(g64hi + kc);
  return cubic_d(lo.x, lo.y, hi.x, hi.y, p);
}

__device__ __forceinline__ double F64(const FTab& T, int32_t r, unsigned int* status) {
  const int k = r >> kRhoCellShift;
  // p = (r mod 2^17) * 2^-17, built in the exponent field: 1 + m 2^-17 minus 1 (both exact)
  const double p = __hiloint2double(0x3FF00000 | ((r & kRhoFracMask) << 3), 0) - 1.0;
  const unsigned kk = static_cast<unsigned>(k - T.kw0);
  if (kk < static_cast<unsigned>(kFWin)) {
    const double2 lo = reinterpret_cast<const double2*>(T.win)[kk];
    const double2 hi = reinterpret_cast<const double2*>(T.win)[kFWin + kk];
    return cubic_d(lo.x, lo.y, hi.x, hi.y, p);
  }
  return F64_far(T.pot->F64lo, T.pot->F64hi, status, r, p);
}

// A cell known to lie inside the shared-memory window.
__device__ __forceinline__ double F64win(const FTab& T, int32_t r) {
  const int kk = (r >> kRhoCellShift) - T.kw0;
  const double p = __hiloint2double(0x3FF00000 | ((r & kRhoFracMask) << 3), 0) - 1.0;
  const double2 lo = reinterpret_cast<const double2*>(T.win)[kk];
  const double2 hi = reinterpret_cast<const double2*>(T.win)[kFWin + kk];
  return cubic_d(lo.x, lo.y, hi.x, hi.y, p);
}
__device__ __forceinline__ FCell32 cell32win(const FTab& T, int32_t r) {
  const int kk = (r >> kRhoCellShift) - T.kw0;
  const float4 a = reinterpret_cast<const float4*>(T.win)[kk];
  FCell32 c;
  c.hi = a.x; c.lo = a.y; c.c1 = a.z; c.c2 = a.w;
  c.c3 = reinterpret_cast<const float*>(T.win + kFWin * 16)[kk];
  c.pad0 = c.pad1 = c.pad2 = 0.f;
  return c;
}

__device__ __forceinline__ FCell32 cell32(const FTab& T, int32_t r, unsigned int* status) {
  const int k = r >> kRhoCellShift;
  const unsigned kk = static_cast<unsigned>(k - T.kw0);
  float4 a;
  float c3;
  if (kk < static_cast<unsigned>(kFWin)) {
    a = reinterpret_cast<const float4*>(T.win)[kk];
    c3 = reinterpret_cast<const float*>(T.win + kFWin * 16)[kk];
  } else {
    int kc = k;
    if (r < 0 || k > kTabN - 2) {
      if (status) atomicOr(status, kErrRhoRange);
      kc = r < 0 ? 0 : kTabN - 2;
    }
    a = __ldg(T.pot->F32a + kc);
    c3 = __ldg(T.pot->F32b + kc);
  }
  FCell32 c;
  c.hi = a.x; c.lo = a.y; c.c1 = a.z; c.c2 = a.w; c.c3 = c3;
  c.pad0 = c.pad1 = c.pad2 = 0.f;
  return c;
}

// Codes 1, 2, 4 and 8 (the mask's bits), or 2, 4 and 8: one test, without a compare for each.
__device__ __forceinline__ bool code_in(uint8_t c, uint32_t mask) { return c <= kMn && ((mask >> c) & 1u) != 0; }
constexpr uint32_t kAtoms = 1u << kFe | 1u << kCu | 1u << kNi | 1u << kMn, kSolutes = kAtoms & ~(1u << kFe);

// The rate of a jump with energy change dE onto a site with code Xc, into the record of vacancy k and jump b: 0 unless
// the code is an atom's (a vacancy's is not, nor are others that a reloaded lattice may hold).
__device__ __forceinline__ void put_rate(Smem& sm, int k, int b, uint8_t Xc, bool atom, double dE, double* de_out) {
  const double rate = arrhenius_rk(sm.job.nu, sm.job.kT, sm.job.rkT, sm.e0[atom ? Xc : 0], dE);
  sm.rates[k][b] = atom ? rate : 0.0;
  sm.vX[k][b] = Xc;
  if (de_out) de_out[k * 8 + b] = atom ? dE : 0.0;  // akmc_calculate only
}

// Pair bond: the rates of vacancy k at local site l, by one warp.  Lanes 4 b + 0..3 run the four bond
// counts of VacRatesSolver::deltaE (vacancy_rates_solver.cpp:45-116) for jump b, each summed in the
// reference order.  A single warp runs this on the hop loop's chain, so it counts instructions: the bond
// tables are indexed by occupancy code, and the neighbours of both x parities are the same offsets from a
// corner (ly, lyz: the row and plane pitch).
__device__ __forceinline__ void pair_rates(Smem& sm, const uint8_t* occ_s, int k, int l, int ly, int lyz, double* de_out) {
  const int lane = threadIdx.x & 31, b = lane >> 2, q = lane & 3;
  const int p = l & 1;
  const int tl = l + sm.d1[8 * p + b].x;
  const uint8_t Xc = occ_s[tl];
  const bool at_t = (q & 1) != 0;
  const uint8_t* c = occ_s + (at_t ? tl : l);
  const int src = (q == 0 || q == 3) ? 0 : 32 - __clz(Xc);  // bond index of V, or of the moving atom
  // after the hop (q = 2, 3) the other end of the jump, neighbour b or its opposite, holds the other one
  const int over = q == 2 ? b : q == 3 ? 7 - b : 8;
  const int over_code = q == 2 ? 0 : Xc;
  const uint8_t* corner = c - ((p ^ (at_t ? 1 : 0)) ? 0 : ly + lyz);
  const double* t1 = sm.b1 + src;
  const double* t2 = sm.b2 + src;
  double energy = 0.0;
#pragma unroll
  for (int b2 = 0; b2 < 8; ++b2) {  // 1nn order: dX, then dy, then dz rising
    int o = corner[((b2 & 4) ? 1 : -1) + ((b2 & 2) ? ly : 0) + ((b2 & 1) ? lyz : 0)];
    o = b2 == over ? over_code : o;
    energy += t1[o * 5];
  }
  // 2nn -x, -y, -z, +z, +x (PeriodLatticeList::get2nn2 order under the mask of get2nnStatus)
  energy += t2[c[-2] * 5];
  energy += t2[c[-ly] * 5];
  energy += t2[c[-lyz] * 5];
  energy += t2[c[lyz] * 5];
  energy += t2[c[2] * 5];
  const double pair = energy + __shfl_down_sync(kFull, energy, 1);  // q0: e_before, q2: e_after
  const double after = __shfl_down_sync(kFull, pair, 2);
  if (q == 0) put_rate(sm, k, b, Xc, code_in(Xc, kAtoms), after - pair, de_out);
}

// FP32 F cell at density r: the node and the polynomial part of dF32.
struct F32Val {
  float hi, lo, q;
};
__device__ __forceinline__ F32Val F32part(const FCell32& c, int32_t r) {
  const float p = static_cast<float>(r & kRhoFracMask) * 0x1p-17f;
  F32Val v;
  v.hi = c.hi;
  v.lo = c.lo;
  v.q = fma_f(fma_f(c.c3, p, c.c2), p, c.c1) * p;
  return v;
}
// F(r1) - F(r0) from the two parts: dF32's sums.
__device__ __forceinline__ float F32diff(const F32Val& a1, const F32Val& a0) {
  const float node = (a1.hi - a0.hi) + (a1.lo - a0.lo);
  return node + (a1.q - a0.q);
}

// One slot of the dE terms of the vacancy at local site l for moving Fe atoms, into term set `set`;
// all 32 lanes of a warp.  With REFRESH the vacancy has just come here from local site `from` by jump
// b of an atom X, and the slot's leader first brings its site's density up to date (the 78 density
// deltas of the hop all lie on the slots' sites; no other warp touches them before the next barrier).
// `inside`: the vacancy is still in its sector; one that left it needs no terms, and some of its sites lie
// past the region's 2-cell halo (the refreshed ones never do).
// What bounds this: the instructions of one chain (a hop waits for it), and four 16-byte reads of random F
// cells a lane (about 10 shared-memory wavefronts a warp and read).  Each jump's 76 sites evaluated on their
// own took 1232 F evaluations a vacancy; the shared terms take 447.
template <int KIND, bool REFRESH>
__device__ __forceinline__ void foot_terms(Smem& sm, int set, const uint8_t* occ_s, int32_t* rho_s, int l, const Slot& c,
                                           int slot, const FTab& FT, int b, int X, int from, bool inside) {
  const int lead = (c.tA >> 10) & 31, raw = c.tA >> 15;
  int j = l + ((l & 1) ? c.off[1] : c.off[0]);
  int code = 0;
  if (REFRESH) {
    code = sm.rf[b][slot];
    if (!inside && !code) j = l;  // outside the staged halo: only the deltas are wanted
  }
  int o = occ_s[j];
  int32_t r = rho_s[j];
  if (REFRESH) {
    r += sm.dfq[atom_index(static_cast<uint8_t>(X)) * 64 + code];  // code 0: + 0
    if (j == from) o = X;
    __syncwarp();
    if (code && lead == (threadIdx.x & 31)) rho_s[j] = r;
  }
  const int32_t rA = r + c.dA, rB = r + c.dB;
  static_assert((kFWin & (kFWin - 1)) == 0, "one test for both cells");
  const bool win = static_cast<unsigned>(((rA >> kRhoCellShift) - FT.kw0) | ((rB >> kRhoCellShift) - FT.kw0)) <
                   static_cast<unsigned>(kFWin);
  // A density itself is range-checked (hA = 0).  The terms are not: one that a jump of a Fe atom uses cannot leave the
  // table when the density does not (the atom's own share is part of it), and one that no jump uses, its target being
  // another atom or a vacancy, may: nothing reads it.
  unsigned int* const status = c.hA == 0 ? FT.status : nullptr;
  const bool atom = o != kV;
  const int y = atom ? atom_index(static_cast<uint8_t>(o)) * 64 : 0;
  if (KIND == kEam64) {
    double FA, FB;
    if (win) {
      FA = F64win(FT, rA);
      FB = F64win(FT, rB);
    } else {
      FA = F64(FT, rA, status);
      FB = F64(FT, rB, nullptr);
    }
    const double F0 = __shfl_sync(kFull, FA, lead);
    const double tA = (FA - F0) + sm.dphi64[y + c.hA], tB = (FB - F0) + sm.dphi64[y + c.hB];
    double* const T = sm.term[set];
    T[c.tA & 1023] = atom ? tA : 0.0;
    T[c.tB] = atom ? tB : 0.0;
    if (raw) T[kTermN + raw - 1] = FA;
  } else {
    F32Val a, bb;
    if (win) {
      a = F32part(cell32win(FT, rA), rA);
      bb = F32part(cell32win(FT, rB), rB);
    } else {
      a = F32part(cell32(FT, rA, status), rA);
      bb = F32part(cell32(FT, rB, nullptr), rB);
    }
    F32Val f0;
    f0.hi = __shfl_sync(kFull, a.hi, lead);
    f0.lo = __shfl_sync(kFull, a.lo, lead);
    f0.q = __shfl_sync(kFull, a.q, lead);
    const float tA = F32diff(a, f0) + sm.dphi32[y + c.hA], tB = F32diff(bb, f0) + sm.dphi32[y + c.hB];
    float2* const T = reinterpret_cast<float2*>(sm.term[set]);
    const float on = atom ? 1.f : 0.f;
    T[c.tA & 1023] = make_float2(tA, on);
    T[c.tB] = make_float2(tB, on);
    if (raw) sm.fx[set][raw - 1] = make_float4(a.hi, a.lo, a.q, 0.f);
  }
}

// Rates of jumps 4 half .. 4 half + 3 of vacancy k at local site l from term set `set`, by one warp, for
// Fe targets and those that hold no atom; solutes' jumps are left to solute_rate.  Eight lanes take a jump:
// lane sub the partial sums sub + 8 g (g = 0..3) of the 32 interleaved ones (entries i = q, q + 32, q + 64
// of the jump's list; ix: their terms, 10 bits each), merged in the order of the 32-lane xor butterfly
// (16, 8, 4, 2, 1).  A vacancy's site adds 0.0, which leaves every partial sum as it is: a sum that
// starts at a term (never -0.0) cannot become -0.0.
template <int KIND>
__device__ __forceinline__ void jump_rates(Smem& sm, int set, const uint8_t* occ_s, int k, int l, int half,
                                           const int4 (&ix)[2], double* de_out) {
  const int lane = threadIdx.x & 31, b = 4 * half + (lane >> 3);
  const int p = l & 1;
  const uint8_t Xc = occ_s[l + sm.d1[8 * p + b].x];
  const int32_t w0 = p ? ix[1].x : ix[0].x, w1 = p ? ix[1].y : ix[0].y, w2 = p ? ix[1].z : ix[0].z,
                w3 = p ? ix[1].w : ix[0].w;
  const int i[10] = {w0 & 1023, (w0 >> 10) & 1023, (w0 >> 20) & 1023, w1 & 1023, (w1 >> 10) & 1023,
                     (w1 >> 20) & 1023, w2 & 1023, (w2 >> 10) & 1023, (w2 >> 20) & 1023, w3 & 1023};
  double dE;
  if (KIND == kEam64) {
    const double* T = sm.term[set];
    double t[10];
#pragma unroll
    for (int q = 0; q < 10; ++q) t[q] = T[i[q]];
    const double EX = T[kTermN] - T[kTermN + 1 + b];
    const double g0 = (t[0] + t[1]) + t[2], g1 = (t[3] + t[4]) + t[5], g2 = t[6] + t[7], g3 = t[8] + t[9];
    double x = (g0 + g2) + (g1 + g3);
#pragma unroll
    for (int m = 4; m >= 1; m >>= 1) x = x + __shfl_xor_sync(kFull, x, m);
    dE = EX + x;
  } else {
    const float2* T = reinterpret_cast<const float2*>(sm.term[set]);
    float2 t[10];
#pragma unroll
    for (int q = 0; q < 10; ++q) t[q] = T[i[q]];
    const float4 f1 = sm.fx[set][0], f0 = sm.fx[set][1 + b];
    const F32Val e1 = {f1.x, f1.y, f1.z}, e0 = {f0.x, f0.y, f0.z};
    const float EX = F32diff(e1, e0);
    Comp32 g[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      g[q].s = g[q].c = 0.f;
      const int first = q < 2 ? 3 * q : 6 + 2 * (q - 2), n = q < 2 ? 3 : 2;
#pragma unroll
      for (int v = 0; v < 3; ++v)
        if (v < n && t[first + v].y != 0.f) kahan_add(g[q], t[first + v].x);
    }
    Comp32 x = comp_merge(comp_merge(g[0], g[2]), comp_merge(g[1], g[3]));
#pragma unroll
    for (int m = 4; m >= 1; m >>= 1) {
      Comp32 o;
      o.s = __shfl_xor_sync(kFull, x.s, m);
      o.c = __shfl_xor_sync(kFull, x.c, m);
      x = comp_merge(x, o);
    }
    dE = static_cast<double>(EX + (x.s - x.c));
  }
  if ((lane & 7) == 0 && !code_in(Xc, kSolutes)) put_rate(sm, k, b, Xc, Xc == kFe, dE, de_out);
}

// Jumps of the vacancy at local site l whose target holds a solute, one bit each; all lanes of a warp.
__device__ __forceinline__ unsigned solute_jumps(const Smem& sm, const uint8_t* occ_s, int l) {
  const int lane = threadIdx.x & 31;
  return __ballot_sync(kFull, lane < 8 && code_in(occ_s[l + sm.d1[8 * (l & 1) + (lane & 7)].x], kSolutes));
}
// Rate of jump b of vacancy k at local site l with an atom as target, by one warp: for solutes (solute_jumps; the
// shared terms are those of a moving Fe atom), and for every atom in a job rich in solutes.  Lane q sums sites i = q,
// q + 32, q + 64 of the jump's list; the 32 partials merge by a xor butterfly (16, 8, 4, 2, 1), then the moving atom's
// own embedding change is added.
template <int KIND>
__device__ __forceinline__ void solute_rate(Smem& sm, const uint8_t* occ_s, const int32_t* rho_s, int k, int l, int b,
                                            int LX, int LY, const Geometry& G, const FTab& FT, double* de_out) {
  const int q = threadIdx.x & 31;
  const int p = l & 1;
  const int tl = l + sm.d1[8 * p + b].x;
  const uint8_t Xc = occ_s[tl];
  const int X = atom_index(Xc);
  uint8_t o[3];
  int32_t r0[3], r1[3];
  int h[3];
  bool in[3];
#pragma unroll
  for (int u = 0; u < 3; ++u) {
    in[u] = q + 32 * u < kJumpN;
    const int32_t e = in[u] ? __ldg(&G.jump[p][b][q + 32 * u]) : 0;  // outside the list: the vacancy's own site
    const int j = l + local_delta(e, LX, LY);
    h[u] = unpack_sh_s(e) * 8 + unpack_sh_t(e);
    o[u] = occ_s[j];
    r0[u] = rho_s[j];
    r1[u] = r0[u] + sm.dfq[X * 64 + h[u]];
  }
  const int32_t rx1 = rho_s[l] - sm.fq1[X], rx0 = rho_s[tl];
  // every cell inside the shared-memory window (nearly always): one straight run of loads
  // and polynomials; otherwise the general path, which reads far cells from global memory
  bool win = static_cast<unsigned>((rx1 >> kRhoCellShift) - FT.kw0) < static_cast<unsigned>(kFWin) &&
             static_cast<unsigned>((rx0 >> kRhoCellShift) - FT.kw0) < static_cast<unsigned>(kFWin);
#pragma unroll
  for (int u = 0; u < 3; ++u)
    win = win && (!in[u] || (static_cast<unsigned>((r0[u] >> kRhoCellShift) - FT.kw0) < static_cast<unsigned>(kFWin) &&
                             static_cast<unsigned>((r1[u] >> kRhoCellShift) - FT.kw0) < static_cast<unsigned>(kFWin)));
  double dE;
  if (KIND == kEam64) {
    double t[3], EX;
    if (win) {
      EX = F64win(FT, rx1) - F64win(FT, rx0);
#pragma unroll
      for (int u = 0; u < 3; ++u) t[u] = in[u] ? F64win(FT, r1[u]) - F64win(FT, r0[u]) : 0.0;
    } else {
      EX = F64(FT, rx1, FT.status) - F64(FT, rx0, FT.status);
#pragma unroll
      for (int u = 0; u < 3; ++u) t[u] = in[u] ? F64(FT, r1[u], FT.status) - F64(FT, r0[u], FT.status) : 0.0;
    }
    // site term (F(r+d) - F(r)) + (phi_s - phi_t), summed in list order
    double acc = 0.0;
#pragma unroll
    for (int u = 0; u < 3; ++u)
      if (in[u] && o[u] != kV) acc += t[u] + sm.dphi64[(X * 4 + atom_index(o[u])) * 64 + h[u]];
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) acc = acc + __shfl_xor_sync(kFull, acc, m);
    dE = EX + acc;
  } else {
    float t[3], EX;
    if (win) {
      EX = dF32(cell32win(FT, rx1), cell32win(FT, rx0), rx1, rx0);
#pragma unroll
      for (int u = 0; u < 3; ++u) t[u] = in[u] ? dF32(cell32win(FT, r1[u]), cell32win(FT, r0[u]), r1[u], r0[u]) : 0.f;
    } else {
      EX = dF32(cell32(FT, rx1, FT.status), cell32(FT, rx0, FT.status), rx1, rx0);
#pragma unroll
      for (int u = 0; u < 3; ++u)
        t[u] = in[u] ? dF32(cell32(FT, r1[u], FT.status), cell32(FT, r0[u], FT.status), r1[u], r0[u]) : 0.f;
    }
    Comp32 acc;
    acc.s = 0.f;
    acc.c = 0.f;
#pragma unroll
    for (int u = 0; u < 3; ++u)
      if (in[u] && o[u] != kV) kahan_add(acc, t[u] + sm.dphi32[(X * 4 + atom_index(o[u])) * 64 + h[u]]);
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
      Comp32 v;
      v.s = __shfl_xor_sync(kFull, acc.s, m);
      v.c = __shfl_xor_sync(kFull, acc.c, m);
      acc = comp_merge(acc, v);
    }
    dE = static_cast<double>(EX + (acc.s - acc.c));
  }
  if (q == 0) put_rate(sm, k, b, Xc, true, dE, de_out);
}
// Rates of the vacancies of masks m0 and m1 in a job rich in solutes, a warp a jump (W = 4: two), without the shared
// terms: nearly every jump is summed on its own anyway, and all warps take part.  Vacancy ksel is at local site snew.
// In a box of Cu with 20 vacancies, 128 rounds took 14.5 ms jump by jump on 8 warps, 19.5 with shared terms and the
// solutes' jumps left to 4 of them, and 13.4 so (FP64; FP32-comp 15.1, 21.2, 12.4).  Out of line: the loop of the other
// jobs keeps its code.
template <int KIND, int W>
__device__ __noinline__ void rich_rates(Smem& sm, const uint8_t* occ_s, const int32_t* rho_s, unsigned m0, unsigned m1,
                                        int ksel, int snew, int LX, int LY, const Geometry* geo, const Potential* pot,
                                        unsigned int* status, double* de_out) {
  FTab FT;
  FT.win = sm.fwin;
  FT.kw0 = sm.job.fwin0;
  FT.pot = pot;
  FT.status = status;
  while (m0 | m1) {
    const int k = m0 ? __ffs(static_cast<int>(m0)) - 1 : 31 + __ffs(static_cast<int>(m1));
    if (m0) m0 &= m0 - 1;
    else m1 &= m1 - 1;
    const int l = k == ksel ? snew : sm.vpk[k][0].x;
    for (int b = threadIdx.x >> 5; b < 8; b += W) {
      const uint8_t Xc = occ_s[l + sm.d1[8 * (l & 1) + b].x];
      if (code_in(Xc, kAtoms)) solute_rate<KIND>(sm, occ_s, rho_s, k, l, b, LX, LY, *geo, FT, de_out);
      else if ((threadIdx.x & 31) == 0) put_rate(sm, k, b, Xc, false, 0.0, de_out);
    }
  }
}

// The CTA's copy of job `job`'s record (constant while a launch runs); CTA-wide, uniform.
__device__ __forceinline__ void load_job(Smem& sm, const RoundArgs& a, int job) {
  if (sm.job_key == job) return;
  __syncthreads();  // every thread has read the key; the previous job's readers are done
  static_assert(sizeof(JobDev) % 16 == 0, "copied in 16-byte words");
  if (threadIdx.x < sizeof(JobDev) / 16)
    reinterpret_cast<int4*>(&sm.job)[threadIdx.x] = __ldcg(reinterpret_cast<const int4*>(a.jobs + job) + threadIdx.x);
  if (threadIdx.x == 0) sm.job_key = job;
  __syncthreads();
}

// Issues the copies of a region into shared memory (CTA-wide, no wait: stage_wait).  A region that does not
// wrap in y or z is one tensor copy per array of the job's box from entry (kHaloL + R.ox, R.oy, R.oz) of the
// lattice (x a multiple of 16 entries: 16-byte aligned in both arrays), laid out with the box as pitch; parts of
// the box past the region are staged too and never read, parts past the array are filled with zeros.  The others
// go row by row, 16 bytes a copy (cp.async), half a warp a row where its copies fit: one bulk copy per row and
// array measured 15 cycles each through the copy unit, 5.9K cycles for the 14 x 14 rows of a 20-cell block.
template <int KIND, int W>
__device__ __forceinline__ void stage_region(Smem& sm, const RoundArgs& a, const Region& R, uint8_t* occ_s, int32_t* rho_s) {
  AKMC_SHAPE(W);
  constexpr bool eam = KIND != kPairBond;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const JobDev& J = sm.job;
  if (R.tma) {
    if (tid == kCtl) {
      bulk_expect(&sm.mbar_st, static_cast<uint32_t>(R.n) * (eam ? 5u : 1u));
      asm volatile("fence.proxy.async;" ::: "memory");  // generic accesses before, copies after
      const unsigned char* m = static_cast<const unsigned char*>(a.tmaps) + static_cast<size_t>(sm.job_key) * 256;
      const int x = kHaloL + R.ox, y = R.oy, z = R.oz;
      asm volatile(
          "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
              smem_u32(occ_s)),
          "l"(m), "r"(x), "r"(y), "r"(z), "r"(smem_u32(&sm.mbar_st))
          : "memory");
      if (eam)
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                smem_u32(rho_s)),
            "l"(m + 128), "r"(x), "r"(y), "r"(z), "r"(smem_u32(&sm.mbar_st))
            : "memory");
    }
  } else if (R.bulk) {
    const int no = R.bo >> 4, nc = no + (eam ? R.br >> 2 : 0);  // 16-byte copies of a row
    const int per = nc <= 16 ? 2 : 1;                           // rows a warp takes at a time (nc <= 32)
    const int c = per == 2 ? lane & 15 : lane, sub = per == 2 ? lane >> 4 : 0;
    const int nrows = R.ey * R.ez;
    int row = warp * per + sub;
    int lz = row / R.ey, ly = row - lz * R.ey;
    const int step = kThreads / 32 * per, dz = step / R.ey, dy = step - dz * R.ey;
    for (; row < nrows; row += step) {
      const int gy = wrap1(R.oy + ly, J.sy), gz = wrap1(R.oz + lz, J.sz);
      const int64_t first = static_cast<int64_t>(J.px) * (gy + static_cast<int64_t>(J.sy) * gz) + kHaloL + R.ox;
      const int l = R.LX * (ly + R.LY * lz);  // the shared row (pitch LX, LY)
      if (c < nc) {
        const bool o = c < no;
        const void* src = o ? static_cast<const void*>(J.occ + first + 16 * c) : static_cast<const void*>(J.rho + first + 4 * (c - no));
        const uint32_t dst = o ? smem_u32(occ_s + l + 16 * c) : smem_u32(rho_s + l + 4 * (c - no));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
      }
      ly += dy;
      lz += dz;
      if (ly >= R.ey) {
        ly -= R.ey;
        ++lz;
      }
    }
  } else {
    // row loads, where shared memory cannot hold the rounded rows: warp w takes rows w, w + W, ...;
    // kStageRows rows of loads are issued before any shared-memory store so they are all in flight (rows hold
    // <= 64 sites; the halo holds the sites past either end)
    const int gx0 = kHaloL + R.ox + lane, gx1 = gx0 + 32;
    const bool has0 = lane < R.LX, has1 = lane + 32 < R.LX;
    constexpr int kW = kThreads / 32;
    const int nrows = R.LY * R.LZ;
    for (int row0 = warp; row0 < nrows; row0 += kStageRows * kW) {
      uint8_t ov[kStageRows][2];
      int32_t rv[kStageRows][2];
#pragma unroll
      for (int k = 0; k < kStageRows; ++k) {
        const int row = row0 + kW * k;
        if (row < nrows) {
          const int ly = row % R.LY, lz = row / R.LY;
          const int gy = wrap1(R.oy + ly, J.sy), gz = wrap1(R.oz + lz, J.sz);
          const int64_t base = static_cast<int64_t>(J.px) * (gy + static_cast<int64_t>(J.sy) * gz);
          if (has0) {
            ov[k][0] = __ldcg(J.occ + base + gx0);
            if (eam) rv[k][0] = __ldcg(J.rho + base + gx0);
          }
          if (has1) {
            ov[k][1] = __ldcg(J.occ + base + gx1);
            if (eam) rv[k][1] = __ldcg(J.rho + base + gx1);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < kStageRows; ++k) {
        const int row = row0 + kW * k;
        if (row < nrows) {
          const int l = lane + R.LX * row;
          if (has0) {
            occ_s[l] = ov[k][0];
            if (eam) rho_s[l] = rv[k][0];
          }
          if (has1) {
            occ_s[l + 32] = ov[k][1];
            if (eam) rho_s[l + 32] = rv[k][1];
          }
        }
      }
    }
  }
}

// Vacancy record k of the running sector: vacancy v at site s = (X, y, z).
__device__ __forceinline__ void put_record(Smem& sm, const Region& R, int k, int v, int32_t s, int X, int y, int z) {
  const int lx = X - R.ox, ly = y - R.oy, lz = z - R.oz;
  sm.vidx[k] = v;
  sm.vact[k] = 1;
  sm.vpk[k][0] = make_int4(lx + R.LX * (ly + R.LY * lz), lx, ly, lz);
  sm.vpk[k][1] = make_int4(X, y, z, s);
}

// Phase profile (builds with -DAKMC_PHASE_PROFILE): thread 0 accumulates the cycles
// between consecutive CTA barriers into counters[8 + phase].
#ifdef AKMC_PHASE_PROFILE
#define AKMC_PHASE(i)                                                                           \
  do {                                                                                          \
    if (threadIdx.x == 0) {                                                                     \
      const long long t_ = clock64();                                                           \
      atomicAdd(a.counters + 8 + (i), static_cast<unsigned long long>(t_ - tph));               \
      tph = t_;                                                                                 \
    }                                                                                           \
  } while (0)
#else
#define AKMC_PHASE(i) \
  do {              \
  } while (0)
#endif
// Advances the running state of stream lane (0 selection, 1 residence time) by one draw into ring
// slot `slot`: the raw draw and the state after it.  Called by lanes 0 and 1 of one warp.
__device__ __forceinline__ void draw_ahead(Smem& sm, uint64_t (&x)[4], int lane, int slot) {
  sm.raw[lane][slot] = xoshiro_next(x);
  ulonglong2* const st = reinterpret_cast<ulonglong2*>(sm.sts[slot][lane]);
  st[0] = make_ulonglong2(x[0], x[1]);
  st[1] = make_ulonglong2(x[2], x[3]);
}
// What a batch's draws stand for, one draw a lane: the selection uniform in [0, 1) (lanes 0-7) and
// -ln of the residence-time uniform in (0, 1] (lanes 8-15; sublattice.inl:118-120).
__device__ __forceinline__ void draw_values(Smem& sm, int lane, int slot0) {
  if (lane < kDrawBatch) {
    sm.du[slot0 + lane] = static_cast<double>(sm.raw[0][slot0 + lane] >> 11) * 0x1p-53;
  } else if (lane < 2 * kDrawBatch) {
    const int k = slot0 + lane - kDrawBatch;
    sm.dl[k] = -port_log(static_cast<double>((sm.raw[1][k] >> 11) + 1) * 0x1p-53);
  }
}

// The hop loop of the active sector of one block, round C (or, with API, one per-hop API step), CTA-collective.
// Before the call, after a CTA barrier that ended all earlier use of shared memory: sm.job holds the block's
// job, the region's copies are issued (stage_region), and threads outside the last warp have written the records
// of the sector's sm.fnv vacancies (put_record, any order).  Returns, uniformly, the number of vacancies, or -1
// when the sector's clock is already past its window: nothing ran.
//
// Every warp selects for itself, all lanes alike (the ordered sums are deterministic, so no broadcast
// is needed); the hop's updates are spread over the warps.
template <int KIND, int W, bool API>
__device__ __forceinline__ int run_block(const RoundArgs& a, Smem& sm, Round& C, const Region& R, uint8_t* occ_s,
                                         int32_t* rho_s, int sec) {
  AKMC_SHAPE(W);
  constexpr int kClk = Shape<W>::kClk, kOrdWarp = Shape<W>::kOrdWarp;
  constexpr bool eam = KIND != kPairBond;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
#ifdef AKMC_PHASE_PROFILE
  long long tph = clock64();
#endif
  const JobDev& J = sm.job;
  const int64_t round_now = C.r;
  const double thr = API ? 0.0 : static_cast<double>((round_now >> 3) + 1) * J.window - C.evo;
  const bool runs = API || 0.0 < thr;  // else sector_time stays 0 (sublattice.inl:82)
  const Potential& P = a.pots[J.pot];
  JobC jc;
  jc.occ = J.occ;
  jc.rho = J.rho;
  jc.sx = J.sx;
  jc.sy = J.sy;
  jc.sz = J.sz;
  jc.px = J.px;
  // F-table window: one bulk copy per plane issued by the control thread, overlapped with the staging
  const int win_key = J.pot * 2 + (KIND == kEam32 ? 1 : 0);
  const bool need_win = eam && runs && sm.win_pot != win_key;
  // the shell tables depend on the potential, the kind and the region's row strides only: kept
  // from the CTA's previous block when those match
  const int tab0 = J.pot * 4 + KIND, tab1 = R.LX | (R.LY << 16);
  const bool need_tab = runs && (sm.tab_key[0] != tab0 || sm.tab_key[1] != tab1);
  if (need_win && tid == kCtl) {
    if (KIND == kEam32) {
      bulk_expect(&sm.mbar, kFWin * 20u);
      bulk_copy(sm.fwin, P.F32a + J.fwin0, kFWin * 16u, &sm.mbar);
      bulk_copy(sm.fwin + kFWin * 16, P.F32b + J.fwin0, kFWin * 4u, &sm.mbar);
    } else {
      bulk_expect(&sm.mbar, kFWin * 32u);
      bulk_copy(sm.fwin, P.F64lo + J.fwin0, kFWin * 16u, &sm.mbar);
      bulk_copy(sm.fwin + kFWin * 16, P.F64hi + J.fwin0, kFWin * 16u, &sm.mbar);
    }
  }
  if (need_tab) load_tables<W>(sm, P, *a.geo, R, KIND);
  FTab FT;
  FT.win = sm.fwin;
  FT.kw0 = J.fwin0;
  FT.pot = &P;
  FT.status = a.status;
  uint64_t dst[4] = {0, 0, 0, 0};  // last warp, lanes 0 and 1: a stream's running state
  if (warp == kEvalWarps - 1) {
    if (!API) {  // the first batch of draws, while the others order the vacancies and the copies fly
      if (lane < 2) {
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = C.str[lane][i];
#pragma unroll 1
        for (int k = 0; k < kDrawBatch; ++k) draw_ahead(sm, dst, lane, k);
        if (KIND == kPairBond)  // the pair-bond loop of one vacancy draws in warp 1
#pragma unroll
          for (int i = 0; i < 4; ++i) sm.str[lane][i] = dst[i];
      }
      __syncwarp();
      draw_values(sm, lane, 0);
    }
  } else {
    asm volatile("bar.sync 3, %0;" ::"n"(kThreads - 32) : "memory");  // the records, written by these warps
    const int n = sm.fnv;
    if (tid < n) {
      // z-y-x scan order of ABVIModel::calcRates = ascending site id inside a sector
      const int s = sm.vpk[tid][1].w;
      int rank = 0;
      for (int i = 0; i < n; ++i) rank += sm.vpk[i][1].w < s ? 1 : 0;
      sm.ord[0][rank] = tid;
    }
    if (tid == 64) {
      sm.nord[0] = n;
      sm.ctl_ok = 1;
      sm.ctl_stop = 0;
      if (need_win) {
        if (mbar_wait(&sm.mbar, sm.mbar_phase)) {
          sm.mbar_phase ^= 1u;
          sm.win_pot = win_key;
        } else {
          atomicOr(a.status, kErrTimeout);
          mbar_wait(&sm.mbar, sm.mbar_phase);  // bounded second wait for the copy in flight
          sm.win_pot = -1;
          sm.ctl_ok = 0;
        }
      }
      if (R.tma) {
        if (mbar_wait(&sm.mbar_st, sm.mbst_phase)) {
          sm.mbst_phase ^= 1u;
        } else {
          atomicOr(a.status, kErrTimeout);
          if (mbar_wait(&sm.mbar_st, sm.mbst_phase)) sm.mbst_phase ^= 1u;  // bounded second wait
          sm.ctl_ok = 0;
        }
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");  // this thread's copies of the region's rows
  AKMC_PHASE(0);
  __syncthreads();
  AKMC_PHASE(1);
  if (need_tab && tid == 0) {
    sm.tab_key[0] = tab0;
    sm.tab_key[1] = tab1;
  }
  if (!runs) return -1;
  const int cnt = sm.fnv;
  if (!sm.ctl_ok) return cnt;
  // this lane's share of the dE terms and of the jump sums (taken by the even and odd warps of a pair)
  Slot sl[kJumpsPerWarp];
  int4 ix[2];
  if (eam) {
#pragma unroll
    for (int q = 0; q < kJumpsPerWarp; ++q) sl[q] = sm.slot[tid + kThreads * q];
    ix[0] = sm.ix[tid & 63][0];
    ix[1] = sm.ix[tid & 63][1];
  }
  double* const de_out = API && a.mode == kModeCalc ? a.api->de : nullptr;
  constexpr int D = eam ? 4 : 3;  // a hop changes the rates of vacancies within D cells of its origin

  // Density site i of 78 of a hop: jump b of parity p from the site with local index s and global
  // coordinates (gX, gY, gZ).  UPDATE: the delta of moving atom X is applied first; the density is
  // written through.
  auto refresh = [&](int i, int p, int b, int s, int X, int gX, int gY, int gZ, bool update) {
    const int32_t e = sm.rl[p][b][i];
    const int j = s + local_delta(e, R);
    int32_t v = rho_s[j];
    if (update) {
      v += sm.dfq[atom_index(static_cast<uint8_t>(X)) * 64 + unpack_sh_s(e) * 8 + unpack_sh_t(e)];
      rho_s[j] = v;
    }
    const int gx = wrap1(gX + unpack_dx(e), jc.sx), gy = wrap1(gY + unpack_dy(e), jc.sy),
              gz = wrap1(gZ + unpack_dz(e), jc.sz);
    lattice_put(jc.rho + static_cast<int64_t>(jc.px) * (gy + static_cast<int64_t>(jc.sy) * gz), jc.sx, gx, v);
  };
  // Occupancy o of the site (gX, gY, gZ), written through.
  auto put_occ = [&](int gX, int gY, int gZ, uint8_t o) {
    lattice_put(jc.occ + static_cast<int64_t>(jc.px) * (gY + static_cast<int64_t>(jc.sy) * gZ), jc.sx, gX, o);
  };
  // local coordinates inside the sector
  const int slx = 2 * R.hx, swx = 2 * R.w[0];
  auto in_sector = [&](int lx, int ly, int lz) -> bool {
    return static_cast<unsigned>(lx - slx) < static_cast<unsigned>(swx) &&
           static_cast<unsigned>(ly - 2) < static_cast<unsigned>(R.w[1]) &&
           static_cast<unsigned>(lz - 2) < static_cast<unsigned>(R.w[2]);
  };
  // The ordered total of one vacancy's rates and its selection (ABVIModel::calcRates, kmc.cpp:68-115,
  // and select, kmc.cpp:242-309), alike in every lane: the first of the running sums above u * total wins.
  // Jumps onto a vacancy hold 0.0.  Returns the jump, -1 for none.
  auto select_one = [&](const double2 (&r2)[4], double u, double& total) -> int {
    const double v0 = r2[0].x, v1 = v0 + r2[0].y, v2 = v1 + r2[1].x, v3 = v2 + r2[1].y, v4 = v3 + r2[2].x,
                 v5 = v4 + r2[2].y, v6 = v5 + r2[3].x, v7 = v6 + r2[3].y;
    total = v7;
    const double expected = u * v7;  // ModelAdapter::selectAndPerform
    int b = v7 > expected ? 7 : -1;
    b = v6 > expected ? 6 : b;
    b = v5 > expected ? 5 : b;
    b = v4 > expected ? 4 : b;
    b = v3 > expected ? 3 : b;
    b = v2 > expected ? 2 : b;
    b = v1 > expected ? 1 : b;
    b = v0 > expected ? 0 : b;
    return b;
  };
  // The clock thread's values of the block-round: the sector's clock, hops, n_act sum and evaluations, selections
  // made; left in shared memory by clock_end.
  double time = 0.0;
  int64_t nh = 0, nact_sum = 0, evals = cnt;
  int nsel = 0;
  // The selection used draw `it`; advances the sector's clock and decides whether its window is reached.  Returns
  // the residence time.
  auto clock_step = [&](int it, double total, bool hop, int n_act) -> double {
    const double dt = sm.dl[it & (kDrawRing - 1)] / total;
    time += dt;
    int stop = time < thr ? 0 : 1;
    nsel = it + 1;
    if (hop) {
      nact_sum += n_act;
      nh += 1;
      if (nh >= a.hop_cap) {
        atomicOr(a.status, kErrHopCap);
        stop = 1;
      }
    }
    sm.ctl_stop = stop;
    return dt;
  };
  auto clock_end = [&]() {
    if (tid != kClk) return;
    sm.c_time = time;
    sm.c_sel = nsel;
    sm.c_nh = nh;
    sm.c_nact = nact_sum;
    sm.c_evals = evals;
  };
  // The event record of the hop-th hop of this block-round (from 1).
  auto log_event = [&](int64_t hop, int from, int to, int X, double u, double total, double dt, int n_act, int nd) {
    const unsigned long long slot = atomicAdd(a.log_count, 1ull);
    if (slot < static_cast<unsigned long long>(a.log_cap)) {
      akmc_event* e = a.log + slot;
      e->round = round_now;
      e->hop = C.hops + hop - 1;
      e->from_site = from;
      e->to_site = to;
      e->block = C.local;
      e->species = X;
      e->u = u;
      e->total = total;
      e->dt = dt;
      e->n_act = n_act;
      e->n_dirty = nd;
      e->job = C.job;
      e->reserved = 0;
    } else {
      atomicOr(a.status, kErrLogOverflow);
    }
  };
  // One draw of each stream ahead of its use, a batch after the one in use; the batch's values when
  // it is complete.  Iteration `it`, by the last warp, whose lanes 0 and 1 hold the streams' states.
  auto draw_step = [&](int it) {
    if (lane < 2) draw_ahead(sm, dst, lane, (it + kDrawBatch) & (kDrawRing - 1));
    if ((it & (kDrawBatch - 1)) == kDrawBatch - 1) {
      __syncwarp();
      draw_values(sm, lane, (it + 1) & (kDrawRing - 1));
    }
  };
  if (!API && cnt == 1 && !eam) {
    // One vacancy, pair bond: warp 0 runs the whole hop loop without a CTA barrier (32 lanes hold the 4
    // bond counts of all 8 jumps); warp 1 draws ahead, a batch at a time.  Only occupancies change: the
    // path is kept and its sites written through when the loop ends (or the list is full).
    int2* const path = reinterpret_cast<int2*>(&sm.term[0][0]);  // (local site, site id)
    constexpr int kPath = 512;
    static_assert(kPath * sizeof(int2) <= sizeof(sm.term), "the path fits in the term sets");
    auto put_path = [&](int n, int t0, int nt) {
      for (int i = t0; i < n; i += nt) {
        const int2 e = path[i];
        const int t = e.y / jc.sx;
        put_occ(e.y % jc.sx, t % jc.sy, t / jc.sy, occ_s[e.x]);
      }
    };
    if (warp == 1) {
      // batch n is ready at the n-th meeting of the two warps; warp 0 leaves at the one it names
      for (int n = 1;; ++n) {
        if (lane < 2) {
          uint64_t x[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) x[i] = sm.str[lane][i];
#pragma unroll 1
          for (int k = 0; k < kDrawBatch; ++k) draw_ahead(sm, x, lane, (n * kDrawBatch + k) & (kDrawRing - 1));
#pragma unroll
          for (int i = 0; i < 4; ++i) sm.str[lane][i] = x[i];
        }
        __syncwarp();
        draw_values(sm, lane, (n * kDrawBatch) & (kDrawRing - 1));
        asm volatile("bar.sync 2, 64;" ::: "memory");
        if (*reinterpret_cast<volatile int32_t*>(&sm.ctl_stop) == n) break;
      }
    } else if (warp == 0) {
      const int4 pa = sm.vpk[0][0], pb = sm.vpk[0][1];
      int s = pa.x, lx = pa.y, ly = pa.z, lz = pa.w, gX = pb.x, gY = pb.y, gZ = pb.z, gid = pb.w;
      int it = 0, np = 1, meets = 0;
      if (lane == 0) path[0] = make_int2(s, gid);
      for (;; ++it) {
        pair_rates(sm, occ_s, 0, s, R.LX, R.LX * R.LY, nullptr);
        __syncwarp();
        const double2* r = reinterpret_cast<const double2*>(sm.rates[0]);
        const double2 r2[4] = {r[0], r[1], r[2], r[3]};
        double total;
        if (it > 0 && (it & (kDrawBatch - 1)) == 0) {
          // the next batch of draws, once it is sure that one is used: the meeting lets warp 1 write over the
          // batch before, which holds the streams' state after draw it - 1, the one a sector without events keeps
          select_one(r2, 0.0, total);
          if (fabs(total) < DBL_EPSILON) {
            time = thr;
            break;
          }
          asm volatile("bar.sync 2, 64;" ::: "memory");
          ++meets;
        }
        const double u = sm.du[it & (kDrawRing - 1)];
        const int b = select_one(r2, u, total);
        if (fabs(total) < DBL_EPSILON) {  // sublattice.inl:108-112
          time = thr;
          break;
        }
        const double dt = sm.dl[it & (kDrawRing - 1)] / total;
        time += dt;
        bool stop = !(time < thr);
        if (b >= 0) {  // else: a selection that finds no jump advances the clock only
          const int X = sm.vX[0][b];
          const int4 d = sm.d1[8 * (s & 1) + b];
          lx += d.y;
          ly += d.z;
          lz += d.w;
          gX = wrap1(gX + d.y, jc.sx);
          gY = wrap1(gY + d.z, jc.sy);
          gZ = wrap1(gZ + d.w, jc.sz);
          const int snew = s + d.x;
          const int nid = gX + jc.sx * (gY + jc.sy * gZ);
          const bool nact = in_sector(lx, ly, lz);
          nh += 1;
          evals += nact ? 1 : 0;
          __syncwarp();
          if (lane == 0) {
            occ_s[snew] = kV;
            occ_s[s] = static_cast<uint8_t>(X);
            path[np] = make_int2(snew, nid);
            if (a.log_cap > 0) log_event(nh, gid, nid, X, u, total, dt, 1, nact ? 1 : 0);
          }
          __syncwarp();
          s = snew;
          gid = nid;
          if (++np == kPath) {  // the list is full: write it through and start over from here
            put_path(np, lane, 32);
            __syncwarp();
            if (lane == 0) path[0] = make_int2(s, gid);
            np = 1;
          }
          if (nh >= a.hop_cap) {
            if (lane == 0) atomicOr(a.status, kErrHopCap);
            stop = true;
          }
          if (!nact && !stop) {  // the sector is empty now: its clock jumps to the window
            time = thr;
            stop = true;
          }
        }
        if (stop) {
          ++it;
          break;
        }
      }
      if (lane == 0) {
        sm.vpk[0][0] = make_int4(s, lx, ly, lz);
        sm.vpk[0][1] = make_int4(gX, gY, gZ, gid);
        sm.c_time = time;
        sm.c_sel = it;
        sm.c_nh = nh;
        sm.c_nact = nh;
        sm.c_evals = evals;
        sm.c_path = np;
        // the next meeting is warp 1's last
        *reinterpret_cast<volatile int32_t*>(&sm.ctl_stop) = meets + 1;
      }
      __syncwarp();
      asm volatile("bar.sync 2, 64;" ::: "memory");
    }
    __syncthreads();
    put_path(sm.c_path, tid, kThreads);
  } else if (!API && cnt == 1) {
    // One vacancy, EAM (nearly every block-round at dilute concentrations): its record lives in
    // registers, alike in every thread.  A hop is two phases, a CTA barrier after each:
    //  A  warps 0 and 1: the 8 jump sums and rates from the dE terms; the others: jumps with a solute
    //     target, then what the last hop left to do off the chain (its clock, the draws ahead, the
    //     write-through of its 78 densities and two occupancies);
    //  B  every warp selects, then the density deltas and dE terms at the vacancy's new site.
    constexpr int kWt0 = 64, kWtN = kEvalWarps == 8 ? 96 : 64;  // write-through threads (densities)
    constexpr int kOc = kEvalWarps == 8 ? 160 : 96;             // and of the two occupancies
    const int4 pa = sm.vpk[0][0], pb = sm.vpk[0][1];
    int s = pa.x, lx = pa.y, ly = pa.z, lz = pa.w, gX = pb.x, gY = pb.y, gZ = pb.z, gid = pb.w;
#pragma unroll
    for (int q = 0; q < kJumpsPerWarp; ++q)
      foot_terms<KIND, false>(sm, 0, occ_s, rho_s, s, sl[q], tid + kThreads * q, FT, 0, 0, 0, true);
    __syncthreads();
    // the last selection: its uniform, total, jump, atom and origin; g*: the vacancy's global record,
    // kept by the warps that write (not 0 and 1)
    bool hop = false, nact = true;
    int b = 0, X = 0, os = 0;
    int4 d = make_int4(0, 0, 0, 0);
    double u = 0.0, total = 0.0;
    for (int it = 0;; ++it) {
      if (warp < 2) {
        if (nact) jump_rates<KIND>(sm, 0, occ_s, 0, s, warp, ix, nullptr);
      } else {
        if (nact) {
          unsigned solutes = solute_jumps(sm, occ_s, s);
          for (int q = 2; solutes; ++q) {  // the k-th of them to warp 2 + k
            if ((q - 2) % (kEvalWarps - 2) == warp - 2)
              solute_rate<KIND>(sm, occ_s, rho_s, 0, s, __ffs(static_cast<int>(solutes)) - 1, R.LX, R.LY, *a.geo, FT,
                                nullptr);
            solutes &= solutes - 1;
          }
        }
        if (it > 0) {
          const int oX = gX, oY = gY, oZ = gZ, oid = gid;
          if (hop) {
            gX = wrap1(gX + d.y, jc.sx);
            gY = wrap1(gY + d.z, jc.sy);
            gZ = wrap1(gZ + d.w, jc.sz);
            gid = gX + jc.sx * (gY + jc.sy * gZ);
          }
          if (tid == kClk) {
            const double dt = clock_step(it - 1, total, hop, 1);
            if (hop) {
              evals += nact ? 1 : 0;
              if (a.log_cap > 0) log_event(nh, oid, gid, X, u, total, dt, 1, nact ? 1 : 0);
            }
          }
          if (hop) {
            if (tid >= kWt0 && tid < kWt0 + kWtN)
              for (int i = tid - kWt0; i < kRefreshN; i += kWtN) refresh(i, os & 1, b, os, X, oX, oY, oZ, false);
            if (tid == kOc || tid == kOc + 1) {
              const bool to = tid == kOc;
              put_occ(to ? gX : oX, to ? gY : oY, to ? gZ : oZ, to ? static_cast<uint8_t>(kV) : static_cast<uint8_t>(X));
            }
          }
          if (warp == kEvalWarps - 1) draw_step(it - 1);
        }
      }
      __syncthreads();
      AKMC_PHASE(2);
      if (it > 0 && sm.ctl_stop) break;
      if (!nact) {  // the sector is empty now: its clock jumps to the window
        time = thr;
        break;
      }
      const double2* r = reinterpret_cast<const double2*>(sm.rates[0]);
      const double2 r2[4] = {r[0], r[1], r[2], r[3]};
      u = sm.du[it & (kDrawRing - 1)];
      const int sel = select_one(r2, u, total);
      if (fabs(total) < DBL_EPSILON) {  // sublattice.inl:108-112
        time = thr;
        break;
      }
      hop = sel >= 0;  // else: a selection that finds no jump advances the clock only
      if (hop) {
        b = sel;
        X = sm.vX[0][b];
        d = sm.d1[8 * (s & 1) + b];
        os = s;
        s += d.x;
        lx += d.y;
        ly += d.z;
        lz += d.w;
        nact = in_sector(lx, ly, lz);
        // perform (ABVIModel::perform, kmc.cpp:358-396) on the staged region
        if (tid == kCtl) {
          occ_s[s] = kV;
          occ_s[os] = static_cast<uint8_t>(X);
        }
#pragma unroll
        for (int q = 0; q < kJumpsPerWarp; ++q)
          foot_terms<KIND, true>(sm, 0, occ_s, rho_s, s, sl[q], tid + kThreads * q, FT, b, X, os, nact);
      }
      __syncthreads();
      AKMC_PHASE(5);
    }
    if (tid == 64) {
      sm.vpk[0][0] = make_int4(s, lx, ly, lz);
      sm.vpk[0][1] = make_int4(gX, gY, gZ, gid);
    }
    clock_end();
  } else {
    const bool rich = eam && sm.job.rich != 0;
    // vacancy k lies within D cells of the cell (qx, qy, qz) and in the sector
    auto dirty = [&](int k, int qx, int qy, int qz) -> bool {
      const int4 v = sm.vpk[k][0];
      return sm.vact[k] && abs((v.y >> 1) - qx) <= D && abs(v.z - qy) <= D && abs(v.w - qz) <= D;
    };
    int c = 0;  // set of the ordered list in use
    int ksel = -1, snew = 0;
    // vacancies to evaluate: all of them at first, then those the last hop made dirty
    unsigned m0 = cnt >= 32 ? kFull : (1u << cnt) - 1u, m1 = cnt > 32 ? (cnt >= 64 ? kFull : (1u << (cnt - 32)) - 1u) : 0u;
    for (int it = 0;; ++it) {
      auto next = [&]() -> int {  // takes one vacancy off the masks, -1 when there is none
        if (m0) {
          const int k = __ffs(static_cast<int>(m0)) - 1;
          m0 &= m0 - 1;
          return k;
        }
        if (m1) {
          const int k = 31 + __ffs(static_cast<int>(m1));
          m1 &= m1 - 1;
          return k;
        }
        return -1;
      };
      auto site = [&](int k) -> int { return k == ksel ? snew : sm.vpk[k][0].x; };
      if (!eam) {  // a warp takes a vacancy
        for (int n = 0;; ++n) {
          const int k = next();
          if (k < 0) break;
          if (n % kEvalWarps == warp) pair_rates(sm, occ_s, k, site(k), R.LX, R.LX * R.LY, de_out);
        }
      } else if (rich) {
        rich_rates<KIND, W>(sm, occ_s, rho_s, m0, m1, ksel, snew, R.LX, R.LY, a.geo, a.pots + sm.job.pot, a.status, de_out);
        m0 = m1 = 0;
      } else {
        // two vacancies at a time: their dE terms by all warps, a barrier, then the jump sums of the
        // first by warps 0 and 1 and of the second by warps 2 and 3, solute targets by the last warps
        while (m0 | m1) {
          const int ka = next(), kb = next();
          const int la = site(ka), lb = kb >= 0 ? site(kb) : la;
#pragma unroll
          for (int q = 0; q < kJumpsPerWarp; ++q)
            foot_terms<KIND, false>(sm, 0, occ_s, rho_s, la, sl[q], tid + kThreads * q, FT, 0, 0, 0, true);
          if (kb >= 0)
#pragma unroll
            for (int q = 0; q < kJumpsPerWarp; ++q)
              foot_terms<KIND, false>(sm, 1, occ_s, rho_s, lb, sl[q], tid + kThreads * q, FT, 0, 0, 0, true);
          __syncthreads();
          if (warp < 4) {
            if (warp < 2) jump_rates<KIND>(sm, 0, occ_s, ka, la, warp & 1, ix, de_out);
            else if (kb >= 0) jump_rates<KIND>(sm, 1, occ_s, kb, lb, warp & 1, ix, de_out);
          }
          constexpr int kw = kEvalWarps == 8 ? 4 : 0;
          if (warp >= kw) {
            unsigned sol = solute_jumps(sm, occ_s, la) | (kb >= 0 ? solute_jumps(sm, occ_s, lb) << 8 : 0u);
            for (int n = 0; sol; ++n) {  // the solute targets of both, one after another to these warps
              const int q = __ffs(static_cast<int>(sol)) - 1;
              if (n % (kEvalWarps - kw) == warp - kw)
                solute_rate<KIND>(sm, occ_s, rho_s, q < 8 ? ka : kb, q < 8 ? la : lb, q & 7, R.LX, R.LY, *a.geo, FT,
                                  de_out);
              sol &= sol - 1;
            }
          }
          if (m0 | m1) __syncthreads();  // the term sets are written again
        }
      }
      __syncthreads();
      AKMC_PHASE(2);
      // ordered total over the z-y-x sorted list; lane i keeps the running sum through its vacancy
      // (i or i + 32 of the list)
      const int nord = sm.nord[c];
      double total = 0.0, s0 = 0.0, s1 = 0.0;
      for (int i = 0; i < nord; ++i) {
        const double2* r2 = reinterpret_cast<const double2*>(sm.rates[sm.ord[c][i]]);
        const double2 a0 = r2[0], a1 = r2[1], a2 = r2[2], a3 = r2[3];
        total += a0.x;
        total += a0.y;
        total += a1.x;
        total += a1.y;
        total += a2.x;
        total += a2.y;
        total += a3.x;
        total += a3.y;
        if (i == lane) s0 = total;
        if (i == lane + 32) s1 = total;
      }
      if (API && a.mode == kModeCalc) {  // akmc_calculate: the sector's vacancies with their jump rates
        if (tid < cnt) a.api->sites[tid] = sm.vpk[tid][1].w;
        for (int i = tid; i < 8 * cnt; i += kThreads) a.api->rates[i] = (&sm.rates[0][0])[i];
        if (tid == kClk) {
          a.api->total = total;
          a.api->count = cnt;
        }
        break;
      }
      if (fabs(total) < DBL_EPSILON) {  // sublattice.inl:108-112
        if (tid == kClk) {
          if (API) {
            a.api->event.from_site = -1;
            a.api->event.total = total;
          } else {
            time = thr;
          }
        }
        break;
      }
      const double u = API ? a.api_u : sm.du[it & (kDrawRing - 1)];
      const double expected = u * total;  // ModelAdapter::selectAndPerform
      // the first vacancy whose running sum is above u * total (the sums never fall), then the jump
      const unsigned f0 = __ballot_sync(kFull, lane < nord && s0 > expected);
      const unsigned f1 = __ballot_sync(kFull, lane + 32 < nord && s1 > expected);
      const bool hop = (f0 | f1) != 0;
      const int pos = f0 ? __ffs(static_cast<int>(f0)) - 1 : f1 ? 31 + __ffs(static_cast<int>(f1)) : 0;
      double x = 0.0;
      if (pos > 0) x = __shfl_sync(kFull, pos <= 32 ? s0 : s1, (pos - 1) & 31);
      ksel = sm.ord[c][pos];
      {
        const double2* r2 = reinterpret_cast<const double2*>(sm.rates[ksel]);
        const double2 a0 = r2[0], a1 = r2[1], a2 = r2[2], a3 = r2[3];
        const double rr[8] = {a0.x, a0.y, a1.x, a1.y, a2.x, a2.y, a3.x, a3.y};
#pragma unroll
        for (int q = 0; q < 8; ++q) x += q <= lane ? rr[q] : 0.0;
      }
      const unsigned above = __ballot_sync(kFull, lane < 8 && x > expected);
      const int b = hop ? __ffs(static_cast<int>(above)) - 1 : 0;
      const int X = sm.vX[ksel][b];
      const int4 pa = sm.vpk[ksel][0], pb = sm.vpk[ksel][1];
      const int s = pa.x, p = s & 1;
      const int qx = pa.y >> 1, qy = pa.z, qz = pa.w;  // the hop's origin cell
      const int4 d = sm.d1[8 * p + b];
      const int nlx = pa.y + d.y, nly = qy + d.z, nlz = qz + d.w;
      snew = s + d.x;
      const bool nact = in_sector(nlx, nly, nlz);
      const int nX = wrap1(pb.x + d.y, jc.sx), nY = wrap1(pb.y + d.z, jc.sy), nZ = wrap1(pb.z + d.w, jc.sz);
      const int32_t nid = nX + jc.sx * (nY + jc.sy * nZ);
      double dt = 0.0;
      if (warp < 3) {
        if (eam && hop && tid < kRefreshN) refresh(tid, p, b, s, X, pb.x, pb.y, pb.z, true);
      } else {
        if (tid == 96 && hop) {
          occ_s[snew] = kV;
          occ_s[s] = static_cast<uint8_t>(X);
          put_occ(nX, nY, nZ, kV);
          put_occ(pb.x, pb.y, pb.z, static_cast<uint8_t>(X));
        }
        if (warp == kOrdWarp && hop) {
          // the hopped vacancy leaves its place in the ordered list and re-enters at its new site
          // id if it is still inside the sector; every other one moves by at most one place
          int less = 0;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int i = lane + 32 * h;
            const bool other = i < nord && i != pos;
            const int k = other ? sm.ord[c][i] : 0;
            const bool before = other && sm.vpk[k][1].w < nid;
            less += __popc(__ballot_sync(kFull, before));
            if (other) sm.ord[c ^ 1][i - (i > pos ? 1 : 0) + (nact && !before ? 1 : 0)] = k;
          }
          if (lane == 0) {
            if (nact) sm.ord[c ^ 1][less] = ksel;
            sm.nord[c ^ 1] = nord - 1 + (nact ? 1 : 0);
          }
        }
        if (tid == kClk) {
          if (API) {
            if (hop) {
              nh = 1;
              nact_sum += nord;
            }
            sm.ctl_stop = 1;  // the per-hop entry point stops after one selection
          } else {
            dt = clock_step(it, total, hop, nord);
          }
        }
        if (!API && warp == kEvalWarps - 1) draw_step(it);
      }
      __syncthreads();
      AKMC_PHASE(4);
      if (hop) {
        m0 = __ballot_sync(kFull, lane < cnt && (lane == ksel ? nact : dirty(lane, qx, qy, qz)));
        if (cnt > 32) m1 = __ballot_sync(kFull, lane + 32 < cnt && (lane + 32 == ksel ? nact : dirty(lane + 32, qx, qy, qz)));
        c ^= 1;
        if (tid == 96) {
          sm.vpk[ksel][0] = make_int4(snew, nlx, nly, nlz);
          sm.vpk[ksel][1] = make_int4(nX, nY, nZ, nid);
          sm.vact[ksel] = nact ? 1 : 0;
        }
      }
      if (tid == kClk && hop) {
        const int nd = __popc(m0) + __popc(m1);
        evals += nd;
        if (!API && a.log_cap > 0) log_event(nh, pb.w, nid, X, u, total, dt, nord, nd);
      }
      if (API && tid == kClk) {
        akmc_event* e = &a.api->event;
        e->round = 0;
        e->hop = C.hops;
        e->from_site = hop ? pb.w : -1;
        e->to_site = hop ? nid : -1;
        e->block = C.local;
        e->species = hop ? X : 0;
        e->u = u;
        e->total = total;
        e->dt = 0.0;
        e->n_act = nord;
        e->n_dirty = hop ? __popc(m0) + __popc(m1) : 0;
        e->job = C.job;
        e->reserved = 0;
      }
      if (sm.ctl_stop) break;
    }
    clock_end();
  }
  __syncthreads();
  AKMC_PHASE(6);
  if (API && a.mode == kModeCalc) return cnt;
  // The lattice was written through at every hop (or at the end of the pair-bond loop); the vacancy positions,
  // the block's record and the counters remain.
  if (tid < cnt) a.vac_site[sm.vidx[tid]] = sm.vpk[tid][1].w;
  if (tid == 0) {
    BlockDev& B = a.blocks[C.gb];
    if (!API) {
      B.evo[sec] = C.evo + sm.c_time;
      const int n = sm.c_sel;  // draws the selections used: the streams move on by as many
      if (n > 0) {
        const int slot = (n - 1) & (kDrawRing - 1);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          B.xs[i] = C.str[0][i] = sm.sts[slot][0][i];
          B.xt[i] = C.str[1][i] = sm.sts[slot][1][i];
        }
      }
    }
    C.hops += sm.c_nh;
    B.hops = C.hops;
  }
  if (tid == 32) {
    const int64_t nh = sm.c_nh;
    if (sm.acc_job != C.job) {
      if (sm.acc_job >= 0 && sm.acc_job_hops)
        atomicAdd(reinterpret_cast<unsigned long long*>(&a.jobs[sm.acc_job].hops), sm.acc_job_hops);
      sm.acc_job = C.job;
      sm.acc_job_hops = 0;
    }
    sm.acc_job_hops += static_cast<unsigned long long>(nh);
    sm.acc[0] += static_cast<unsigned long long>(nh);
    sm.acc[1] += static_cast<unsigned long long>(sm.c_evals);
    sm.acc[2] += 1ull;
    sm.acc[3] += static_cast<unsigned long long>(sm.c_nact);
    sm.acc[4] += static_cast<unsigned long long>(R.nt);
    sm.acc[5] += static_cast<unsigned long long>(nh * (eam ? 2 + kRefreshN : 2));
  }
  return cnt;
}

// The region's arrays after Smem, each starting on a 128-byte boundary of the shared window
// (tensor copies want it; hop_smem_bytes leaves room for the padding).
__device__ __forceinline__ void carve(uint8_t* smem, int nreg, Smem*& sm, uint8_t*& occ_s, int32_t*& rho_s) {
  sm = reinterpret_cast<Smem*>(smem);
  uint8_t* p = smem + sizeof(Smem);
  p += (128u - (smem_u32(p) & 127u)) & 127u;
  rho_s = reinterpret_cast<int32_t*>(p);
  occ_s = occ_of(rho_s, nreg);
}

// The site's coordinates and whether it lies in the region's sector.
__device__ __forceinline__ bool region_site(const Region& R, const JobDev& J, int32_t s, int& X, int& y, int& z) {
  const int t = s / J.sx;
  X = s - t * J.sx;
  z = t / J.sy;
  y = t - z * J.sy;
  return static_cast<unsigned>((X >> 1) - R.slo[0]) < static_cast<unsigned>(R.w[0]) &&
         static_cast<unsigned>(y - R.slo[1]) < static_cast<unsigned>(R.w[1]) &&
         static_cast<unsigned>(z - R.slo[2]) < static_cast<unsigned>(R.w[2]);
}

// Block gb's record as round[0] (kernels whose blocks no sweep hands over); CTA-wide, no barrier.
__device__ __forceinline__ void load_block(Smem& sm, const RoundArgs& a, int gb, int sec) {
  const int tid = threadIdx.x;
  const BlockDev& B = a.blocks[gb];
  Round& C = sm.round[0];
  if (tid == 0) {
    C.gb = gb;
    C.job = B.job;
    C.local = B.local_id;
    C.r = B.round;
    C.hops = B.hops;
    C.evo = B.evo[sec];
  } else if (tid >= 32 && tid < 35) {
    C.c0[tid - 32] = B.c0[tid - 32];
    C.c1[tid - 32] = B.c1[tid - 32];
  } else if (tid >= 64 && tid < 72) {
    const int q = tid - 64;
    C.str[q >> 2][q & 3] = q < 4 ? B.xs[q] : B.xt[q - 4];
  }
}

// One block whose sector's vacancies k_bucket listed (k_hop), CTA-wide.
template <int KIND, int W>
__device__ __forceinline__ void listed_block(const RoundArgs& a, int gb, int sec, uint8_t* smem) {
  Smem& sm0 = *reinterpret_cast<Smem*>(smem);
  const int tid = threadIdx.x;
  __syncthreads();  // the previous block's readers are done
  load_block(sm0, a, gb, sec);
  if (tid == 0) sm0.fnv = min(a.blocks[gb].cnt, kMaxV);
  __syncthreads();
  Round& C = sm0.round[0];
  load_job(sm0, a, C.job);
  Region R;
  make_region(C.c0, C.c1, sm0.job, sec, R);
  Smem* sm;
  uint8_t* occ_s;
  int32_t* rho_s;
  carve(smem, R.n, sm, occ_s, rho_s);
  stage_region<KIND, W>(*sm, a, R, occ_s, rho_s);
  if (tid < sm->fnv) {
    const int v = a.blk_list[static_cast<int64_t>(gb) * kMaxV + tid];
    const int32_t s = a.vac_site[v];
    int X, y, z;
    region_site(R, sm->job, s, X, y, z);
    put_record(*sm, R, tid, v, s, X, y, z);
  }
  run_block<KIND, W, false>(a, *sm, C, R, occ_s, rho_s, sec);
}

__global__ void k_bucket(RoundArgs a) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= a.nvac) return;
  const int j = a.vac_job[v];
  if (j < 0) return;  // a free entry of the vacancy table (a context with room for admitted jobs)
  const JobDev& J = a.jobs[j];
  if (J.done) return;
  const int sec = sector_of_round(J.round);
  const int s = a.vac_site[v];
  const int X = s % J.sx;
  const int t = s / J.sx;
  const int c[3] = {X >> 1, t % J.sy, t / J.sy};
  int k[3];
  for (int d = 0; d < 3; ++d) k[d] = block_of(c[d], J.n[d], J.nb[d]);
  const int gb = J.block0 + k[0] + J.nb[0] * (k[1] + J.nb[1] * k[2]);
  BlockDev& B = a.blocks[gb];
  for (int d = 0; d < 3; ++d) {
    const int half = (B.c1[d] - B.c0[d]) / 2;
    const int hi = (c[d] - B.c0[d]) >= half ? 1 : 0;
    if (hi != ((sec >> d) & 1)) return;
  }
  const int slot = atomicAdd(&B.cnt, 1);
  if (slot >= kMaxV) {
    atomicOr(a.status, kErrVacOverflow);
    return;
  }
  a.blk_list[static_cast<int64_t>(gb) * kMaxV + slot] = v;
  if (slot == 0) {
    const int q = atomicAdd(a.n_active, 1);
    a.active[q] = gb;
  }
}

__device__ void init_cta_smem(uint8_t* smem) {
  Smem* sm = reinterpret_cast<Smem*>(smem);
  if (threadIdx.x == 0) {
    sm->win_pot = -1;
    sm->job_key = -1;
    sm->fnv = 0;
    sm->tab_key[0] = sm->tab_key[1] = -1;
    sm->mbar_phase = 0;
    sm->mbst_phase = 0;
    mbar_init(&sm->mbar);
    mbar_init(&sm->mbar_st);
    for (int i = 0; i < 6; ++i) sm->acc[i] = 0;
    sm->acc_job = -1;
    sm->acc_job_hops = 0;
  }
  __syncthreads();
}

// Adds the CTA's counters (summed by the control thread) to the device counters; CTA-wide.
template <int W>
__device__ void cta_flush(const RoundArgs& a, uint8_t* smem) {
  AKMC_SHAPE(W);
  Smem* sm = reinterpret_cast<Smem*>(smem);
  __syncthreads();
  if (threadIdx.x == kCtl) {
    const int idx[6] = {0, 1, 3, 4, 5, 6};
    for (int i = 0; i < 6; ++i)
      if (sm->acc[i]) atomicAdd(a.counters + idx[i], sm->acc[i]);
    if (sm->acc_job >= 0 && sm->acc_job_hops)
      atomicAdd(reinterpret_cast<unsigned long long*>(&a.jobs[sm->acc_job].hops), sm->acc_job_hops);
  }
}

__device__ __forceinline__ int job_kind(const JobDev& J) {
  return J.model == AKMC_MODEL_PAIRBOND ? kPairBond : (J.precision == AKMC_FP32C ? kEam32 : kEam64);
}

// One kernel per energy kind, so each holds only its own hop loop (instruction-cache
// footprint); items of other kinds are left to their kernel.
template <int KIND, int W>
__global__ void __launch_bounds__(Shape<W>::kThreads, Shape<W>::kCtasPerSm) k_hop(RoundArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int na = *a.n_active;
  if (static_cast<int>(blockIdx.x) >= na) return;
  init_cta_smem(smem);
  for (int item = blockIdx.x; item < na; item += gridDim.x) {
    const int gb = a.active[item];
    const BlockDev& B = a.blocks[gb];
    if (job_kind(a.jobs[B.job]) != KIND) continue;
    listed_block<KIND, W>(a, gb, sector_of_round(B.round), smem);
  }
  cta_flush<W>(a, smem);
}

// ---------------------------------------------------------------------------
// Asynchronous round schedule.  A block's round r may run once, for every neighbour
// offset d in {-1,0,1}^3, the neighbour block has completed its latest earlier round
// whose staged region (sector plus a 2-cell halo) meets region r (flow_lag); rounds of
// different blocks then run in any order and the result equals the round-by-round
// schedule (sublattice.inl:61-179): a round reads and writes only its region, every
// write that a region can see comes from an earlier round that it waits for, and rounds
// that run at the same time have disjoint regions.  Each block keeps the ids of the
// vacancies in its area in kFlowSlots slots; a hop that carries a vacancy into a
// neighbour's area moves the id there.
//
// k_flow is persistent.  Each sweep a thread looks at one block.  A ready round whose sector holds
// no vacancy is one compare-and-swap: the clock's jumps to the window (sublattice.inl:108-112) are
// caught up when the sector next holds one, or when the launch ends (flow_clock).  A ready round
// with vacancies is handed to the CTA, which runs the hop loop for it.  A block is held with a
// lease while anything works on it, and nothing waits while holding a lease.
//
// A block's word (fstate = rounds << 9 | sector mask << 1 | lease) holds its completed rounds, a
// bit for each sector that has a vacancy, and the lease, so that one compare-and-swap checks all
// three: a neighbour that brought a vacancy into the sector after the word was read makes it fail.
// One add after a fence publishes a round run and frees the lease.  A block at its target keeps
// the lease bit, so a sweep reads nothing else of it.  B.round is refreshed from the word when the
// launch ends.
// A single-block job's rounds depend on nothing else, so the CTA that ran one runs the next
// straight away when it holds no other round of the sweep (its hop budget is checked here, at
// each time-step boundary).

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Release/acquire fence at GPU scope (lighter than the sequentially consistent __threadfence).
__device__ __forceinline__ void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void add_release_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p));
  return v;
}

__host__ __device__ constexpr int flow_sector(int phase) {
  constexpr int ring[8] = {0, 7, 2, 5, 3, 4, 1, 6};  // sector_of_round
  return ring[phase & 7];
}
// The neighbours a round waits for.  Per dimension a +1 neighbour's regions meet ours only between our high half
// and its low half (block edges >= 8 cells, halos of 2), a -1 neighbour's only between our low half and its high
// half.  So the round of sector s meets seven neighbours: those in the directions that s points to (bit a of s:
// + in dimension a, else -), in any nonempty set m of the dimensions, each in the rounds whose sector differs from
// s in every dimension of m.  Bits 4m..4m+3 of flow_lags: rounds back to the latest such round.
__host__ __device__ constexpr uint32_t flow_lags(int phase) {
  uint32_t v = 0;
  for (int m = 1; m < 8; ++m)
    for (int k = 7; k >= 1; --k)
      if (((flow_sector(phase + 8 - k) ^ flow_sector(phase)) & m) == m)
        v = (v & ~(15u << (4 * m))) | (static_cast<uint32_t>(k) << (4 * m));
  return v;
}
__constant__ const uint32_t kFlowLags[8] = {flow_lags(0), flow_lags(1), flow_lags(2), flow_lags(3),
                                            flow_lags(4), flow_lags(5), flow_lags(6), flow_lags(7)};

__device__ __forceinline__ int wrapb(int v, int m) { return v < 0 ? v + m : (v >= m ? v - m : v); }

// Global index of the neighbour of block local_id one step (dir = -1 or 1) along dimension d.
__device__ __forceinline__ int flow_neighbour(const JobDev& J, int local_id, int d, int dir) {
  int b[3] = {local_id % J.nb[0], (local_id / J.nb[0]) % J.nb[1], local_id / (J.nb[0] * J.nb[1])};
  b[d] = wrapb(b[d] + dir, J.nb[d]);
  return J.block0 + b[0] + J.nb[0] * (b[1] + J.nb[1] * b[2]);
}

// A multi-block job with a hop budget ends at the end of the first time step at which the hops
// of all its blocks reach the budget, so its round b at a time-step boundary (b = 8, 16, ...)
// runs only once every block of the job has reached b; the blocks' hops at b (hops_at, written
// when each reached b) then decide.  Blocks of the job are thus never a whole time step apart,
// and the two hops_at slots never hold a boundary someone still reads.  Returns 0 while a block
// is behind, 1 to run round b, 2 when the job ends at b.
__device__ int budget_gate(const RoundArgs& a, const JobDev& J, int64_t b) {
  if (J.hop_budget <= 0 || J.nblocks == 1 || b == 0 || (b & 7)) return 1;
  bool all = true;
  for (int k = 0; k < J.nblocks; ++k)
    all &= static_cast<int64_t>(ld_relaxed_u64(&a.fstate[J.block0 + k]) >> kWordShift) >= b;
  if (!all) return 0;
  fence_acq_rel();  // the hops_at written before those rounds were published
  const int slot = static_cast<int>((b >> 3) & 1);
  int64_t sum = 0;
  for (int k = 0; k < J.nblocks; ++k) sum += __ldcg(&a.blocks[J.block0 + k].hops_at[slot]);
  return sum >= J.hop_budget ? 2 : 1;
}

// A block's row of RoundArgs::nbr, one 32-byte sector: the index differences to its six face neighbours (-x, +x,
// -y, +y, -z, +z; 0 where the dimension has one block), a flags word and the job.  Flags: the energy kind (kNbrFree
// for a free block slot); kNbrGate: the job's hop budget gates its rounds at time-step boundaries (budget_gate);
// kNbrSolo: a single-block job, whose rounds wait for no other block.
constexpr int kNbrFree = 3, kNbrKindMask = 3, kNbrGate = 4, kNbrSolo = 8;

// Whether the round the word w of block gb is at may run: the seven neighbours it meets have completed the rounds it
// waits for.  Their words are read with relaxed loads, all in flight at once, as wide as every other access to them (the
// loads pair with the publishing adds); the caller fences afterwards (an acquire) before it relies on anything those
// rounds wrote.  Only the low halves are compared: neighbours are within a few rounds of each other, so the
// difference of 23 bits of the rounds is exact.
// Bounded by the SM's path to L2: a sweep of 256 blocks that read all 26 neighbours' words and a 128-byte row of
// their indices took 2.5K cycles for the rows and 3.8K for the words (256^3 lattice). One 32-byte
// sector and seven words, and empty rounds passed over in the word alone instead of under a lease with their
// record: 1024 rounds of the 256^3 lattice 27.9 -> 24.1 ms, 512 rounds of 180 pair-bond blocks 10.8 -> 10.0.
__device__ __forceinline__ bool flow_ready(const RoundArgs& a, int gb, unsigned long long w, const int4& d0, const int4& d1) {
  const int ph = static_cast<int>(w >> kWordShift) & 7, s = sector_of_round(ph);
  const uint32_t lags = kFlowLags[ph];
  const int d[3] = {s & 1 ? d0.y : d0.x, s & 2 ? d0.w : d0.z, s & 4 ? d1.y : d1.x};
  int o[8];
  uint32_t lo[8];
#pragma unroll
  for (int m = 1; m < 8; ++m) {
    o[m] = gb + (m & 1 ? d[0] : 0) + (m & 2 ? d[1] : 0) + (m & 4 ? d[2] : 0);
    lo[m] = static_cast<uint32_t>(ld_relaxed_u64(&a.fstate[o[m]]));
  }
  const uint32_t base = static_cast<uint32_t>(w) >> kWordShift << kWordShift;
  bool ok = true;
#pragma unroll
  for (int m = 1; m < 8; ++m) {
    const int ahead = static_cast<int32_t>((lo[m] >> kWordShift << kWordShift) - base) >> kWordShift;
    ok = ok && (o[m] == gb || ahead + static_cast<int>((lags >> (4 * m)) & 15u) > 0);
  }
  return ok;
}

// A sector's clock e, which accounts for `from` of its rounds, after `to` of them when those between found no
// vacancy (total = 0: the clock jumps to the window if it is behind, sublattice.inl:108-112).
__device__ __forceinline__ double flow_clock(double e, int64_t from, int64_t to, double window) {
  for (int64_t t = from; t < to; ++t) {
    const double thr = static_cast<double>(t + 1) * window - e;
    double sector_time = 0.0;
    if (sector_time < thr) sector_time = thr;
    e += sector_time;
  }
  return e;
}
// Rounds of the sector of phase p among a block's first r.
__device__ __forceinline__ int64_t flow_steps(int64_t r, int p) { return (r + 7 - p) >> 3; }

// Block whose area holds site s (the reference's rank split, as k_bucket) and the sector of that
// block the site lies in.
__device__ __noinline__ int owner_sector(const JobDev& J, int32_t s, int* sec) {
  const int X = s % J.sx;
  const int t = s / J.sx;
  const int c[3] = {X >> 1, t % J.sy, t / J.sy};
  int k[3];
  int q = 0;
  for (int d = 0; d < 3; ++d) {
    k[d] = block_of(c[d], J.n[d], J.nb[d]);
    const int lo = k[d] * (J.n[d] / J.nb[d]) + min(k[d], J.n[d] % J.nb[d]);  // the rank split
    const int hi = (k[d] + 1) * (J.n[d] / J.nb[d]) + min(k[d] + 1, J.n[d] % J.nb[d]);
    if (c[d] - lo >= (hi - lo) / 2) q |= 1 << d;
  }
  *sec = q;
  return J.block0 + k[0] + J.nb[0] * (k[1] + J.nb[1] * k[2]);
}

// A block's vacancy slot: the vacancy's id and site in one word, so that one store or compare-and-swap moves it.
constexpr unsigned long long kNoVacancy = ~0ull;
__device__ __forceinline__ unsigned long long slot_word(int v, int32_t site) {
  return static_cast<unsigned long long>(static_cast<uint32_t>(v)) << 32 | static_cast<uint32_t>(site);
}
// Puts vacancy v into a free slot of block o, then marks its sector occupied.  The word becomes readable as a
// whole; a round of o that can see the vacancy waits for this block's round, which is published after both.
__device__ void flow_give(const RoundArgs& a, int o, int v, int32_t site, int osec) {
  unsigned long long* const slots = a.vslot + static_cast<int64_t>(o) * kFlowSlots;
  for (int k = 0; k < a.flow_slots; ++k) {
    const int i = (v + k) & (a.flow_slots - 1);
    if (atomicCAS(slots + i, kNoVacancy, slot_word(v, site)) == kNoVacancy) {
      atomicOr(&a.fstate[o], 2ull << osec);
      return;
    }
  }
  atomicOr(a.status, kErrVacOverflow);
}

// Adds n completed rounds to a held block's word and keeps (keep) or frees the lease, in one release: cumulative, so
// writes of other threads of the CTA that a barrier ordered before this call are released too.  `reached`: this
// lease holder moved the block onto its target (each block is counted once), where the lease stays.
__device__ __forceinline__ void flow_publish(const RoundArgs& a, int gb, int64_t n, bool keep, bool reached, int kind) {
  const unsigned long long v = (static_cast<unsigned long long>(n) << kWordShift) - (keep || reached ? 0 : 1);
  if (v != 0) add_release_u64(&a.fstate[gb], v);
  if (reached) atomicAdd(&a.flow_done[kind], 1);
}

// Lease held, one thread, block gb of job `job`, w its word, its round ready: passes over the rounds whose sectors
// hold no vacancy (one for a multi-block job; for a single-block job, whose rounds wait for nothing, all up to the
// next that has some) and leaves the block's round in *rn (the caller publishes it).  Returns true when it stops at
// a round with vacancies, which is then described in *C (C null: in the next entry of sm.round, false when `take`
// are full); false when the target is reached, the next round has to be looked at anew, or a budget holds it back.
// *reached: this call moved the block onto its target (by passing over rounds, or by a budget moving the target).
__device__ __forceinline__ bool flow_advance(const RoundArgs& a, Smem& sm, int gb, int job, bool solo,
                                             unsigned long long w, Round* C,
                                             int take, int64_t* rn, bool* reached) {
  BlockDev& B = a.blocks[gb];
  const JobDev& J = a.jobs[job];
  const int64_t r0 = static_cast<int64_t>(w >> kWordShift);
  *rn = r0;
  *reached = false;
  const unsigned mask = static_cast<unsigned>(w >> 1) & 255u;
  int skip = 0;  // rounds from r0 on without vacancies, up to the limit above
  while (skip < 8 && !((mask >> sector_of_round(r0 + skip)) & 1u)) ++skip;
  if (!solo) skip = min(skip, 1);
  const int sec = sector_of_round(r0 + skip);
  // one round of loads, all in flight together: the block's record (the lease is held: nothing else writes it) and
  // the job's constants
  static_assert(sizeof(BlockDev) % 16 == 0 && offsetof(BlockDev, xs) % 16 == 0 && offsetof(BlockDev, c0) == 8 &&
                    offsetof(BlockDev, c1) == 20,
                "16-byte reads of the record");
  const int4* head = reinterpret_cast<const int4*>(&B);
  const int4 h0 = __ldcg(head), h1 = __ldcg(head + 1);  // job, local id, c0[0..1] | c0[2], c1
  int64_t target = __ldcg(&B.target);
  const int64_t hops = __ldcg(&B.hops);  // empty rounds add none
  ulonglong2 st[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) st[k] = __ldcg(reinterpret_cast<const ulonglong2*>(B.xs) + k);
  const double evo = __ldcg(&B.evo[sec]);
  const int64_t step = __ldcg(&B.step[sec]);
  const int nidle = *reinterpret_cast<volatile int*>(a.flow_idle);
  const int64_t budget = J.hop_budget;
  const double window = J.window;
  if (budget > 0) {
    int64_t end = target;
    if (solo) {
      // a single-block job with a hop budget ends at the end of the first time step at which its
      // hops reached the budget: once they have, its target moves down to the next boundary at or
      // after r0 (never below r0)
      if (hops >= budget) end = min(end, (r0 + 7) & ~static_cast<int64_t>(7));
    } else {
      const int g = budget_gate(a, J, r0);
      if (g == 0) return false;
      if (g == 2) end = r0;  // the job ends at this boundary: the block's target moves down to it
    }
    if (end < target) {
      target = end;
      B.target = end;
      B.budget_end = 1;
    }
  }
  const int64_t r = min(skip < 8 ? r0 + skip : target, target);
  if (!solo && budget > 0 && r > r0 && (r & 7) == 0) B.hops_at[(r >> 3) & 1] = hops;
  *rn = r;
  *reached = r >= target;  // the lease holder alone moves the target
  if (*reached || (!solo && skip > 0)) return false;  // (here skip is 8 only without a vacancy: the target is reached)
  if (!C) {
    // Rounds a CTA takes per sweep: `take` when the context sets it.  Else every one its threads find while nearly
    // all CTAs have rounds to run (512 boxes: 22.5 ms for 256 rounds; 25.0 with two, 28.2 with one), but two
    // while more than 1 in 8 found none in their last sweep (1024 rounds of the 256^3 lattice: 28.1 against 29.7
    // ms with all) and one while more than half did (64 boxes: 12.7 against 14.1 ms): an idle CTA runs a round
    // sooner than this one, which runs its own one after another.
    const int ctas = static_cast<int>(gridDim.x);
    const int most = a.flow_take > 0 || nidle * 8 <= ctas ? take : nidle * 2 > ctas ? 1 : 2;
    const int i = atomicAdd(&sm.flow_ncand, 1);
    if (i >= most) {
      if (i < take) sm.round[i].gb = -1;  // an entry left out
      return false;
    }
    C = &sm.round[i];
  }
  C->r = r;
  C->t = target;
  C->hops = hops;
  C->evo = flow_clock(evo, step, r >> 3, window);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    C->str[k >> 1][2 * (k & 1)] = st[k].x;
    C->str[k >> 1][2 * (k & 1) + 1] = st[k].y;
  }
  C->gb = gb;
  C->job = job;
  C->local = h0.y;
  C->c0[0] = h0.z;
  C->c0[1] = h0.w;
  C->c0[2] = h1.x;
  C->c1[0] = h1.y;
  C->c1[1] = h1.z;
  C->c1[2] = h1.w;
  return true;
}

template <int KIND, int W>
__global__ void __launch_bounds__(Shape<W>::kThreads, Shape<W>::kCtasPerSm) k_flow(RoundArgs a) {
  AKMC_SHAPE(W);
  const int take = a.flow_take > 0 ? min(a.flow_take, kMaxTake) : kMaxTake;
  bool idle = false;  // thread 0: the CTA is counted in flow_idle
  extern __shared__ __align__(16) uint8_t smem[];
  Smem& sm0 = *reinterpret_cast<Smem*>(smem);
  const int tid = threadIdx.x;
  init_cta_smem(smem);
  const int nb = a.nblocks;
  const int watch = max(1, min(min(kThreads, nb), static_cast<int>((static_cast<int64_t>(nb) * kSweepWatch) / gridDim.x)));
  int cursor = static_cast<int>((static_cast<int64_t>(blockIdx.x) * nb) / gridDim.x);
  const uint64_t t_begin = globaltimer_ns();  // a time-boxed launch takes no new round after its budget
#ifdef AKMC_PHASE_PROFILE
  long long t_sweep = 0, t_hop = 0, n_sweep = 0, n_full = 0, t0 = 0;
#endif
  for (int64_t sweep = 0;; ++sweep) {
#ifdef AKMC_PHASE_PROFILE
    if (tid == 0) t0 = clock64();
#endif
    if (tid == 0) {
      sm0.flow_ncand = 0;
      sm0.flow_progress = 0;
    }
    __syncthreads();
    // thread 0 reads the launch's progress and status before its visit, and decides after it whether the CTA
    // stops after this sweep's rounds
    int need = 0, done = 0;
    unsigned st = 0;
    if (tid == 0) {
      need = *reinterpret_cast<volatile int*>(&a.flow_need[KIND]);
      done = *reinterpret_cast<volatile int*>(&a.flow_done[KIND]);
      st = *reinterpret_cast<volatile unsigned*>(a.status);
    }

    // sweep: thread tid looks after block (cursor + tid) mod nb.  One round of loads (the block's word and row) ends
    // most visits to a block that is held, a second (the neighbours' words) those to one that waits.
    if (tid < watch) {
      int gb = cursor + tid;
      if (gb >= nb) gb -= nb;
      const int4* row = reinterpret_cast<const int4*>(a.nbr + static_cast<int64_t>(gb) * kNbrStride);
      const int4 d0 = __ldg(row), d1 = __ldg(row + 1);
      const unsigned long long w = ld_acquire_u64(&a.fstate[gb]);
      if (!(w & 1ull) && (d1.z & kNbrKindMask) == KIND) {
        const int64_t r = static_cast<int64_t>(w >> kWordShift);
        const int64_t target = __ldcg(&a.blocks[gb].target);
        bool ok = (d1.z & kNbrSolo) || flow_ready(a, gb, w, d0, d1);
        // a multi-block job with a hop budget: its round at a time-step boundary waits for the job's
        // other blocks (a job that ends there is taken, to mark it)
        if (ok && (d1.z & kNbrGate) && budget_gate(a, a.jobs[d1.w], r) == 0) ok = false;
        const bool empty = !(d1.z & kNbrSolo) && !((w >> (1 + sector_of_round(r))) & 1ull);
        // A neighbour that carried a vacancy into this sector marked it in the word before it published the round that
        // flow_ready saw.  The fence orders the two for this thread, so that the compare-and-swap below finds the mark
        // and fails, whatever w was read as.  (It costs 2-3%: 1024 rounds of the resident 256^3 lattice took 21.9 ms
        // without it, 22.4 with.)
        if (ok && empty) fence_acq_rel();
        if (ok && empty && !(d1.z & kNbrGate)) {
          // no vacancy: the round is passed over, and the block keeps the lease bit at its target.  Nothing is read
          // or written but the word, so nothing else is fenced: rounds that read what this block's or its
          // neighbours' rounds wrote wait for those blocks themselves.
          const bool end = r + 1 >= target;
          if (atomicCAS(&a.fstate[gb], w, w + (1ull << kWordShift) + (end ? 1 : 0)) == w) {
            sm0.flow_progress = 1;
            if (end) atomicAdd(&a.flow_done[KIND], 1);
          }
        } else if (ok && atomicCAS(&a.fstate[gb], w, w | 1ull) == w) {
          // the lease, then one fence: the reads of the words become acquires
          fence_acq_rel();
          int64_t rn = r;
          bool reached = false;
          const bool keep = flow_advance(a, sm0, gb, d1.w, (d1.z & kNbrSolo) != 0, w, nullptr, take, &rn, &reached);
          if (rn > r) sm0.flow_progress = 1;
          flow_publish(a, gb, rn - r, keep, reached, KIND);
        }
      }
    }
    if (tid == 0) {
      int stop = done >= need || (st & (kErrVacOverflow | kErrRhoRange | kErrHopCap | kErrTimeout)) != 0;
      if (a.time_budget_ns > 0 && globaltimer_ns() - t_begin >= static_cast<uint64_t>(a.time_budget_ns)) stop = 1;
      if (!stop && sweep + 1 >= a.flow_sweep_limit) {  // watchdog; the default 2^25 no launch of <= 1024 rounds needs
        atomicOr(a.status, kErrTimeout);
        stop = 1;
      }
      sm0.flow_stop = stop;
    }
    __syncthreads();
#ifdef AKMC_PHASE_PROFILE
    if (tid == 0) {
      const long long t1 = clock64();
      t_sweep += t1 - t0;
      t0 = t1;
      ++n_sweep;
    }
#endif

    // the hop loop for each round handed over; a single-block job's next rounds follow while
    // the launch's target allows (empty ones in between run on thread 0)
    const int ncand = min(sm0.flow_ncand, take);
    const bool last = sm0.flow_stop;  // written again after the next sweep's first barrier only
    if (tid == 0 && (ncand == 0) != idle) {
      idle = ncand == 0;
      atomicAdd(a.flow_idle, idle ? 1 : -1);
    }
    for (int c = 0; c < ncand; ++c) {
      Round& C = sm0.round[c];
      while (C.gb >= 0) {
#ifdef AKMC_PHASE_PROFILE
        long long tw = clock64();
#endif
        // the thread that found this round ready read the neighbours' round counters and then
        // fenced (an acquire), and a CTA barrier followed: every thread's reads come after the
        // rounds it waits for (shared data is read at L2)
        load_job(sm0, a, C.job);
        const int gb = C.gb, sec = sector_of_round(C.r);
        Region R;
        make_region(C.c0, C.c1, sm0.job, sec, R);
        Smem* sm;
        uint8_t* occ_s;
        int32_t* rho_s;
        carve(smem, R.n, sm, occ_s, rho_s);
        unsigned long long word = kNoVacancy;  // the block's vacancy slots, read while the region's copies are issued
        const unsigned long long* const slots = a.vslot + static_cast<int64_t>(gb) * kFlowSlots;
        constexpr int kReaders = kThreads - 32;  // not the last warp: the records' barrier leaves it out
        static_assert(kReaders >= kFlowSlots, "one slot a thread at the usual number");
        const int nslots = tid < kReaders ? a.flow_slots : 0;
        if (tid < nslots) word = ld_relaxed_u64(slots + tid);  // a neighbour may be filling another of them
        stage_region<KIND, W>(*sm, a, R, occ_s, rho_s);
        for (int k = tid; k < nslots; k += kReaders) {
          if (k != tid) word = ld_relaxed_u64(slots + k);
          if (word == kNoVacancy) continue;
          const int32_t s = static_cast<int32_t>(word & 0xffffffffu);
          int X, y, z;
          if (!region_site(R, sm->job, s, X, y, z)) continue;
          const int i = atomicAdd(&sm->fnv, 1);
          if (i < kMaxV) {
            sm->fslot[i] = k;
            put_record(*sm, R, i, static_cast<int>(word >> 32), s, X, y, z);
          } else {  // more than a sector may hold
            atomicSub(&sm->fnv, 1);
            atomicOr(a.status, kErrVacOverflow);
          }
        }
#ifdef AKMC_PHASE_PROFILE
        if (tid == 0) {
          atomicAdd(a.counters + 12, static_cast<unsigned long long>(clock64() - tw));  // [4] before the hop loop
          tw = clock64();
        }
#endif
        const int cnt = run_block<KIND, W, false>(a, *sm, C, R, occ_s, rho_s, sec);
        const bool ran = cnt >= 0;
#ifdef AKMC_PHASE_PROFILE
        if (tid == 0) tw = clock64();
#endif
        // Vacancies carried into a neighbour's area change owner, the others' sites and sectors are kept up to
        // date (only if the round ran).  The sector's bit of the block's mask goes first and comes back for
        // each vacancy still in it.  With one vacancy, thread 0 does it all and publishes the round.
        unsigned long long* const fw = a.fstate + gb;
        if (ran && cnt != 1 && tid == 0) atomicAnd(fw, ~(2ull << sec));
        if (ran && cnt > 1) __syncthreads();
        if (ran && tid < cnt) {
          const int4 g = sm->vpk[tid][1];
          const int cx = g.x >> 1, cy = g.y, cz = g.z;
          const bool inside = cx >= C.c0[0] && cx < C.c1[0] && cy >= C.c0[1] && cy < C.c1[1] && cz >= C.c0[2] && cz < C.c1[2];
          unsigned long long* const own = a.vslot + static_cast<int64_t>(gb) * kFlowSlots + sm->fslot[tid];
          int osec = 0, o = gb;
          if (inside)
            osec = (cx - C.c0[0] >= (C.c1[0] - C.c0[0]) / 2 ? 1 : 0) | (cy - C.c0[1] >= (C.c1[1] - C.c0[1]) / 2 ? 2 : 0) |
                   (cz - C.c0[2] >= (C.c1[2] - C.c0[2]) / 2 ? 4 : 0);
          else
            o = owner_sector(sm->job, g.w, &osec);
          if (o == gb) {
            *reinterpret_cast<volatile unsigned long long*>(own) = slot_word(sm->vidx[tid], g.w);
            if (cnt == 1 && osec != sec) atomicAnd(fw, ~(2ull << sec));
            if (cnt > 1 || osec != sec) atomicOr(fw, 2ull << osec);
          } else {
            flow_give(a, o, sm->vidx[tid], g.w, osec);
            *reinterpret_cast<volatile unsigned long long*>(own) = kNoVacancy;
            if (cnt == 1) atomicAnd(fw, ~(2ull << sec));
          }
        }
        if (ran && cnt > 1) __syncthreads();
        if (tid == 0) {
          // round C.r ran (it was below the target when handed over); the target is the lease
          // holder's to move, and it is this CTA
          const int64_t r1 = C.r + 1;
          int64_t rn = r1;
          a.blocks[gb].step[sec] = (C.r >> 3) + 1;
          if ((rn & 7) == 0) a.blocks[gb].hops_at[(rn >> 3) & 1] = C.hops;
          bool more = false, reached = rn >= C.t;
          const bool in_time =
              a.time_budget_ns <= 0 || globaltimer_ns() - t_begin < static_cast<uint64_t>(a.time_budget_ns);
          if (!reached && sm->job.nblocks == 1 && c + 1 == ncand && in_time) {
            // a single-block job: its next rounds wait for nothing, so keep the lease and run on
            // -- when no other round this CTA took in the sweep is waiting for it
            const unsigned long long w = ld_relaxed_u64(fw) + (1ull << kWordShift);
            more = flow_advance(a, *sm, gb, C.job, true, w, &C, 0, &rn, &reached);
          }
          const int64_t ran_rounds = rn - r1 + 1;
          sm->flow_progress = 1;
          sm->flow_more = more;
          sm->fnv = 0;
          flow_publish(a, gb, ran_rounds, more, reached, KIND);
        }
        __syncthreads();
#ifdef AKMC_PHASE_PROFILE
        if (tid == 0) {
          ++n_full;
          atomicAdd(a.counters + 15, static_cast<unsigned long long>(clock64() - tw));  // [7] after the hop loop
        }
#endif
        if (!sm0.flow_more) break;
      }
    }
#ifdef AKMC_PHASE_PROFILE
    if (tid == 0) t_hop += clock64() - t0;
#endif
    if (last) break;
    if (AKMC_SWEEP_SLEEP_NS > 0 && !sm0.flow_progress) __nanosleep(AKMC_SWEEP_SLEEP_NS);
    cursor += watch;
    if (cursor >= nb) cursor %= nb;
  }
  if (tid == 0 && idle) atomicAdd(a.flow_idle, -1);  // the next kind's kernel of the launch counts from zero
  cta_flush<W>(a, smem);
#ifdef AKMC_PHASE_PROFILE
  if (tid == 0) {  // scheduler profile: [12] sweep cycles, [13] hop-loop cycles, [14] sweeps, [15] full rounds
    atomicAdd(a.counters + 20, static_cast<unsigned long long>(t_sweep));
    atomicAdd(a.counters + 21, static_cast<unsigned long long>(t_hop));
    atomicAdd(a.counters + 22, static_cast<unsigned long long>(n_sweep));
    atomicAdd(a.counters + 23, static_cast<unsigned long long>(n_full));
  }
#endif
}

// Per block: target round of this launch, word and row; counts the blocks with
// rounds to run per energy kind.
__global__ void k_flow_prep(RoundArgs a) {
  const int gb = blockIdx.x * blockDim.x + threadIdx.x;
  if (gb >= a.nblocks) return;
  BlockDev& B = a.blocks[gb];
  B.cnt = 0;
  a.vcount[gb] = 0;
  int32_t* row = a.nbr + static_cast<int64_t>(gb) * kNbrStride;
  if (B.job < 0) {  // a free block slot: nothing to run
    B.target = B.round;
    a.fstate[gb] = (static_cast<unsigned long long>(B.round) << kWordShift) | 1ull;
    row[6] = kNbrFree;
    return;
  }
  const JobDev& J = a.jobs[B.job];
  for (int k = 0; k < 6; ++k) row[k] = flow_neighbour(J, B.local_id, k >> 1, k & 1 ? 1 : -1) - gb;
  row[7] = B.job;
  row[6] = job_kind(J) | (J.nblocks == 1 ? kNbrSolo : J.hop_budget > 0 ? kNbrGate : 0);
  // up to flow_rounds of the block's remaining rounds (hop budgets are checked by the kernel,
  // at time-step boundaries); a block sitting at a boundary records its hops there
  int64_t L = B.remaining < a.flow_rounds ? B.remaining : a.flow_rounds;
  if ((B.round & 7) == 0) B.hops_at[(B.round >> 3) & 1] = B.hops;
  int64_t t = B.done ? B.round : B.round + L;
  B.budget_end = 0;  // a budget that ends the job moves this target down again inside the launch
  if (J.max_rounds > 0 && t > J.max_rounds) t = J.max_rounds > B.round ? J.max_rounds : B.round;
  B.remaining -= t - B.round;
  B.target = t;
  for (int p = 0; p < 8; ++p) B.step[sector_of_round(p)] = flow_steps(B.round, p);
  a.fstate[gb] = (static_cast<unsigned long long>(B.round) << kWordShift) | (t > B.round ? 0ull : 1ull);
  if (t > B.round) atomicAdd(&a.flow_need[job_kind(J)], 1);
}

// Per vacancy: into the slots of the block whose area holds it.
__global__ void k_flow_slots(RoundArgs a) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= a.nvac || a.vac_job[v] < 0) return;
  const JobDev& J = a.jobs[a.vac_job[v]];
  int osec = 0;
  const int o = owner_sector(J, a.vac_site[v], &osec);
  const int slot = atomicAdd(&a.vcount[o], 1);
  if (slot >= a.flow_slots) {
    atomicOr(a.status, kErrVacOverflow);
    return;
  }
  a.vslot[static_cast<int64_t>(o) * kFlowSlots + slot] = slot_word(v, a.vac_site[v]);
  atomicOr(&a.fstate[o], 2ull << osec);
}

// After the flow kernels: the sectors' clocks caught up (8 threads a block, one a sector), job round and done flags as
// k_finalize leaves them.
__global__ void k_flow_finalize(RoundArgs a) {
  const int gb = (blockIdx.x * blockDim.x + threadIdx.x) >> 3, p = threadIdx.x & 7;
  if (gb < a.nblocks && a.blocks[gb].job >= 0) {
    BlockDev& B = a.blocks[gb];
    const int sec = sector_of_round(p);
    B.evo[sec] = flow_clock(B.evo[sec], B.step[sec], flow_steps(static_cast<int64_t>(a.fstate[gb] >> kWordShift), p),
                            a.jobs[B.job].window);
  }
  if (p != 0) return;
  if (gb == 0 && a.time_budget_ns <= 0) atomicAdd(a.counters + 2, static_cast<unsigned long long>(a.flow_rounds));
  if (gb >= a.nblocks) return;
  BlockDev& B = a.blocks[gb];
  B.cnt = 0;
  B.round = static_cast<int64_t>(a.fstate[gb] >> kWordShift);
  if (B.job < 0) return;
  // rounds of the call a time-boxed launch left to run go back to the block's remaining ones
  if (B.target > B.round) B.remaining += B.target - B.round;
  JobDev& J = a.jobs[B.job];
  // a hop budget ended the job inside the launch (the block reached the boundary its budget set);
  // or, when every block ran to the call's target (no time box), the job's hops (J.hops, added
  // when k_flow ended) reach the budget on a time-step boundary, as the round-by-round finalize
  // decides
  const int done = B.done || (J.max_rounds > 0 && B.round >= J.max_rounds) || (B.budget_end && B.round >= B.target) ||
                   (a.time_budget_ns <= 0 && J.hop_budget > 0 && (B.round & 7) == 0 && J.hops >= J.hop_budget);
  B.done = done;
  if (B.local_id == 0) {
    J.round = B.round;
    J.done = done;
  }
}

__global__ void k_finalize(RoundArgs a) {
  const int gb = blockIdx.x * blockDim.x + threadIdx.x;
  if (gb == 0) {
    *a.n_active = 0;
    atomicAdd(a.counters + 2, 1ull);
  }
  if (gb >= a.nblocks) return;
  BlockDev& B = a.blocks[gb];
  const int had = B.cnt;
  B.cnt = 0;
  if (B.job < 0) return;  // a free block slot
  JobDev& J = a.jobs[B.job];
  // J.done is only written here, by the job's block 0, so other blocks read their own flag
  if (B.done) return;
  if (had == 0) {  // no vacancy in the sector: total = 0, sector_time = threshold (sublattice.inl:108-112)
    const int sec = sector_of_round(B.round);
    const int64_t step = B.round >> 3;
    const double thr = static_cast<double>(step + 1) * J.window - B.evo[sec];
    double sector_time = 0.0;
    if (sector_time < thr) sector_time = thr;
    B.evo[sec] += sector_time;
  }
  B.round += 1;
  // a hop budget is checked at time-step boundaries (every 8 rounds)
  const int done = (J.hop_budget > 0 && (B.round & 7) == 0 && J.hops >= J.hop_budget) ||
                   (J.max_rounds > 0 && B.round >= J.max_rounds);
  B.done = done;
  if (B.local_id == 0) {
    J.round = B.round;
    J.done = done;
  }
}

// One per-hop API step (akmc_calculate, akmc_select_and_perform) of a single-domain job in one launch: the CTA finds
// the sector's vacancies itself and leaves the answer, the status word included, in one record.
template <int KIND>
__global__ void __launch_bounds__(Shape<8>::kThreads, 1) k_api(RoundArgs a) {
  constexpr int kThreads = Shape<8>::kThreads;
  extern __shared__ __align__(16) uint8_t smem[];
  Smem& sm0 = *reinterpret_cast<Smem*>(smem);
  const int tid = threadIdx.x;
  init_cta_smem(smem);
  // one trip for the job's record, the block's and the vacancies' sites, not one each behind a barrier (a kernel of
  // 8.0 us instead of 8.8 on 20^3 cells, pair bond)
  int4 job = make_int4(0, 0, 0, 0);
  if (tid < sizeof(JobDev) / 16) job = __ldcg(reinterpret_cast<const int4*>(a.jobs + a.api_job) + tid);
  const int32_t first = tid < a.api_nvac ? __ldcg(a.vac_site + a.api_vac0 + tid) : 0;
  load_block(sm0, a, a.api_block, a.api_sector);
  if (tid < sizeof(JobDev) / 16) reinterpret_cast<int4*>(&sm0.job)[tid] = job;
  __syncthreads();
  if (tid == 0) sm0.job_key = a.api_job;
  Round& C = sm0.round[0];
  Region R;
  make_region(C.c0, C.c1, sm0.job, a.api_sector, R);
  Smem* sm;
  uint8_t* occ_s;
  int32_t* rho_s;
  carve(smem, R.n, sm, occ_s, rho_s);
  const int nvac = sm->job.done ? 0 : a.api_nvac;  // a finished job has no event left, as in the rounds
  for (int i = tid; i < nvac; i += kThreads) {
    const int v = a.api_vac0 + i;
    const int32_t s = i == tid ? first : a.vac_site[v];
    int X, y, z;
    if (!region_site(R, sm->job, s, X, y, z)) continue;
    const int k = atomicAdd(&sm->fnv, 1);
    if (k < kMaxV) put_record(*sm, R, k, v, s, X, y, z);
  }
  __syncthreads();
  const int n = sm->fnv;
  if (n > kMaxV) {
    __syncthreads();
    if (tid == 0) {
      atomicOr(a.status, kErrVacOverflow);
      sm->fnv = kMaxV;
    }
    __syncthreads();
  }
  if (n == 0) {  // no vacancy in the sector
    if (tid == 0) {
      a.api->total = 0.0;
      if (a.mode == kModeCalc) {
        a.api->count = 0;
      } else {
        a.api->event.from_site = -1;
        a.api->event.total = 0.0;
      }
    }
  } else {
    stage_region<KIND, 8>(*sm, a, R, occ_s, rho_s);
    run_block<KIND, 8, true>(a, *sm, C, R, occ_s, rho_s, a.api_sector);
    cta_flush<8>(a, smem);
  }
  __syncthreads();
  if (tid == 0) a.api->status = *reinterpret_cast<volatile unsigned int*>(a.status);
}

// Density cache of a whole lattice: rho_i = sum over the 58 neighbours j within the cutoff of
// f_{X_j}(shell) in Q.24, exact integers, so the term order does not matter.  A CTA takes tiles of 64 x 16 x 8
// sites (x doubled).  Nearly all atoms are Fe: every density starts as that of a lattice of Fe, and each other
// site of the tile and its halo (4 sites in x, 2 rows in y and z) adds its difference to its 58 neighbours in
// shared memory, a warp a site.  So the work is the reads (16 bytes a thread, 2.1 of them a site with the halo),
// the writes and 58 additions per solute, not per site.  The additions are shared-memory atomics, a cycle a lane,
// and bound it: the 256^3 lattice with 2.3% solutes takes 215 us.  A tile with more than kRhoList such sites (12% of
// them) is summed site by site (rho_gather), part by part: a precipitate's, say.  A lattice that is rich in solutes
// all over, or small, is left to k_init_rho<GatherSmem>, whose tiles are an eighth (rho_by_site).
constexpr int kRhoHX = 4, kRhoHY = 2, kRhoHZ = 2;
constexpr int kGatLX = kGatTX + 2 * kRhoHX, kGatLY = kGatTY + 2 * kRhoHY, kGatLZ = kGatTZ + 2 * kRhoHZ;

struct RhoNb {
  int off, sh;  // tile offset, shell code 1..5
};
// Squared distance of sites (X0, 0, 0) and (X0 + dX, dy, dz) in (a/2)^2 units: corner sites
// (X even) sit at (X, 2y, 2z), centre sites at (X, 2y + 1, 2z + 1).
__host__ __device__ constexpr int rho_d2(int p0, int dX, int dy, int dz) {
  const int p1 = (p0 + dX) & 1;
  const int hy = 2 * dy + p1 - p0, hz = 2 * dz + p1 - p0;
  return dX * dX + hy * hy + hz * hz;
}
__host__ __device__ constexpr int rho_shell(int d2) {
  return d2 == 3 ? 1 : d2 == 4 ? 2 : d2 == 8 ? 3 : d2 == 11 ? 4 : d2 == 12 ? 5 : 0;
}
// k-th neighbour (k < 58) of a site of x parity p within the 5 shells.
__host__ __device__ constexpr RhoNb rho_nbr(int p, int k) {
  int n = 0;
  for (int dz = -2; dz <= 2; ++dz)
    for (int dy = -2; dy <= 2; ++dy)
      for (int dX = -4; dX <= 4; ++dX) {
        const int sh = (dX || dy || dz) ? rho_shell(rho_d2(p, dX, dy, dz)) : 0;
        if (!sh) continue;
        if (n == k) return RhoNb{dX + kGatLX * (dy + kGatLY * dz), sh};
        ++n;
      }
  return RhoNb{0, 0};
}
__host__ __device__ constexpr int rho_count(int p) {
  int n = 0;
  for (int dz = -2; dz <= 2; ++dz)
    for (int dy = -2; dy <= 2; ++dy)
      for (int dX = -4; dX <= 4; ++dX) n += (dX || dy || dz) && rho_shell(rho_d2(p, dX, dy, dz)) ? 1 : 0;
  return n;
}
static_assert(rho_count(0) == kShellNb && rho_count(1) == kShellNb, "58 neighbours in the 5 BCC shells");

template <int P, int K>
__device__ __forceinline__ int32_t rho_terms(const uint8_t* t, const int32_t* fqc) {
  if constexpr (K == kShellNb) {
    return 0;
  } else {
    constexpr RhoNb e = rho_nbr(P, K);
    return fqc[t[e.off] * 8 + e.sh] + rho_terms<P, K + 1>(t, fqc);
  }
}

// f in Q.24 by occupancy code and shell into shared memory; V and other codes 0.
__device__ void rho_table(int32_t* fqc, const Potential* pot) {
  for (int i = threadIdx.x; i < 16 * 8; i += blockDim.x) {
    const int code = i >> 3;
    const bool atom = code == 1 || code == 2 || code == 4 || code == 8;
    fqc[i] = atom ? pot->fq[species_index(static_cast<uint8_t>(code))][i & 7] : 0;
  }
}

// The tile of kGatTX x kGatTY x kGatTZ sites at (x0, y0, z0) summed site by site: its bytes with their halo in
// shared memory, every term one byte read and one read of the f table (by occupancy code) at immediate offsets.
// CTA-collective, 256 threads.
__device__ void rho_gather(const uint8_t* occ, int32_t* rho, int32_t sx, int32_t sy, int32_t sz, int32_t px, int x0, int y0,
                           int z0, uint8_t* tile, const int32_t* fqc) {
  const int tid = threadIdx.x;
  __syncthreads();  // table written; the previous tile's readers are done
  for (int i = tid; i < kGatLX * kGatLY * kGatLZ; i += blockDim.x) {
    const int lx = i % kGatLX, t = i / kGatLX, ly = t % kGatLY, lz = t / kGatLY;
    // periodic wrap without division: coordinates start at most one halo below 0 and end
    // below 3 box lengths (sx >= 16 sites, sy, sz >= 8 cells)
    int gx = x0 - kRhoHX + lx, gy = y0 - kRhoHY + ly, gz = z0 - kRhoHZ + lz;
    gx += gx < 0 ? sx : 0;
    gy += gy < 0 ? sy : 0;
    gz += gz < 0 ? sz : 0;
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      gx -= gx >= sx ? sx : 0;
      gy -= gy >= sy ? sy : 0;
      gz -= gz >= sz ? sz : 0;
    }
    const uint8_t c = __ldg(occ + kHaloL + gx + static_cast<int64_t>(px) * (gy + static_cast<int64_t>(sy) * gz));
    tile[i] = c < 16 ? c : static_cast<uint8_t>(kV);  // the f table's rows; no code above 8 is an atom's
  }
  __syncthreads();
  // each warp takes sites of one x parity (both parities' sums are unrolled code): warp w
  // covers rows 2 (w / 2) and 2 (w / 2) + 1, the 16 sites of parity w % 2 of each
  for (int k = tid; k < kGatTX * kGatTY * kGatTZ; k += blockDim.x) {
    const int w = k >> 5, ln = k & 31;
    const int p = w & 1, row = ((w >> 1) << 1) + (ln >> 4);
    const int lx = 2 * (ln & 15) + p, ly = row % kGatTY, lz = row / kGatTY;
    const int gx = x0 + lx, gy = y0 + ly, gz = z0 + lz;
    if (gx >= sx || gy >= sy || gz >= sz) continue;
    const uint8_t* t = tile + (lx + kRhoHX) + kGatLX * ((ly + kRhoHY) + kGatLY * (lz + kRhoHZ));
    const int32_t acc = p ? rho_terms<1, 0>(t, fqc) : rho_terms<0, 0>(t, fqc);
    lattice_put(rho + static_cast<int64_t>(px) * (gy + static_cast<int64_t>(sy) * gz), sx, gx, acc);
  }
}

constexpr int kRhoEX = kRhoTX + 2 * kRhoHX, kRhoEY = kRhoTY + 2 * kRhoHY, kRhoEZ = kRhoTZ + 2 * kRhoHZ;
constexpr int kRhoList = 2048;
static_assert(kRhoEX < 128 && kRhoEY < 32 && kRhoEZ < 16, "packed list entries");
static_assert(kRhoTX % kGatTX == 0 && kRhoTY % kGatTY == 0 && kRhoTZ % kGatTZ == 0, "whole gather tiles");

struct RhoSmem {
  union {
    alignas(16) int32_t rho[kRhoTX * kRhoTY * kRhoTZ];
    uint8_t tile[kGatLX * kGatLY * kGatLZ];
  };
  uint32_t list[kRhoList];  // lx | ly << 7 | lz << 12 | code << 16, in the tile with its halo
  int32_t fqc[16 * 8];      // f by occupancy code and shell
  int32_t df[16 * 8];       // minus that of Fe
  int32_t base;             // the density of a site among Fe
  uint32_t n;
};

// The f tables of a potential; CTA-collective.
__device__ void rho_tables(RhoSmem& m, const Potential* pot) {
  __syncthreads();
  rho_table(m.fqc, pot);
  __syncthreads();
  for (int i = threadIdx.x; i < 16 * 8; i += blockDim.x) m.df[i] = m.fqc[i] - m.fqc[kFe * 8 + (i & 7)];
  if (threadIdx.x == 0) {
    const int32_t* f = m.fqc + kFe * 8;
    m.base = 8 * f[1] + 6 * f[2] + 12 * f[3] + 24 * f[4] + 8 * f[5];
  }
}

// One tile of the density build (tix-th tile of the lattice); CTA-collective, 256 threads.  nb: the neighbours of
// a site by its x parity, entries lane and lane + 32 (packed dX, dy, dz and shell; 0: none).
__device__ void rho_tile(const uint8_t* occ, int32_t* rho, int32_t sx, int32_t sy, int32_t sz, int32_t px, int64_t tix,
                         RhoSmem& m, const int32_t (&nb)[2][2]) {
  const int tid = threadIdx.x, warp = tid >> 5;
  const int nx = (sx + kRhoTX - 1) / kRhoTX, ny = (sy + kRhoTY - 1) / kRhoTY;
  const int x0 = static_cast<int>(tix % nx) * kRhoTX;
  const int y0 = static_cast<int>((tix / nx) % ny) * kRhoTY;
  const int z0 = static_cast<int>(tix / (static_cast<int64_t>(nx) * ny)) * kRhoTZ;
  const int ex = min(kRhoTX, sx - x0), ey = min(kRhoTY, sy - y0), ez = min(kRhoTZ, sz - z0);
  __syncthreads();  // tables written; the previous tile's readers are done
  if (tid == 0) m.n = 0;
  const int4 b4 = make_int4(m.base, m.base, m.base, m.base);
  for (int i = tid; i < kRhoTX * kRhoTY * kRhoTZ / 4; i += blockDim.x) reinterpret_cast<int4*>(m.rho)[i] = b4;
  __syncthreads();
  // the sites that are not Fe: rows of the tile and its halo, 16 entries a thread from entry x0 (site x0 - 16; the
  // row's halo entries hold the sites past either end)
  const int nv = (ex + kRhoHX + 16 + 15) / 16, nrows = (ey + 2 * kRhoHY) * (ez + 2 * kRhoHZ);
  for (int i = tid; i < nv * nrows; i += blockDim.x) {
    const int v = i % nv, t = i / nv, lz = t / (ey + 2 * kRhoHY), ly = t - lz * (ey + 2 * kRhoHY);
    const int gy = wrap1(y0 - kRhoHY + ly, sy), gz = wrap1(z0 - kRhoHZ + lz, sz);
    const uint4 w4 = __ldg(reinterpret_cast<const uint4*>(occ + x0 + 16 * v + static_cast<int64_t>(px) * (gy + static_cast<int64_t>(sy) * gz)));
    const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t d = w[q] ^ (0x01010101u * kFe);
      while (d) {
        const int k = (__ffs(static_cast<int>(d)) - 1) >> 3;
        d &= ~(0xffu << (8 * k));
        const int lx = 16 * v + 4 * q + k - (16 - kRhoHX);  // site x0 - kRhoHX + lx
        if (lx < 0 || lx >= ex + 2 * kRhoHX) continue;
        const uint32_t code = (w[q] >> (8 * k)) & 0xffu;
        const uint32_t e = atomicAdd(&m.n, 1u);
        if (e < kRhoList) m.list[e] = lx | ly << 7 | lz << 12 | (code < 16 ? code : 0u) << 16;
      }
    }
  }
  __syncthreads();
  const int n = static_cast<int>(m.n);
  if (n > kRhoList) {
    for (int z = 0; z < ez; z += kGatTZ)
      for (int y = 0; y < ey; y += kGatTY)
        for (int x = 0; x < ex; x += kGatTX) rho_gather(occ, rho, sx, sy, sz, px, x0 + x, y0 + y, z0 + z, m.tile, m.fqc);
    return;
  }
  for (int i = warp; i < n; i += blockDim.x >> 5) {
    const uint32_t e = m.list[i];
    const int lx = e & 127, ly = (e >> 7) & 31, lz = (e >> 12) & 15;
    const int32_t* df = m.df + (e >> 16) * 8;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int32_t w = lx & 1 ? nb[1][u] : nb[0][u];  // x0 and the halo are even
      const int tx = lx - kRhoHX + unpack_dx(w), ty = ly - kRhoHY + unpack_dy(w), tz = lz - kRhoHZ + unpack_dz(w);
      if (w && static_cast<unsigned>(tx) < static_cast<unsigned>(ex) && static_cast<unsigned>(ty) < static_cast<unsigned>(ey) &&
          static_cast<unsigned>(tz) < static_cast<unsigned>(ez))
        atomicAdd(&m.rho[tx + kRhoTX * (ty + kRhoTY * tz)], df[unpack_sh_s(w)]);
    }
  }
  __syncthreads();
  const bool edge = x0 < kHaloR || x0 + ex > sx - kHaloL;  // sites with halo copies
  for (int i = tid; i < kRhoTX * kRhoTY * kRhoTZ / 4; i += blockDim.x) {
    const int lx = 4 * (i % (kRhoTX / 4)), t = i / (kRhoTX / 4), ly = t % kRhoTY, lz = t / kRhoTY;
    if (lx >= ex || ly >= ey || lz >= ez) continue;
    int32_t* const row = rho + static_cast<int64_t>(px) * (y0 + ly + static_cast<int64_t>(sy) * (z0 + lz));
    if (lx + 4 <= ex) *reinterpret_cast<int4*>(row + kHaloL + x0 + lx) = reinterpret_cast<const int4*>(m.rho)[i];
    if (edge || lx + 4 > ex)
      for (int k = 0; k < 4 && lx + k < ex; ++k) lattice_put(row, sx, x0 + lx + k, m.rho[4 * i + k]);
  }
}

__device__ void rho_neighbours(const Geometry* geo, int32_t (&nb)[2][2]) {
  const int lane = threadIdx.x & 31;
  for (int p = 0; p < 2; ++p)
    for (int u = 0; u < 2; ++u) nb[p][u] = lane + 32 * u < kShellNb ? __ldg(&geo->nbr[p][lane + 32 * u]) : 0;
}

// A dense job's tiles: summed site by site, many small ones (one CTA's share of a larger tile is gone through in turn).
struct GatherSmem {
  uint8_t tile[kGatLX * kGatLY * kGatLZ];
  int32_t fqc[16 * 8];
};
__device__ void rho_tables(GatherSmem& m, const Potential* pot) {
  __syncthreads();
  rho_table(m.fqc, pot);
}
__device__ void rho_tile(const uint8_t* occ, int32_t* rho, int32_t sx, int32_t sy, int32_t sz, int32_t px, int64_t tix,
                         GatherSmem& m, const int32_t (&)[2][2]) {
  const int nx = (sx + kGatTX - 1) / kGatTX, ny = (sy + kGatTY - 1) / kGatTY;
  const int64_t t = tix / nx;
  rho_gather(occ, rho, sx, sy, sz, px, static_cast<int>(tix % nx) * kGatTX, static_cast<int>(t % ny) * kGatTY,
             static_cast<int>(t / ny) * kGatTZ, m.tile, m.fqc);
}

template <typename M>
__global__ void __launch_bounds__(256) k_init_rho(const uint8_t* occ, int32_t* rho, int32_t sx, int32_t sy,
                                                  int32_t sz, int32_t px, const Potential* pot, const Geometry* geo) {
  __shared__ M m;
  int32_t nb[2][2];
  rho_neighbours(geo, nb);
  rho_tables(m, pot);
  const int64_t ntiles = rho_tiles(sx, sy, sz, std::is_same_v<M, GatherSmem>);
  for (int64_t tix = blockIdx.x; tix < ntiles; tix += gridDim.x) rho_tile(occ, rho, sx, sy, sz, px, tix, m, nb);
}

// The density build of every EAM job of a context of one sort in one launch: global tile t belongs to the
// job k with tile0[k] <= t < tile0[k + 1] (jobs[k] its index).
template <typename M>
__global__ void __launch_bounds__(256) k_init_rho_jobs(RoundArgs a, const int64_t* tile0, const int32_t* jobs,
                                                       int32_t njobs) {
  __shared__ M m;
  int32_t nb[2][2];
  rho_neighbours(a.geo, nb);
  int pot = -1;
  for (int64_t t = blockIdx.x; t < tile0[njobs]; t += gridDim.x) {
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {  // last k with tile0[k] <= t
      const int mid = (lo + hi + 1) >> 1;
      if (tile0[mid] <= t) lo = mid;
      else hi = mid - 1;
    }
    const JobDev& J = a.jobs[jobs[lo]];
    if (J.pot != pot) {  // uniform over the CTA
      rho_tables(m, a.pots + J.pot);
      pot = J.pot;
    }
    rho_tile(J.occ, J.rho, J.sx, J.sy, J.sz, J.px, t - tile0[lo], m, nb);
  }
}

// Sixteen entries of a lattice row (entry 16 v on, 16-byte aligned in the device layout) from the row's sx sites
// at src (even addresses and sizes), the halo entries on either side included.
__device__ __forceinline__ uint4 row_vector(const uint8_t* src, int sx, int v) {
  const int x0 = 16 * v - kHaloL;
  uint32_t w[4];
  if (x0 >= 0 && x0 + 16 <= sx) {
    const uint16_t* s = reinterpret_cast<const uint16_t*>(src + x0);
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = s[2 * q] | static_cast<uint32_t>(s[2 * q + 1]) << 16;
  } else {
    int x = x0 % sx;
    x += x < 0 ? sx : 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      w[q] = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        w[q] |= static_cast<uint32_t>(src[x]) << (8 * k);
        x = x + 1 == sx ? 0 : x + 1;
      }
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
// Calls f(x) for every vacancy among the row's own sites in vector v.
template <typename F>
__device__ __forceinline__ void for_vacancies(const uint4& w4, int sx, int v, F f) {
  const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
  const int x0 = 16 * v - kHaloL;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t z = (w[q] - 0x01010101u) & ~w[q] & 0x80808080u;  // nonzero when a byte is 0
    if (!z) continue;
    for (int k = 0; k < 4; ++k) {
      const int x = x0 + 4 * q + k;
      if (((w[q] >> (8 * k)) & 0xffu) == kV && x >= 0 && x < sx) f(x);
    }
  }
}

// Rows of a lattice, row0 the first, from the staging buffer into a job's device rows, halos included; with vac_site
// their vacancies go to the job's slice of the vacancy table (cap entries; count: vacancies found).
__global__ void k_load_lattice(const uint8_t* __restrict__ stage, uint8_t* occ, int32_t sx, int32_t px, int64_t row0,
                               int64_t nrows, int32_t* vac_site, int32_t* vac_job, int32_t job, int32_t cap, int32_t* count) {
  const int vpr = px / 16;
  const int64_t n = nrows * vpr;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t row = i / vpr;
    const int v = static_cast<int>(i - row * vpr);
    const uint4 w = row_vector(stage + row * sx, sx, v);
    *reinterpret_cast<uint4*>(occ + (row0 + row) * px + 16 * v) = w;
    if (vac_site)
      for_vacancies(w, sx, v, [&](int x) {
        const int k = atomicAdd(count, 1);
        if (k < cap) {
          vac_site[k] = static_cast<int32_t>((row0 + row) * sx + x);
          vac_job[k] = job;
        }
      });
  }
}

// Whole-context lattice load: chunk c (whole rows of one job) goes from the staging buffer into its job's device
// rows, and its vacancies to the job's slice of the vacancy table.
__global__ void k_scatter_collect(RoundArgs a, const uint8_t* __restrict__ stage, const SiteChunk* chunks, int32_t* counts) {
  const SiteChunk c = chunks[blockIdx.x];
  const JobDev& J = a.jobs[c.job];
  const int sx = J.sx, px = J.px, vpr = px / 16, n = c.nrows * vpr;
  uint8_t* const occ = J.occ + static_cast<int64_t>(px) * c.row0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int row = i / vpr, v = i - row * vpr;
    const uint4 w = row_vector(stage + c.stage0 + static_cast<int64_t>(row) * sx, sx, v);
    *reinterpret_cast<uint4*>(occ + static_cast<int64_t>(row) * px + 16 * v) = w;
    for_vacancies(w, sx, v, [&](int x) {
      const int k = atomicAdd(counts + c.job, 1);
      if (k < c.nvac) {
        a.vac_site[c.vac0 + k] = (c.row0 + row) * sx + x;
        a.vac_job[c.vac0 + k] = c.job;
      }
    });
  }
}

__global__ void k_check_counts(const int32_t* counts, const int32_t* want, int32_t njobs, unsigned int* status) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < njobs && counts[j] != want[j]) atomicOr(status, kErrVacCount);
}

// One thread a word: a read-out moves 72 bytes a block over PCIe, not its whole record.
__global__ void k_gather_clocks(const BlockDev* __restrict__ blocks, int32_t n, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 8 * n)
    out[i] = blocks[i >> 3].evo[i & 7];
  else if (i < 9 * n)
    reinterpret_cast<int64_t*>(out)[i] = blocks[i - 8 * n].hops;
}

// Whole-context lattice read-back: the reverse copy into the staging buffer (rows of sx sites, an even number).
__global__ void k_gather(RoundArgs a, uint8_t* stage, const SiteChunk* chunks) {
  const SiteChunk c = chunks[blockIdx.x];
  const JobDev& J = a.jobs[c.job];
  const int sx = J.sx, px = J.px, vpr = (sx + 15) / 16, n = c.nrows * vpr;
  const uint8_t* const occ = J.occ + static_cast<int64_t>(px) * c.row0 + kHaloL;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int row = i / vpr, v = i - row * vpr;
    const uint4 w4 = *reinterpret_cast<const uint4*>(occ + static_cast<int64_t>(row) * px + 16 * v);
    const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
    uint16_t* const d = reinterpret_cast<uint16_t*>(stage + c.stage0 + static_cast<int64_t>(row) * sx + 16 * v);
    const int left = (sx - 16 * v) / 2;
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (q < left) d[q] = static_cast<uint16_t>(w[q >> 1] >> (16 * (q & 1)));
  }
}

__global__ void k_device_math(const double* x, int64_t n, double* e, double* l) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  e[i] = port_exp(x[i]);
  l[i] = port_log(x[i]);
}

}  // namespace

size_t hop_smem_bytes(int max_region_sites) {
  return sizeof(Smem) + 128 + ((static_cast<size_t>(max_region_sites) * 4 + 127) & ~static_cast<size_t>(127)) +
         static_cast<size_t>(max_region_sites) + 16;
}

template <int W>
void launch_hops(const RoundArgs& a, int hop_grid, size_t smem, cudaStream_t st) {
  constexpr int T = Shape<W>::kThreads;
  if (a.kind_mask & (1 << kEam64)) k_hop<kEam64, W><<<hop_grid, T, smem, st>>>(a);
  if (a.kind_mask & (1 << kEam32)) k_hop<kEam32, W><<<hop_grid, T, smem, st>>>(a);
  if (a.kind_mask & (1 << kPairBond)) k_hop<kPairBond, W><<<hop_grid, T, smem, st>>>(a);
}
template <int W>
void launch_flows(const RoundArgs& a, int grid, size_t smem, cudaStream_t st) {
  constexpr int T = Shape<W>::kThreads;
  if (a.kind_mask & (1 << kEam64)) k_flow<kEam64, W><<<grid, T, smem, st>>>(a);
  if (a.kind_mask & (1 << kEam32)) k_flow<kEam32, W><<<grid, T, smem, st>>>(a);
  if (a.kind_mask & (1 << kPairBond)) k_flow<kPairBond, W><<<grid, T, smem, st>>>(a);
}

int launch_round(const RoundArgs& a, int hop_grid, size_t smem, void* stream, void* ev0, void* ev1) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (a.nvac > 0) k_bucket<<<(a.nvac + 127) / 128, 128, 0, st>>>(a);
  if (ev0) cudaEventRecord(static_cast<cudaEvent_t>(ev0), st);
  if (a.eval_warps == 4) launch_hops<4>(a, hop_grid, smem, st);
  else launch_hops<8>(a, hop_grid, smem, st);
  if (ev1) cudaEventRecord(static_cast<cudaEvent_t>(ev1), st);
  k_finalize<<<(a.nblocks + 127) / 128, 128, 0, st>>>(a);
  return static_cast<int>(cudaGetLastError());
}

int launch_api(const RoundArgs& a, int kind, size_t smem, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  constexpr int T = Shape<8>::kThreads;
  if (kind == kPairBond) k_api<kPairBond><<<1, T, smem, st>>>(a);
  else if (kind == kEam32) k_api<kEam32><<<1, T, smem, st>>>(a);
  else k_api<kEam64><<<1, T, smem, st>>>(a);
  return static_cast<int>(cudaGetLastError());
}

__global__ void k_flow_begin(RoundArgs a, int64_t n) {
  const int gb = blockIdx.x * blockDim.x + threadIdx.x;
  if (gb < a.nblocks) a.blocks[gb].remaining = n;
}

int launch_flow_begin(const RoundArgs& a, int64_t n, void* stream) {
  k_flow_begin<<<(a.nblocks + 127) / 128, 128, 0, static_cast<cudaStream_t>(stream)>>>(a, n);
  return static_cast<int>(cudaGetLastError());
}

int launch_flow(const RoundArgs& a, int grid, size_t smem, void* stream, void* ev0, void* ev1) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaMemsetAsync(a.flow_need, 0, 7 * sizeof(int32_t), st);  // and flow_done, flow_idle behind it
  // (a context with one block uses the slots up to kSoloSlots past its first)
  cudaMemsetAsync(a.vslot, 0xff,
                  (static_cast<size_t>(a.nblocks - 1) * kFlowSlots + a.flow_slots) * sizeof(unsigned long long), st);
  k_flow_prep<<<(a.nblocks + 127) / 128, 128, 0, st>>>(a);
  if (a.nvac > 0) k_flow_slots<<<(a.nvac + 127) / 128, 128, 0, st>>>(a);
  if (ev0) cudaEventRecord(static_cast<cudaEvent_t>(ev0), st);
  if (a.eval_warps == 4) launch_flows<4>(a, grid, smem, st);
  else launch_flows<8>(a, grid, smem, st);
  if (ev1) cudaEventRecord(static_cast<cudaEvent_t>(ev1), st);
  k_flow_finalize<<<(a.nblocks + 15) / 16, 128, 0, st>>>(a);
  return static_cast<int>(cudaGetLastError());
}

int hop_ctas_per_sm(int eval_warps) { return eval_warps == 4 ? Shape<4>::kCtasPerSm : Shape<8>::kCtasPerSm; }

int configure_hop_smem(size_t smem) {
  const void* kernels[] = {
      reinterpret_cast<const void*>(k_hop<kEam64, 8>),     reinterpret_cast<const void*>(k_hop<kEam32, 8>),
      reinterpret_cast<const void*>(k_hop<kPairBond, 8>),  reinterpret_cast<const void*>(k_hop<kEam64, 4>),
      reinterpret_cast<const void*>(k_hop<kEam32, 4>),     reinterpret_cast<const void*>(k_hop<kPairBond, 4>),
      reinterpret_cast<const void*>(k_flow<kEam64, 8>),    reinterpret_cast<const void*>(k_flow<kEam32, 8>),
      reinterpret_cast<const void*>(k_flow<kPairBond, 8>), reinterpret_cast<const void*>(k_flow<kEam64, 4>),
      reinterpret_cast<const void*>(k_flow<kEam32, 4>),    reinterpret_cast<const void*>(k_flow<kPairBond, 4>),
      reinterpret_cast<const void*>(k_api<kEam64>),        reinterpret_cast<const void*>(k_api<kEam32>),
      reinterpret_cast<const void*>(k_api<kPairBond>)};
  cudaError_t e = cudaSuccess;
  for (const void* f : kernels)
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  return static_cast<int>(e);
}

int launch_gather_clocks(const BlockDev* blocks, int32_t n, double* out, void* stream) {
  k_gather_clocks<<<(9 * n + 127) / 128, 128, 0, static_cast<cudaStream_t>(stream)>>>(blocks, n, out);
  return static_cast<int>(cudaGetLastError());
}
int launch_init_rho(uint8_t* occ, int32_t* rho, int32_t sx, int32_t sy, int32_t sz, bool dense, const Potential* pot,
                    const Geometry* geo, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int blocks = static_cast<int>(std::min<int64_t>(rho_tiles(sx, sy, sz, dense), 148 * 16));
  if (dense) k_init_rho<GatherSmem><<<blocks, 256, 0, st>>>(occ, rho, sx, sy, sz, lattice_pitch(sx), pot, geo);
  else k_init_rho<RhoSmem><<<blocks, 256, 0, st>>>(occ, rho, sx, sy, sz, lattice_pitch(sx), pot, geo);
  return static_cast<int>(cudaGetLastError());
}

__global__ void k_check_vacancy_count(const int32_t* count, int32_t want, unsigned int* status) {
  if (*count != want) atomicOr(status, kErrVacCount);
}

int launch_init_rho_jobs(const RoundArgs& a, const JobsLoad& L, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto blocks = [](const JobsLoad::RhoJobs& r) { return static_cast<int>(std::min<int64_t>(r.tiles, 148 * 16)); };
  const JobsLoad::RhoJobs &s = L.rho[0], &d = L.rho[1];
  if (s.n > 0) k_init_rho_jobs<RhoSmem><<<blocks(s), 256, 0, st>>>(a, s.tile0, s.jobs, s.n);
  if (d.n > 0) k_init_rho_jobs<GatherSmem><<<blocks(d), 256, 0, st>>>(a, d.tile0, d.jobs, d.n);
  return static_cast<int>(cudaGetLastError());
}

int launch_load_jobs(const RoundArgs& a, const JobsLoad& L, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(L.counts, 0, sizeof(int32_t) * L.njobs, st);
  if (e != cudaSuccess) return static_cast<int>(e);
  k_scatter_collect<<<L.nchunks, 256, 0, st>>>(a, L.stage, L.chunks, L.counts);
  k_check_counts<<<(L.njobs + 127) / 128, 128, 0, st>>>(L.counts, L.want, L.njobs, a.status);
  return launch_init_rho_jobs(a, L, stream);
}


int launch_gather_jobs(const RoundArgs& a, const JobsLoad& L, void* stream) {
  k_gather<<<L.nchunks, 256, 0, static_cast<cudaStream_t>(stream)>>>(a, L.stage, L.chunks);
  return static_cast<int>(cudaGetLastError());
}

int launch_load_lattice(const uint8_t* stage, uint8_t* occ, int32_t sx, int64_t row0, int64_t n, int64_t nrows,
                        int32_t* vac_site, int32_t* vac_job, int32_t job, int32_t cap, int32_t* count,
                        unsigned int* status, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int32_t px = lattice_pitch(sx);
  const int blocks = static_cast<int>(std::min<int64_t>((n * (px / 16) + 255) / 256, 148 * 32));
  if (vac_site && row0 == 0) cudaMemsetAsync(count, 0, sizeof(int32_t), st);
  k_load_lattice<<<blocks, 256, 0, st>>>(stage, occ, sx, px, row0, n, vac_site, vac_job, job, cap, count);
  if (vac_site && row0 + n == nrows) k_check_vacancy_count<<<1, 1, 0, st>>>(count, cap, status);
  return static_cast<int>(cudaGetLastError());
}

int launch_device_math(const double* x, int64_t n, double* e, double* l, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  k_device_math<<<static_cast<int>((n + 255) / 256), 256, 0, st>>>(x, n, e, l);
  return static_cast<int>(cudaGetLastError());
}

// Round scratch of akmc_run_rounds_noalloc (2.1 MB): block vacancy lists, active-block
// list and active count for kNoAllocMaxBlocks blocks, with the count 256-byte aligned.
constexpr size_t kNoAllocWords = static_cast<size_t>(kNoAllocMaxBlocks) * (kMaxV + 1) + 64;
static __device__ __align__(256) int32_t g_noalloc_scratch[kNoAllocWords];

int noalloc_scratch(int32_t** base) {
  void* p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  *base = e == cudaSuccess ? static_cast<int32_t*>(p) : nullptr;
  return static_cast<int>(e);
}

}  // namespace akmc
