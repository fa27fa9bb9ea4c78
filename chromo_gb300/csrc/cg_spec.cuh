// cg_spec.cuh -- the production MC kernel: several moves of a replica in flight.
//
// One CTA per replica, W warps, each warp split into 32 / G groups of G lanes
// (G = 8, 16 or 32).  A group evaluates one move, so up to S <= W * 32 / G moves
// are in flight (the default FP32 shape has 3/4 as many moves as warps; short
// tangent rotations take 8 or 16 lanes and more moves).  Within one controller's
// cycle (same move kind, fixed amplitudes) the next B <= S attempted moves are
// evaluated at once, group s taking move t0 + s, all against the state before
// the batch.  Then:
//
//   * each move's read/write footprint -- the beads it reads or writes and
//     the voxels it touches -- is compared with the footprints of the earlier
//     moves of the batch (beads by index range, voxels through a block-wide
//     voxel -> move-bitmask table);
//   * walking the batch in order, move s stands iff no earlier *accepted*
//     move's footprint meets its own; the first move that fails, and every
//     later one, is evaluated again in the next batch on the updated state;
//   * the standing accepted moves are committed; their footprints are
//     disjoint, so the commits do not interact.
//
// The result is exactly that of applying the moves one after the other (a
// rejected move changes nothing; an accepted move only changes its own
// footprint), for every W and G: each attempted move takes its random numbers
// from its own Philox4x32-10 sub-stream, indexed by (replica, move number,
// draw number), and dE is summed exactly in fixed point (FP32 storage: every term;
// FP64 storage: the field's, whose number and order of voxels vary, the bonds' in a
// fixed order), so neither the spread of beads and voxels over lanes nor the order
// of hash claims changes a bit.  Acceptance statistics and the controllers' amplitude updates
// are applied in move order as in the one-move-at-a-time loop
// (chromo/mc/mc_sim.pyx:88-182).
//
// Several moves per warp: a move of a few beads (the mean segment of the
// benchmark's moves is 4-20 beads) leaves most of a warp's lanes idle, and the
// scalar part of a move (draws, bead selection, rotation, Metropolis) is
// computed redundantly by all lanes of its group; with G = 16 or 8 one warp
// instruction serves 2 or 4 moves.  Every warp-collective operation below is
// executed by the whole warp with per-group masks, so groups may diverge only
// in code without collectives.
//
// Loops of run-time length are not unrolled: the kernel is large and few warps
// share an SM, and a fifth of its instruction fetches missed the first cache
// with them unrolled (a tenth of the kernel's time on 256 chains).  Exceptions,
// measured: the binder columns of add_corner.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

#include "cg_device.cuh"
#include "cg_exact.h"
#include "cg_kernels.h"
#include "cg_move.cuh"

namespace cg {

// Draw j (>= kDrawCache) of a move's sub-stream: word j & 3 of Philox block
// j >> 2.  Out of line: few moves draw this many numbers, and inlined at every
// draw site the rounds would fill the instruction cache.
static __device__ __noinline__ unsigned move_draw_slow(uint2 key, unsigned tlo, unsigned thi,
                                                       unsigned long long j) {
  uint4 o = philox(make_uint4((unsigned)(j >> 2), tlo, thi, 0x2545F491u), key);
  return comp4(o, (unsigned)j & 3u) >> 1;
}

// Random numbers of one attempted move (its own counter space).  Draw j is
// word j & 3 of Philox block j >> 2.  The first kDrawCache draws are computed
// at init by the move's G lanes into its shared-memory buffer, so a move's
// draws cost one Philox latency instead of a chain of them; init() must be
// called by the whole warp.
struct MoveRng {
  uint2 key, keyb;
  unsigned tlo, thi;
  unsigned long long pos, bpos;
  const unsigned* buf;
  bool fail;
  template <int G>
  __device__ void init(unsigned long long seed, int rep, unsigned long long t, unsigned* draws, int gl) {
    key = make_uint2((unsigned)seed ^ (unsigned)rep * 0x85EBCA6Bu, (unsigned)(seed >> 32) ^ 0x1B873593u);
    keyb = make_uint2(key.x ^ 0x68E31DA4u, key.y ^ 0xB5297A4Du);
    tlo = (unsigned)t;
    thi = (unsigned)(t >> 32);
    pos = 0; bpos = 0; fail = false;
    #pragma unroll 1
    for (int j = gl; j < kDrawCache / 4; j += G) {
      uint4 o = philox(make_uint4((unsigned)j, tlo, thi, 0x2545F491u), key);
      reinterpret_cast<uint4*>(draws)[j] = o;
    }
    __syncwarp();
    buf = draws;
  }
  __device__ __forceinline__ unsigned next() { return word(pos++); }
  // draw j, from the cache when it holds it
  __device__ __forceinline__ unsigned word(unsigned long long j) const {
    if (j < (unsigned long long)kDrawCache) return buf[j] >> 1;
    return move_draw_slow(key, tlo, thi, j);
  }
  __device__ __forceinline__ int state_at(unsigned long long k, int nt, bool& ok) const {
    ok = true;
    uint4 o = philox(make_uint4((unsigned)(k >> 2), tlo, thi, 0x7F4A7C15u), keyb);
    return (int)__umulhi(comp4(o, (unsigned)(k & 3)), (unsigned)(nt + 1));
  }
};

__device__ __forceinline__ int block_insert(int* bkeys, int logHB, int key) {
  const unsigned mask = (1u << logHB) - 1u;
  unsigned h = ((unsigned)key * 0x9E3779B1u) >> (32 - logHB);
  #pragma unroll 1
  for (int it = 0; it < 64; it++) {
    int prev = atomicCAS(&bkeys[h], -1, key);
    if (prev == -1 || prev == key) return (int)h;
    h = (h + 1) & mask;
  }
  return -1;
}

// Empty the block voxel table (thread tid of nt), 16 bytes a store.
__device__ __forceinline__ void clear_block_table(int* bkeys, unsigned* bmask, int logHB, int tid, int nt) {
  int4* k = reinterpret_cast<int4*>(bkeys);
  int4* m = reinterpret_cast<int4*>(bmask);
#pragma unroll 1
  for (int i = tid; i < (1 << logHB) / 4; i += nt) {
    k[i] = make_int4(-1, -1, -1, -1);
    m[i] = make_int4(0, 0, 0, 0);
  }
}

// Scratch of one move slot: its shared-memory region, or the slot's global
// region for moves too large for shared memory.
struct SlotScratch {
  int* keys;
  int* used;
  int* bslot;
  long long* vals;
  int logH;
  void* stage;
  int* idx;
};

// Drop the entries a move left in a voxel table (keys, values, block slots).
__device__ __forceinline__ void clear_table(const SlotScratch& T, int hcol, int nu, int gl, int G) {
  #pragma unroll 1
  for (int i = gl; i < nu; i += G) {
    const int slot = T.used[i];
    T.keys[slot] = -1;
    #pragma unroll 1
    for (int cc = 0; cc < hcol; cc++) T.vals[(long long)slot * hcol + cc] = 0;
    T.bslot[i] = -1;
  }
}

// A position move's bead data in global memory (one replica).
template <typename Pos>
struct ChainView {
  const V4<Pos>* r4;
  const V4<Pos>* t34;
  const V4<Pos>* t24;
  const unsigned* st;
  const double* bonds;
  const float* bonds32;
  const double* twist;  // (eps_twist, omega0) per bond, SSTWLC replicas only
  // lean: the caller's instantiation has no SSTWLC replica (twist stays null)
  __device__ ChainView(const KArgs& a, const RepDev& rd, bool lean)
      : r4(reinterpret_cast<const V4<Pos>*>(a.r4) + rd.bead_off),
        t34(reinterpret_cast<const V4<Pos>*>(a.t34) + rd.bead_off),
        t24(reinterpret_cast<const V4<Pos>*>(a.t24) + rd.bead_off),
        st(a.states + rd.bead_off), bonds(a.bonds + rd.bead_off * 6), bonds32(a.bonds32 + rd.bead_off * 8),
        twist(!lean && rd.twist ? a.twist + rd.bead_off * 2 : nullptr) {}
};

// Largest position move of a shared voxel table (the split counters' bound,
// see add_delta), halved for each axis of a single voxel, on which a bead's
// lower and upper corners fall in the same voxel.
constexpr int kPoolMaxBeads = 256;

// Lanes that share one bead's trilinear corners in the block-wide deposit,
// each with kCornersPerLane corners (two neighbours along x).
constexpr int kLanesPerBead = 4;
constexpr int kCornersPerLane = 8 / kLanesPerBead;

// New position (and, but for a slide, which only translates, new tangents) of
// a bead under a move's transform M.
template <typename Pos>
__device__ __forceinline__ void move_bead(int kind, const Pos (&M)[3][4], const Pos (&r)[3], const Pos (&t3)[3],
                                          const Pos (&t2)[3], Pos (&tr)[3], Pos (&tt3)[3], Pos (&tt2)[3]) {
  if (kind == CG_SLIDE) {
    for (int j = 0; j < 3; j++) { tr[j] = r[j] + M[j][3]; tt3[j] = t3[j]; tt2[j] = t2[j]; }
  } else {
    for (int j = 0; j < 3; j++) {
      Pos er = 0, e3 = 0, e2 = 0;
      for (int q = 0; q < 3; q++) { er += M[j][q] * r[q]; e3 += M[j][q] * t3[q]; e2 += M[j][q] * t2[q]; }
      tr[j] = er + M[j][3]; tt3[j] = e3; tt2[j] = e2;
    }
  }
}

template <typename Pos>
__device__ __forceinline__ void load_transform(const MovePlan& P, Pos (&M)[3][4]) {
  const Pos* Mp = reinterpret_cast<const Pos*>(P.M);
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 4; j++) M[i][j] = Mp[4 * i + j];
}

// Elastic dE of one boundary bond of a position move: the bond to the fixed
// neighbour left of the segment (side 0) or right of it (side 1); zero where the
// segment ends the chain.  The move's plan holds its segment and transform.
template <typename Pos, typename Acc, int LEAN>
static __device__ __forceinline__ Acc boundary_term(const KArgs& a, const RepDev& rd, const MovePlan& P, int kind,
                                                 int side) {
  const ChainView<Pos> cv(a, rd, LEAN);
  const long long N = rd.n_beads;
  Acc out = acc_zero<Acc>();
  const long long i = side == 0 ? P.ind0 : P.indf - 1;
  const long long in = side == 0 ? i - 1 : i + 1;
  if (in < 0 || in >= N) return out;
  Pos M[3][4];
  load_transform(P, M);
  const V4<Pos> R = cv.r4[i], T3 = cv.t34[i], RN = cv.r4[in], TN = cv.t34[in];
  const Bond<Pos> bn = bond_at(cv.bonds, cv.bonds32, side == 0 ? in : i, (Pos)0);
  const Pos r[3] = {R.x, R.y, R.z}, t3[3] = {T3.x, T3.y, T3.z};
  const Pos rn[3] = {RN.x, RN.y, RN.z}, tn[3] = {TN.x, TN.y, TN.z};
  const Pos t2[3] = {0, 0, 0};
  Pos tr[3], tt3[3], tt2[3];
  move_bead(kind, M, r, t3, t2, tr, tt3, tt2);
  if (side == 0) acc_add(out, pair_dE_fwd(bn, rn, r, tr, tn, t3, tt3));
  else acc_add(out, pair_dE_rev(bn, r, tr, rn, t3, tt3, tn));
  return out;
}

// FP64 storage: elastic energy of the same bond before the move (after = false)
// or after it.
static __device__ __forceinline__ double boundary_energy(const KArgs& a, const RepDev& rd, const MovePlan& P, int kind,
                                                   int side, bool after) {
  const ChainView<double> cv(a, rd, true);
  const long long i = side == 0 ? P.ind0 : P.indf - 1;
  const long long in = side == 0 ? i - 1 : i + 1;
  if (in < 0 || in >= rd.n_beads) return 0.0;
  double r[3], t3[3], rn[3], tn[3];
  ld3(cv.r4, i, r); ld3(cv.t34, i, t3); ld3(cv.r4, in, rn); ld3(cv.t34, in, tn);
  if (after) {
    double M[3][4], tr[3], tt3[3], tt2[3];
    const double t2[3] = {0, 0, 0};
    load_transform(P, M);
    move_bead(kind, M, r, t3, t2, tr, tt3, tt2);
    for (int j = 0; j < 3; j++) { r[j] = tr[j]; t3[j] = tt3[j]; }
  }
  const bool left = side == 0;
  double ra[3], rb[3], ta[3], tb[3];
  for (int j = 0; j < 3; j++) {
    ra[j] = left ? rn[j] : r[j];
    rb[j] = left ? r[j] : rn[j];
    ta[j] = left ? tn[j] : t3[j];
    tb[j] = left ? t3[j] : tn[j];
  }
  return bond_e(load_bond<double>(cv.bonds, left ? in : i), ra, rb, ta, tb);
}

// SSTWLC: twist energy of the same bond before the move (after = false) or
// after it.
template <typename Pos>
static __device__ __forceinline__ double boundary_twist(const KArgs& a, const RepDev& rd, const MovePlan& P, int kind,
                                                  int side, bool after) {
  const ChainView<Pos> cv(a, rd, false);
  const long long i = side == 0 ? P.ind0 : P.indf - 1;
  const long long in = side == 0 ? i - 1 : i + 1;
  if (in < 0 || in >= rd.n_beads) return 0.0;
  V4<Pos> T2 = cv.t24[i], T3 = cv.t34[i];
  const V4<Pos> N2 = cv.t24[in], N3 = cv.t34[in];
  if (after) {
    Pos M[3][4];
    load_transform(P, M);
    const Pos r[3] = {0, 0, 0}, t3[3] = {T3.x, T3.y, T3.z}, t2[3] = {T2.x, T2.y, T2.z};
    Pos tr[3], tt3[3], tt2[3];
    move_bead(kind, M, r, t3, t2, tr, tt3, tt2);
    T2.x = tt2[0]; T2.y = tt2[1]; T2.z = tt2[2];
    T3.x = tt3[0]; T3.y = tt3[1]; T3.z = tt3[2];
  }
  const bool left = side == 0;
  return twist_bond_energy(cv.twist + 2 * (left ? in : i), frame_of(left ? N2 : T2, left ? N3 : T3),
                           frame_of(left ? T2 : N2, left ? T3 : N3));
}

// Where one bead's weights lie before (0) and after (1) a move: the voxel of
// the lowest corner, the axes on which the upper voxel wraps to 0 (bit j), and
// the lower voxel's weight per axis.
template <typename Pos>
struct BeadCells {
  int v0, v1;
  unsigned wrap0, wrap1;
  Pos wl0[3], wl1[3];
};

// One lane's bead i = ind0 + k of a position move (transform M): moves it,
// stages its new vectors for the commit, counts the confinement crossings and
// finds its cells.  Returns false (and E_NONFINITE in e) for a position that
// is not finite.
template <typename Pos, int LEAN>
__device__ __forceinline__ bool place_bead(const RepDev& rd, const GridF& gf, const ChainView<Pos>& cv, int kind,
                                           const Pos (&M)[3][4], long long i, V4<Pos>* stage, bool density,
                                           bool conf, BeadCells<Pos>& c, unsigned& e, int& oob) {
  const V4<Pos> R = cv.r4[i];
  const Pos r[3] = {R.x, R.y, R.z};
  Pos t3[3] = {0, 0, 0}, t2[3] = {0, 0, 0}, tr[3], tt3[3], tt2[3];
  if (kind != CG_SLIDE) {
    const V4<Pos> T3 = cv.t34[i], T2 = cv.t24[i];
    t3[0] = T3.x; t3[1] = T3.y; t3[2] = T3.z;
    t2[0] = T2.x; t2[1] = T2.y; t2[2] = T2.z;
  }
  move_bead(kind, M, r, t3, t2, tr, tt3, tt2);
  stage[0] = V4<Pos>{tr[0], tr[1], tr[2], (Pos)0};
  if (kind != CG_SLIDE) {  // a slide's commit writes positions only
    stage[1] = V4<Pos>{tt3[0], tt3[1], tt3[2], (Pos)0};
    stage[2] = V4<Pos>{tt2[0], tt2[1], tt2[2], (Pos)0};
  }
  oob = conf ? out_of_bounds(rd, tr, true) * 65536 + out_of_bounds(rd, r, false) : 0;
  if (!(isfinite(tr[0]) && isfinite(tr[1]) && isfinite(tr[2]))) {
    e |= E_NONFINITE;
    return false;
  }
  if (density) {
    int lo[3], hi[3];
    move_axes<LEAN == 1>(rd, gf, r, c.wl0, lo, hi);
    c.v0 = lo[0] + gf.nx * lo[1] + gf.nxy * lo[2];
    c.wrap0 = (hi[0] == 0 ? 1u : 0u) | (hi[1] == 0 ? 2u : 0u) | (hi[2] == 0 ? 4u : 0u);
    move_axes<LEAN == 1>(rd, gf, tr, c.wl1, lo, hi);
    c.v1 = lo[0] + gf.nx * lo[1] + gf.nxy * lo[2];
    c.wrap1 = (hi[0] == 0 ? 1u : 0u) | (hi[1] == 0 ? 2u : 0u) | (hi[2] == 0 ? 4u : 0u);
  }
  return true;
}

// Voxels and fixed-point weights of the two corners (y, z bits of cl) a lane
// takes of one set of cells.
template <typename Pos>
__device__ __forceinline__ void corner_pair(const GridF& gf, int v, unsigned wrap, const Pos (&wl)[3], int cl,
                                            int& va, int& vb, long long& qa, long long& qb) {
  const bool by = cl & 1, bz = cl & 2;
  const Pos fy = by ? 1 - wl[1] : wl[1], fz = bz ? 1 - wl[2] : wl[2];
  if (by) v += (wrap & 2u) ? gf.nx - gf.nxy : gf.nx;
  if (bz) v += (wrap & 4u) ? gf.nxy - gf.nxy * gf.n[2] : gf.nxy;
  va = v;
  vb = v + ((wrap & 1u) ? 1 - gf.nx : 1);
  qa = q40(wl[0] * fy * fz);
  qb = q40((1 - wl[0]) * fy * fz);
}

// Voxel-table contributions of corners (cl, two along x) of a bead: q[2j] at
// vq[2j] (old weight removed; the weight change when the old and new cells
// are the same eight voxels) and q[2j+1] at vq[2j+1] (new weight otherwise).
template <typename Pos>
__device__ __forceinline__ void corner_terms(const GridF& gf, const BeadCells<Pos>& c, int cl,
                                             int (&vq)[2 * kCornersPerLane], long long (&q)[2 * kCornersPerLane]) {
  corner_pair(gf, c.v0, c.wrap0, c.wl0, cl, vq[0], vq[2], q[0], q[2]);
  corner_pair(gf, c.v1, c.wrap1, c.wl1, cl, vq[1], vq[3], q[1], q[3]);
  const bool same = c.v0 == c.v1;
#pragma unroll
  for (int j = 0; j < kCornersPerLane; j++) {
    const long long qo = q[2 * j], qn = q[2 * j + 1];
    q[2 * j] = same ? qn - qo : -qo;
    q[2 * j + 1] = same ? 0 : qn;
  }
}

template <typename Pos>
__device__ __forceinline__ BeadCells<Pos> shfl_cells(const BeadCells<Pos>& c, unsigned wraps, int src,
                                                     unsigned& got_wraps) {
  BeadCells<Pos> o;
  o.v0 = __shfl_sync(kFull, c.v0, src);
  o.v1 = __shfl_sync(kFull, c.v1, src);
  got_wraps = __shfl_sync(kFull, wraps, src);
#pragma unroll
  for (int j = 0; j < 3; j++) {
    o.wl0[j] = __shfl_sync(kFull, c.wl0[j], src);
    o.wl1[j] = __shfl_sync(kFull, c.wl1[j], src);
  }
  return o;
}

// A bond term kept in a move plan (fixed-point part and FP64 part).
__device__ __forceinline__ void store_acc(long long& q, double& h, const Fx& v) { q = v.q; h = v.hard; }
__device__ __forceinline__ void store_acc(long long& q, double& h, double v) { q = 0; h = v; }
template <typename Acc> __device__ __forceinline__ Acc load_acc(long long q, double h);
template <> __device__ __forceinline__ Fx load_acc<Fx>(long long q, double h) { return Fx{q, h}; }
template <> __device__ __forceinline__ double load_acc<double>(long long, double h) { return h; }

// Deposit of the batch's position moves that use a shared voxel table
// (plan.blk), by every thread of the CTA.  The moves' beads, in move order,
// are dealt out to the warps in runs of at most 32.  Each warp first takes one
// bead per lane (load, transform, staging, cells), then four lanes per bead:
// the cells go round by shuffles and each lane adds two corners (old weights
// out, new weights in) to the voxel table.  The last warp also takes the
// moves' boundary bonds, one per lane.  (Four lanes per bead for the whole
// task, each repeating the bead's transform and cells, issue three times the
// instructions; bonds on the lanes of a segment's end beads are executed by
// nearly every warp: together a ninth of a pass over 256 chains, and a third of
// one over SSTWLC chains, whose FP64 twist terms of a batch's bonds so share their
// warp's issue.)  The table is the CTA's pooled table (keys voxel * 32 + slot,
// one used list) or the slot's own table.  The bond terms, confinement counts
// and error bits go to the move's plan.  A move
// whose optimistic table overflows (E_OVF: a pool or a table past 3/4 load) is
// skipped from then on; its group deposits it again in its global table.
// Called by every thread.
template <typename Pos, int LEAN>
__device__ void block_deposit(const KArgs& a, SpecShared& sh, int rep, int B, int kind) {
  using Acc = typename AccOf<Pos>::type;
  unsigned char* smem = reinterpret_cast<unsigned char*>(&sh);
  const RepDev& rd = sh.ws.rd;
  const GridF& gf = sh.ws.gf;
  const ChainView<Pos> cv(a, rd, LEAN);
  const bool conf = rd.field_kind != 0 && rd.confine_kind;
  const int Hs = 1 << a.logH, hcol = a.hcol;
  const bool pool = a.pool_on != 0;
  const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5), W = (int)(blockDim.x >> 5);
  // lane j of every warp holds the end of move j's beads in the batch's bead
  // list (the moves with plan.blk)
  int end = (lane < B && sh.plan[lane].blk) ? sh.plan[lane].m : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, end, o);
    if (lane >= o) end += y;
  }
  const int total = __shfl_sync(kFull, end, 31);
  // One lane's two corners of a bead of move t (-1: none) with states inf.
  auto corner_pass = [&](const BeadCells<Pos>& d, int t, unsigned inf) {
    const int tt = t < 0 ? 0 : t;
    MovePlan& P = sh.plan[tt];
    const bool act = t >= 0 && !(P.derr & E_OVF);
    unsigned char* wb = smem + a.spec_off_warps + (size_t)tt * a.warp_smem;
    int vq[2 * kCornersPerLane];
    long long q[2 * kCornersPerLane];
    corner_terms(gf, d, lane % kLanesPerBead, vq, q);
    // the pooled table (one used list for the whole CTA, keys voxel * 32 +
    // slot), or the move's own table (one used list per move)
    int* keys = reinterpret_cast<int*>(pool ? smem + a.off_pkeys : wb + a.off_keys);
    int* used = reinterpret_cast<int*>(wb + a.off_used);
    unsigned short* pu = reinterpret_cast<unsigned short*>(smem + a.off_pused);
    long long* vals = reinterpret_cast<long long*>(pool ? smem + a.off_pvals : wb + a.off_vals);
    bool want[2 * kCornersPerLane];
#pragma unroll
    for (int j = 0; j < 2 * kCornersPerLane; j++) {
      want[j] = act && q[j] != 0;
      if (pool) vq[j] = vq[j] * 32 + tt;
    }
    const bool sure = P.sure && !pool;
    const unsigned full_bit = sure ? E_SPIN : E_OVF;
    const int lh = pool ? a.pool_logH : a.logH;
    int slot[2 * kCornersPerLane];
    unsigned e = 0;
    if (pool)
      claim_slots<2 * kCornersPerLane>(keys, pu, &sh.npool, lh, vq, want, slot, e, (3 << lh) / 4, full_bit);
    else
      claim_slots<2 * kCornersPerLane>(keys, used, &sh.nused[tt], lh, vq, want, slot, e,
                                       sure ? Hs : (3 << lh) / 4, full_bit);
    if (!(e & full_bit)) {
#pragma unroll
      for (int j = 0; j < 2 * kCornersPerLane; j++)
        if (want[j]) add_corner(vals, hcol, slot[j], q[j], inf, rd.nb, true);
    }
    if (e && t >= 0) atomicOr(&P.derr, e);
  };
  // warps of the beads: all, without those of an SSTWLC batch's bonds (below)
  // where at least half remain
  const bool twist = !LEAN && cv.twist != nullptr;
  const int tws = twist ? (4 * B + 31) >> 5 : 0, WD = 2 * tws <= W ? W - tws : W;
  constexpr int BP = 32 / kLanesPerBead;
  if constexpr (sizeof(Pos) == 8) {
    // FP64 holds its pipe for ~60 cycles an operation whatever the number of
    // lanes, so the four lanes of a bead take an axis each (the fourth repeats
    // the third's), 8 beads a warp and pass: one row of the transform, one
    // coordinate's cells.
    #pragma unroll 1
    for (int b0 = warp < WD ? warp * BP : total; b0 < total; b0 += WD * BP) {
      const int b = b0 + (lane >> 2), quad = lane & 28, ax = lane & 3, j = ax < 3 ? ax : 2;
      int s = 0;
      #pragma unroll 1
      for (int u = 0; u < B; u++) s += __shfl_sync(kFull, end, u) <= b ? 1 : 0;
      int base = __shfl_sync(kFull, end, s > 0 ? s - 1 : 0);
      if (s == 0) base = 0;
      bool on = b < total;
      if (!on) s = 0;
      MovePlan& P = sh.plan[s];
      double r[3] = {0, 0, 0}, tr = 0;
      unsigned sw = 0;
      if (on) {
        const long long k = b - base, i = P.ind0 + k;
        double* stage = reinterpret_cast<double*>(
            (P.gstage ? reinterpret_cast<V4<Pos>*>(a.g_stage) + ((long long)rep * a.spec_s + s) * a.g_stage_cap * 3
                      : reinterpret_cast<V4<Pos>*>(smem + a.spec_off_warps + (size_t)s * a.warp_smem + a.off_stage)) +
            3 * k);
        const double* M = reinterpret_cast<const double*>(P.M) + 4 * j;
        sw = cv.st[i];
        ld3(cv.r4, i, r);
        if (kind == CG_SLIDE) {  // a slide's commit writes positions only
          tr = (j == 0 ? r[0] : j == 1 ? r[1] : r[2]) + M[3];
        } else {
          double t3[3], t2[3];
          ld3(cv.t34, i, t3);
          ld3(cv.t24, i, t2);
          tr = M[0] * r[0] + M[1] * r[1] + M[2] * r[2] + M[3];
          const double tt3 = M[0] * t3[0] + M[1] * t3[1] + M[2] * t3[2];
          const double tt2 = M[0] * t2[0] + M[1] * t2[1] + M[2] * t2[2];
          stage[4 + ax] = ax < 3 ? tt3 : 0.0;
          stage[8 + ax] = ax < 3 ? tt2 : 0.0;
        }
        stage[ax] = ax < 3 ? tr : 0.0;
      }
      const unsigned bad = __ballot_sync(kFull, !isfinite(tr)) >> quad & 15u;
      const bool fast = LEAN != 1 && rd.fast_n > 0;
      double t[3] = {0, 0, 0};
      if (conf || fast)
        for (int q = 0; q < 3; q++) t[q] = __shfl_sync(kFull, tr, quad + q);
      if (conf && on && ax == 0) {
        const int oob = out_of_bounds(rd, t, true) * 65536 + out_of_bounds(rd, r, false);
        if (oob) atomicAdd(&P.oob, oob);
      }
      if (bad) {
        if (ax == 0) atomicOr(&P.derr, (unsigned)E_NONFINITE);
        on = false;
        tr = 0;
      }
      double w0, w1;
      int lo0, hi0, lo1, hi1;
      if (fast) {
        if (bad) t[0] = t[1] = t[2] = 0;
        double wa[3], wb[3];
        int la[3], ha[3], lb[3], hb[3];
        fast_axes_ool(rd, gf, r, wa, la, ha);
        fast_axes_ool(rd, gf, t, wb, lb, hb);
        w0 = j == 0 ? wa[0] : j == 1 ? wa[1] : wa[2];
        w1 = j == 0 ? wb[0] : j == 1 ? wb[1] : wb[2];
        lo0 = j == 0 ? la[0] : j == 1 ? la[1] : la[2];
        lo1 = j == 0 ? lb[0] : j == 1 ? lb[1] : lb[2];
        hi0 = j == 0 ? ha[0] : j == 1 ? ha[1] : ha[2];
        hi1 = j == 0 ? hb[0] : j == 1 ? hb[1] : hb[2];
      } else {
        const double w = *(j == 0 ? &rd.wx : j == 1 ? &rd.wy : &rd.wz), d = *(j == 0 ? &rd.dx : j == 1 ? &rd.dy : &rd.dz);
        const float iw = gf.inv_w[j];
        const double id = gf.inv_dd[j];
        const int n = gf.n[j];
        w0 = voxel_axis(j == 0 ? r[0] : j == 1 ? r[1] : r[2], w, d, iw, id, n, lo0, hi0);
        w1 = voxel_axis(tr, w, d, iw, id, n, lo1, hi1);
      }
      const int stride = ax == 0 ? 1 : ax == 1 ? gf.nx : ax == 2 ? gf.nxy : 0;
      BeadCells<Pos> c;
      c.v0 = lo0 * stride;
      c.v1 = lo1 * stride;
#pragma unroll
      for (int o = 1; o <= 2; o <<= 1) {
        c.v0 += __shfl_xor_sync(kFull, c.v0, o);
        c.v1 += __shfl_xor_sync(kFull, c.v1, o);
      }
      c.wrap0 = __ballot_sync(kFull, hi0 == 0) >> quad & 7u;
      c.wrap1 = __ballot_sync(kFull, hi1 == 0) >> quad & 7u;
#pragma unroll
      for (int q = 0; q < 3; q++) {
        c.wl0[q] = __shfl_sync(kFull, w0, quad + q);
        c.wl1[q] = __shfl_sync(kFull, w1, quad + q);
      }
      corner_pass(c, on ? s : -1, sw & 0xFFFFFFu);
    }
  } else {
    // beads per warp and round: an even share, in whole passes of the corners
    // (by steps: a batch has a few hundred beads)
    int per = WD;  // warps times rounds
    while (32 * per < total) per += WD;
    int run = BP;
    while (run * per < total) run += BP;
    #pragma unroll 1
    for (int b0 = warp < WD ? warp * run : total; b0 < total; b0 += WD * run) {
      const int b = b0 + lane;
      // the bead's move: the number of moves whose beads end at or before b
      int s = 0;
      #pragma unroll 1
      for (int j = 0; j < B; j++) s += __shfl_sync(kFull, end, j) <= b ? 1 : 0;
      int base = __shfl_sync(kFull, end, s > 0 ? s - 1 : 0);
      if (s == 0) base = 0;
      bool on = lane < run && b < total;
      if (!on) s = 0;
      BeadCells<Pos> c;
      c.v0 = c.v1 = 0;
      c.wrap0 = c.wrap1 = 0;
      for (int j = 0; j < 3; j++) c.wl0[j] = c.wl1[j] = 0;
      unsigned info = 0;  // states (three bytes), wrap bits of the cells before and after
      if (on) {
        MovePlan& P = sh.plan[s];
        const long long k = b - base, i = P.ind0 + k;
        Pos M[3][4];
        load_transform(P, M);
        V4<Pos>* stage = P.gstage ? reinterpret_cast<V4<Pos>*>(a.g_stage) +
                                        ((long long)rep * a.spec_s + s) * a.g_stage_cap * 3
                                  : reinterpret_cast<V4<Pos>*>(smem + a.spec_off_warps + (size_t)s * a.warp_smem +
                                                               a.off_stage);
        const unsigned sw = cv.st[i];
        unsigned e = 0;
        int oob;
        on = place_bead<Pos, LEAN>(rd, gf, cv, kind, M, i, stage + 3 * k, true, conf, c, e, oob);
        info = (sw & 0xFFFFFFu) | c.wrap0 << 24 | c.wrap1 << 27;
        if (oob) atomicAdd(&P.oob, oob);
        if (e) atomicOr(&P.derr, e);
      }
      const int sl = on ? s : -1;
      const int left = total - b0 < run ? total - b0 : run;
      #pragma unroll 1
      for (int p = 0; p < left; p += BP) {
        const int src = p + lane / kLanesPerBead;
        unsigned inf;
        BeadCells<Pos> d = shfl_cells(c, info, src, inf);
        const int t = __shfl_sync(kFull, sl, src);
        d.wrap0 = (inf >> 24) & 7u;
        d.wrap1 = (inf >> 27) & 7u;
        corner_pass(d, t, inf);
      }
    }
  }
  // boundary bonds of the moves, two per move
  if (twist || sizeof(Pos) == 8) {
    // a bond's energies before and after the move on two lanes each, four a move:
    // an energy of FP64 storage is ~45 FP64 operations, a twist energy ~150, which
    // issue at 1/64 of the FP32 rate whatever the number of lanes.  SSTWLC: by
    // warps without beads, where a batch's deposit waited for the two twist
    // energies of each bond (64 SSTWLC chains of 2,000 beads, 10 steps, kernel
    // only, with short_tangent_twist: 7.60 -> 4.82 ms)
    #pragma unroll 1
    for (int j0 = 32 * (W - 1 - warp); j0 < 4 * B; j0 += 32 * W) {
      const int j = j0 + lane, side = (j >> 1) & 1;
      MovePlan& P = sh.plan[j < 4 * B ? j >> 2 : 0];
      const bool on = j < 4 * B && P.blk;
      Acc t = acc_zero<Acc>();
      if constexpr (sizeof(Pos) == 8) {
        const double e = on ? boundary_energy(a, rd, P, kind, side, j & 1) : 0.0;
        t = __shfl_xor_sync(kFull, e, 1) - e;
      } else {
        if (on && !(j & 1)) t = boundary_term<Pos, Acc, LEAN>(a, rd, P, kind, side);
      }
      if (!LEAN && twist) {
        const double e = on ? boundary_twist<Pos>(a, rd, P, kind, side, j & 1) : 0.0;
        acc_add_d(t, __shfl_xor_sync(kFull, e, 1) - e);
      }
      if (on && !(j & 1)) store_acc(P.pq[side], P.ph[side], t);
    }
  } else if (warp == W - 1)
    for (int j = lane; j < 2 * B; j += 32) {
      MovePlan& P = sh.plan[j >> 1];
      if (P.blk) store_acc(P.pq[j & 1], P.ph[j & 1], boundary_term<Pos, Acc, LEAN>(a, rd, P, kind, j & 1));
    }
}

// One pooled entry's field term: FP32 storage in fixed point, FP64 storage in
// FP64.
__device__ __forceinline__ void pool_voxel_dE(const WarpShared& ws, const KArgs& a, const long long (&row)[4], int v,
                                              long long* d, Fx& part, long long& huge) {
  voxel_dE_f32(ws, a, row, v, d, true, part, huge);
}
__device__ __forceinline__ void pool_voxel_dE(const WarpShared& ws, const KArgs& a, const long long (&row)[4], int v,
                                              long long* d, double& part, long long& huge) {
  voxel_dE_f64(ws, a, row, v, d, true, part, huge);
}

// FP64 storage: a move's field dE is summed exactly (cg_exact.h), so that it does not
// depend on the order of its voxels, which the claims of a table, the warps of a pass
// and an overflow to another table change.  Terms beyond the limbs' range, 2^-108 ..
// 2^32, are added in FP64 to `beyond`, order-dependent in their last place.  The limbs
// are in the move slot's draw buffer, whose last draw was taken when the move was
// proposed.  (FP64 reductions of a warp's terms, and an FP64 shared atomic each, took
// 1.90 ms against 1.81 for 200 moves of each of 64 chains of 1,000 beads.)
static_assert(CGX_LIMBS <= kDrawCache && CGX_LIMBS <= 32, "the limbs share a slot's draw buffer, a lane clears one");
__device__ __forceinline__ int* move_limbs(const KArgs& a, SpecShared& sh, int s) {
  return reinterpret_cast<int*>(reinterpret_cast<unsigned char*>(&sh) + a.spec_off_warps +
                                (size_t)s * a.warp_smem + a.off_draws);
}
__device__ __forceinline__ void add_exact(int* L, double* beyond, double x) {
  int v[4];
  const int i = cgx_split((unsigned long long)__double_as_longlong(x), v);
  if (i < 0) {
    if (!is_zero64(x)) atomicAdd(beyond, x);
    return;
  }
#pragma unroll
  for (int k = 0; k < 4; k++) atomicAdd(L + i + k, v[k]);
}

// Add a lane's field term to its move's plan (s; -1: none).  Fixed point: q = l2
// 2^40 + l1 2^20 + l0 with l0, l1 in [0, 2^20); the limbs of at most 4,096 entries
// sum within 32 bits (|q| < 2^51), so each lane adds its own with four 32-bit
// shared atomics (a warp's entries belong to a handful of moves; reducing them move
// by move first took longer: the field phase of a batch of ~5 moves on 256 chains
// 12.0 k against 8.5 k cycles).
__device__ __forceinline__ void add_plan_part(MovePlan& P, const Fx& part) {
  atomicAdd(&P.fl0, (unsigned)(part.q & 0xFFFFF));
  atomicAdd(&P.fl1, (unsigned)((part.q >> 20) & 0xFFFFF));
  atomicAdd(&P.fl2, (int)(part.q >> 40));
  if (!is_zero64(part.hard)) atomicAdd(&P.fh, part.hard);
}
__device__ __forceinline__ void add_pool_part(const KArgs&, SpecShared& sh, int s, const Fx& part) {
  if (s < 0) return;
  MovePlan& P = sh.plan[s];
  add_plan_part(P, part);
  atomicAdd(&P.fn, 1);
}
__device__ __forceinline__ void add_pool_part(const KArgs& a, SpecShared& sh, int s, double part) {
  if (s < 0) return;
  MovePlan& P = sh.plan[s];
  add_exact(move_limbs(a, sh, s), &P.fh, part);
  atomicAdd(&P.fn, 1);
}

// Field dE and conflict registration of the batch's pooled voxel entries, by
// every thread of the CTA: entry -> (voxel, move slot s); the voxel's field
// term (which also leaves the voxel's post-move row in the entry for the
// commit); its registration in the block voxel table, whose atomicOr returns
// the moves that registered the voxel first (an earlier one is a conflict of
// s, a later one learns of s through its plan's mask).  Entries of moves that
// overflowed the pool are skipped (their groups redo them in their global
// tables).  Called by every thread.
template <typename Pos>
static __device__ void block_field_pool(const KArgs& a, SpecShared& sh, unsigned char* smem, int* bkeys,
                                 unsigned* bmask) {
  using Acc = typename AccOf<Pos>::type;
  const WarpShared& ws = sh.ws;
  const RepDev& rd = ws.rd;
  const int* pkeys = reinterpret_cast<const int*>(smem + a.off_pkeys);
  const unsigned short* pused = reinterpret_cast<const unsigned short*>(smem + a.off_pused);
  long long* pvals = reinterpret_cast<long long*>(smem + a.off_pvals);
  const long long* grid = a.grid + rd.vox_off * a.ncol;
  const int n = sh.npool;
  const int lane = (int)(threadIdx.x & 31u);
  // entry e's slot and key (-1: none, or of a move that overflowed) and its
  // voxel's grid row
  auto fetch = [&](int e, int& slot, int& key, long long (&row)[4]) {
    key = -1;
    slot = 0;
    if (e < n) {
      slot = pused[e];
      key = pkeys[slot];
      if (sh.plan[key & 31].derr & E_OVF) key = -1;
    }
    if (key >= 0) load_row(grid + (long long)(key >> 5) * a.ncol, a.ncol, row);
  };
  // an entry's row is under way while its voxel is registered (fetching the next
  // entry's ahead as well spilled registers and cost 1 %)
  #pragma unroll 1
  for (int e0 = (int)(threadIdx.x & ~31u); e0 < n; e0 += (int)blockDim.x) {
    int slot, key;
    long long row[4];
    fetch(e0 + lane, slot, key, row);
    const int s = key < 0 ? -1 : key & 31;
    Acc part = acc_zero<Acc>();
    if (key >= 0) {
      const int v = key >> 5;
      MovePlan& P = sh.plan[s];
      const int b = block_insert(bkeys, a.spec_logHB, v);
      if (b < 0) {
        atomicOr(&P.freg, 1);
      } else {
        const unsigned prior = atomicOr(&bmask[b], 1u << s);
        const unsigned below = (1u << s) - 1u, above = ~((2u << s) - 1u);
        if (prior & below) atomicOr(&P.cmask, prior & below);
        #pragma unroll 1
        for (unsigned later = prior & above; later; later &= later - 1)
          atomicOr(&sh.plan[__ffs((int)later) - 1].cmask, 1u << s);
      }
      long long hp = 0;
      pool_voxel_dE(ws, a, row, v, pvals + (long long)slot * a.hcol, part, hp);
      if (hp) atomicAdd(reinterpret_cast<unsigned long long*>(&P.fH), (unsigned long long)hp);
    }
    add_pool_part(a, sh, s, part);
  }
}

// Commit of the pooled entries after the batch is resolved, by every thread:
// the post-move rows of the standing accepted moves (the first `cut`, bits of
// `acc`) go to the grid with 16-byte stores; every entry is cleared, and so
// is the block voxel table.
static __device__ void block_commit_pool(const KArgs& a, SpecShared& sh, unsigned char* smem, int cut, unsigned acc,
                                  int* bkeys, unsigned* bmask) {
  // the last two warps keep the batch's books meanwhile (with two or fewer they
  // do both)
  const int tid = (int)threadIdx.x, nt = (int)blockDim.x > 64 ? (int)blockDim.x - 64 : (int)blockDim.x;
  if (tid >= nt) return;
  const RepDev& rd = sh.ws.rd;
  int* pkeys = reinterpret_cast<int*>(smem + a.off_pkeys);
  const unsigned short* pused = reinterpret_cast<const unsigned short*>(smem + a.off_pused);
  long long* pvals = reinterpret_cast<long long*>(smem + a.off_pvals);
  long long* grid = a.grid + rd.vox_off * a.ncol;
  const int n = sh.npool, hcol = a.hcol, ncol = a.ncol;
  #pragma unroll 1
  for (int e = tid; e < n; e += nt) {
    const int slot = pused[e];
    const int key = pkeys[slot];
    const int s = key & 31;
    long long* src = pvals + (long long)slot * hcol;
    if (s < cut && ((acc >> s) & 1u) && !(sh.plan[s].derr & E_OVF)) {
      longlong2* dst = reinterpret_cast<longlong2*>(grid + (long long)(key >> 5) * ncol);
      dst[0] = make_longlong2(src[0], src[1]);
      if (ncol == 4) dst[1] = make_longlong2(hcol > 2 ? src[2] : 0, hcol > 3 ? src[3] : 0);
    }
    pkeys[slot] = -1;
    #pragma unroll 1
    for (int cc = 0; cc < hcol; cc++) src[cc] = 0;
  }
  clear_block_table(bkeys, bmask, a.spec_logHB, tid, nt);
}

// Move-log terms of a plan (out of line: the log is off in production runs).
static __device__ __noinline__ void log_terms_d(MovePlan& P, double dEp, unsigned long long pos) {
  P.dEp = dEp;
  P.ndraw = (int)pos;
}
__device__ __forceinline__ void log_terms(MovePlan& P, double dEp, unsigned long long pos) {
  log_terms_d(P, dEp, pos);
}
__device__ __forceinline__ void log_terms(MovePlan& P, const Fx& dEp, unsigned long long pos) {
  log_terms_d(P, acc_d(dEp), pos);
}

// Record of move t (its plan) in the move log, when t is within the log.
static __device__ __noinline__ void log_move(const KArgs& a, int rep, unsigned long long k, const MovePlan& P) {
  if (k >= (unsigned long long)a.mlog_cap) return;
  cg_move_record rec;
  rec.kind = P.kind;
  rec.n_inds = P.empty ? 0 : P.m;
  rec.ind0 = P.ind0;
  rec.indf = P.indf;
  rec.dE_poly = P.empty ? 0.0 : P.dEp;
  rec.dE_field = P.empty ? 0.0 : dE_value(P.dq, P.dE) - P.dEp;
  rec.accepted = P.empty ? -1 : P.dec;
  rec.n_draws = P.ndraw;
  a.mlog[(long long)rep * a.mlog_cap + (long long)k] = rec;
}

// A move's field dE from its plan: fixed point into `soft` (FP32 storage) or
// FP64 into `hard` (limbs: move_limbs).
__device__ __forceinline__ void plan_field(const MovePlan& P, const int*, Fx& soft, double&) {
  soft.q = P.fq + (long long)P.fl2 * 1099511627776LL + (long long)P.fl1 * 1048576LL + (long long)P.fl0;
  soft.hard = P.fh;
}
__device__ __forceinline__ void plan_field(const MovePlan& P, const int* limbs, double&, double& hard) {
  hard = cgx_value(limbs);
  if (!is_zero64(P.fh)) hard += P.fh;
}

// Scratch of move slot `slot`: its shared-memory region, or its region of the
// global scratch (tables, staging and lists of any size the move can have).
__device__ __forceinline__ SlotScratch shared_slot(const KArgs& a, SpecShared& sh, int slot) {
  unsigned char* wb = reinterpret_cast<unsigned char*>(&sh) + a.spec_off_warps + (size_t)slot * a.warp_smem;
  SlotScratch S;
  S.keys = reinterpret_cast<int*>(wb + a.off_keys);
  S.used = reinterpret_cast<int*>(wb + a.off_used);
  S.bslot = reinterpret_cast<int*>(wb + a.off_bslot);
  S.vals = reinterpret_cast<long long*>(wb + a.off_vals);
  S.logH = a.logH;
  S.stage = wb + a.off_stage;
  S.idx = reinterpret_cast<int*>(wb + a.off_idx);
  return S;
}
template <typename Pos>
__device__ __forceinline__ SlotScratch global_slot(const KArgs& a, int rep, int slot) {
  const long long gi = (long long)rep * a.spec_s + slot, Hg = 1LL << a.g_logH;
  SlotScratch S;
  S.keys = a.g_keys + gi * Hg;
  S.used = a.g_used + gi * Hg;
  S.bslot = a.g_bslot + gi * Hg;
  S.vals = a.g_vals + gi * Hg * a.hcol;
  S.logH = a.g_logH;
  S.stage = reinterpret_cast<V4<Pos>*>(a.g_stage) + gi * a.g_stage_cap * 3;
  S.idx = a.g_idx + gi * a.g_stage_cap;
  return S;
}

// Field dE over a move's own table (nu entries, slot s) by its group: fixed point
// into `soft` (FP32 storage), or into the move's limbs and P.fh (FP64 storage; the
// limbs and P.fh are zero).
template <int G>
__device__ __forceinline__ void own_field(const KArgs& a, SpecShared& sh, int s, const SlotScratch& S, int nu, int gl,
                                          bool split, long long& nvox, Fx& soft, long long& huge) {
  double hard = 0;
  field_dE_voxels<G>(sh.ws, a, a.hcol, S.keys, S.used, S.vals, nu, gl, nvox, soft, hard, huge, split);
}
template <int G>
__device__ __forceinline__ void own_field(const KArgs& a, SpecShared& sh, int s, const SlotScratch& S, int nu, int gl,
                                          bool split, long long& nvox, double&, long long& huge) {
  static_assert(G == 32, "a move of FP64 storage has a warp");
  const long long* grid = a.grid + sh.ws.rd.vox_off * a.ncol;
  int* limbs = move_limbs(a, sh, s);
  long long hp = 0;
  int room = CGX_TERMS;  // terms that the limbs still hold
  #pragma unroll 1
  for (int i0 = 0; i0 < nu; i0 += 32) {
    const int i = i0 + gl;
    if (i < nu) {
      const int slot = S.used[i], v = S.keys[slot];
      long long row[4];
      load_row(grid + (long long)v * a.ncol, a.ncol, row);
      double part = 0;
      voxel_dE_f64(sh.ws, a, row, v, S.vals + (long long)slot * a.hcol, split, part, hp);
      add_exact(limbs, &sh.plan[s].fh, part);
    }
    room -= 32;
    if (room < 32) {
      __syncwarp();
      if (gl == 0) cgx_carry(limbs);
      __syncwarp();
      room = CGX_TERMS;
    }
  }
  nvox = nu;
  huge += gsum<32>(hp);
  __syncwarp();
}
// Field terms of a move left in its plan by own_path.
__device__ __forceinline__ void store_field(MovePlan& P, const Fx& soft) { P.fq = soft.q; P.fh = soft.hard; }
__device__ __forceinline__ void store_field(MovePlan&, double) {}

// A position move taken by its own group: its deposit (`dep`: the CTA did not
// deposit it, or it overflowed the shared table it was deposited in) in its
// shared or global table, the field dE over that table and the registration of
// its voxels, all left in its plan.  The moves of the pooled table need it
// only when they are long (over kPoolMaxBeads) or overflowed the pool; chains
// in no density field take it for the bond terms.  Out of line: with the pooled
// table it is rare, and inline it cost every batch ~3.6 k cycles of empty
// passes and reductions.  Called by the whole warp; `run` is false for groups
// without such a move.
template <typename Pos, int G, int LEAN>
static __device__ __noinline__ void own_path(const KArgs& a, SpecShared& sh, int rep, int s, int gl, bool run,
                                             int kind, int* bkeys, unsigned* bmask) {
  using Acc = typename AccOf<Pos>::type;
  const RepDev& rd = sh.ws.rd;
  const GridF& gf = sh.ws.gf;
  const ChainView<Pos> cv(a, rd, LEAN);
  MovePlan& P = sh.plan[s];
  const int hcol = a.hcol;
  const bool density = rd.field_kind == 2, check_field = rd.field_kind != 0;
  const long long m = run ? P.m : 0, ind0 = run ? P.ind0 : 0;
  const int Hs = 1 << a.logH;
  const bool sure = run && P.sure;
  int gtab = run ? P.gtab : 0;
  bool ovf = run && (P.derr & E_OVF) != 0;
  bool dep = run && (!P.blk || ovf);
  int* nused = &sh.nused[s];
  SlotScratch S = gtab ? global_slot<Pos>(a, rep, s) : shared_slot(a, sh, s);
  V4<Pos>* stage = reinterpret_cast<V4<Pos>*>(run && P.gstage ? global_slot<Pos>(a, rep, s).stage
                                                              : shared_slot(a, sh, s).stage);
  Pos M[3][4];
  load_transform(P, M);
  unsigned err = 0;
  int oob = 0;
  // pass 0: moves the CTA did not deposit; pass 1: overflowed ones
  for (int pass = 0; pass < 2; pass++) {
    if (pass == 1) {
      if (!__any_sync(kFull, ovf)) break;
      if (ovf && !gtab) clear_table(S, hcol, *nused, gl, G);
      __syncwarp();
      if (ovf) {
        if (gl == 0) *nused = 0;
        S = global_slot<Pos>(a, rep, s);
        gtab = 1;
        oob = 0;
      }
      __syncwarp();
    }
    const bool go = pass == 0 ? (dep && !ovf) : ovf;
    const int cap = gtab ? (1 << a.g_logH) : (sure ? Hs : (3 * Hs) / 4);
    const unsigned full_bit = (gtab || sure) ? E_SPIN : E_OVF;
    unsigned e = 0;
    // one bead per lane, its corners two by two
    #pragma unroll 1
    for (long long kb = 0; __any_sync(kFull, go && kb < m && !(e & E_OVF)); kb += G) {
      const long long k = kb + gl;
      bool act = go && k < m && !(e & E_OVF);
      BeadCells<Pos> c = {};
      unsigned sw = 0;
      if (act) {
        int ob;
        if (density) sw = cv.st[ind0 + k];
        act = place_bead<Pos, LEAN>(rd, gf, cv, kind, M, ind0 + k, stage + 3 * k, density, check_field && rd.confine_kind, c,
                         e, ob);
        oob += ob;
      }
      if (density) {
        for (int cl = 0; cl < kLanesPerBead; cl++) {
          int vq[2 * kCornersPerLane];
          long long q[2 * kCornersPerLane];
          corner_terms(gf, c, cl, vq, q);
          bool want[2 * kCornersPerLane];
#pragma unroll
          for (int j = 0; j < 2 * kCornersPerLane; j++) want[j] = act && q[j] != 0 && !(e & E_OVF);
          int slot[2 * kCornersPerLane];
          claim_slots<2 * kCornersPerLane>(S.keys, S.used, nused, S.logH, vq, want, slot, e, cap, full_bit);
          if (!(e & full_bit)) {
#pragma unroll
            for (int j = 0; j < 2 * kCornersPerLane; j++)
              if (want[j]) add_corner(S.vals, hcol, slot[j], q[j], sw, rd.nb, !gtab);
          }
        }
        e = gor<G>(e);  // a full table ends the group's passes together
      }
    }
    e = gor<G>(e);
    if (go) ovf = pass == 0 && (e & E_OVF) != 0;
    err |= e & ~E_OVF;
  }
  err = gor<G>(err);
  oob = gsum<G>(oob);
  __syncwarp();
  Acc soft = acc_zero<Acc>();
  long long huge = 0, nvox = 0;
  unsigned cmb = 0;
  int regfail = 0;
  if (density) {
    const int nu = run ? *nused : 0;
    own_field<G>(a, sh, s, S, nu, gl, !gtab, nvox, soft, huge);
    // register the touched voxels for the conflict test: the moves that
    // registered a voxel first are this move's conflicts if earlier in the
    // batch; a later move that registered it first learns of this one through
    // its plan's mask
    const int nr = err ? 0 : nu;
    const unsigned below = (1u << s) - 1u, above = ~((2u << s) - 1u);
    #pragma unroll 1
    for (int i = gl; i < nr; i += G) {
      const int b = block_insert(bkeys, a.spec_logHB, S.keys[S.used[i]]);
      S.bslot[i] = b;
      if (b < 0) {
        regfail = 1;
      } else {
        const unsigned prior = atomicOr(&bmask[b], 1u << s);
        cmb |= prior & below;
        #pragma unroll 1
        for (unsigned later = prior & above; later; later &= later - 1)
          atomicOr(&sh.plan[__ffs((int)later) - 1].cmask, 1u << s);
      }
    }
    cmb = gor<G>(cmb);
    regfail = (int)gor<G>((unsigned)regfail);
  }
  Acc bond = acc_zero<Acc>();
  if (dep && gl < 2) {
    bond = boundary_term<Pos, Acc, LEAN>(a, rd, P, kind, gl);
    if (!LEAN && rd.twist)
      acc_add_d(bond, boundary_twist<Pos>(a, rd, P, kind, gl, true) - boundary_twist<Pos>(a, rd, P, kind, gl, false));
  }
  if (dep && gl < 2) store_acc(P.pq[gl], P.ph[gl], bond);
  if (run && gl == 0) {
    if (dep) P.oob = oob;
    if (err) atomicOr(&P.derr, err);  // E_OVF stays: the pooled pass and commit skip this move's entries
    P.gtab = gtab;
    P.fn = (int)nvox;
    P.fH = huge;
    store_field(P, soft);
    if (cmb) atomicOr(&P.cmask, cmb);
    P.freg = regfail;
  }
  __syncwarp();
}

// Tangent rotation of bead i about the axis of draws xa, xb (sine sa, cosine
// ca): its new frame and the dE of its two bonds, the neighbours' frames as they
// are.  Lean: without the twist terms.
template <typename Pos, int LEAN>
__device__ __forceinline__ typename AccOf<Pos>::type rotate_tangent(const KArgs& a, const RepDev& rd, long long i,
                                                                    unsigned xa, unsigned xb, Pos sa, Pos ca,
                                                                    Pos (&tt3)[3], Pos (&tt2)[3]) {
  using Real = Pos;
  using Acc = typename AccOf<Real>::type;
  const long long N = rd.n_beads;
  const V4<Pos>* r4 = reinterpret_cast<const V4<Pos>*>(a.r4) + rd.bead_off;
  const V4<Pos>* t34 = reinterpret_cast<const V4<Pos>*>(a.t34) + rd.bead_off;
  const V4<Pos>* t24 = reinterpret_cast<const V4<Pos>*>(a.t24) + rd.bead_off;
  const double* bonds = a.bonds + rd.bead_off * 6;
  const float* bonds32 = a.bonds32 + rd.bead_off * 8;
  // the bead, both neighbours and both bonds, loaded together (in-range
  // indices at the chain ends, where the term is skipped)
  const bool hl = i != 0, hr = i + 1 != N;
  const long long il = hl ? i - 1 : i, ir = hr ? i + 1 : i;
  Real r[3], t3[3], t2[3], r0[3], t30[3], r1[3], t31[3];
  ld3(r4, i, r); ld3(t34, i, t3); ld3(t24, i, t2);
  ld3(r4, il, r0); ld3(t34, il, t30); ld3(r4, ir, r1); ld3(t34, ir, t31);
  const Bond<Real> bl = bond_at(bonds, bonds32, il, (Real)0), br = bond_at(bonds, bonds32, i, (Real)0);
  Real axis[3];
  sphere_from<Real>(xa, xb, axis);
  const Real origin[3] = {0, 0, 0};
  Real M[3][4];
  axis_rotation_sc(axis, origin, sa, ca, M);
  for (int j = 0; j < 3; j++) {
    Real e3 = 0, e2 = 0;
    for (int q = 0; q < 3; q++) { e3 += M[j][q] * t3[q]; e2 += M[j][q] * t2[q]; }
    tt3[j] = e3; tt2[j] = e2;
  }
  Acc de = acc_zero<Acc>();
  if (hl) acc_add(de, tangent_dE_fwd(bl, r0, r, t30, t3, tt3));
  if (hr) acc_add(de, tangent_dE_rev(br, r, r1, t3, tt3, t31));
  if (!LEAN && rd.twist) {  // SSTWLC: twist terms of both bonds
    const double* tw = a.twist + rd.bead_off * 2;
    const Frame cur = frame_of(t2, t3), nw = frame_of(tt2, tt3);
    double dt = 0;
    if (hl) {
      const Frame l = frame_of(t24[il], t34[il]);
      dt += twist_pair_dE(tw + 2 * il, l, cur, l, nw);
    }
    if (hr) {
      const Frame rr = frame_of(t24[ir], t34[ir]);
      dt += twist_pair_dE(tw + 2 * i, cur, rr, nw, rr);
    }
    acc_add_d(de, dt);
  }
  return de;
}

// ---------------------------------------------------------------- short tangent rotations
// Batches of tangent rotations of few beads (SimpleControl settles at an
// amplitude of ~13, a mean of 7 beads): 8 lanes per move up to 8 beads, 16 beyond,
// instead of 32, so that 2-4 times as many moves are in flight on the same warps,
// and the rotated beads registered in the block table (key: bead), so that a
// move finds the earlier moves that rotate its beads or their neighbours by
// three look-ups a bead instead of comparing lists.  A move's staging, index
// list and draws fit a quarter of a slot's region for up to 16 beads, half of it
// for up to 32.  One 10,000-bead chain,
// 10 MC steps, kernel only: 2.83 -> 2.62 ms; 64 SSTWLC chains of 2,000 beads,
// whose FP64 twist terms fill their warps' lanes: 10.4 -> 9.1 ms (with the
// phases' state kept in the plans); 9-16 beads on 16 lanes instead of 8, one
// pass instead of two: 256 chains 9.90 -> 9.53 ms, the SSTWLC chains 8.46 -> 7.60.
//
// Without twist, amplitudes above 16 + N S / 4000 (S moves in flight) and those with
// amp^2 > 5.4 sqrt(N S) take the path of 32 lanes: on 16 lanes over 16 beads need two
// passes, which pays where more moves stand than the S of 32 lanes, and beads drawn
// twice, likely on short chains, are redrawn by one lane.  320 rotations here / there,
// us: 64 chains (S = 12) of 50 beads, up to 10 / 13 / 16: 1,160 / 1,454 / 1,747 and
// 1,401 / 1,468 / 1,538; of 1,000, up to 17 / 24 / 32: 644 / 1,137 / 1,819 and 832 /
// 1,084 / 1,288; of 5,000: 374 / 555 / 883 and 539 / 700 / 856; 32 of 50,000: 232 / 306 /
// 395 and 411 / 468 / 544.  256 chains (S = 6) of 50 beads, up to 8 / 10 / 13: 928 /
// 1,132 / 1,358 and 1,088 / 1,161 / 1,182; of 5,000, up to 17 / 24 / 32: 432 / 698 / 943
// and 563 / 665 / 795.  The FP64 twist terms outweigh that up to 32 beads and amp^2 =
// 16 N (200 rotations on each of 64 SSTWLC chains of 20 beads, up to 16 / 20: 3,052 /
// 5,464 and 4,978 / 4,760; of 50, up to 26 / 32: 3,811 / 4,787 and 4,360 / 4,247; of
// 200, up to 32: 3,678 and 4,052).
//
// Moves in flight: kShortSpan sqrt(N) / (amp + 1), at which about two of them
// meet an earlier accepted one (3 and 4 measured alike, 6 and 9 were slower on
// 2,000-bead chains).
constexpr float kShortSpan = 4.0f;
struct ShortTangent {
  int GS, s, gl;
  unsigned gmask;  // the group's lanes
  int* idx;
  float* stage;    // new t3, t2 of each bead: 6 floats
  unsigned* draws;
  int ndraw;
  // gs lanes a group; up to cap (16 or 32) beads a move, which take a quarter or
  // a half of a slot's region
  __device__ __forceinline__ ShortTangent(const KArgs& a, SpecShared& sh, int gs, int cap) : GS(gs) {
    const int lane = (int)(threadIdx.x & 31u), per = 64 / cap;
    s = (int)threadIdx.x / gs;
    gl = lane & (gs - 1);
    gmask = (gs == 16 ? 0xFFFFu : 0xFFu) << (lane & ~(gs - 1));
    const int room = ((a.off_idx - a.off_stage + 4 * (int)a.stage_cap) / per) & ~15;
    place(a, sh, s, cap, idx, stage);
    draws = reinterpret_cast<unsigned*>(stage + 6 * cap);
    ndraw = (room - 24 * cap) / 16 * 4;
  }
  // index list and staging of move s
  static __device__ __forceinline__ void place(const KArgs& a, SpecShared& sh, int s, int cap, int*& idx,
                                               float*& stage) {
    const int per = 64 / cap, sub = s % per;
    unsigned char* base =
        reinterpret_cast<unsigned char*>(&sh) + a.spec_off_warps + (size_t)(s / per) * a.warp_smem;
    const int room = ((a.off_idx - a.off_stage + 4 * (int)a.stage_cap) / per) & ~15;
    idx = reinterpret_cast<int*>(base + a.off_draws) + sub * cap;
    stage = reinterpret_cast<float*>(base + a.off_stage + sub * room);
  }
};
static_assert(kDrawCache == 64, "the index lists share a slot's draw buffer: four of 16 or two of 32 beads");

__device__ __forceinline__ unsigned block_find(const int* bkeys, const unsigned* bmask, int logHB, int key) {
  const unsigned mask = (1u << logHB) - 1u;
  unsigned h = ((unsigned)key * 0x9E3779B1u) >> (32 - logHB);
  #pragma unroll 1
  for (int it = 0; it < 64; it++) {  // as far as block_insert probes
    const int k = bkeys[h];
    if (k == key) return bmask[h];
    if (k == -1) return 0u;
    h = (h + 1) & mask;
  }
  return 0u;
}

// Evaluate the batch's B moves (one per group of GS lanes) into their plans.
template <int LEAN>
__device__ void short_tangent_evaluate(const KArgs& a, SpecShared& sh, int rep, const ShortTangent& T, int B,
                                       const cg_move_ctl& c, int* bkeys, unsigned* bmask) {
  const RepDev& rd = sh.ws.rd;
  const int GS = T.GS, gl = T.gl, s = T.s;
  const bool live = s < B;
  if (!__any_sync(kFull, live)) return;
  const unsigned N = (unsigned)rd.n_beads, amp = (unsigned)c.amp_bead;
  const unsigned long long t = sh.t0 + (unsigned long long)s;
  const uint2 key = make_uint2((unsigned)a.seed ^ (unsigned)rep * 0x85EBCA6Bu,
                               (unsigned)(a.seed >> 32) ^ 0x1B873593u);
  const unsigned tlo = (unsigned)t, thi = (unsigned)(t >> 32);
  const int have = min(T.ndraw, (int)(3 * amp + 6) & ~3);  // angle, count, beads, axes, decision
  #pragma unroll 1
  for (int j = gl; 4 * j < have; j += GS)
    reinterpret_cast<uint4*>(T.draws)[j] = philox(make_uint4((unsigned)j, tlo, thi, 0x2545F491u), key);
  __syncwarp();
  auto word = [&](int j) { return j < have ? T.draws[j] >> 1 : move_draw_slow(key, tlo, thi, (unsigned long long)j); };
  const float ang = (float)c.amp_move * (uni<float>(word(0)) - 0.5f);
  const int n = (int)(word(1) % amp) + 1;
  unsigned err = n > (int)N ? E_WINDOW : 0u;
  int m = live && !err ? n : 0;
  // distinct random beads in draw order: nearly always the first m draws are
  int mine[2] = {-1, -1};
#pragma unroll
  for (int p = 0; p < 2; p++) {
    const int k = p * GS + gl;
    if (k < m) T.idx[k] = mine[p] = (int)(word(2 + k) % N);
  }
  __syncwarp();
  bool dup = false;
  const int most = (int)__reduce_max_sync(kFull, (unsigned)m);
  #pragma unroll 1
  for (int q = 0; q + 1 < most; q++) {
    const int v = q < m ? T.idx[q] : -2;
    dup = dup || (v == mine[0] && q < gl) || (v == mine[1] && q < GS + gl);
  }
  const unsigned dups = __ballot_sync(kFull, dup);
  int used = m;  // draws taken for the beads
  if (dups) {    // with redraws: by the group's first lane
    if ((dups & T.gmask) && gl == 0) {
      int got = 0, pos = 0;
      while (got < m) {
        if (pos >= 32 * kMaxIter) { err |= E_SPIN; break; }
        const int x = (int)(word(2 + pos++) % N);
        bool seen = false;
        #pragma unroll 1
        for (int q = 0; q < got; q++) seen = seen || T.idx[q] == x;
        if (!seen) T.idx[got++] = x;
      }
      used = pos;
    }
    const int first = __ffs((int)T.gmask) - 1;
    used = __shfl_sync(kFull, used, first);
    err |= __shfl_sync(kFull, err, first);
    if (err) m = 0;
    __syncwarp();
  }
  float sa, ca;
  rsincos(ang, &sa, &ca);
  Fx part = acc_zero<Fx>();
  int regfail = 0;
  #pragma unroll 1
  for (int k = gl; k < m; k += GS) {
    const int i = T.idx[k];
    const unsigned xa = word(2 + used + 2 * k), xb = word(3 + used + 2 * k);
    float tt3[3], tt2[3];
    acc_add(part, rotate_tangent<float, true>(a, rd, i, xa, xb, sa, ca, tt3, tt2));
    for (int j = 0; j < 3; j++) {
      T.stage[6 * k + j] = tt3[j];
      T.stage[6 * k + 3 + j] = tt2[j];
    }
    const int b = block_insert(bkeys, a.spec_logHB, i);
    if (b < 0) regfail = 1;
    else atomicOr(&bmask[b], 1u << s);
  }
  #pragma unroll 1
  for (int o = GS / 2; o > 0; o >>= 1) {
    part.q += __shfl_xor_sync(kFull, part.q, o);
    regfail |= __shfl_xor_sync(kFull, regfail, o);
  }
  if (__any_sync(kFull, !is_zero64(part.hard)))
    #pragma unroll 1
    for (int o = GS / 2; o > 0; o >>= 1) part.hard += __shfl_xor_sync(kFull, part.hard, o);
  if (live && gl == 0) {
    MovePlan& P = sh.plan[s];
    P.kind = CG_TANGENT_ROTATION;
    P.m = m;
    P.ind0 = m > 0 ? T.idx[0] : 0;
    P.indf = m > 0 ? P.ind0 + 1 : 0;
    P.empty = 0;
    P.err = (int)err;
    P.regfail = regfail;
    P.nvox = 0;
    P.cmask = 0;
    if (!LEAN && rd.twist) {  // decided by short_tangent_twist
      P.xm = word(2 + used + 2 * m);
      P.ndraw = 2 + used + 2 * m + (err ? 0 : 1);
      P.fq = part.q;
      P.fh = part.hard;
      P.fl0 = P.fl1 = 0;
      P.fl2 = 0;
      return;
    }
    bool dec = false;
    if (!err) dec = decide(word(2 + used + 2 * m), part, Fx{0, 0.0}, 0.0, P.dq, P.dE);
    P.dec = dec ? 1 : 0;
    if (!LEAN && a.mlog) log_terms(P, part, (unsigned long long)(2 + used + 2 * m + (err ? 0 : 1)));
  }
}

// SSTWLC: twist terms of the batch's rotated beads, then the decisions.  A
// bead's four bond energies (left and right bond, before and after) are taken by
// four lanes, the batch's beads packed over the CTA's warps: one FP64 energy after
// another in the bead's own lane were 43 k of a batch's 57 k cycles.  Called by
// every thread, after a barrier.
static __device__ __noinline__ void short_tangent_twist(const KArgs& a, SpecShared& sh, int B, int cap) {
  const RepDev& rd = sh.ws.rd;
  const ChainView<float> cv(a, rd, false);
  const int lane = (int)(threadIdx.x & 31u);
  int end = lane < B ? sh.plan[lane].m : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, end, o);
    if (lane >= o) end += y;
  }
  const int total = 4 * __shfl_sync(kFull, end, 31);
  #pragma unroll 1
  for (int j0 = (int)threadIdx.x - lane; j0 < total; j0 += (int)blockDim.x) {
    const int j = j0 + lane;
    int s = 0;
    #pragma unroll 1
    for (int u = 0; u < B; u++) s += __shfl_sync(kFull, end, u) <= (j >> 2) ? 1 : 0;
    int base = __shfl_sync(kFull, end, s > 0 ? (s - 1) & 31 : 0);
    if (s == 0) base = 0;
    const bool on = j < total;
    double e = 0.0;
    if (on) {
      int* idx;
      float* stage;
      ShortTangent::place(a, sh, s, cap, idx, stage);
      const int k = (j >> 2) - base, i = idx[k];
      const bool left = !(j & 2);
      const int in = left ? i - 1 : i + 1;
      if (in >= 0 && in < (int)rd.n_beads) {
        V4<float> T2 = cv.t24[i], T3 = cv.t34[i];
        const V4<float> N2 = cv.t24[in], N3 = cv.t34[in];
        if (j & 1) {
          const float* q = stage + 6 * k;
          T3 = V4<float>{q[0], q[1], q[2], 0.0f};
          T2 = V4<float>{q[3], q[4], q[5], 0.0f};
        }
        e = twist_bond_energy(cv.twist + 2 * (left ? in : i), frame_of(left ? N2 : T2, left ? N3 : T3),
                              frame_of(left ? T2 : N2, left ? T3 : N3));
      }
    }
    const double d = __shfl_xor_sync(kFull, e, 1) - e;       // lanes 0 and 2 of four
    const double dt = d + __shfl_down_sync(kFull, d, 2);     // lane 0
    if (on && !(j & 3)) {
      Fx part = acc_zero<Fx>();
      acc_add_d(part, dt);
      add_plan_part(sh.plan[s], part);
    }
  }
  __syncthreads();
  if ((int)threadIdx.x < B) {
    MovePlan& P = sh.plan[threadIdx.x];
    Fx part;
    double none = 0.0;
    plan_field(P, nullptr, part, none);
    bool dec = false;
    if (!P.err) dec = decide(P.xm, part, Fx{0, 0.0}, 0.0, P.dq, P.dE);
    P.dec = dec ? 1 : 0;
    if (a.mlog) log_terms(P, part, (unsigned long long)P.ndraw);
  }
}

// The earlier moves of the batch that rotate this move's beads or their
// neighbours.
static __device__ __forceinline__ void short_tangent_conflicts(const KArgs& a, SpecShared& sh, const ShortTangent& T, int B,
                                                        const int* bkeys, const unsigned* bmask) {
  const int s = T.s;
  unsigned cm = 0;
  const int m = s < B ? sh.plan[s].m : 0;
  #pragma unroll 1
  for (int k = T.gl; k < m; k += T.GS) {
    const int i = T.idx[k];
#pragma unroll
    for (int d = -1; d <= 1; d++) cm |= block_find(bkeys, bmask, a.spec_logHB, i + d);
  }
  cm &= (1u << s) - 1u;
  if (cm) atomicOr(&sh.plan[s].cmask, cm);
}

static __device__ __forceinline__ void short_tangent_commit(const KArgs& a, SpecShared& sh, const ShortTangent& T, int cut,
                                                     unsigned acc, int* bkeys, unsigned* bmask) {
  const RepDev& rd = sh.ws.rd;
  const int s = T.s;
  if (s < cut && ((acc >> s) & 1u)) {
    V4<float>* t34w = reinterpret_cast<V4<float>*>(a.t34) + rd.bead_off;
    V4<float>* t24w = reinterpret_cast<V4<float>*>(a.t24) + rd.bead_off;
    const int m = sh.plan[s].m;
    #pragma unroll 1
    for (int k = T.gl; k < m; k += T.GS) {
      const float* q = T.stage + 6 * k;
      const int i = T.idx[k];
      t34w[i] = V4<float>{q[0], q[1], q[2], 0.0f};
      t24w[i] = V4<float>{q[3], q[4], q[5], 0.0f};
    }
  }
  clear_block_table(bkeys, bmask, a.spec_logHB, (int)threadIdx.x, (int)blockDim.x);
}

__device__ __forceinline__ void segment_of(long long b0, long long b1, long long N, int& ind0, int& indf) {
  long long i0, i1;
  check_bead_bounds(b0, b1, N, i0, i1);
  ind0 = (int)i0;
  indf = (int)i1;
}

// A move's state between the phases of its batch is in its plan, so little is
// held in registers over them (kept in registers, it was spilled around the
// out-of-line own_path and cost every batch ~5 %).

// Propose position move t of the batch in slot s (group lanes gl = 0..G-1):
// its segment and transform, its table and its Metropolis draw go to its plan.
// `live` is false for the groups of a partly filled batch.  Called by the whole
// warp.
template <typename Pos, int G, int LEAN>
__device__ void propose_position(const KArgs& a, SpecShared& sh, int rep, int s, int gl, bool live, int kind,
                                 const cg_move_ctl& c, unsigned long long t) {
  using Real = Pos;
  const RepDev& rd = sh.ws.rd;
  const long long N = rd.n_beads;
  const V4<Pos>* r4 = reinterpret_cast<const V4<Pos>*>(a.r4) + rd.bead_off;
  MovePlan& P = sh.plan[s];
  MoveRng g;
  if (!__any_sync(kFull, live)) return;
  g.init<G>(a.seed, rep, t,
            reinterpret_cast<unsigned*>(reinterpret_cast<unsigned char*>(&sh) + a.spec_off_warps +
                                        (size_t)s * a.warp_smem + a.off_draws), gl);
  unsigned err = 0;
  const bool density = rd.field_kind == 2;
  int ind0 = 0, indf = 0, m = 0, gstage = 0, gtab = 0;  // chains are limited to 2e9 beads
  bool empty = !live;
  const int Hs = 1 << a.logH;
  const bool pool = a.pool_on != 0;
  // FP64: the sines and the rows of M on lanes of the warp (row gl here, from the
  // column gl on)
  constexpr bool kRows = sizeof(Pos) == 8 && G == 32;
  double row[4] = {1.0, 0.0, 0.0, 0.0};
  Real M[3][4];
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 4; j++) M[i][j] = i == j ? (Real)1 : (Real)0;
  if (live) {
    if (kind == CG_CRANK_SHAFT) {
      Real ang = (Real)c.amp_move * (uni<Real>(g.next()) - (Real)0.5);
      const unsigned xb0 = g.next();
      long long b0 = sizeof(Real) == 4 ? scaled_index(xb0, N) : (long long)(int)(unif(xb0) * (double)N);
      long long b1 = from_point(g, c.amp_bead, N, b0, err);
      if (b1 < 1) b1 = 1;
      segment_of(b0, b1, N, ind0, indf);
      long long ia, ib;
      if (ind0 == indf - 1 && ind0 == 0) { ia = indf; ib = ind0; }
      else if (ind0 == indf - 1 && ind0 == N - 1) { ia = ind0; ib = ind0 - 1; }
      else if (ind0 == 0 && indf == N) { ia = indf - 1; ib = ind0; }
      else if (ind0 == 0) { ia = indf; ib = ind0; }
      else if (indf == N) { ia = indf - 1; ib = ind0 - 1; }
      else { ia = indf; ib = ind0 - 1; }
      if (!err) {
        Real pa[3], pb[3], dir[3], p[3];
        long long ip;  // the fulcrum bead, loaded with the two axis beads
        if (ind0 == 0 && indf != N) ip = indf;
        else if (ind0 != 0 && indf == N) ip = ind0 - 1;
        else if (ind0 == 0 && indf == N) ip = ind0;
        else ip = ind0 - 1;
        ld3(r4, ia, pa); ld3(r4, ib, pb); ld3(r4, ip, p);
        for (int i = 0; i < 3; i++) dir[i] = pa[i] - pb[i];
        Real mag = rsqrt_(dir[0] * dir[0] + dir[1] * dir[1] + dir[2] * dir[2]);
        if (mag < (Real)1E-5) sphere<Real>(g, dir);
        else { Real sc = (Real)1 / mag; for (int i = 0; i < 3; i++) dir[i] = dir[i] * sc; }
        if constexpr (kRows) {
          double sn, cs;
          sincos(ang, &sn, &cs);
          rotation_row(dir, p, sn, cs, gl < 3 ? gl : 0, row);
        } else {
          axis_rotation(dir, p, ang, M);
        }
      }
    } else if (kind == CG_END_PIVOT) {
      Real ang = (Real)c.amp_move * (uni<Real>(g.next()) - (Real)0.5);
      long long lhs = g.next() & 1u;
      if (lhs == 1) { ind0 = 0; indf = (int)from_left(g, c.amp_bead, N, err) + 1; }
      else { ind0 = (int)(N - from_left(g, c.amp_bead, N, err)); indf = (int)N; }
      Real axis[3], p[3];
      double sn, cs;
      if constexpr (kRows) {
        const unsigned xa = g.next(), xb = g.next();
        sphere_and_angle(xa, xb, ang, axis, sn, cs);
      } else {
        sphere<Real>(g, axis);
      }
      long long ip;
      if (ind0 == 0 && indf != N) ip = indf;
      else if (ind0 != 0 && indf == N) ip = ind0 - 1;
      else if (ind0 == 0 && indf == N && lhs == 1) ip = indf - 1;
      else ip = ind0;
      if (!err) {
        ld3(r4, ip, p);
        if constexpr (kRows) rotation_row(axis, p, sn, cs, gl < 3 ? gl : 0, row);
        else axis_rotation(axis, p, ang, M);
      }
    } else {
      Real amp = (Real)c.amp_move * uni<Real>(g.next()), d[3];
      if constexpr (kRows) {
        const unsigned xa = g.next(), xb = g.next();
        double sn, cs;
        sphere_and_angle(xa, xb, 0.0, d, sn, cs);
        row[3] = (gl == 0 ? d[0] : gl == 1 ? d[1] : d[2]) * amp;
      } else {
        sphere<Real>(g, d);
        for (int i = 0; i < 3; i++) M[i][3] = d[i] * amp;
      }
      long long b0 = g.next() % (unsigned)N;
      long long b1 = from_point(g, c.amp_bead, N, b0, err);
      segment_of(b0, b1, N, ind0, indf);
    }
  }
  m = (!live || err) ? 0 : indf - ind0;
  if (live && !err && m == 0) empty = true;
  // the Metropolis draw, taken now: the plan holds all of the move's state from here
  unsigned xm = 0;
  if (live && !err && !empty) xm = g.next();
  if constexpr (sizeof(Pos) == 8) {  // the field sum's limbs
    __syncwarp();
    if (live && gl < CGX_LIMBS) move_limbs(a, sh, s)[gl] = 0;
  }
  if (m > a.stage_cap) gstage = 1;
  // voxel table: the CTA's pooled table for every move of up to
  // kPoolMaxBeads beads, optimistically (a pool past 3/4 load sends the move
  // to its global table); without the pool (a grid of 2^26 voxels and more)
  // the slot's own table when the move's at most 16 m voxels surely fit, or
  // optimistically up to m <= slots / 4 with the same fallback; global beyond
  bool sure = false, blk;
  const int most = kPoolMaxBeads >> ((rd.nx == 1) + (rd.ny == 1) + (rd.nz == 1));
  if (pool) {
    blk = density && m > 0 && m <= most;
    gtab = density && m > 0 && !blk;
  } else {
    sure = 16 * m <= Hs;
    gtab = (!sure && 4 * m > Hs) || m > most;
    blk = density && m > 0 && !gtab;  // moves with a shared table are deposited by the whole CTA
  }
  if (gl == 0 && live) {
    P.blk = blk ? 1 : 0;
    P.sure = sure ? 1 : 0;
    P.kind = kind;
    P.m = m;
    P.ind0 = ind0;
    P.indf = indf;
    P.empty = empty ? 1 : 0;
    P.err = (int)err;
    P.xm = xm;
    if (!LEAN) P.ndraw = (int)g.pos;
    P.gstage = gstage;
    P.gtab = gtab;
    P.oob = 0;
    P.derr = 0;
    P.cmask = 0;
    P.pq[0] = P.pq[1] = 0;
    P.ph[0] = P.ph[1] = 0;
    P.fq = P.fH = 0;
    P.fh = 0;
    P.fl0 = P.fl1 = 0;
    P.fl2 = 0;
    P.fn = P.freg = 0;
    if constexpr (!kRows) {
      Pos* Mp = reinterpret_cast<Pos*>(P.M);  // in the position type: no conversions
      for (int i = 0; i < 3; i++)
        for (int j = 0; j < 4; j++) Mp[4 * i + j] = M[i][j];
    }
  }
  if constexpr (kRows)
    if (gl < 3 && live) {
      double* Mp = reinterpret_cast<double*>(P.M) + 4 * gl;
      Mp[gl] = row[0];
      Mp[gl == 2 ? 0 : gl + 1] = row[1];
      Mp[gl == 0 ? 2 : gl - 1] = row[2];
      Mp[3] = row[3];
    }
}

// Earlier moves u of the batch whose written beads [ind0, indf) meet the beads
// a position move reads (its segment and both neighbours), added to its mask; a
// move with no beads (failed or empty) is never accepted, so it needs no
// exclusion.  Called by the whole warp.
template <int G>
__device__ __forceinline__ void bead_conflicts(SpecShared& sh, int s, int gl, bool live, int B) {
  MovePlan& P = sh.plan[s];
  const int m = live ? P.m : 0, ind0 = P.ind0, indf = P.indf;
  unsigned cmb = 0;
  #pragma unroll 1
  for (int u0 = 0; u0 < B; u0 += G) {
    const int u = u0 + gl;
    bool hit = false;
    if (m > 0 && u < s) {
      const MovePlan& U = sh.plan[u];
      hit = U.m > 0 && U.ind0 <= indf && ind0 <= U.indf;
    }
    cmb |= gballot<G>(hit) << u0;
  }
  if (gl == 0 && live && cmb) atomicOr(&P.cmask, cmb);
}

// The decision on a position move from the results in its plan.
template <typename Pos, int G, int LEAN>
__device__ __forceinline__ void decide_position(const KArgs& a, SpecShared& sh, int s, int gl, bool live) {
  using Acc = typename AccOf<Pos>::type;
  if (!live) return;
  MovePlan& P = sh.plan[s];
  Acc dEp = acc_zero<Acc>(), dEs = acc_zero<Acc>();
  double dEh = 0;
  long long dEH = 0;  // the exact 1e99 penalties, in kHugeUnit units
  unsigned err = (unsigned)P.err;
  int nvox = 0, regfail = 0;
  if (P.m > 0) {
    acc_add(dEp, load_acc<Acc>(P.pq[0], P.ph[0]));
    acc_add(dEp, load_acc<Acc>(P.pq[1], P.ph[1]));
    plan_field(P, move_limbs(a, sh, s), dEs, dEh);
    const int oo = P.oob;
    dEH = P.fH + (((long long)(oo >> 16) - (long long)(oo & 0xFFFF)) << 40);
    err |= P.derr & ~E_OVF;
    nvox = P.fn;
    regfail = P.freg;
  }
  bool dec = false;
  long long dq = 0;
  double dh = 0;
  if (!err && !P.empty) dec = decide(P.xm, dEp, dEs, with_huge(dEh, dEH), dq, dh);
  __syncwarp(group_mask<G>());  // every lane has read the plan
  if (gl == 0) {
    P.dq = dq;
    P.dE = dh;
    P.err = (int)err;
    P.regfail = regfail;
    P.dec = dec ? 1 : 0;
    P.nvox = nvox;
    if (!LEAN && a.mlog) log_terms(P, dEp, (unsigned long long)P.ndraw);
  }
}

// Evaluate tangent rotation or binding move t of the batch in slot s (group
// lanes gl = 0..G-1); `live` is false for the groups of a partly filled batch.
// Called by the whole warp.
template <typename Pos, int G, int LEAN>
__device__ void evaluate_move(const KArgs& a, SpecShared& sh, int rep, int s, int gl, bool live, int kind,
                              const cg_move_ctl& c, unsigned long long t, int* bkeys, unsigned* bmask) {
  using Real = Pos;
  using Acc = typename AccOf<Real>::type;
  const RepDev& rd = sh.ws.rd;
  const GridF& gf = sh.ws.gf;
  const WarpShared& ws = sh.ws;
  const long long N = rd.n_beads;
  const int hcol = a.hcol;  // stride of the voxel-table values
  const V4<Pos>* r4 = reinterpret_cast<const V4<Pos>*>(a.r4) + rd.bead_off;
  const unsigned* st = a.states + rd.bead_off;
  const unsigned* mk = a.marks + rd.bead_off;
  MovePlan& P = sh.plan[s];
  MoveRng g;
  if (!__any_sync(kFull, live)) return;
  g.init<G>(a.seed, rep, t,
            reinterpret_cast<unsigned*>(reinterpret_cast<unsigned char*>(&sh) + a.spec_off_warps +
                                        (size_t)s * a.warp_smem + a.off_draws), gl);
  unsigned err = 0;
  const bool check_field = rd.field_kind != 0 && kind != CG_TANGENT_ROTATION;
  const bool density = rd.field_kind == 2;
  int ind0 = 0, indf = 0, m = 0;  // chains are limited to 2e9 beads
  // dE = dEp (polymer) + dEs (field; fixed point for FP32 storage) + dEh (the
  // FP64 part: confinement penalties, and the whole field dE for FP64 storage)
  Acc dEp = acc_zero<Acc>(), dEs = acc_zero<Acc>();
  double dEh = 0;
  long long dEH = 0;  // the exact 1e99 penalties, in kHugeUnit units
  int nvox = 0;
  const bool empty = !live;
  unsigned xm = 0;  // the decision's draw
  int gtab = 0, gstage = 0, regfail = 0;
  const int Hs = 1 << a.logH;

  if (kind == CG_TANGENT_ROTATION) {
    Real ang = 0;
    long long n = 0;
    if (live) {
      ang = (Real)c.amp_move * (uni<Real>(g.next()) - (Real)0.5);
      n = (long long)(g.next() % (unsigned)c.amp_bead) + 1;
      if (n > N) err |= E_WINDOW;
    }
    m = (!live || err) ? 0 : (int)n;
    if (m > a.stage_cap) gstage = 1;
    const SlotScratch S = gstage ? global_slot<Pos>(a, rep, s) : shared_slot(a, sh, s);
    int* idx = S.idx;
    unsigned* picked = a.picked + a.picked_off[rep] + s * ((N + 31) / 32);
    // n distinct random beads, drawn in order with redraws (get_inds): G
    // candidates per round, the first fresh ones taken in draw order.  Beads
    // taken in a round that another round follows are marked in the slot's
    // bitmap, which later rounds consult (a move of fewer beads than G
    // usually needs one round and touches no bitmap).
    long long got = 0;
    int it = 0, rounds = 0;
    const unsigned lt = (1u << gl) - 1u;
    const unsigned gmask = G == 32 ? kFull : ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31u) & ~(unsigned)(G - 1));
    for (;;) {
      bool want = live && !err && got < m;
      if (want && ++it > kMaxIter) { err |= E_SPIN; want = false; }
      if (!__any_sync(kFull, want)) break;
      const unsigned x = g.word(g.pos + gl);
      const long long cand = want ? (long long)(x % (unsigned)N) : -1 - (long long)(threadIdx.x & 31u);
      const unsigned grp = __match_any_sync(kFull, cand) & gmask;
      const unsigned gshift = G == 32 ? 0u : ((threadIdx.x & 31u) & ~(unsigned)(G - 1));
      const bool first = ((grp >> gshift) & lt) == 0;
      const bool fresh = want && first && !(rounds > 0 && ((picked[cand >> 5] >> (cand & 31)) & 1u));
      const unsigned bal = gballot<G>(fresh);
      const long long need = m - got;
      const int cnt = __popc(bal);
      const int rank = __popc(bal & lt);
      if (fresh && rank < need) {
        idx[got + rank] = (int)cand;
        if (cnt < need) atomicOr(&picked[cand >> 5], 1u << (cand & 31));
      }
      if (want) {
        rounds++;
        long long consumed;
        if (cnt >= need) {
          unsigned b = bal;
          #pragma unroll 1
          for (long long q = 1; q < need; q++) b &= b - 1;
          consumed = __ffs((int)b);
          got = m;
        } else {
          consumed = G;
          got += cnt;
        }
        g.pos += consumed;
      }
      __syncwarp();
    }
    err = gor<G>(err);
    const long long marked = rounds > 1 ? got : 0;  // beads whose marks are cleared below
    if (err) m = 0;
    const unsigned long long axis_base = g.pos;
    V4<Pos>* stage = reinterpret_cast<V4<Pos>*>(S.stage);
    Acc part = acc_zero<Acc>();
    // FP64 without twist: the last rotations of up to 16 by four lanes a bead, 8 beads
    // a pass (~110 FP64 operations instead of ~300): the sines of the sphere's angles
    // and of the rotation, the rows of the rotation, and the two bonds' energies
    // before and after it, the bead's dE on the lane that a whole pass has it on
    // (1,000 beads, 300 moves, kernel only, with block_deposit's bonds: 5.07 -> 4.66
    // ms).  Three such passes take longer than one of 32 beads (80 rotations of up
    // to 100 beads: 4.51 ms by such passes alone, 3.29 by whole ones, 3.17 mixed).
    constexpr bool kQuads = sizeof(Pos) == 8 && G == 32;
    int whole = m;
    if (kQuads && (LEAN || !rd.twist) && (m & 31) <= 16) whole = m & ~31;
    if (whole > 0) {
      Real sa, ca;
      rsincos(ang, &sa, &ca);
      #pragma unroll 1
      for (long long k = gl; k < whole; k += G) {
        const unsigned xa = g.word(axis_base + 2 * k), xb = g.word(axis_base + 2 * k + 1);
        Real tt3[3], tt2[3];
        const Acc de = rotate_tangent<Pos, LEAN>(a, rd, idx[k], xa, xb, sa, ca, tt3, tt2);
        stage[3 * k + 1] = V4<Pos>{(Pos)tt3[0], (Pos)tt3[1], (Pos)tt3[2], (Pos)0};
        stage[3 * k + 2] = V4<Pos>{(Pos)tt2[0], (Pos)tt2[1], (Pos)tt2[2], (Pos)0};
        acc_add(part, de);
      }
    }
    if constexpr (kQuads) {
      #pragma unroll 1
      for (int k0 = whole; k0 < m; k0 += 8) {
        const int lane = gl, quad = lane & 28, ax = lane & 3, j = ax < 3 ? ax : 2;
        const bool on = k0 + (lane >> 2) < m;
        const int k = on ? k0 + (lane >> 2) : 0;
        const long long i = idx[k], in = ax & 2 ? i + 1 : i - 1;
        const unsigned xa = g.word(axis_base + 2 * k), xb = g.word(axis_base + 2 * k + 1);
        const double u = uni<double>(ax == 0 ? xa : xb);
        const double phi = u * (2.0 * 3.141592653589793), theta = acos(u * 2 - 1);
        double sn, cs;
        sincos(ax == 0 ? phi : ax == 1 ? theta : (double)ang, &sn, &cs);
        const double st1 = __shfl_sync(kFull, sn, quad + 1);
        const double axis[3] = {__shfl_sync(kFull, cs, quad) * st1, __shfl_sync(kFull, sn, quad) * st1,
                                __shfl_sync(kFull, cs, quad + 1)};
        const double none[3] = {0, 0, 0};
        double R[4], r[3], t3[3], t2[3];
        rotation_row(axis, none, __shfl_sync(kFull, sn, quad + 2), __shfl_sync(kFull, cs, quad + 2), j, R);
        const double m0 = j == 0 ? R[0] : j == 1 ? R[2] : R[1], m1 = j == 0 ? R[1] : j == 1 ? R[0] : R[2],
                     m2 = j == 0 ? R[2] : j == 1 ? R[1] : R[0];
        const V4<double>* q4 = reinterpret_cast<const V4<double>*>(a.t34) + rd.bead_off;
        ld3(reinterpret_cast<const V4<double>*>(r4), i, r);
        ld3(q4, i, t3);
        ld3(reinterpret_cast<const V4<double>*>(a.t24) + rd.bead_off, i, t2);
        const double tt3 = m0 * t3[0] + m1 * t3[1] + m2 * t3[2], tt2 = m0 * t2[0] + m1 * t2[1] + m2 * t2[2];
        if (on) {
          double* q = reinterpret_cast<double*>(stage + 3 * k);
          q[4 + ax] = ax < 3 ? tt3 : 0.0;
          q[8 + ax] = ax < 3 ? tt2 : 0.0;
        }
        double mine[3];  // the bead's tangent, before (even lanes) or after
        for (int q = 0; q < 3; q++) {
          const double moved = __shfl_sync(kFull, tt3, quad + q);
          mine[q] = ax & 1 ? moved : t3[q];
        }
        double e = 0.0;
        if (in >= 0 && in < N) {
          const bool left = !(ax & 2);
          double rn[3], tn[3], ra[3], rb[3], ta[3], tb[3];
          ld3(reinterpret_cast<const V4<double>*>(r4), in, rn);
          ld3(q4, in, tn);
          for (int q = 0; q < 3; q++) {
            ra[q] = left ? rn[q] : r[q];
            rb[q] = left ? r[q] : rn[q];
            ta[q] = left ? tn[q] : mine[q];
            tb[q] = left ? mine[q] : tn[q];
          }
          e = bond_e(load_bond<double>(a.bonds + rd.bead_off * 6, left ? in : i), ra, rb, ta, tb);
        }
        const double d = __shfl_xor_sync(kFull, e, 1) - e;          // lanes 0 and 2 of four
        const double de = d + __shfl_down_sync(kFull, d, 2);        // lane 0
        const double of = __shfl_sync(kFull, de, 4 * (lane & 7));   // bead k0 + (lane & 7)
        if ((lane >> 3) == ((k0 >> 3) & 3) && k0 + (lane & 7) < m) acc_add(part, of);
      }
    }
    g.pos = axis_base + 2 * (unsigned long long)m;
    dEp = gsum<G>(part);
    // the picked marks only serve the redraws of this move
    #pragma unroll 1
    for (long long k = gl; k < marked; k += G) {
      int i = idx[k];
      atomicAnd(&picked[i >> 5], ~(1u << (i & 31)));
    }
    __syncwarp();
    if (m > 0) {
      ind0 = idx[0];
      indf = ind0 + 1;
    }
  } else {
    int bsel = 0;
    if (live) {
      bsel = (int)(g.next() % (unsigned)rd.nb);
      long long b0 = g.next() % (unsigned)N;
      long long b1 = from_point(g, c.amp_bead, N, b0, err);
      if (!err) segment_of(b0, b1, N, ind0, indf);
    }
    m = (!live || err) ? 0 : indf - ind0;
    if constexpr (sizeof(Pos) == 8) {  // the decision's draw, then the field sum's limbs in the buffer
      if (live) xm = g.word(g.pos);
      __syncwarp();
      if (live && gl < CGX_LIMBS) move_limbs(a, sh, s)[gl] = 0;
      if (live && gl == 0) P.fh = 0;
      __syncwarp();
    }
    const int nt = rd.sites[bsel];
    if (m > a.stage_cap) gstage = 1;
    if (8 * m > Hs) gtab = 1;
    const SlotScratch S = gtab ? global_slot<Pos>(a, rep, s) : shared_slot(a, sh, s);
    int* nused = &sh.nused[s];
    int* idx = gstage ? global_slot<Pos>(a, rep, s).idx : shared_slot(a, sh, s).idx;
    Acc part = acc_zero<Acc>();
    int dbl = 0;
    // eight lanes per bead, one trilinear corner each: corner lane 0 takes
    // the binding free energy, each lane the change of its corner's binder
    // column
    constexpr int BP = G / 8;
    const int kc = gl >> 3, cl = gl & 7;
    #pragma unroll 1
    for (long long kb = 0; __any_sync(kFull, kb < m); kb += BP) {
      const long long k = kb + kc;
      int vq[1] = {0};
      bool want[1] = {false};
      long long q = 0;
      if (k < m) {
        const long long i = ind0 + k;
        bool ok;
        int s_new = g.state_at(g.bpos + k, nt, ok);
        unsigned sw = st[i], mw = mk[i];
        int s_old = (int)((sw >> (8 * bsel)) & 0xFF);
        if (cl == 0) {
          acc_add(part, bead_bind_dE(ws, sw, mw, bsel, s_new, (Real)0));
          dbl += (s_new == 2 ? 1 : 0) - (s_old == 2 ? 1 : 0);
          idx[k] = s_new;
        }
        if (density && s_new != s_old) {
          Real p[3], wl[3], w;
          int lo[3], hi[3];
          ld3(r4, i, p);
          move_axes<LEAN == 1>(rd, gf, p, wl, lo, hi);
          voxel_corner(gf, wl, lo, hi, cl, w, vq[0]);
          q = q40(w) * (long long)(s_new - s_old);
          want[0] = true;
        }
      }
      if (density) {
        int slot[1];
        claim_slots<1>(S.keys, S.used, nused, S.logH, vq, want, slot, err, 1 << S.logH, E_SPIN);
        if (want[0] && slot[0] >= 0) add_delta(S.vals, hcol, slot[0], 1 + bsel, q, !gtab);
      }
    }
    g.bpos += (unsigned long long)m;
    err = gor<G>(err);
    dEp = gsum<G>(part);
    const int ddb = gsum<G>(dbl);
    if (check_field && rd.field_kind == 1 && rd.confine_kind == 2) {
      int oob = 0;
      #pragma unroll 1
      for (long long k = gl; k < m; k += G) {
        double p[3];
        ld3(r4, ind0 + k, p);
        oob += out_of_bounds(rd, p, true);
      }
      dEH += (long long)gsum<G>(oob) << 40;
    }
    __syncwarp();
    if (density) {
      long long nv = 0;
      own_field<G>(a, sh, s, S, *nused, gl, !gtab, nv, dEs, dEH);
      if constexpr (sizeof(Pos) == 8) plan_field(P, move_limbs(a, sh, s), dEs, dEh);
      nvox = (int)nv;
      if (m > 0) add_intra(ws, bsel, ddb, dEs, dEh);
    }
    if (gl == 0 && live) P.bsel = bsel;
    // register the touched voxels for the conflict test
    if (density) {
      const int nu = (live && !err) ? *nused : 0;
      #pragma unroll 1
      for (int i = gl; i < nu; i += G) {
        const int b = block_insert(bkeys, a.spec_logHB, S.keys[S.used[i]]);
        S.bslot[i] = b;
        if (b < 0) regfail = 1;
        else atomicOr(&bmask[b], 1u << s);
      }
      regfail = (int)gor<G>((unsigned)regfail);
    }
  }
  err = gor<G>(err);
  bool dec = false;
  long long dq = 0;
  double dh = 0;
  if (live && !err && !empty) {
    const bool taken = sizeof(Pos) == 8 && kind != CG_TANGENT_ROTATION;
    if (taken) g.pos++;
    else xm = g.next();
    dec = decide(xm, dEp, dEs, with_huge(dEh, dEH), dq, dh);
  }
  if (gl == 0 && live) {
    P.dq = dq;
    P.dE = dh;
    P.kind = kind; P.m = (int)m; P.ind0 = (int)ind0; P.indf = (int)indf;
    P.empty = empty ? 1 : 0; P.err = (int)err; P.regfail = regfail; P.dec = dec ? 1 : 0;
    P.nvox = (int)nvox; P.gtab = gtab; P.gstage = gstage;
    if (!LEAN && a.mlog) log_terms(P, dEp, g.pos);
  }
}

// Bits of earlier moves of the batch (u < s) whose footprint meets move s's.
template <typename Pos, int G>
__device__ void conflict_mask(const KArgs& a, SpecShared& sh, unsigned char* smem, int rep, int s, int gl,
                              bool live, int kind, int B, const unsigned* bmask) {
  MovePlan& P = sh.plan[s];
  const RepDev& rd = sh.ws.rd;
  const bool act = live && !P.err && !P.empty;
  unsigned cm = 0;
  if (rd.field_kind == 2 && kind != CG_TANGENT_ROTATION) {
    const int nu = act ? sh.nused[s] : 0;
    const int* bs = (P.gtab ? global_slot<Pos>(a, rep, s) : shared_slot(a, sh, s)).bslot;
    #pragma unroll 1
    for (int i = gl; i < nu; i += G) {
      int b = bs[i];
      if (b >= 0) cm |= bmask[b];
    }
    cm = gor<G>(cm);
  }
  cm &= (1u << s) - 1u;
  if (kind == CG_TANGENT_ROTATION) {
    // rotated beads of u against those of s and their neighbours
    const int* lw = (P.gstage ? global_slot<Pos>(a, rep, s) : shared_slot(a, sh, s)).idx;
    #pragma unroll 1
    for (int u = 0; u < B; u++) {
      const MovePlan& U = sh.plan[u];
      int hit = 0;
      if (act && u < s && !U.err && !U.empty) {
        const int* lu = U.gstage ? a.g_idx + ((long long)rep * a.spec_s + u) * a.g_stage_cap
                                 : reinterpret_cast<const int*>(smem + a.spec_off_warps +
                                                                (size_t)u * a.warp_smem + a.off_idx);
        #pragma unroll 1
        for (int k = gl; k < P.m && !hit; k += G) {
          int j = lw[k];
          #pragma unroll 1
          for (int q = 0; q < U.m; q++) {
            int d = lu[q] - j;
            if (d >= -1 && d <= 1) { hit = 1; break; }
          }
        }
      }
      if (gany<G>(hit)) cm |= 1u << u;
    }
  } else {
    // lane gl takes the earlier moves u = u0 + gl: beads written by u,
    // [ind0, indf), against the beads read by s -- the segment and, for
    // position moves, its two neighbours
    #pragma unroll 1
    for (int u0 = 0; u0 < B; u0 += G) {
      const int u = u0 + gl;
      bool hit = false;
      if (act && u < s) {
        const MovePlan& U = sh.plan[u];
        if (!U.err && !U.empty) {
          const long long wlo = U.ind0, whi = (long long)U.indf - 1;
          const long long rlo = P.kind == CG_CHANGE_BINDING_STATE ? P.ind0 : (long long)P.ind0 - 1;
          const long long rhi = P.kind == CG_CHANGE_BINDING_STATE ? (long long)P.indf - 1 : (long long)P.indf;
          hit = wlo <= rhi && rlo <= whi;
        }
      }
      cm |= gballot<G>(hit) << u0;
    }
  }
  if (gl == 0 && live) P.cmask = cm;
}

// SimpleControl.update_amplitudes (chromo/mc/mc_controller.py:126-189)
__device__ __forceinline__ void update_amplitudes(cg_move_ctl& c) {
  if (c.ctrl_kind != 1) return;
  double acc = c.acc_rate;
  if (acc < 0.5) {
    double prop = c.amp_move * 0.95;
    if (prop > c.move_lo) c.amp_move = prop;
    else {
      c.amp_move = c.move_hi;
      double nb = (double)(c.amp_bead - 1);
      c.amp_bead = (long long)(c.bead_lo > nb ? c.bead_lo : nb);
    }
  } else if (acc > 0.5) {
    double prop = c.amp_move / 0.95;
    if (prop < c.move_hi) c.amp_move = prop;
    else {
      c.amp_move = c.move_lo;
      double nb = (double)(c.amp_bead + 1);
      c.amp_bead = (long long)(c.bead_hi < nb ? c.bead_hi : nb);
    }
  }
}

template <typename Pos, int G>
__device__ void commit_and_clear(const KArgs& a, SpecShared& sh, int rep, int s, int gl, bool accept, int* bkeys,
                                 unsigned* bmask) {
  const MovePlan& P = sh.plan[s];
  const RepDev& rd = sh.ws.rd;
  const int ncol = a.ncol, hcol = a.hcol;
  V4<Pos>* r4w = reinterpret_cast<V4<Pos>*>(a.r4) + rd.bead_off;
  V4<Pos>* t34w = reinterpret_cast<V4<Pos>*>(a.t34) + rd.bead_off;
  V4<Pos>* t24w = reinterpret_cast<V4<Pos>*>(a.t24) + rd.bead_off;
  unsigned* st = a.states + rd.bead_off;
  const int m = P.m;
  if (accept) {
    const SlotScratch S = P.gstage ? global_slot<Pos>(a, rep, s) : shared_slot(a, sh, s);
    const V4<Pos>* stage = reinterpret_cast<const V4<Pos>*>(S.stage);
    const int* idx = S.idx;
    if (P.kind <= CG_SLIDE) {
      #pragma unroll 1
      for (int k = gl; k < m; k += G) {
        const long long i = (long long)P.ind0 + k;
        r4w[i] = stage[3 * k];
        if (P.kind != CG_SLIDE) {
          t34w[i] = stage[3 * k + 1];
          t24w[i] = stage[3 * k + 2];
        }
      }
    } else if (P.kind == CG_TANGENT_ROTATION) {
      #pragma unroll 1
      for (int k = gl; k < m; k += G) {
        const long long i = idx[k];
        t34w[i] = stage[3 * k + 1];
        t24w[i] = stage[3 * k + 2];
      }
    } else {
      #pragma unroll 1
      for (int k = gl; k < m; k += G) {
        const long long i = (long long)P.ind0 + k;
        unsigned sw = st[i];
        sw = (sw & ~(0xFFu << (8 * P.bsel))) | ((unsigned)idx[k] << (8 * P.bsel));
        st[i] = sw;
      }
    }
  }
  const int nu = sh.nused[s];
  if (nu == 0) return;  // no table of its own
  const SlotScratch T = P.gtab ? global_slot<Pos>(a, rep, s) : shared_slot(a, sh, s);
  int *keys = T.keys, *used = T.used, *bslot = T.bslot;
  long long* vals = T.vals;
  long long* grid = a.grid + rd.vox_off * ncol;
  #pragma unroll 1
  for (int i = gl; i < nu; i += G) {
    int slot = used[i];
    if (accept) {  // the voxel's post-move row, stored with 16-byte stores (padding column stays 0)
      const int v = keys[slot];
      const long long* src = vals + (long long)slot * hcol;
      longlong2* dst = reinterpret_cast<longlong2*>(grid + (long long)v * ncol);
      dst[0] = make_longlong2(src[0], src[1]);
      if (ncol == 4) dst[1] = make_longlong2(hcol > 2 ? src[2] : 0, hcol > 3 ? src[3] : 0);
    }
    keys[slot] = -1;
    #pragma unroll 1
    for (int cc = 0; cc < hcol; cc++) vals[(long long)slot * hcol + cc] = 0;
    int b = bslot[i];
    if (b >= 0) { bkeys[b] = -1; bmask[b] = 0u; }
    bslot[i] = -1;
  }
}

// Moves in flight for the next cycle of a position move: a batch of B costs
// about kBatchFixed + B (its phases' latencies, in units of one more move) and
// stands up to the first move that meets an earlier accepted one.  With p the
// chance of that per pair of moves, as the batches so far met it, E(B) = sum_k
// prod_(j<k) (1 - j p) moves of the batch are expected to stand; the B with the
// least (kBatchFixed + B) / E(B) is taken.  The outcome does not depend on it.
// (128 confined chains of 3,000 beads, of whose 12 moves in flight 4.7 stood: 4.84
// -> 4.16 ms; kBatchFixed of 10, 20 and 40 measured within 1 %.)
constexpr float kBatchFixed = 20.0f;
__device__ __forceinline__ int batch_limit(float met, float pairs, int most) {
  const float p = pairs > 0.0f ? met / pairs : 0.0f;
  float stand = 1.0f, E = 0.0f, best_e = 0.0f, best_c = 1.0f;
  int best = 1;
#pragma unroll 1
  for (int B = 1; B <= most; B++) {
    E += stand;
    const float c = kBatchFixed + (float)B;
    if (c * best_e < best_c * E) {
      best = B;
      best_e = E;
      best_c = c;
    }
    stand = fmaxf(0.0f, stand * (1.0f - (float)B * p));
  }
  return best;
}

// FP32 storage: 128 registers, 16 warps per SM, in CTAs of more warps than
// moves in flight (the block-wide phases use them all).  At 168 registers and 12
// warps: 256 chains, 20 MC steps, kernel only, 10.3 against 9.95 ms, one
// 10,000-bead chain, 10 steps, 2.40 against 2.23.  FP64 storage: 168 registers.
// LEAN (the host picks it per launch, a.lean): 1, the instantiation for launches with
// no SSTWLC or fast_field replica and no move log, whose code for those is left out; 2,
// the same with fast_field; 0, any launch.  The full form's spills cost fast_field
// replicas ~10 % (one 1,000-bead chain, 80 moves: rotations of up to 60 beads 373 us in
// form 2, 410 in form 0; binding moves 93 and 103; cranks of up to 30 beads 147 and 164).
template <typename Pos, int G, int LEAN>
__global__ void __maxnreg__(sizeof(Pos) == 4 ? 128 : 168) spec_kernel(KArgs a) {
  extern __shared__ __align__(32) unsigned char smem[];
  constexpr int GPW = 32 / G;  // move groups per warp
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gl = lane & (G - 1);
  const int slot = warp * GPW + lane / G;
  const int Sn = a.spec_s;
  const int rep = blockIdx.x;
  if (rep >= a.n_reps) return;
  SpecShared& sh = *reinterpret_cast<SpecShared*>(smem);
  int* bkeys = reinterpret_cast<int*>(smem + a.spec_off_bkeys);
  unsigned* bmask = reinterpret_cast<unsigned*>(smem + a.spec_off_bmask);
  const int HB = 1 << a.spec_logHB;
  const int hcol = a.hcol;
  {
    const unsigned* src = reinterpret_cast<const unsigned*>(a.reps + rep);
    unsigned* dst = reinterpret_cast<unsigned*>(&sh.ws.rd);
    for (int i = tid; i < (int)(sizeof(RepDev) / 4); i += blockDim.x) dst[i] = src[i];
    const unsigned* cs = reinterpret_cast<const unsigned*>(a.ctl + (long long)rep * 5);
    unsigned* cd = reinterpret_cast<unsigned*>(sh.ws.ctl);
    for (int i = tid; i < (int)(5 * sizeof(cg_move_ctl) / 4); i += blockDim.x) cd[i] = cs[i];
    for (int i = tid; i < HB; i += blockDim.x) { bkeys[i] = -1; bmask[i] = 0u; }
    for (int i = tid; i < 30; i += blockDim.x) sh.ws.tally[i] = 0;
    if (slot < Sn) {
      const SlotScratch sm = shared_slot(a, sh, slot);
      for (int i = gl; i < (1 << a.logH); i += G) { sm.keys[i] = -1; sm.bslot[i] = -1; }
      for (int i = gl; i < (1 << a.logH) * hcol; i += G) sm.vals[i] = 0;
      if (gl == 0) sh.nused[slot] = 0;
    }
    if (a.pool_on) {
      int* pk = reinterpret_cast<int*>(smem + a.off_pkeys);
      long long* pv = reinterpret_cast<long long*>(smem + a.off_pvals);
      for (int i = tid; i < (1 << a.pool_logH); i += blockDim.x) pk[i] = -1;
      for (int i = tid; i < (1 << a.pool_logH) * hcol; i += blockDim.x) pv[i] = 0;
    }
  }
  __syncthreads();
  // the constants: the lean FP32 form by the warps' first threads (kernel only, 256
  // chains of 2,000-20,000 beads, 20 steps: 9.27 -> 9.18 ms, one 10,000-bead chain
  // 2.04 -> 2.02); in the other forms the call cost the main loop registers (FP64 and
  // SSTWLC chains 0.9 % slower), and one thread takes them
  constexpr bool kSpreadSetup = sizeof(Pos) == 4 && LEAN;
  if (kSpreadSetup && lane == 0)
    #pragma unroll 1
    for (int part = warp; part < kSetupParts; part += (int)(blockDim.x >> 5)) setup_part(sh.ws, part);
  if (tid == 0) {
    const RepDev& rd0 = sh.ws.rd;
    if (!kSpreadSetup)
#pragma unroll
      for (int part = 0; part < kSetupParts; part++) setup_body(sh.ws, part);
    sh.t0 = sh.start[0] = rd0.draw_pos;
    sh.tlog = rd0.draw_pos;
    sh.run_dE = rd0.run_dE;
    sh.run_q = 0;
    for (int k = 0; k < 3; k++) {
      sh.met[k] = sh.pairs[k] = 0.0f;
      sh.limit[k] = Sn;
    }
    sh.stop = 0;
    sh.npool = 0;
    const float n = (float)rd0.n_beads;
    sh.short_amp = !LEAN && rd0.twist ? (int)fminf(32.0f, 4.0f * sqrtf(n))
                                          : (int)fminf(fminf(32.0f, sqrtf(5.4f * sqrtf(n * (float)Sn))),
                                                       16.0f + n * (float)Sn * (1.0f / 4000.0f));
  }
  __syncthreads();

  for (long long step = 0; step < a.n_steps; step++) {
    for (int ci = 0; ci < a.n_ctl; ci++) {
      cg_move_ctl& c = sh.ws.ctl[ci];
      const int kind = (int)c.move_kind;
      if (c.move_on == 1) {
        // the moves left come from the move counter, in shared memory: loop
        // counters held in registers over the phases were spilled in them (144 bytes
        // loaded per thread; kernel only, 256 chains of 2,000-20,000 beads, 20 steps:
        // 9.50 -> 9.28 ms, 128 confined chains 3.93 -> 3.72, one 10,000-bead chain
        // 2.11 -> 2.03)
        for (;;) {
          const long long rest = c.num_per_cycle - (long long)(sh.t0 - sh.start[(((int)step & a.n_ctl) ^ ci) & 1]);
          if (rest <= 0) break;
          // short tangent rotations: groups of 8 or 16 lanes, and as many moves
          // in flight as are likely to stand (a later move meets the ~3/2 (amp + 1)
          // beads of each earlier accepted one with probability ~3/8 (amp + 1)^2 / N)
          constexpr bool kShort = G == 32 && sizeof(Pos) == 4;
          const bool brief = kShort && kind == CG_TANGENT_ROTATION && c.amp_bead >= 1 && c.amp_bead <= sh.short_amp;
          const int gs = c.amp_bead <= 8 ? 8 : 16, cap = c.amp_bead <= 16 ? 16 : 32;  // of a short rotation
          int most = kind <= CG_SLIDE ? sh.limit[kind] : Sn;
          if (brief) {
            const int room = min(min(kMaxS, Sn * (64 / cap)), (int)blockDim.x / gs);
            const int likely = (int)(kShortSpan * sqrtf((float)sh.ws.rd.n_beads) / (float)(c.amp_bead + 1));
            most = min(room, max(Sn, likely));
          }
          const int B = (int)(rest < most ? rest : most);
          const bool wlive = warp * GPW < B;  // the warp has a move of this batch
          const bool live = slot < B;
          if constexpr (kShort) {
            if (brief) {
              const ShortTangent T(a, sh, gs, cap);
              short_tangent_evaluate<LEAN>(a, sh, rep, T, B, c, bkeys, bmask);
              __syncthreads();
              if (!LEAN && sh.ws.rd.twist) short_tangent_twist(a, sh, B, cap);
              short_tangent_conflicts(a, sh, T, B, bkeys, bmask);
              __syncthreads();
            }
          }
          if (kind <= CG_SLIDE) {
            if (tid == 0) sh.npool = 0;  // every reader of the last batch's pool passed a barrier since
            propose_position<Pos, G, LEAN>(a, sh, rep, slot, gl, live, kind, c, sh.t0 + (unsigned long long)slot);
            __syncthreads();
            block_deposit<Pos, LEAN>(a, sh, rep, B, kind);
            bead_conflicts<G>(sh, slot, gl, live, B);
            __syncthreads();
            const bool pool = a.pool_on != 0, density = sh.ws.rd.field_kind == 2;
            if (pool && density) block_field_pool<Pos>(a, sh, smem, bkeys, bmask);
            {
              const MovePlan& P = sh.plan[slot];
              const bool own = live && P.m > 0 && (!P.blk || !pool || (P.derr & E_OVF));
              if (__any_sync(kFull, own)) own_path<Pos, G, LEAN>(a, sh, rep, slot, gl, own, kind, bkeys, bmask);
            }
            if (pool && density) __syncthreads();  // the pooled field pass is complete
            decide_position<Pos, G, LEAN>(a, sh, slot, gl, live);
            __syncthreads();
          } else if (!brief) {
            evaluate_move<Pos, G, LEAN>(a, sh, rep, slot, gl, live, kind, c, sh.t0 + (unsigned long long)slot, bkeys,
                                        bmask);
            __syncthreads();
            if (wlive) conflict_mask<Pos, G>(a, sh, smem, rep, slot, gl, live, kind, B, bmask);
            __syncthreads();
          }
          // Resolve, computed by every warp from the plans (lane u reads move u):
          // the batch stands up to the first move that failed or meets an
          // earlier accepted move (everything before it stands, so "earlier
          // accepted" is the accepted moves below it), or up to and including
          // the first move whose voxels could not be registered.
          const bool valid = lane < B;
          const MovePlan& Pl = sh.plan[valid ? lane : 0];
          const bool p_err = valid && Pl.err != 0;
          const unsigned D = __ballot_sync(kFull, valid && !Pl.empty && Pl.dec);
          const unsigned F = __ballot_sync(kFull, p_err || (valid && (Pl.cmask & D & ((1u << lane) - 1u))));
          const unsigned RF = __ballot_sync(kFull, valid && Pl.regfail);
          const int first_fail = F ? __ffs((int)F) - 1 : B;
          int cut = first_fail;
          if (RF && __ffs((int)RF) < cut) cut = __ffs((int)RF);
          const unsigned acc = cut >= 32 ? D : (D & ((1u << cut) - 1u));
          // bookkeeping of the standing moves by the last two warps (which, with
          // more warps than moves in flight, have no move to commit): one the
          // acceptance rate, an FP64 chain in move order, the other the sums
          const int last = (int)(blockDim.x >> 5) - 1;
          if (warp == last) {
            const unsigned empties = __ballot_sync(kFull, lane < cut && Pl.empty);
            if (lane == 0) {
              c.num_attempt += cut;
              c.num_success += __popc(acc);
              // acc = alpha * x + (1 - alpha) * acc with x in {0, 1}: one FP64
              // multiply a move, and an add of alpha where it was accepted
              double rate = c.acc_rate;
              const double alpha = c.alpha, beta = 1 - c.alpha;
#pragma unroll 1
              for (int w = 0; w < cut; w++) {
                if (!LEAN && a.mlog) log_move(a, rep, sh.t0 + (unsigned long long)w - sh.tlog, sh.plan[w]);
                if ((empties >> w) & 1u) continue;
                rate = beta * rate;
                if ((D >> w) & 1u) rate = alpha + rate;
              }
              c.acc_rate = rate;
              if (kind <= CG_SLIDE) {
                const bool met = first_fail < B;
                sh.met[kind] = 0.9f * sh.met[kind] + (met ? 1.0f : 0.0f);
                sh.pairs[kind] = 0.9f * sh.pairs[kind] + (float)(cut * (cut - 1) / 2 + (met ? cut : 0));
              }
              sh.t0 += (unsigned long long)cut;
              if (cut == first_fail && first_fail < B && sh.plan[first_fail].err) sh.stop = sh.plan[first_fail].err;
              // every batch attempts at least one move or stops the run; a loop
              // that did not would end with an error status instead of spinning
              else if (cut == 0) sh.stop = E_SPIN;
            }
          }
          if (warp == (last > 0 ? last - 1 : 0)) {
            const bool stand = lane < cut;
            const bool took = (acc >> lane) & 1u;
            const unsigned sm_m = __reduce_add_sync(kFull, stand ? (unsigned)Pl.m : 0u);
            const unsigned sm_v = __reduce_add_sync(kFull, stand ? (unsigned)Pl.nvox : 0u);
            const unsigned ac_m = __reduce_add_sync(kFull, took ? (unsigned)Pl.m : 0u);
            const unsigned ac_v = __reduce_add_sync(kFull, took ? (unsigned)Pl.nvox : 0u);
            // running sum of accepted dE, penalised moves left out: the
            // fixed-point parts exactly (32-bit reductions of 16-bit pieces of
            // the two's complement), moves with an FP64 part one by one
            const unsigned hards = __ballot_sync(kFull, took && !is_zero64(Pl.dE));
            if constexpr (sizeof(Pos) == 4) {
              const unsigned long long q = took && !((hards >> lane) & 1u) ? (unsigned long long)Pl.dq : 0ull;
              unsigned long long sum = 0;
#pragma unroll
              for (int k = 0; k < 4; k++)
                sum += (unsigned long long)__reduce_add_sync(kFull, (unsigned)(q >> (16 * k)) & 0xFFFFu) << (16 * k);
              if (lane == 0) {
                sh.run_q += (long long)sum;
                if (sh.run_q > (1LL << 61) || sh.run_q < -(1LL << 61)) {  // far from the int64 range
                  sh.run_dE += (double)sh.run_q * kFxEInv;
                  sh.run_q = 0;
                }
              }
            }
            if (lane == 0) {
              unsigned long long* t = sh.ws.tally + kind * 6;
              t[0] += (unsigned long long)cut;
              t[1] += (unsigned long long)__popc(acc);
              t[2] += sm_m;
              t[3] += sm_v;
              t[4] += ac_m;
              t[5] += ac_v;
#pragma unroll 1
              for (unsigned left = hards; left; left &= left - 1) {
                const MovePlan& P = sh.plan[__ffs((int)left) - 1];
                const double dE = dE_value(P.dq, P.dE);
                if (soft_dE(dE)) sh.run_dE += dE;
              }
            }
          }
          if constexpr (kShort)
            if (brief) short_tangent_commit(a, sh, ShortTangent(a, sh, gs, cap), cut, acc, bkeys, bmask);
          if (!brief) {
            if (wlive && live)
              commit_and_clear<Pos, G>(a, sh, rep, slot, gl, slot < cut && ((acc >> slot) & 1u), bkeys, bmask);
            __syncwarp();
            if (live && gl == 0) sh.nused[slot] = 0;
          }
          if (kind <= CG_SLIDE && a.pool_on && sh.ws.rd.field_kind == 2)
            block_commit_pool(a, sh, smem, cut, acc, bkeys, bmask);
          __syncthreads();
          if (sh.stop) break;
        }
      }
      if (sh.stop) break;
      if (tid == 0) {
        update_amplitudes(c);
        sh.start[((((int)step & a.n_ctl) ^ ci) & 1) ^ 1] = sh.t0;
        if (kind <= CG_SLIDE) sh.limit[kind] = batch_limit(sh.met[kind], sh.pairs[kind], Sn);
      }
      __syncthreads();
    }
    if (sh.stop) break;
  }
  __syncthreads();
  {
    unsigned* cd = reinterpret_cast<unsigned*>(a.ctl + (long long)rep * 5);
    const unsigned* cs = reinterpret_cast<const unsigned*>(sh.ws.ctl);
    for (int i = tid; i < (int)(5 * sizeof(cg_move_ctl) / 4); i += blockDim.x) cd[i] = cs[i];
  }
  if (tid == 0) {
    RepDev* out = a.reps + rep;
    out->draw_pos = sh.t0;
    out->run_dE = sh.run_dE + (double)sh.run_q * kFxEInv;
    out->err = (unsigned)sh.stop;
    unsigned long long* t = a.tally + (long long)rep * 30;
    for (int i = 0; i < 30; i++) t[i] += sh.ws.tally[i];
  }
}

}  // namespace cg

// Launch, shared-memory opt-in and register count of one storage / lanes
// pair (all its forms).
#define CG_SPEC_INSTANTIATE(Pos, G, NAME)                                                          \
  void cg_launch_spec_##NAME(const cg::KArgs& a, size_t smem, cudaStream_t s) {                    \
    auto* kernel = a.lean == 1 ? cg::spec_kernel<Pos, G, 1>                                        \
                   : a.lean == 2 ? cg::spec_kernel<Pos, G, 2> : cg::spec_kernel<Pos, G, 0>;        \
    kernel<<<a.n_reps, 32 * a.spec_w, smem, s>>>(a);                                               \
  }                                                                                                \
  cudaError_t cg_spec_smem_##NAME(int bytes) {                                                     \
    for (auto* kernel : {cg::spec_kernel<Pos, G, 0>, cg::spec_kernel<Pos, G, 1>, cg::spec_kernel<Pos, G, 2>}) { \
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); \
      if (e != cudaSuccess) return e;                                                              \
    }                                                                                              \
    return cudaSuccess;                                                                            \
  }                                                                                                \
  int cg_spec_regs_##NAME() { /* of the code, the same on every device: asked for once */          \
    static std::atomic<int> known{0};                                                              \
    int regs = known.load(std::memory_order_relaxed);                                              \
    if (regs > 0) return regs;                                                                     \
    for (auto* kernel : {cg::spec_kernel<Pos, G, 0>, cg::spec_kernel<Pos, G, 1>, cg::spec_kernel<Pos, G, 2>}) { \
      cudaFuncAttributes at;                                                                       \
      if (cudaFuncGetAttributes(&at, kernel) != cudaSuccess) return 0;                             \
      if (at.numRegs > regs) regs = at.numRegs;                                                    \
    }                                                                                              \
    known.store(regs, std::memory_order_relaxed);                                                  \
    return regs;                                                                                   \
  }
