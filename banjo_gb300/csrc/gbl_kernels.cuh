// Kernels of the bonded-lattice substep.
//
// Device layout (one lattice, or many independent lattices concatenated):
//   nodes  u[i]   = (u.xyz, inv_mass)   v[i] = (v.xyz, mass)   x0[i] = (x0.xyz, 0)
//          up[i]  = u_prev              strain[2i..2i+1] = (e0..e3 | e4, e5, valid, 0)
//          rinv   9 x N, unm 3 x N      (component-major, coalesced per node)
//          nbr[k*N+i] = (rest.xyz, the slot's weight, negated once its bond has failed; 0 when padded)
//          nbr_other[k*N+i] (i itself for a padded slot), nbr_bond[k*N+i]
//   bonds  rec[d] = (a | dead | last-of-a, b | last-of-b, rest_length_sq_minus, rest_length)
//          geo[d] = (rest_edge.xyz, compliance)
//          prev[d] = (prev_tensile, prev_compressive, prev_shear, damage)
//          plastic[d] = (extension, strain), thr4/thr2 = six damage thresholds
// Bonds are stored level-major. A level is the set of bonds at one depth of
// the reference's serial sweep order (CpuLatticeBackend.cpp:336-348, 395-407),
// depth being one more than the deepest earlier bond at either end: a level
// shares no node, and every node meets its bonds in the serial order, so any
// thread mapping inside a level reproduces the serial sweep bit for bit.
// dev2sched maps storage index d to schedule index j; everything a caller
// sees (events, downloads, failure lists) is in schedule order.
#pragma once

#include "gbl_math.cuh"

#include <cfloat>
#include <cstdint>
#include <type_traits>

namespace gbl {

template <class R> struct BondRec;
template <> struct alignas(16) BondRec<float> { std::uint32_t a, b; float rsm, rest; };
template <> struct alignas(8) BondRec<double> { std::uint32_t a, b; double rsm, rest; };

template <class R> __device__ __forceinline__ std::uint32_t endA(const BondRec<R> &r) { return r.a & kNodeMask; }
template <class R> __device__ __forceinline__ std::uint32_t endB(const BondRec<R> &r) { return r.b & kNodeMask; }

// ---------------------------------------------------------------------------
// The bounds-checked build (GBL_BOUNDS_CHECK defined: libgbl_checked.so). Every
// index the kernels read out of device data -- bond ends, neighbour slots,
// candidate, dirty, event, load, halo and isolated-node lists -- is checked
// against the length of the array it indexes before it is used. A violation is
// counted in g_bounds_violation, with the first one's site, index and length,
// and the access is skipped; nothing traps, so the context stays usable and
// the host reads the record (gbl_bounds_report). In the normal build the check
// is the constant true.
// ---------------------------------------------------------------------------
enum BoundsSite : unsigned {
    kSiteSolve = 1, kSiteStrain, kSiteDirty, kSiteDirtyBond, kSiteEndSample, kSiteCandidate, kSiteEvent,
    kSiteEventEnd, kSiteLoad, kSiteIsolated, kSiteHalo, kSiteDamp
};
#ifdef GBL_BOUNDS_CHECK
__device__ unsigned long long g_bounds_violation[4]; // count, then the first's site, index, length
__device__ __noinline__ bool boundsViolated(std::uint64_t i, std::uint64_t n, unsigned site) {
    if (atomicAdd(&g_bounds_violation[0], 1ULL) == 0) {
        g_bounds_violation[1] = site;
        g_bounds_violation[2] = i;
        g_bounds_violation[3] = n;
    }
    return false;
}
__device__ __forceinline__ bool inBounds(std::uint64_t i, std::uint64_t n, unsigned site) {
    return i < n || boundsViolated(i, n, site);
}
#else
__device__ __forceinline__ constexpr bool inBounds(std::uint64_t, std::uint64_t, unsigned) { return true; }
#endif
template <class R> __device__ __forceinline__ bool endsInBounds(const BondRec<R> &r, std::uint32_t n, unsigned site) {
    return inBounds(endA(r), n, site) && inBounds(endB(r), n, site);
}

// Streaming loads for data read once per pass (bond records), so that they do
// not evict the node arrays the gathers keep re-reading from L2.
__device__ __forceinline__ BondRec<float> ldStream(const BondRec<float> *p) {
    const uint4 v = __ldcs(reinterpret_cast<const uint4 *>(p));
    return {v.x, v.y, __uint_as_float(v.z), __uint_as_float(v.w)};
}
__device__ __forceinline__ BondRec<double> ldStream(const BondRec<double> *p) {
    const uint2 ab = __ldcs(reinterpret_cast<const uint2 *>(p));
    const double *d = reinterpret_cast<const double *>(p);
    return {ab.x, ab.y, __ldcs(d + 1), __ldcs(d + 2)};
}
__device__ __forceinline__ Q4<float> ldStream(const Q4<float> *p) {
    const float4 v = __ldcs(reinterpret_cast<const float4 *>(p));
    return {v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ Q4<double> ldStream(const Q4<double> *p) {
    const double2 *q = reinterpret_cast<const double2 *>(p);
    const double2 lo = __ldcs(q), hi = __ldcs(q + 1);
    return {lo.x, lo.y, hi.x, hi.y};
}
// L2-only loads for node data gathered once per pass by a different thread.
__device__ __forceinline__ Q4<float> ldShared(const Q4<float> *p) {
    const float4 v = __ldcg(reinterpret_cast<const float4 *>(p));
    return {v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ Q4<double> ldShared(const Q4<double> *p) {
    const double2 *q = reinterpret_cast<const double2 *>(p);
    const double2 lo = __ldcg(q), hi = __ldcg(q + 1);
    return {lo.x, lo.y, hi.x, hi.y};
}

// Serial bookkeeping (ContactAccumulators, LatticePhysics.hpp:379-388).
struct ContactAcc {
    unsigned long long impulse_contacts;
    double impulse_x, impulse_y, impulse_z, dissipated, max_penetration, max_correction, max_center_shift;
    unsigned long long candidate_overflow, ball_support_events;
};

struct LoadLedger {
    unsigned long long steps;
    double elapsed, req_imp[3], imp[3], req_ang[3], ang[3], work;
};

// NodeContactAccumulators (LatticePhysics.hpp:204-221).
struct NodeAcc {
    unsigned long long contacts, pair_tests, rebuilds, pairs_listed, pair_overflow;
    double dissipated, max_overlap, max_correction, momentum[3];
};

// One device control block per lattice: the RunStatus accumulators, the
// RunControl exit rules, and the substep's transient counters.
struct Ctl {
    unsigned long long total_steps, first_failure_step, last_failure_step, last_energy_gain_step, last_damage_gain_step;
    unsigned failure_rounds, broken_bonds, rank_deficient, exit_reason;
    double removed_energy, max_damage, plastic_work;
    float damage_floor; // the largest float not above max_damage + 1e-6
    unsigned max_t, max_c, max_s, max_plastic; // non-negative float bit patterns
    ContactAcc contact;
    LoadLedger ext;
    // RunControl
    unsigned stop, error;
    unsigned long long quiet_steps, min_steps, no_failure_steps, energy_flat_steps, calm_steps;
    double energy_flat_fraction, calm_damage_margin, removable_energy;
    unsigned long long loads_remaining;
    unsigned long long step_limit; // a served lattice's substep count (0: none); reaching it is exit 3 (max steps)
    // transient
    unsigned full_restart, dirty_count, ffb_count, loads_kicked;
    unsigned event_count, ext_count; // broken bonds this substep; loaded nodes (set between runs)
    unsigned dmg_count, energy_gain;  // damage-record candidates; any broken bond passed the gain test
    double plastic_substep, removed_substep;
    // Node-to-node contact: its accumulators; whether the pair list is rebuilt
    // this substep (set at upload, after a failure round, or by the drift
    // test; cleared by the narrow phase), the list's length, and the bucket
    // fill of the build in progress.
    NodeAcc node;
    unsigned nc_rebuild, nc_pairs, nc_members;
    // The energy audit: the kinetic energy before the phase being measured,
    // and what the damping sweep and the striker passes took out.
    double ke_mark, damping_dissipated, striker_dissipated;
    // External wrenches: how many are set, and the count of sources kicked
    // since upload (a new source's place in the status order).
    unsigned wrench_count, source_seq;
    // Bond projections the sweeps ran: per substep, the bonds alive when its
    // sweep starts (alive at upload less those broken since) times the
    // solver iterations.
    unsigned long long projections, live_bonds;
};

// An external wrench on the device (ExternalWrench, FastLattice.hpp:153-157):
// its nodes (a range of the load list, sources in name order, nodes ascending),
// its source ledger slot, and its point, force and torque.
struct WrenchDev {
    std::uint32_t begin, end, slot, pad;
    double point[3], force[3], torque[3];
};
// A source's ledger (ExternalWrenchLedger) and its place in the status order.
struct SourceSlot {
    LoadLedger load;
    unsigned long long order;
};

constexpr unsigned kErrExternalOverflow = 1;
constexpr unsigned kErrWrench = 2;

template <class R> struct Staged;
template <class R> struct Dev {
    std::uint32_t N, B, D, blocks, tiles_b;
    Q4<R> *u, *v, *x0, *up, *strain;
    R *rinv, *unm, *approach;
    std::uint8_t *dirty, *engaged, *candidate;
    std::uint32_t *cand_bits;
    Q4<R> *nbr;
    std::uint32_t *nbr_other, *nbr_bond;
    std::uint32_t *slot_a, *slot_b;
    BondRec<R> *rec;
    Q4<R> *geo, *prev, *thr4;
    Q2<R> *thr2, *plastic;
    R *lambda;
    std::uint8_t *mode;
    // Substep ledger scratch. ev_*: broken bonds (bit per bond, whole tiles of
    // words; per-tile offset; removed energy by bond); dmg_*: bonds whose
    // damage passed the run maximum (the candidates of the damage-record
    // scan, their values in bond order); tile_*: per end-sample tile plastic
    // work, per tile the prefix of the removed energy.
    std::uint32_t *ev_bits, *ev_tile;
    double *ev_removed;
    uint2 *ev_ends;               // the two nodes of a broken bond, by schedule index
    std::uint32_t *dev2sched;     // bond storage order (level-major) -> schedule index
    std::uint32_t *isolated;      // nodes without bonds (their support projection has no sweep to ride on)
    std::uint32_t isolated_count;
    std::uint32_t *level_begin;   // sweep level boundaries in storage order (level_count + 1), when level_count fits
    std::uint32_t level_count;
    std::uint32_t *dmg_bits, *dmg_tile;
    float *ev_damage, *dmg_value;
    double *tile_plastic, *tile_removed;
    std::uint32_t *blk_ev, *blk_dmg;   // per scan block of tiles: totals, then offsets
    double *blk_removed, *blk_plastic;
    std::uint32_t *node_block_begin, *cand_list, *cand_count, *dirty_list, *ffb;
    Staged<R> *cand_stage; // the listed candidates' records, slab by slab (allocated when the settings have a sphere)
    // Contact halo of the substep (stamped with the substep's number + 1): the
    // listed sphere candidates and their neighbours, and the end-sample tiles
    // holding a bond at one of them. Everything outside it is final before the
    // second contact pass, so its strain and end sample run beside that pass.
    std::uint32_t *halo_stamp, *late_tile_stamp;
    Q4<R> *ext_force;     // applied force (backend precision), w != 0 marks a loaded node
    double *ext_req;      // requested force, 3 per node
    double *ext_contrib;  // 13 per node: impulse 3, angular 3, work, requested 3, requested angular 3
    std::uint32_t *ext_nodes;
    WrenchDev *wrench;    // the set wrenches (their count is in the control block)
    SourceSlot *sources;  // every source kicked since upload
    // Node-to-node contact scratch, allocated when the settings turn contact
    // on: positions at the last build, each node's grid cell (w: its bucket),
    // the hashed grid (per bucket: count, then scatter cursor; first member;
    // members ascending within a bucket), pairs per owner and per 256-node
    // tile (then the tile's first pair), and the pair list in narrow-phase
    // order (owner, partner, bond or kNoBond).
    Q4<R> *nc_built;
    int4 *nc_cell;
    std::uint32_t *nc_count, *nc_start, *nc_members, *nc_fill, *nc_tile;
    std::uint32_t *nc_pa, *nc_pb, *nc_pbond;
    std::uint32_t nc_mask;
    double origin[3];
    Sphere<R> *sphere;
    Ctl *ctl;
    unsigned *running; // lattices of the engine still running this call; a lattice that stops takes itself off
};

constexpr int kThreads = 256;

// Programmatic dependent launch (sm_90+): the kernels of a substep are launched
// while the one before still runs, so that launch latency and CTA start-up
// (1 to 1.5 us, most of what the small ones take) overlap it. Each waits for
// the previous grid to finish, its writes visible, before it touches anything
// an earlier kernel writes, and lets the next one launch only after its own
// wait: at most two overlap, and all before the previous one is complete.
__device__ __forceinline__ void waitPreviousGrid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allowNextGrid() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void startAfterPrevious() {
    waitPreviousGrid();
    allowNextGrid();
}

// One CTA's share of a launch: a range of one lattice's nodes, bonds, tiles or
// scan blocks (what the range indexes is the kernel's).
struct Work {
    std::uint32_t lattice, begin, end;
};

// What a launch covers. With many lattices (Many = true) every CTA reads its
// item from `list` and its lattice's descriptor from `table`, so one launch
// advances any number of independent lattices. A launch over one lattice
// (Many = false) carries that lattice's descriptor in `one`, in the kernel's
// parameter space, and CTA b covers [base + b*per, min(base + (b+1)*per, end)):
// no dependent loads before the work itself.
template <class R> struct Grid {
    const Dev<R> *table;
    const Work *list;
    std::uint32_t base, end, per;
    Dev<R> one;
};

template <bool Many, class R> __device__ __forceinline__ Work item(const Grid<R> &g) {
    if (Many) return g.list[blockIdx.x];
    const std::uint32_t b = g.base + blockIdx.x * g.per;
    return Work{0U, b, b + g.per < g.end ? b + g.per : g.end};
}

template <class R, bool Many> __device__ __forceinline__ Dev<R> descriptor(const Grid<R> &g, const Work &w) {
    if (Many) return g.table[w.lattice];
    return g.one;
}

// The descriptor as a reference a long kernel reads its fields through: for
// many lattices, the CTA's lattice's descriptor copied once into shared
// memory (its fields are then read from there as needed, not held in
// registers across the kernel); for one lattice, the launch's own. Every
// thread of the CTA must call it (it synchronises).
template <class R> struct SharedDesc {
    __align__(16) unsigned char bytes[sizeof(Dev<R>)];
};
template <class R, bool Many>
__device__ __forceinline__ const Dev<R> &descriptorIn(const Grid<R> &g, const Work &w, SharedDesc<R> &smem) {
    if (!Many) return g.one;
    const unsigned *src = reinterpret_cast<const unsigned *>(g.table + w.lattice);
    unsigned *dst = reinterpret_cast<unsigned *>(smem.bytes);
    for (unsigned k = threadIdx.x; k < sizeof(Dev<R>) / sizeof(unsigned); k += blockDim.x) dst[k] = src[k];
    __syncthreads();
    return *reinterpret_cast<const Dev<R> *>(smem.bytes);
}

template <class R> __device__ __forceinline__ V3<R> pos(const Dev<R> &L, std::uint32_t i) {
    return xyz(L.x0[i]) + xyz(L.u[i]);
}

// The node arrays a bond's sample reads.
template <class R> struct NodeView {
    const Q4<R> *u, *x0, *strain;
};
template <class R> __device__ __forceinline__ NodeView<R> viewOf(const Dev<R> &L) { return {L.u, L.x0, L.strain}; }
template <class R> __device__ __forceinline__ V3<R> pos(const NodeView<R> &V, std::uint32_t i) {
    return xyz(V.x0[i]) + xyz(V.u[i]);
}

// ---------------------------------------------------------------------------
// Nonlocal node strain (LatticePhysics.hpp:791-907, plate bending off).
// ---------------------------------------------------------------------------
// A slot's weight while its bond is alive, else 0 (LatticeArrays::nbr_alive
// gating nbr_weight); the raw weight stays in the slot, sign-flipped, for the
// rest geometry of plate bending.
template <class R> __device__ __forceinline__ R liveWeight(R w) { return signbit(w) ? R(0) : w; }

// Bending strain of a sheet one cell thick (plateBendingStrain,
// LatticePhysics.hpp:575-777): the rest neighbourhood (every bond built, alive
// or not) says whether the node lies in a sheet and which way it faces; a
// tilt fit and then a curvature fit over the live neighbours; a fit that
// explains no more than 0.9 of the out-of-plane motion claims no bending; the
// tension fibre of |K| at half the thickness, capped at the yield stretch, is
// added to E in the sheet's frame.
template <class R, bool Direct>
__device__ __noinline__ void plateBending(const Dev<R> &L, std::uint32_t i, V3<R> xi, R half_thickness,
                                          R yield_stretch, R *e) {
    const std::size_t N = L.N;
    R rest_cov[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (std::uint32_t k = 0; k < L.D; ++k) {
        const std::size_t slot = k * N + i;
        if (L.nbr_bond[slot] == kNoBond) continue;
        const Q4<R> q = L.nbr[slot];
        const R w = absR(q.w);
        if (w <= R(0)) continue;
        const R rr[3] = {q.x, q.y, q.z};
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c) rest_cov[r * 3 + c] += w * rr[r] * rr[c];
    }
    R rest_inv[9], flat[3];
    if (pseudoInverse3(rest_cov, rest_inv, flat) >= 3) return; // a solid neighbourhood, not a sheet
    const V3<R> normal{flat[0], flat[1], flat[2]};
    if (!(dot(normal, normal) > R(0))) return;
    R inv[9];
    for (int k = 0; k < 9; ++k) inv[k] = L.rinv[k * N + i];
    auto neighbour = [&](std::uint32_t k, R &w, V3<R> &rest, V3<R> &d) {
        const std::size_t slot = k * N + i;
        const bool present = L.nbr_bond[slot] != kNoBond;
        const Q4<R> q = L.nbr[slot];
        std::uint32_t other = present ? L.nbr_other[slot] : i;
        if (!inBounds(other, N, kSiteStrain)) other = i;
        w = present ? liveWeight(q.w) : R(0);
        rest = present ? V3<R>{q.x, q.y, q.z} : V3<R>{R(0), R(0), R(0)};
        const V3<R> xo = Direct ? pos(L, other) : xyz(L.u[other]);
        d = Direct ? (xo - xi) - rest : xo - xi;
    };
    R rhs[3] = {0, 0, 0};
    for (std::uint32_t k = 0; k < L.D; ++k) {
        R w;
        V3<R> rest, d;
        neighbour(k, w, rest, d);
        const R out = w * dot(d, normal);
        rhs[0] += out * rest.x;
        rhs[1] += out * rest.y;
        rhs[2] += out * rest.z;
    }
    R tilt[3];
    for (int r = 0; r < 3; ++r) {
        R acc = R(0);
        for (int k = 0; k < 3; ++k) acc += inv[r * 3 + k] * rhs[k];
        tilt[r] = acc;
    }
    const R ax = normal.x < R(0) ? -normal.x : normal.x;
    const R ay = normal.y < R(0) ? -normal.y : normal.y;
    const R az = normal.z < R(0) ? -normal.z : normal.z;
    const V3<R> axis = (ax <= ay && ax <= az) ? V3<R>{R(1), R(0), R(0)}
                     : (ay <= az)             ? V3<R>{R(0), R(1), R(0)}
                                              : V3<R>{R(0), R(0), R(1)};
    V3<R> e1 = cross(normal, axis);
    const R e1len = length(e1);
    if (!(e1len > R(0))) return;
    e1 = (R(1) / e1len) * e1;
    const V3<R> e2 = cross(normal, e1);
    R A[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    R g[3] = {0, 0, 0};
    R out2 = R(0);
    for (std::uint32_t k = 0; k < L.D; ++k) {
        R w;
        V3<R> rest, d;
        neighbour(k, w, rest, d);
        const R left = dot(d, normal) - (tilt[0] * rest.x + tilt[1] * rest.y + tilt[2] * rest.z);
        const R p1 = dot(rest, e1), p2 = dot(rest, e2);
        const R psi[3] = {R(0.5) * p1 * p1, p1 * p2, R(0.5) * p2 * p2};
        for (int r = 0; r < 3; ++r) {
            for (int c = 0; c < 3; ++c) A[r * 3 + c] += w * psi[r] * psi[c];
            g[r] += w * psi[r] * left;
        }
        out2 += w * left * left;
    }
    R ev[3], axes[9];
    jacobi3(A, ev, axes);
    R biggest = absR(ev[0]);
    for (int k = 1; k < 3; ++k) biggest = absR(ev[k]) > biggest ? absR(ev[k]) : biggest;
    const R determined = R(1.0e-3) * biggest;
    R c[3] = {0, 0, 0};
    int along = 0;
    for (int k = 0; k < 3; ++k) {
        if (!(ev[k] > determined)) continue;
        ++along;
        R projected = R(0);
        for (int r = 0; r < 3; ++r) projected += axes[r * 3 + k] * g[r];
        const R amount = projected / ev[k];
        for (int r = 0; r < 3; ++r) c[r] += amount * axes[r * 3 + k];
    }
    if (along < 1) return;
    const R explained = c[0] * g[0] + c[1] * g[1] + c[2] * g[2];
    if (!(explained > R(0.9) * out2)) return;
    const R half_trace = R(0.5) * (c[0] + c[2]);
    const R det = c[0] * c[2] - c[1] * c[1];
    R under = half_trace * half_trace - det;
    if (under < R(0)) under = R(0);
    const R disc = sqrtR(under);
    const R l1 = half_trace + disc, l2 = half_trace - disc;
    const R a1 = l1 < R(0) ? -l1 : l1, a2 = l2 < R(0) ? -l2 : l2;
    const R most = yield_stretch > R(0) ? yield_stretch : R(-1);
    R s1 = half_thickness * a1, s2 = half_thickness * a2;
    if (most > R(0)) {
        if (s1 > most) s1 = most;
        if (s2 > most) s2 = most;
    }
    const R alpha = R(0.5) * (s1 + s2), beta = R(0.5) * (s1 - s2);
    const R ratio = disc > R(0) ? beta / disc : R(0);
    const R b11 = alpha + ratio * (c[0] - half_trace);
    const R b12 = ratio * c[1];
    const R b22 = alpha + ratio * (c[2] - half_trace);
    const R u1[3] = {e1.x, e1.y, e1.z}, u2[3] = {e2.x, e2.y, e2.z};
    const int rows[6] = {0, 1, 2, 0, 0, 1};
    const int cols[6] = {0, 1, 2, 1, 2, 2};
    for (int q = 0; q < 6; ++q)
        e[q] += b11 * u1[rows[q]] * u1[cols[q]] + b22 * u2[rows[q]] * u2[cols[q]] +
                b12 * (u1[rows[q]] * u2[cols[q]] + u2[rows[q]] * u1[cols[q]]);
}

template <class R, bool Direct, bool Plate = false, int Ahead = 2>
__device__ void nodeStrain(const Dev<R> &L, std::uint32_t i, R plate_half_thickness = R(0), R plate_yield = R(0)) {
    const std::size_t N = L.N;
    if (L.dirty[i]) {
        R cov[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        std::uint32_t live = 0;
        // A slot that is dead, padded or a degenerate rest edge has no weight
        // and adds zeros, which change nothing: no branch, so the slots' loads
        // are in flight together.
#pragma unroll 6
        for (std::uint32_t k = 0; k < L.D; ++k) {
            const Q4<R> q = L.nbr[k * N + i];
            const R w = liveWeight(q.w);
            const bool counts = !(w <= R(0));
            const R rr[3] = {counts ? q.x : R(0), counts ? q.y : R(0), counts ? q.z : R(0)};
            for (int r = 0; r < 3; ++r)
                for (int c = 0; c < 3; ++c) cov[r * 3 + c] += w * rr[r] * rr[c];
            live += counts ? 1U : 0U;
        }
        R valid = R(0);
        if (live >= 1U) {
            R inv[9], un[3];
            const int rank = pseudoInverse3(cov, inv, un);
            if (rank >= 2) {
                for (int k = 0; k < 9; ++k) L.rinv[k * N + i] = inv[k];
                for (int k = 0; k < 3; ++k) L.unm[k * N + i] = un[k];
                valid = R(1);
            }
            if (rank < 3) atomicAdd(&L.ctl->rank_deficient, 1U);
        }
        L.strain[2 * i + 1].z = valid;
        L.dirty[i] = 0;
        if (valid == R(0)) return;
    } else if (L.strain[2 * i + 1].z == R(0)) {
        return;
    }
    R acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const V3<R> xi = Direct ? pos(L, i) : xyz(L.u[i]);
#pragma unroll Ahead
    for (std::uint32_t k = 0; k < L.D; ++k) {
        const std::size_t slot = k * N + i;
        const Q4<R> q = L.nbr[slot];
        const std::uint32_t other = L.nbr_other[slot];
        if (!inBounds(other, N, kSiteStrain)) continue;
        const V3<R> rest{q.x, q.y, q.z};
        const V3<R> xo = Direct ? pos(L, other) : xyz(L.u[other]);
        const V3<R> cur = Direct ? (xo - xi) - rest : xo - xi;
        const R w = liveWeight(q.w);
        const R cc[3] = {cur.x, cur.y, cur.z};
        const R rr[3] = {rest.x, rest.y, rest.z};
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c) acc[r * 3 + c] += w * cc[r] * rr[c];
    }
    R inv[9], un[3], e[6];
    for (int k = 0; k < 9; ++k) inv[k] = L.rinv[k * N + i];
    for (int k = 0; k < 3; ++k) un[k] = L.unm[k * N + i];
    strainFromMoments(acc, inv, un, e);
    // What a coplanar neighbourhood's plane cannot hold: the bending of a
    // sheet one cell thick (LatticePhysics.hpp:896-905).
    if (Plate && plate_half_thickness > R(0) && un[0] * un[0] + un[1] * un[1] + un[2] * un[2] > R(0))
        plateBending<R, Direct>(L, i, xi, plate_half_thickness, plate_yield, e);
    L.strain[2 * i] = Q4<R>{e[0], e[1], e[2], e[3]};
    L.strain[2 * i + 1] = Q4<R>{e[4], e[5], R(1), R(0)};
}

// The stamp of the running substep in the halo marks (never 0, the cleared value).
template <class R> __device__ __forceinline__ std::uint32_t substepStamp(const Dev<R> &L) {
    return static_cast<std::uint32_t>(L.ctl->total_steps) + 1U;
}

template <class R, bool Many, bool Direct, bool Plate>
__global__ void __launch_bounds__(kThreads) kStrainAll(const Grid<R> launch, int part, R plate, R yield) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    __shared__ SharedDesc<R> desc;
    const Dev<R> &L = descriptorIn<R, Many>(launch, w, desc);
    if (L.ctl->stop) return;
    const std::uint32_t i = w.begin + threadIdx.x;
    if (i >= w.end) return;
    // part 0: every node; 1: the nodes outside the contact halo; 2: inside it.
    if (part != 0) {
        const bool halo = L.halo_stamp[i] == substepStamp(L);
        if (halo != (part == 2)) return;
    }
    nodeStrain<R, Direct, Plate>(L, i, plate, yield);
}

// The start-of-substep restart after an upload (every node) or after a failure
// round (the dirty nodes only: every other node's strain is unchanged, since
// positions have not moved since the end sample and its bonds are the same;
// src/fastlattice/ParallelCpuLatticeBackend.cpp:1718-1757 relies on the same fact).
// It reads the substep's starting positions: before the kick from u, or after
// it (beside the first contact pass) from u_prev, where the kick copied them.
// After an upload every node is dirty, and what bounds the kernel is one
// thread's chain: covariance loads, 12 Jacobi sweeps, moment loads. Six slots'
// loads in flight and an eigen-solve in registers: 32x8x8 33 -> 27 us,
// 128x32x32 62 -> 54 us, 128 mixed lattices 89 -> 70 us. (The end sample, which
// solves no eigensystem for most nodes, is bound by memory: 3, 6 or 9 slots
// ahead there measured the same as 2.)
template <class R, bool Many, bool Direct, bool Plate>
__global__ void __launch_bounds__(kThreads) kRestartStrain(const Grid<R> launch, int after_kick, R plate, R yield) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    Dev<R> L = descriptor<R, Many>(launch, w);
    if (after_kick) L.u = L.up; // the kick kept the substep's starting positions there
    if (L.ctl->stop) return;
    // Items cover the node index range; a dirty list is never longer.
    const std::uint32_t t = w.begin + threadIdx.x;
    if (t >= w.end) return;
    if (L.ctl->full_restart) nodeStrain<R, Direct, Plate, 6>(L, t, plate, yield);
    else if (t < L.ctl->dirty_count) {
        const std::uint32_t node = L.dirty_list[t];
        if (inBounds(node, L.N, kSiteDirty)) nodeStrain<R, Direct, Plate, 6>(L, node, plate, yield);
    }
}

// ---------------------------------------------------------------------------
// Bond samples (LatticePhysics.hpp:921-959, 1116-1126).
// ---------------------------------------------------------------------------
template <class R, bool Direct>
__device__ __forceinline__ V3<R> bondVector(const NodeView<R> &V, std::uint32_t a, std::uint32_t b, V3<R> edge) {
    if (Direct) return pos(V, b) - pos(V, a);
    return edge + (xyz(V.u[b]) - xyz(V.u[a]));
}

template <class R, bool Direct, class M>
__device__ __forceinline__ void sampleBond(M &m, const NodeView<R> &V, std::uint32_t a, std::uint32_t b, const BondRec<R> &rec,
                                           V3<R> edge, R len, R &t, R &c, R &s) {
    const R rest = rec.rest;
    R stretch;
    if (Direct) {
        stretch = m.div(len, rest) - R(1);
    } else {
        const V3<R> du = xyz(V.u[b]) - xyz(V.u[a]);
        const R num = rec.rsm + R(2) * dot(edge, du) + dot(du, du);
        stretch = m.div(num, (len + rest) * rest);
    }
    t = stretch;
    c = -stretch;
    s = R(0);
    const R rl = m.root(dot(edge, edge));
    if (rl > R(1.0e-9)) {
        const V3<R> dir = edge * m.div(R(1), rl);
        const std::uint32_t ends[2] = {a, b};
        for (int q = 0; q < 2; ++q) {
            const Q4<R> s0 = V.strain[2 * ends[q]], s1 = V.strain[2 * ends[q] + 1];
            if (s1.z == R(0)) continue;
            const R e[6] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y};
            R nn, sh;
            resolveAlong(m, e, dir, nn, sh);
            t = maxR(t, nn);
            c = maxR(c, -nn);
            s = maxR(s, sh);
        }
    }
}

// The current length of a bond and its sample, branch-free in the float lane
// where its operands allow.
template <class R> struct BondSample {
    R len, t, c, s;
};
template <class R, bool Direct, class M>
__device__ __forceinline__ BondSample<R> lengthAndSample(M &m, const NodeView<R> &V, std::uint32_t a, std::uint32_t b,
                                                         const BondRec<R> &rec, V3<R> edge) {
    BondSample<R> o;
    const V3<R> now = bondVector<R, Direct>(V, a, b, edge);
    o.len = m.root(dot(now, now));
    sampleBond<R, Direct>(m, V, a, b, rec, edge, o.len, o.t, o.c, o.s);
    return o;
}
template <class R, bool Direct>
__device__ __noinline__ BondSample<R> sampleAnywhere(NodeView<R> V, std::uint32_t a, std::uint32_t b, R rsm, R rest,
                                                     V3<R> edge) {
    PlainMath<R> plain;
    return lengthAndSample<R, Direct>(plain, V, a, b, BondRec<R>{a, b, rsm, rest}, edge);
}
template <class R, bool Direct>
__device__ __forceinline__ BondSample<R> sampleOf(const NodeView<R> &V, std::uint32_t a, std::uint32_t b, const BondRec<R> &rec,
                                                  V3<R> edge) {
    if constexpr (std::is_same<R, float>::value && !Direct) {
        QuickMath quick;
        const BondSample<R> o = lengthAndSample<R, Direct>(quick, V, a, b, rec, edge);
        return quick.good ? o : sampleAnywhere<R, Direct>(V, a, b, rec.rsm, rec.rest, edge);
    } else {
        PlainMath<R> plain;
        return lengthAndSample<R, Direct>(plain, V, a, b, rec, edge);
    }
}

template <class R, bool Direct>
__device__ __forceinline__ void startSample(const Dev<R> &L, const NodeView<R> &V, std::uint32_t j) {
    const BondRec<R> rec = L.rec[j];
    if (rec.a & kDeadBit) return;
    const Q4<R> g = L.geo[j];
    const BondSample<R> o = sampleOf<R, Direct>(V, endA(rec), endB(rec), rec, V3<R>{g.x, g.y, g.z});
    Q4<R> p = L.prev[j];
    p.x = maxR(R(0), o.t);
    p.y = maxR(R(0), o.c);
    p.z = maxR(R(0), o.s);
    L.prev[j] = p;
}

// Every live bond after an upload, or the live bonds at each dirty node after a
// failure round: items cover the bond storage range, kRestartPer bonds a CTA
// (most substeps have few dirty nodes, and a CTA per 256 bonds spent 111 us of
// a 128-trial substep starting CTAs, 88,000 of them; 21 now), and the
// lattice's threads share the (slot, dirty node) pairs, consecutive threads
// on consecutive dirty nodes. A bond with both ends dirty is sampled twice to the same values. (One
// thread per dirty node walking its slots was a chain of 18 or 32 samples: 39
// us a substep in the 32x8x8 beam, now 8; 100 in the 128x32x32 bar, now 11.)
constexpr unsigned kRestartPer = 8 * kThreads;
template <class R, bool Many, bool Direct>
__global__ void __launch_bounds__(kThreads) kRestartBonds(const Grid<R> launch, int after_kick) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    __shared__ SharedDesc<R> desc;
    const Dev<R> &L = descriptorIn<R, Many>(launch, w, desc);
    if (L.ctl->stop) return;
    const NodeView<R> V{after_kick ? L.up : L.u, L.x0, L.strain};
    if (L.ctl->full_restart) {
        for (std::uint32_t d = w.begin + threadIdx.x; d < w.end; d += kThreads) startSample<R, Direct>(L, V, d);
        return;
    }
    const std::uint32_t dirty = L.ctl->dirty_count;
    const std::uint64_t pairs = static_cast<std::uint64_t>(dirty) * L.D;
    const std::uint64_t threads = static_cast<std::uint64_t>((L.B + kRestartPer - 1) / kRestartPer) * kThreads;
    for (std::uint64_t q = w.begin / kRestartPer * kThreads + threadIdx.x; q < pairs; q += threads) {
        const std::uint32_t k = static_cast<std::uint32_t>(q / dirty);
        const std::uint32_t node = L.dirty_list[q - static_cast<std::uint64_t>(k) * dirty];
        if (!inBounds(node, L.N, kSiteDirty)) continue;
        const std::uint32_t bond = L.nbr_bond[static_cast<std::size_t>(k) * L.N + node];
        if (bond != kNoBond && inBounds(bond, L.B, kSiteDirtyBond)) startSample<R, Direct>(L, V, bond);
    }
}

// ---------------------------------------------------------------------------
// Kick and classify (LatticePhysics.hpp:1702-1719), with the external force
// kick before it (ExternalLoads.hpp:79-148).
// ---------------------------------------------------------------------------
template <class R>
__device__ __forceinline__ bool sphereCandidate(const Settings<R> &S, const Sphere<R> &sp, V3<R> x, V3<R> vel, R mass) {
    if (mass <= R(0)) return false;
    const V3<R> r = x - sp.center;
    const R distance = length(r);
    const R gap = distance - (sp.radius + S.c_node_radius);
    const R bound = length(vel - sp.velocity) + length(sp.angular) * distance;
    const R reach = maxR(S.c_margin, bound * S.dt) + S.c_slack;
    return gap <= reach;
}

template <class R, bool Many>
__global__ void __launch_bounds__(kThreads) kKick(const Grid<R> launch, Settings<R> S) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    __shared__ SharedDesc<R> desc;
    const Dev<R> &L = descriptorIn<R, Many>(launch, w, desc);
    if (L.ctl->stop) return;
    const std::uint32_t i = w.begin + threadIdx.x; // items start on multiples of 256: warps cover whole bit words
    bool cand = false;
    if (i < w.end) {
        Q4<R> vq = L.v[i];
        const Q4<R> uq = L.u[i];
        V3<R> vel = xyz(vq);
        if (L.ctl->ext_count && L.ctl->loads_remaining > 0) {
            const Q4<R> f = L.ext_force[i];
            if (f.w != R(0)) {
                const V3<R> before = vel;
                const V3<R> after = before + (S.dt * uq.w) * V3<R>{f.x, f.y, f.z};
                if (!finiteR(after.x) || !finiteR(after.y) || !finiteR(after.z)) {
                    atomicOr(&L.ctl->error, kErrExternalOverflow);
                } else {
                    vel = after;
                    const double m = static_cast<double>(vq.w);
                    const double o[3] = {double(before.x), double(before.y), double(before.z)};
                    const double n[3] = {double(after.x), double(after.y), double(after.z)};
                    const double imp[3] = {m * (n[0] - o[0]), m * (n[1] - o[1]), m * (n[2] - o[2])};
                    const V3<R> p = xyz(L.x0[i]) + xyz(uq);
                    const double wp[3] = {L.origin[0] + double(p.x), L.origin[1] + double(p.y), L.origin[2] + double(p.z)};
                    const double dt = static_cast<double>(S.dt);
                    const double rq[3] = {dt * L.ext_req[3 * i], dt * L.ext_req[3 * i + 1], dt * L.ext_req[3 * i + 2]};
                    double *c = L.ext_contrib + 13 * static_cast<std::size_t>(i);
                    c[0] = imp[0]; c[1] = imp[1]; c[2] = imp[2];
                    c[3] = wp[1] * imp[2] - wp[2] * imp[1];
                    c[4] = wp[2] * imp[0] - wp[0] * imp[2];
                    c[5] = wp[0] * imp[1] - wp[1] * imp[0];
                    c[6] = imp[0] * (.5 * (o[0] + n[0])) + imp[1] * (.5 * (o[1] + n[1])) + imp[2] * (.5 * (o[2] + n[2]));
                    c[7] = rq[0]; c[8] = rq[1]; c[9] = rq[2];
                    c[10] = wp[1] * rq[2] - wp[2] * rq[1];
                    c[11] = wp[2] * rq[0] - wp[0] * rq[2];
                    c[12] = wp[0] * rq[1] - wp[1] * rq[0];
                }
            }
        }
        vel = vel + S.dt * S.gravity;
        L.v[i] = Q4<R>{vel.x, vel.y, vel.z, vq.w};
        L.up[i] = uq;
        L.engaged[i] = 0;
        L.engaged[L.N + i] = 0;
        if (S.sphere_enabled) {
            Sphere<R> kicked = *L.sphere;
            kicked.velocity = kicked.velocity + S.dt * S.gravity;
            cand = sphereCandidate(S, kicked, xyz(L.x0[i]) + xyz(uq), vel, vq.w);
        }
        L.candidate[i] = cand ? 1 : 0;
        if (!cand) {
            for (std::uint32_t p = 0; p < S.plane_count; ++p) L.approach[p * L.N + i] = dot(vel, S.planes[p].normal);
            const V3<R> un = xyz(uq) + S.dt * vel;
            L.u[i] = Q4<R>{un.x, un.y, un.z, uq.w};
        }
    }
    if (S.sphere_enabled) {
        const unsigned bits = __ballot_sync(0xffffffffU, cand);
        if ((threadIdx.x & 31) == 0 && i / 32 < (L.N + 31) / 32) L.cand_bits[i / 32] = bits;
    }
}

// ---------------------------------------------------------------------------
// A serial FP64 sum, by one warp: what s = (((s + x[0]) + x[1]) + ...) gives,
// rounding by rounding, without its chain of dependent adds (38 ns each here).
//
// While the running sum stays inside one binade, it is an integer number M of
// that binade's ulps, and adding x rounds M + x/ulp to the nearest integer:
// unless x/ulp lies half-way between two integers, that is M + rint(x/ulp),
// whatever M is. So the roundings are known before the sums, and the running
// sums are integer prefix sums, which any order forms alike. A run of terms
// is taken up to the first one that is a tie, is too large for the integers,
// or takes the sum to the end of its binade (a sum that rounds to a binade's
// own bound may have rounded in the one below); that term is added by the
// hardware, and the next run starts from there. Sums of one sign cross few
// binades. One that keeps crossing goes on term by term, longer each time
// (FoldPace): then it is the chain, by one lane. Cantilevers loaded by forces of
// any sign, ms a substep, this and a chain alone: 48x12x12 0.27 and 0.27,
// 64x16x16 0.60 and 0.60, 96x24x24 1.96 and 1.97; under their weight, which goes
// by runs, 0.22-0.26 and 0.32, 0.38-0.44 and 0.66, 0.91-0.99 and 2.05.
//
// All of a run is integer arithmetic on the terms' bits (this GPU has two FP64
// lanes an SM: the same run with FP64 scaling, rint and conversions was slower
// than the chain). `x` is in shared memory; every lane calls with the same
// arguments and gets the sum.
// ---------------------------------------------------------------------------
// How a sum goes on, kept from chunk to chunk: the terms still to be added one
// by one, and how many that are after the next run that comes to little (a run
// costs about as much as 30 adds, whatever it comes to). At most 1,024: at 256,
// 512 and 2,048 the 64x16x16 cantilever takes 0.63, 0.61 and 0.59 ms a substep
// with forces of any sign, 0.37, 0.37 and 0.42 under its weight.
constexpr unsigned kFoldWorth = 32, kFoldMost = 1024;
struct FoldPace {
    unsigned owed = kFoldWorth, patience = kFoldWorth;
};

// Whether a sum goes by runs from here: not when it is zero, subnormal or not
// finite. Zero terms leave a zero sum as it is (it is never -0 here: it started
// as +0 or is a cancellation) and are passed over, `at` moved up.
__device__ __forceinline__ bool foldRuns(double s, const double *x, unsigned &at, unsigned n) {
    using u64 = unsigned long long;
    const u64 sb = static_cast<u64>(__double_as_longlong(s));
    const int exponent = static_cast<int>((sb >> 52) & 0x7ff);
    if (exponent != 0 && exponent != 0x7ff) return true;
    if ((sb << 1) != 0) return false;
    const u64 *bits = reinterpret_cast<const u64 *>(x);
    const unsigned lane = threadIdx.x & 31;
    for (; at < n; at += 32) {
        const bool some = at + lane < n && (bits[at + lane] << 1) != 0;
        const unsigned mask = __ballot_sync(0xffffffffU, some);
        if (mask == 0) continue;
        at += static_cast<unsigned>(__ffs(mask) - 1);
        break;
    }
    return false;
}

// One run from term `at`: the terms it took, at most kFoldRun, `s` with them.
constexpr unsigned kFoldPer = 8; // consecutive terms per lane
constexpr unsigned kFoldRun = 32 * kFoldPer;
__device__ __forceinline__ unsigned foldRun(double &s, const double *x, unsigned at, unsigned n) {
    using u64 = unsigned long long;
    constexpr unsigned kPer = kFoldPer;
    constexpr u64 kOne = 1ULL << 52;
    const unsigned lane = threadIdx.x & 31;
    const u64 *bits = reinterpret_cast<const u64 *>(x);
    const u64 sb = static_cast<u64>(__double_as_longlong(s));
    const int exponent = static_cast<int>((sb >> 52) & 0x7ff);
    const bool negative = (sb >> 63) != 0;
    const unsigned first = at + lane * kPer;
    // The running sums in ulps, signed as the sum is: M positive.
    long long upto[kPer], sum = 0;
    unsigned bad = kPer; // the first of the lane's terms that ends a run by itself
#pragma unroll
    for (unsigned k = 0; k < kPer; ++k) {
        const u64 b = first + k < n ? bits[first + k] : 0ULL;
        const int e = static_cast<int>((b >> 52) & 0x7ff);
        const u64 mantissa = (b & (kOne - 1)) | (e ? kOne : 0ULL);
        const int shift = exponent - (e ? e : 1); // x = mantissa / 2^shift ulps
        const int by = shift < 0 ? 0 : shift > 55 ? 55 : shift;
        const u64 low = mantissa & ((1ULL << by) - 1), half = (1ULL << by) >> 1;
        const long long r = static_cast<long long>((mantissa >> by) + (low > half ? 1 : 0));
        if (bad == kPer && (shift < 0 || (low == half && half != 0) || first + k >= n)) bad = k;
        sum += ((b >> 63) != 0) != negative ? -r : r;
        upto[k] = sum;
    }
    long long before = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffU, before, o);
        if (lane >= static_cast<unsigned>(o)) before += y;
    }
    before += static_cast<long long>((sb & (kOne - 1)) | kOne) - sum;
#pragma unroll
    for (unsigned k = 0; k < kPer; ++k) {
        const long long total = before + upto[k];
        if (bad > k && !(total > static_cast<long long>(kOne) && total < static_cast<long long>(2 * kOne))) bad = k;
    }
    const unsigned stop = __reduce_min_sync(0xffffffffU, bad < kPer ? lane * kPer + bad : 32 * kPer);
    if (stop) {
        const unsigned pick = (stop - 1) % kPer;
        long long mine = upto[0];
#pragma unroll
        for (unsigned k = 1; k < kPer; ++k)
            if (pick == k) mine = upto[k];
        const u64 total = static_cast<u64>(__shfl_sync(0xffffffffU, before + mine, static_cast<int>((stop - 1) / kPer)));
        s = __longlong_as_double(static_cast<long long>((sb & (0xfffULL << 52)) | (total & (kOne - 1))));
    }
    return stop;
}

__device__ __forceinline__ double foldSerial(double s, const double *x, unsigned n, FoldPace &pace) {
    for (unsigned at = 0; at < n;) {
        if (pace.owed == 0) {
            if (foldRuns(s, x, at, n)) {
                const unsigned stop = foldRun(s, x, at, n);
                at += stop;
                if (at < n && stop < kFoldRun) { // the term it ended at is added by the hardware
                    pace.owed = stop >= kFoldWorth ? 1 : pace.patience;
                    if (stop < kFoldWorth) pace.patience = pace.patience < kFoldMost ? 2 * pace.patience : kFoldMost;
                    else if (stop >= 2 * kFoldWorth) pace.patience = kFoldWorth;
                }
            } else {
                pace.owed = 1;
            }
        }
        if (pace.owed && at < n) {
            const unsigned upto = n - at < pace.owed ? n : at + pace.owed;
            pace.owed -= upto - at;
            if ((threadIdx.x & 31) == 0) {
                // Two terms a load: a load between dependent adds costs them 8 cycles of 72.
                unsigned k = at;
                if (__cvta_generic_to_shared(x + k) & 8U) s += x[k++];
#pragma unroll 8
                for (; k + 2 <= upto; k += 2) {
                    const double2 t = *reinterpret_cast<const double2 *>(x + k);
                    s += t.x;
                    s += t.y;
                }
                if (k < upto) s += x[k];
            }
            s = __shfl_sync(0xffffffffU, s, 0);
            at = upto;
        }
    }
    return s;
}

// The same for terms of one sign: their sum crosses a binade once, so the next
// run soon pays.
__device__ __forceinline__ double foldOneSign(double s, const double *x, unsigned n) {
    unsigned patience = 16;
    for (unsigned at = 0; at < n;) {
        unsigned owed = 1;
        if (foldRuns(s, x, at, n)) {
            const unsigned stop = foldRun(s, x, at, n);
            at += stop;
            owed = stop == kFoldRun ? 0 : stop < 16 ? patience : 1;
            patience = stop < 16 ? 2 * patience : stop >= 64 ? 16 : patience;
        }
        for (; owed && at < n; --owed, ++at) s += x[at];
    }
    return s;
}

// ---------------------------------------------------------------------------
// External wrenches (ExternalLoads.hpp:171-238): each wrench's force and
// torque spread over its nodes by mass about their mass centre, from the
// current positions, before every kick. One CTA per wrench. The region's sums
// (mass, centre, inertia tensor, the resultant checks) are the reference's
// serial folds in node order: the CTA forms a chunk's terms, a node per thread,
// and a warp folds each sum (foldSerial). (Formed by the folding thread, a
// node's divisions and norms cost it a microsecond each: 410 us a kick with 81
// and 18 nodes, 160 now, most of it the eigen-solve.) The eigen-solve of the tensor is the
// reference's cyclic Jacobi in double. apply 1 writes the kick's forces (when
// loads remain); a wrench the current geometry cannot carry then stops the
// lattice before the kick changes anything, with kErrWrench set (the reference
// throws there). apply 0 only validates, into *verdict.
// ---------------------------------------------------------------------------
constexpr unsigned kWrenchThreads = 256;

__device__ inline double normD(double x, double y, double z) { return norm3d(x, y, z); }

template <class R>
__device__ __forceinline__ void wrenchSpread(const Dev<R> &L, const WrenchDev *ws, const std::uint32_t *lists,
                                             unsigned *verdict, int apply, unsigned index) {
    Ctl &c = *L.ctl;
    if (apply && (c.stop || c.loads_remaining == 0 || index >= c.wrench_count)) return;
    const WrenchDev w = ws[index];
    const std::uint32_t *list = lists + w.begin;
    const std::uint32_t n = w.end - w.begin;
    const unsigned t = threadIdx.x, warp = t / 32;
    __shared__ double terms[8][kWrenchThreads]; // a chunk's terms of up to eight sums
    __shared__ double sums[8], mass, center[3], tensor[9], alpha[3], moment[3];
    __shared__ int bad;
    if (t == 0) bad = 0;
    const std::uint32_t a0 = list[0];
    const V3<R> p0 = xyz(L.x0[a0]) + xyz(L.u[a0]);
    const double anchor[3] = {double(p0.x), double(p0.y), double(p0.z)};
    __syncthreads();
    // One pass over the region: form(k, j) writes node k's terms at place j of
    // the first `count` sums; warp q folds sum q, left in sums[q].
    auto pass = [&](unsigned count, auto &&form) {
        double acc = 0.0;
        FoldPace pace;
        for (std::uint32_t base = 0; base < n; base += kWrenchThreads) {
            if (base + t < n) form(base + t, t);
            __syncthreads();
            if (warp < count)
                acc = foldSerial(acc, terms[warp], n - base < kWrenchThreads ? n - base : kWrenchThreads, pace);
            __syncthreads();
        }
        if (warp < count && t % 32 == 0) sums[warp] = acc;
        __syncthreads();
    };
    // Mass, and position relative to the anchor; movable, finite nodes only.
    auto node = [&](std::uint32_t k, double &m, double r[3]) {
        const std::uint32_t i = list[k];
        const Q4<R> u = L.u[i], v = L.v[i]; // w: inverse mass, mass
        const V3<R> p = xyz(L.x0[i]) + xyz(u);
        m = double(v.w);
        r[0] = double(p.x) - anchor[0];
        r[1] = double(p.y) - anchor[1];
        r[2] = double(p.z) - anchor[2];
        if (!(v.w > R(0)) || !(u.w > R(0)) || !isfinite(v.w) || !isfinite(u.w) || !isfinite(r[0]) || !isfinite(r[1]) ||
            !isfinite(r[2]))
            bad = 1;
    };
    pass(1, [&](std::uint32_t k, unsigned j) {
        double m, r[3];
        node(k, m, r);
        terms[0][j] = m;
    });
    if (t == 0) {
        mass = sums[0];
        if (!(mass > 0) || !isfinite(mass)) bad = 1;
    }
    __syncthreads();
    pass(3, [&](std::uint32_t k, unsigned j) {
        double m, r[3];
        node(k, m, r);
        const double share = m / mass;
        for (int q = 0; q < 3; ++q) terms[q][j] = r[q] * share;
    });
    if (t < 3) center[t] = sums[t];
    __syncthreads();
    // The tensor is symmetric: xx, yy, zz, xy, xz, yz.
    pass(6, [&](std::uint32_t k, unsigned j) {
        double m, p[3];
        node(k, m, p);
        const double r[3] = {p[0] - center[0], p[1] - center[1], p[2] - center[2]};
        const double share = m / mass;
        for (int a = 0; a < 3; ++a)
            terms[a][j] = share * (r[(a + 1) % 3] * r[(a + 1) % 3] + r[(a + 2) % 3] * r[(a + 2) % 3]);
        terms[3][j] = share * (-r[0] * r[1]);
        terms[4][j] = share * (-r[0] * r[2]);
        terms[5][j] = share * (-r[1] * r[2]);
    });
    if (t < 9) {
        const unsigned a = t / 3, b = t % 3;
        tensor[t] = sums[a == b ? a : a + b + 2];
    }
    __syncthreads();
    if (t == 0) {
        const double arm[3] = {((w.point[0] - L.origin[0]) - anchor[0]) - center[0],
                               ((w.point[1] - L.origin[1]) - anchor[1]) - center[1],
                               ((w.point[2] - L.origin[2]) - anchor[2]) - center[2]};
        moment[0] = w.torque[0] + (arm[1] * w.force[2] - arm[2] * w.force[1]);
        moment[1] = w.torque[1] + (arm[2] * w.force[0] - arm[0] * w.force[2]);
        moment[2] = w.torque[2] + (arm[0] * w.force[1] - arm[1] * w.force[0]);
        for (int q = 0; q < 3; ++q)
            if (!isfinite(center[q]) || !isfinite(moment[q])) bad = 1;
        double scale = 0.0;
        for (int e = 0; e < 9; ++e) {
            if (!isfinite(tensor[e])) bad = 1;
            const double x = fabs(tensor[e]);
            scale = scale < x ? x : scale;
        }
        double al[3] = {0.0, 0.0, 0.0};
        const double mn = normD(moment[0], moment[1], moment[2]);
        if (!bad && scale > 0) {
            double m9[9], eig[3], axes[9];
            for (int e = 0; e < 9; ++e) m9[e] = tensor[e] / scale;
            jacobi3(m9, eig, axes);
            double largest = fabs(eig[0]);
            largest = largest < fabs(eig[1]) ? fabs(eig[1]) : largest;
            largest = largest < fabs(eig[2]) ? fabs(eig[2]) : largest;
            double un[3] = {moment[0], moment[1], moment[2]};
#pragma unroll
            for (int axis = 0; axis < 3; ++axis) {
                if (!(eig[axis] > 1e-10 * largest)) continue;
                const double dir[3] = {axes[axis], axes[3 + axis], axes[6 + axis]};
                const double component = dir[0] * moment[0] + dir[1] * moment[1] + dir[2] * moment[2];
                const double sc = component / mass / scale / eig[axis];
                for (int q = 0; q < 3; ++q) {
                    un[q] = un[q] - dir[q] * component;
                    al[q] = al[q] + dir[q] * sc;
                }
            }
            if (normD(un[0], un[1], un[2]) > 1024 * DBL_EPSILON * mn) bad = 1;
        } else if (!bad && mn > 0) {
            bad = 1; // a torque with no sampled lever arm
        }
        for (int q = 0; q < 3; ++q) {
            if (!isfinite(al[q])) bad = 1;
            alpha[q] = al[q];
        }
    }
    __syncthreads();
    // Node forces, written for the kick, and the resultant checks.
    pass(8, [&](std::uint32_t k, unsigned j) {
        double m, p[3];
        node(k, m, p);
        const double share = m / mass;
        const double r[3] = {p[0] - center[0], p[1] - center[1], p[2] - center[2]};
        const double cr[3] = {alpha[1] * r[2] - alpha[2] * r[1], alpha[2] * r[0] - alpha[0] * r[2],
                              alpha[0] * r[1] - alpha[1] * r[0]};
        double f[3];
        for (int q = 0; q < 3; ++q) f[q] = w.force[q] * share + cr[q] * m;
        const R fx = R(f[0]), fy = R(f[1]), fz = R(f[2]);
        if (!isfinite(f[0]) || !isfinite(f[1]) || !isfinite(f[2]) || !isfinite(fx) || !isfinite(fy) || !isfinite(fz))
            bad = 1;
        if (apply) {
            const std::uint32_t i = list[k];
            L.ext_force[i] = Q4<R>{fx, fy, fz, R(1)};
            L.ext_req[3 * static_cast<std::size_t>(i)] = f[0];
            L.ext_req[3 * static_cast<std::size_t>(i) + 1] = f[1];
            L.ext_req[3 * static_cast<std::size_t>(i) + 2] = f[2];
        }
        const double mo[3] = {r[1] * f[2] - r[2] * f[1], r[2] * f[0] - r[0] * f[2], r[0] * f[1] - r[1] * f[0]};
        for (int q = 0; q < 3; ++q) {
            terms[q][j] = f[q];
            terms[3 + q][j] = mo[q];
        }
        terms[6][j] = normD(f[0], f[1], f[2]);
        terms[7][j] = normD(mo[0], mo[1], mo[2]);
    });
    if (t == 0) {
        for (int q = 0; q < 8; ++q)
            if (!isfinite(sums[q])) bad = 1;
        const double fn = normD(w.force[0], w.force[1], w.force[2]);
        const double mn = normD(moment[0], moment[1], moment[2]);
        const double df = normD(sums[0] - w.force[0], sums[1] - w.force[1], sums[2] - w.force[2]);
        const double dm = normD(sums[3] - moment[0], sums[4] - moment[1], sums[5] - moment[2]);
        if (df > 1e-10 * (fn < sums[6] ? sums[6] : fn) || dm > 1e-10 * (mn < sums[7] ? sums[7] : mn)) bad = 1;
        if (bad) {
            if (!apply) {
                atomicOr(verdict, 1U);
            } else if (!(atomicOr(&c.error, kErrWrench) & kErrWrench)) {
                c.stop = 1;
                atomicSub(L.running, 1U);
            }
        }
    }
}

// One lattice's wrenches: one CTA per wrench.
template <class R>
__global__ void __launch_bounds__(kWrenchThreads)
kWrench(const Dev<R> L, const WrenchDev *ws, const std::uint32_t *lists, unsigned *verdict, int apply) {
    startAfterPrevious();
    wrenchSpread(L, ws, lists, verdict, apply, blockIdx.x);
}

// A batch's wrenches in one launch: one CTA per (lattice, wrench) item.
template <class R>
__global__ void __launch_bounds__(kWrenchThreads) kWrenchMany(const Grid<R> launch) {
    startAfterPrevious();
    const Work w = launch.list[blockIdx.x];
    const Dev<R> &L = launch.table[w.lattice];
    wrenchSpread(L, L.wrench, L.ext_nodes, nullptr, 1, w.begin);
}

// Ordered candidate lists per slab, capped at 1024 (CpuLatticeBackend.cpp:375-386):
// one CTA per slab scans its bit words in node order.
template <class R, bool Many>
__global__ void __launch_bounds__(1024) kCandidates(const Grid<R> launch) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    if (L.ctl->stop) return;
    __shared__ std::uint32_t warp_total[32];
    __shared__ std::uint32_t carry;
    const std::uint32_t blk = w.begin; // one item per (lattice, slab)
    const std::uint32_t nb = L.node_block_begin[blk], ne = L.node_block_begin[blk + 1];
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const std::uint32_t w0 = nb / 32, w1 = ne == nb ? w0 : (ne - 1) / 32 + 1;
    for (std::uint32_t base = w0; base < w1; base += blockDim.x) {
        const std::uint32_t word = base + threadIdx.x;
        std::uint32_t bits = 0;
        if (word < w1) {
            bits = L.cand_bits[word];
            const std::uint32_t lo = word * 32, hi = lo + 32;
            if (nb > lo) bits &= ~0U << (nb - lo);
            if (ne < hi) bits &= (ne - lo) >= 32 ? ~0U : ((1U << (ne - lo)) - 1U);
        }
        const std::uint32_t n = __popc(bits);
        // Block exclusive scan of n.
        std::uint32_t x = n;
        for (int o = 1; o < 32; o <<= 1) {
            const std::uint32_t y = __shfl_up_sync(0xffffffffU, x, o);
            if ((threadIdx.x & 31) >= static_cast<unsigned>(o)) x += y;
        }
        if ((threadIdx.x & 31) == 31) warp_total[threadIdx.x / 32] = x;
        __syncthreads();
        if (threadIdx.x < 32) {
            std::uint32_t t = warp_total[threadIdx.x];
            for (int o = 1; o < 32; o <<= 1) {
                const std::uint32_t y = __shfl_up_sync(0xffffffffU, t, o);
                if (threadIdx.x >= static_cast<unsigned>(o)) t += y;
            }
            warp_total[threadIdx.x] = t;
        }
        __syncthreads();
        std::uint32_t before = carry + x - n + (threadIdx.x >= 32 ? warp_total[threadIdx.x / 32 - 1] : 0U);
        while (bits) {
            const int b = __ffs(bits) - 1;
            bits &= bits - 1;
            if (before < kCandidatesPerBlock) L.cand_list[blk * kCandidatesPerBlock + before] = word * 32 + b;
            ++before;
        }
        __syncthreads();
        if (threadIdx.x == 0) carry += warp_total[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const std::uint32_t total = carry;
        L.cand_count[blk] = total < kCandidatesPerBlock ? total : kCandidatesPerBlock;
        // Slabs of one lattice finish in any order: the count is shared.
        if (total > kCandidatesPerBlock)
            atomicAdd(&L.ctl->contact.candidate_overflow,
                      static_cast<unsigned long long>(total - kCandidatesPerBlock));
    }
}

// The contact halo of the substep: per (lattice, slab) item, its listed
// candidates, their neighbours, and the end-sample tiles of every bond at one
// of those nodes. Threads that mark the same entry write the same stamp. A
// slab's CTAs along y share its candidates' slots: each slot is a chain of
// loads (the neighbour, then its bonds) that one CTA walked one after another
// (kick, lists and halo of the 256x128x128 impact 245 us, now 117; of
// 128x64x64 147, now 49).
constexpr unsigned kHaloParts = 9;
template <class R, bool Many>
__global__ void __launch_bounds__(1024) kMarkHalo(const Grid<R> launch) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    if (L.ctl->stop) return;
    const std::uint32_t stamp = substepStamp(L);
    const std::uint32_t n = L.cand_count[w.begin];
    const std::uint32_t *list = L.cand_list + w.begin * kCandidatesPerBlock;
    for (std::uint32_t k = threadIdx.x; k < n; k += blockDim.x) {
        const std::uint32_t c = list[k];
        if (!inBounds(c, L.N, kSiteHalo)) continue;
        if (blockIdx.y == 0) L.halo_stamp[c] = stamp;
        for (std::uint32_t q = blockIdx.y; q < L.D; q += gridDim.y) {
            const std::size_t slot = static_cast<std::size_t>(q) * L.N + c;
            const std::uint32_t o = L.nbr_other[slot];
            if (!inBounds(o, L.N, kSiteHalo)) continue;
            L.halo_stamp[o] = stamp;
#pragma unroll 6
            for (std::uint32_t r = 0; r < L.D; ++r) {
                const std::uint32_t bd = L.nbr_bond[static_cast<std::size_t>(r) * L.N + o];
                if (bd != kNoBond && inBounds(bd, L.B, kSiteHalo)) L.late_tile_stamp[bd / kThreads] = stamp;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Sphere contact (LatticePhysics.hpp:1322-1428): candidates in slab, then node
// order, one contact at a time -- every contact moves the sphere the next one
// sees, so that chain is serial by definition. It runs on one warp of one
// CTA per lattice (kSpherePass); everything that does not depend on the
// sphere's changing state is done before it, on every SM (kSphereStage).
//
// A candidate's record: in pass 1 the sphere centre cannot move (only pass 2
// corrects positions), so the offset r, its length and unit normal, the gap,
// the inverse masses and the effective inverse mass along the normal are the
// stage's, with the reference's expressions, and the chain starts at the
// relative velocity. In pass 2 they are the node's position and masses.
// ---------------------------------------------------------------------------
template <class R> struct Staged {
    V3<R> p;       // position x0 + u (pass 2), or r = p - centre (pass 1)
    V3<R> normal;  // pass 1: normalized(r)
    R gap;         // pass 1: |r| - (sphere radius + node contact radius)
    R eff_n;       // pass 1: effective inverse mass along the normal
    R inm;         // 1 / mass
    R before;      // the node's kinetic energy as the pass reaches it
    Q4<R> u, v;    // u (w: inv_mass), v (w: mass)
};

// What one hit leaves: its candidate (for the write-back) and what it adds to
// the contact ledger's FP64 sums, in backend precision. The chain writes it to
// a log in shared memory and goes on, and the fold lanes widen and add it in
// log order (LatticePhysics.hpp:1354-1381), so the FP64 adds stay off the
// serial chain.
template <class R> struct ContactLog {
    R normal_imp[3], friction_imp[3];
    R lost;         // the node's kinetic energy before minus after
    unsigned flags; // kLogFriction: friction_imp applies; kLogImpulse: the sums do; candidate << 8
};
constexpr unsigned kLogFriction = 1, kLogImpulse = 2;

// Candidates a staging buffer of the contact pass holds, and its bytes: the
// records of a chunk of a slab's candidates and the log of its hits. Two
// buffers fit the shared memory a CTA may take.
template <class R> constexpr unsigned kSphereChunk = sizeof(R) == 4 ? kCandidatesPerBlock : 480;
template <class R>
constexpr unsigned kSphereChunkBytes = kSphereChunk<R> * static_cast<unsigned>(sizeof(Staged<R>) + sizeof(ContactLog<R>));

template <class R>
__device__ __forceinline__ void contactApply(V3<R> imp, V3<R> r, R inm, R ism, R iin, V3<R> &nv, V3<R> &sv, V3<R> &sw) {
    nv = nv + inm * imp;
    sv = sv - ism * imp;
    const V3<R> ti = -cross(r, imp);
    sw = sw + iin * ti;
}

// A candidate's geometry against the sphere's centre.
template <class R> struct ContactGeometry {
    V3<R> r, normal;
    R gap, eff_n; // |r| - (sphere radius + node contact radius); effective inverse mass along the normal
};
template <class R, class M>
__device__ __forceinline__ ContactGeometry<R> contactGeometry(M &m, V3<R> r, R cr, R inm, R ism, R iin) {
    ContactGeometry<R> g;
    g.r = r;
    const R sq = dot(r, r), distance = m.root(sq);
    g.normal = distance > R(1.0e-12) ? m.div(r, distance) : mk<R>(1, 0, 0); // normalized(r)
    const V3<R> rn = cross(r, g.normal);
    g.eff_n = inm + ism + iin * dot(rn, rn);
    g.gap = distance - cr;
    return g;
}

// A candidate against the current sphere state, carried through as if it were
// the next contact (LatticePhysics.hpp:1338-1386): 0 outside the contact gate
// (nothing happens), 1 a graze (past the gate, but no normal impulse and no
// position correction: it only raises the penetration record), 2 a hit, with
// the node's and the sphere's velocities after it.
template <class R> struct ContactTry {
    int kind;
    bool impulse;       // a normal impulse (else only a position correction)
    V3<R> nv, sv, sw;   // the node's velocity, the sphere's velocities
    ContactLog<R> log;
};
template <class R, class M>
__device__ __forceinline__ ContactTry<R> contactTry(M &m, const Settings<R> &S, const Sphere<R> &sp, V3<R> nv,
                                                    const ContactGeometry<R> &g, R mass, R inm, R before, R ism, R iin,
                                                    bool correct) {
    ContactTry<R> o;
    const V3<R> rel = nv - sp.velocity - cross(sp.angular, g.r);
    const R vn = dot(rel, g.normal);
    const bool outside = g.gap > maxR(S.c_margin, -vn * S.dt);
    const R restitution = -vn > S.c_threshold ? S.c_restitution : R(0);
    const R desired = g.gap > S.c_margin ? m.div(-g.gap, S.dt) : -restitution * minR(vn, R(0));
    const R ni = maxR(R(0), m.div(desired - vn, g.eff_n));
    o.impulse = ni > R(0);
    o.kind = outside ? 0 : (o.impulse || (correct && g.gap < -S.c_margin)) ? 2 : 1;
    o.nv = nv;
    o.sv = sp.velocity;
    o.sw = sp.angular;
    const V3<R> imp = ni * g.normal;
    if (!(o.kind == 2 && o.impulse)) return o;
    contactApply(imp, g.r, inm, ism, iin, o.nv, o.sv, o.sw);
    o.log.normal_imp[0] = imp.x;
    o.log.normal_imp[1] = imp.y;
    o.log.normal_imp[2] = imp.z;
    o.log.flags = kLogImpulse;
    const V3<R> after = o.nv - o.sv - cross(o.sw, g.r);
    const V3<R> tangent = after - dot(after, g.normal) * g.normal;
    // A tangential speed of at most 1e-12 takes no friction; a square below
    // 2^-80 is under it whatever its root's rounding.
    const R sq = dot(tangent, tangent);
    if (!(sq < R(0x1p-80))) {
        const R ts = m.root(sq);
        if (ts > R(1.0e-12)) {
            const V3<R> d = m.div(tangent, ts);
            const V3<R> rd = cross(g.r, d);
            const R stick = m.div(ts, inm + ism + iin * dot(rd, rd));
            const R fi = stick <= S.c_static * ni ? stick : minR(stick, S.c_dynamic * ni);
            const V3<R> fimp = -fi * d;
            contactApply(fimp, g.r, inm, ism, iin, o.nv, o.sv, o.sw);
            o.log.friction_imp[0] = fimp.x;
            o.log.friction_imp[1] = fimp.y;
            o.log.friction_imp[2] = fimp.z;
            o.log.flags = kLogImpulse | kLogFriction;
        }
    }
    o.log.lost = before - R(0.5) * mass * dot(o.nv, o.nv);
    return o;
}

// The position correction of a deep hit (second pass): the node's new
// displacement and the sphere centre's.
template <class R>
__device__ __forceinline__ R contactCorrect(const Settings<R> &S, const Sphere<R> &sp, const ContactGeometry<R> &g, R inm,
                                            R ism, Q4<R> &u, V3<R> &center) {
    const R corr = minR(-g.gap - S.c_margin, R(0.2) * maxR(S.c_node_radius, sp.radius * R(0.01)));
    const R sum = inm + ism;
    const V3<R> ns = (corr * inm / sum) * g.normal;
    const V3<R> ss = -((corr * ism / sum) * g.normal);
    const V3<R> un = xyz(u) + ns;
    u = Q4<R>{un.x, un.y, un.z, u.w};
    center = sp.center + ss;
    return corr;
}

// A candidate's node arrays after the pass: pass 1 predicts its position and
// keeps its approach speeds, pass 2 gives it the support planes' response.
template <class R>
__device__ __forceinline__ void contactSettle(const Dev<R> &L, const Settings<R> &S, int pass, std::uint32_t i,
                                              const Q4<R> &uq, const Q4<R> &vq) {
    if (pass == 1) {
        for (std::uint32_t p = 0; p < S.plane_count; ++p) L.approach[p * L.N + i] = dot(xyz(vq), S.planes[p].normal);
        const V3<R> un = xyz(uq) + S.dt * xyz(vq);
        L.u[i] = Q4<R>{un.x, un.y, un.z, uq.w};
        L.v[i] = vq;
    } else {
        V3<R> vel = xyz(vq);
        for (std::uint32_t p = 0; p < S.plane_count; ++p)
            if (L.engaged[p * L.N + i]) vel = supportVelocity(S.planes[p], vel, L.approach[p * L.N + i]);
        L.u[i] = uq;
        L.v[i] = Q4<R>{vel.x, vel.y, vel.z, vq.w};
    }
}

// The candidates of one slab, one CTA of the parts along y: their records, and
// their node arrays as the pass leaves them if the chain does not touch them
// (it rewrites the nodes it hits). The chain's CTA then only copies records,
// where it used to gather and divide for them: in the double lane, whose
// divisions one SM is slow at, a pass of 75 hits took 962 us, now 817.
constexpr unsigned kStageThreads = 128;
constexpr unsigned kStageParts = kCandidatesPerBlock / kStageThreads;
template <class R, bool Many>
__global__ void __launch_bounds__(kStageThreads) kSphereStage(const Grid<R> launch, Settings<R> S, int pass) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    __shared__ SharedDesc<R> desc;
    const Dev<R> &L = descriptorIn<R, Many>(launch, w, desc);
    if (L.ctl->stop) return;
    const std::uint32_t b = w.begin;
    const std::uint32_t k = blockIdx.y * kStageThreads + threadIdx.x;
    if (k >= L.cand_count[b]) return;
    const std::uint32_t i = L.cand_list[b * kCandidatesPerBlock + k];
    Staged<R> &out = L.cand_stage[b * kCandidatesPerBlock + k];
    if (!inBounds(i, L.N, kSiteCandidate)) {
        out = Staged<R>{}; // no mass: the chain passes it by
        return;
    }
    const Sphere<R> sp = *L.sphere;
    const R ism = R(1) / sp.mass, iin = R(1) / sp.inertia, cr = sp.radius + S.c_node_radius;
    Staged<R> c;
    c.u = L.u[i];
    c.v = L.v[i];
    const R mass = c.v.w;
    const V3<R> p = xyz(L.x0[i]) + xyz(c.u);
    c.inm = R(1) / mass;
    c.before = R(0.5) * mass * dot(xyz(c.v), xyz(c.v));
    if (pass == 1) {
        const V3<R> r = p - sp.center;
        const R distance = length(r);
        const V3<R> normal = normalized(r);
        const V3<R> rn = cross(r, normal);
        c.p = r;
        c.normal = normal;
        c.gap = distance - cr;
        c.eff_n = c.inm + ism + iin * dot(rn, rn);
    } else {
        c.p = p;
        c.normal = V3<R>{};
        c.gap = c.eff_n = R(0);
    }
    out = c;
    contactSettle(L, S, pass, i, c.u, c.v);
}

// The CTA takes nearly all of an SM's registers, so no other kernel's CTAs come
// to share the SM the chain runs on (with 256 threads the kernels beside it
// did: 1,460 against 966 us).
template <class R> constexpr unsigned kSphereThreads = sizeof(R) == 4 ? 512 : 320;
// Two staging buffers: the chain of one chunk of candidates runs on warp 0 while
// warp 1 folds the ledger log of the chunk before it and the other warps
// write back that chunk's hits and then copy the next chunk's records into the
// same buffer (after a barrier of their own and the fold's).

// The chain runs on warp 0, with every lane holding the same sphere state.
// Only a candidate that passes the contact gate changes anything. The lanes
// hold the next 32 candidates in registers and each carries its own through
// against the current state as if it were the next contact; the first lane
// that hits has done the serial chain's next step, its sphere state goes to
// every lane, and the lanes after it try again. The candidates before it were
// tested against exactly the state the serial order shows them, so the result
// is the serial chain's; the records (deepest penetration, largest
// correction) are maxima, which any order forms alike. What a hit costs is its
// own dependent arithmetic -- three divisions and a root, without branches in
// the float lane -- a ballot and six shuffles. Both passes of a substep, with
// what runs beside them: impact 256x128x128 (2,700 hits) 1,500 us, 1,902
// before; 128x64x64 471 us, 572 before.
// Slabs are disjoint sets of nodes: staging one slab's candidates, running
// another's chain and writing back a third's touch different nodes.
//
// The ledger's four FP64 sums (impulse x, y, z and dissipated energy) are four
// independent serial folds; lanes 0-3 of warp 1 run one each over the hit
// logs, slab after slab, in the order the chain wrote them.
template <class R, bool Many>
__global__ void __launch_bounds__(kSphereThreads<R>) kSpherePass(const Grid<R> launch, Settings<R> S, int pass) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    constexpr unsigned kChunk = kSphereChunk<R>;
    extern __shared__ __align__(16) unsigned char sphere_smem[];
    Staged<R> *stage_base = reinterpret_cast<Staged<R> *>(sphere_smem);
    ContactLog<R> *log_base = reinterpret_cast<ContactLog<R> *>(sphere_smem + 2 * kChunk * sizeof(Staged<R>));
    __shared__ unsigned log_count[2];
    __shared__ double folded[4];
    if (L.ctl->stop) return;
    const unsigned lane = threadIdx.x & 31U;
    const bool chain = threadIdx.x < 32;
    const bool fold = threadIdx.x >= 32 && threadIdx.x < 36;
    Sphere<R> sp = *L.sphere;
    const R ism = R(1) / sp.mass; // constant over the pass, as is the inertia
    const R iin = R(1) / sp.inertia;
    const R cr = sp.radius + S.c_node_radius;
    ContactAcc acc{};
    V3<R> c0{};
    R e0 = R(0), max_pen = R(0), max_corr = R(0);
    double sum = 0.0; // the fold lane's ledger sum
    if (chain) {
        if (pass == 1) sp.velocity = sp.velocity + S.dt * S.gravity; // the kicked sphere becomes the state
        acc = L.ctl->contact;
        max_pen = R(acc.max_penetration);
        max_corr = R(acc.max_correction);
        c0 = sp.center;
        e0 = R(0.5) * sp.mass * dot(sp.velocity, sp.velocity) + R(0.5) * sp.inertia * dot(sp.angular, sp.angular);
    } else if (fold) {
        const ContactAcc &a = L.ctl->contact;
        sum = lane == 0 ? a.impulse_x : lane == 1 ? a.impulse_y : lane == 2 ? a.impulse_z : a.dissipated;
    }

    // A chunk: candidates [off, off + count) of slab b (b == L.blocks: none).
    struct Chunk {
        std::uint32_t b, off, count;
    };
    auto chunkAt = [&](std::uint32_t b, std::uint32_t off) {
        for (; b < L.blocks; ++b, off = 0) {
            const std::uint32_t n = L.cand_count[b];
            if (off < n) return Chunk{b, off, n - off < kChunk ? n - off : kChunk};
        }
        return Chunk{b, 0U, 0U};
    };
    // Its records into a buffer, 16 bytes at a time, by threads [t0, t0 + nt).
    auto copyIn = [&](const Chunk &c, Staged<R> *st, unsigned t0, unsigned nt) {
        const uint4 *src = reinterpret_cast<const uint4 *>(L.cand_stage + c.b * kCandidatesPerBlock + c.off);
        uint4 *dst = reinterpret_cast<uint4 *>(st);
        const std::uint32_t words = c.count * static_cast<std::uint32_t>(sizeof(Staged<R>) / sizeof(uint4));
#pragma unroll 8
        for (std::uint32_t k = threadIdx.x - t0; k < words; k += nt) dst[k] = __ldcg(src + k);
    };
    // Its hits back to the node arrays, by threads [t0, t0 + nt).
    auto writeBack = [&](const Chunk &c, const Staged<R> *st, const ContactLog<R> *lg, unsigned hits, unsigned t0,
                         unsigned nt) {
        for (unsigned e = threadIdx.x - t0; e < hits; e += nt) {
            const std::uint32_t k = lg[e].flags >> 8;
            const std::uint32_t i = L.cand_list[c.b * kCandidatesPerBlock + c.off + k];
            if (inBounds(i, L.N, kSiteCandidate)) contactSettle(L, S, pass, i, st[k].u, st[k].v);
        }
    };
    // Its hit log into the fold lanes' sums (lane q: sum q).
    auto foldLog = [&](const ContactLog<R> *lg, unsigned n) {
        for (unsigned e = 0; e < n; ++e) {
            const unsigned flags = lg[e].flags;
            if (!(flags & kLogImpulse)) continue;
            if (lane < 3) {
                sum += static_cast<double>(lg[e].normal_imp[lane]);
                if (flags & kLogFriction) sum += static_cast<double>(lg[e].friction_imp[lane]);
            } else {
                sum += static_cast<double>(lg[e].lost);
            }
        }
    };
    // The serial chain over a chunk, on warp 0; its hits go to `lg`.
    auto runChain = [&](std::uint32_t n, Staged<R> *st, ContactLog<R> *lg, unsigned &logged) {
        unsigned hits = 0, impulses = 0;
        for (std::uint32_t k0 = 0; k0 < n; k0 += 32) {
            const std::uint32_t k = k0 + lane;
            Staged<R> c{};
            if (k < n) c = st[k];
            const bool movable = k < n && c.v.w > R(0);
            ContactGeometry<R> g{c.p, c.normal, c.gap, c.eff_n};
            unsigned from = 0;
            bool moved = pass == 2; // the sphere's centre since `g` was formed
            for (;;) {
                ContactTry<R> t{};
                if (movable && lane >= from) {
                    auto attempt = [&](auto &m) {
                        if (pass == 2 && moved) g = contactGeometry<R>(m, c.p - sp.center, cr, c.inm, ism, iin);
                        t = contactTry<R>(m, S, sp, xyz(c.v), g, c.v.w, c.inm, c.before, ism, iin, pass == 2);
                    };
                    if constexpr (std::is_same<R, float>::value) {
                        QuickMath quick;
                        attempt(quick);
                        if (!quick.good) {
                            PlainMath<R> plain;
                            attempt(plain);
                        }
                    } else {
                        PlainMath<R> plain;
                        attempt(plain);
                    }
                }
                const unsigned mask = __ballot_sync(0xffffffffU, t.kind == 2);
                const unsigned j = mask ? static_cast<unsigned>(__ffs(mask) - 1) : 32U;
                if (t.kind != 0 && lane <= j && -g.gap > max_pen) max_pen = -g.gap;
                if (mask == 0) break;
                const bool mine = lane == j;
                const bool impulse = __ballot_sync(0xffffffffU, mine && t.impulse) != 0;
                const int src = static_cast<int>(j);
                sp.velocity = {__shfl_sync(0xffffffffU, t.sv.x, src), __shfl_sync(0xffffffffU, t.sv.y, src),
                               __shfl_sync(0xffffffffU, t.sv.z, src)};
                sp.angular = {__shfl_sync(0xffffffffU, t.sw.x, src), __shfl_sync(0xffffffffU, t.sw.y, src),
                              __shfl_sync(0xffffffffU, t.sw.z, src)};
                if (mine) {
                    if (impulse) st[k].v = Q4<R>{t.nv.x, t.nv.y, t.nv.z, c.v.w};
                    else t.log.flags = 0;
                    t.log.flags |= k << 8;
                    lg[hits] = t.log;
                }
                ++hits;
                impulses += impulse ? 1U : 0U;
                moved = false;
                if (pass == 2) {
                    V3<R> center = sp.center;
                    const bool deep = mine && g.gap < -S.c_margin;
                    if (deep) {
                        Q4<R> uq = c.u;
                        const R corr = contactCorrect<R>(S, sp, g, c.inm, ism, uq, center);
                        st[k].u = uq;
                        if (corr > max_corr) max_corr = corr;
                    }
                    moved = __any_sync(0xffffffffU, deep);
                    if (moved)
                        sp.center = {__shfl_sync(0xffffffffU, center.x, src), __shfl_sync(0xffffffffU, center.y, src),
                                     __shfl_sync(0xffffffffU, center.z, src)};
                }
                from = j + 1;
                if (from == 32) break;
            }
        }
        acc.impulse_contacts += impulses;
        if (lane == 0) logged = hits;
    };
    Chunk cur = chunkAt(0, 0), prev{L.blocks, 0U, 0U};
    if (cur.b < L.blocks) copyIn(cur, stage_base, 0, blockDim.x);
    __syncthreads();
    unsigned cb = 0;
    while (cur.b < L.blocks) {
        const Chunk nxt = chunkAt(cur.b, cur.off + cur.count);
        const unsigned ob = cb ^ 1U;
        Staged<R> *const other = stage_base + ob * kChunk;
        ContactLog<R> *const other_log = log_base + ob * kChunk;
        if (chain) {
            runChain(cur.count, stage_base + cb * kChunk, log_base + cb * kChunk, log_count[cb]);
        } else if (threadIdx.x < 64) {
            if (fold && prev.b < L.blocks) foldLog(other_log, log_count[ob]);
        } else {
            if (prev.b < L.blocks) writeBack(prev, other, other_log, log_count[ob], 64, blockDim.x - 64);
            // The write-back reads the buffer the copy fills.
            asm volatile("bar.sync 1, %0;" ::"r"(blockDim.x - 64) : "memory");
            if (nxt.b < L.blocks) copyIn(nxt, other, 64, blockDim.x - 64);
        }
        __syncthreads();
        prev = cur;
        cur = nxt;
        cb = ob;
    }
    if (prev.b < L.blocks) {
        const unsigned ob = cb ^ 1U;
        if (fold) foldLog(log_base + ob * kChunk, log_count[ob]);
        writeBack(prev, stage_base + ob * kChunk, log_base + ob * kChunk, log_count[ob], 0, blockDim.x);
    }
    if (fold) folded[lane] = sum;
    if (chain) {
        for (int o = 16; o > 0; o >>= 1) {
            max_pen = maxR(max_pen, __shfl_xor_sync(0xffffffffU, max_pen, o));
            max_corr = maxR(max_corr, __shfl_xor_sync(0xffffffffU, max_corr, o));
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // The records only ever hold a widened R.
        if (max_pen > R(acc.max_penetration)) acc.max_penetration = static_cast<double>(max_pen);
        if (max_corr > R(acc.max_correction)) acc.max_correction = static_cast<double>(max_corr);
        acc.impulse_x = folded[0];
        acc.impulse_y = folded[1];
        acc.impulse_z = folded[2];
        acc.dissipated = folded[3];
        const R e1 = R(0.5) * sp.mass * dot(sp.velocity, sp.velocity) + R(0.5) * sp.inertia * dot(sp.angular, sp.angular);
        acc.dissipated += static_cast<double>(e0 - e1);
        const R shift = length(sp.center - c0);
        if (shift > R(acc.max_center_shift)) acc.max_center_shift = static_cast<double>(shift);
        *L.sphere = sp;
        L.ctl->contact = acc;
    }
}

// ---------------------------------------------------------------------------
// XPBD projection of one level (LatticePhysics.hpp:1132-1168), one bond per
// thread over the level's contiguous storage range [begin, end).
//
// Support (LatticePhysics.hpp:1255-1261) rides on the sweep: the reference
// projects every node out of the support planes after the whole sweep; here a
// node is projected by the thread that ran its last bond of the sweep (the
// record's last-of flags), right after that bond. Nothing later in the sweep
// touches the node and the projection reads only the node itself, so the
// result is the reference's, and the separate pass over the nodes is gone. A
// broken or degenerate last bond still carries its nodes' projection.
// ---------------------------------------------------------------------------
template <class R>
__device__ __forceinline__ bool supportProject(const Dev<R> &L, const Settings<R> &S, std::uint32_t i, V3<R> &u) {
    const V3<R> x0 = xyz(L.x0[i]);
    bool projected = false;
    for (std::uint32_t p = 0; p < S.plane_count; ++p) {
        bool here = false;
        const R depth = projectSupport(S.planes[p], x0, u, L.approach[p * L.N + i], S.dt, here);
        if (depth > R(0)) L.engaged[p * L.N + i] = 1;
        projected = projected || here;
    }
    return projected;
}

// One bond per thread. Float: 256-thread CTAs, six to an SM (sweep of
// 256x128x128, ms per substep: six 2.47, four or five 2.58, eight, spilling at
// 32 registers, 3.02; two bonds a thread 2.81. A level too small for all the
// SMs waits for latency, not for work: 128, 64 and 32 threads measured the same
// there, and 64 and 32 slower on large levels). Double: an SM has two FP64
// lanes, so what bounds a level is its busiest SM's bonds, and a level is dealt
// out in single warps; no spilling at up to 80 registers. Sweep of 48x24x40 in
// 27 levels of 59 CTAs of 256 threads, us per substep: 1,302 at the 40
// registers of the float lane's six CTAs, 1,176 without spills, 1,010, 916 and
// 864 in 128, 64 and 32 threads, 818 with the rest positions and the compliance
// term fetched ahead (bondAhead). 128x64x64: 3,880 in 256 threads, 3,627 in 32.
template <class R> constexpr unsigned kSolveThreads = sizeof(R) == 8 ? 32U : static_cast<unsigned>(kThreads);
template <class R> constexpr unsigned kSolveBlocks = sizeof(R) == 8 ? 24U : 6U;

// A sweep level (programmatic dependent launch, startAfterPrevious) loads what
// no earlier kernel of the substep writes -- records, geometry, multipliers,
// plastic extension, the double lane's rest positions, the stop flag -- before
// it waits for the previous grid; at most two levels overlap.

// The projection of one live bond (LatticePhysics.hpp:1132-1168): its unit
// direction and the multiplier's change, with the reference's expressions;
// alpha is the compliance over dt^2. Returns whether the nodes move (a
// degenerate bond leaves them).
template <class R, bool Direct, bool Plastic>
__device__ __forceinline__ bool bondStep(V3<R> x0a, V3<R> x0b, V3<R> ua, V3<R> ub, V3<R> edge, R rsm, R original,
                                         R alpha, R wa, R wb, R lambda, R plastic, V3<R> &dir, R &dl) {
    const V3<R> delta = Direct ? (x0b + ub) - (x0a + ua) : edge + (ub - ua);
    const R cl = length(delta);
    if (!(cl > R(1.0e-12))) return false;
    const R rest = Plastic ? original + plastic : original;
    R constraint;
    if (Direct) {
        constraint = cl - rest;
    } else {
        const V3<R> du = ub - ua;
        const R num = rsm + R(2) * dot(edge, du) + dot(du, du);
        constraint = (Plastic ? num - plastic * (rest + original) : num) / (cl + rest);
    }
    dir = delta / cl;
    dl = (-constraint - alpha * lambda) / (wa + wb + alpha);
    return true;
}
// The float lane's step where an operand is outside the branch-free range.
struct FloatStep {
    V3<float> dir;
    float dl;
    bool moves;
};
template <bool Plastic>
__device__ __noinline__ FloatStep floatStepAnywhere(V3<float> ua, V3<float> ub, V3<float> edge, float rsm,
                                                    float original, float compliance, float wa, float wb, float lambda,
                                                    float plastic, float dt) {
    FloatStep s{};
    s.moves = bondStep<float, false, Plastic>(V3<float>{}, V3<float>{}, ua, ub, edge, rsm, original,
                                              compliance / (dt * dt), wa, wb, lambda, plastic, s.dir, s.dl);
    return s;
}
// The float lane's step. The same values from the branch-free quotients: the
// six divisions and the root of a bond took most of a round (a beam of 135
// nodes swept in one CTA: 0.78 us a level with them, 0.40 without).
template <bool Plastic>
__device__ __forceinline__ FloatStep floatStep(const Settings<float> &S, V3<float> ua, V3<float> ub, V3<float> edge,
                                               float rsm, float original, float compliance, float wa, float wb,
                                               float lambda, float plastic) {
    const V3<float> du = ub - ua;
    const V3<float> delta = edge + du;
    const float sq = dot(delta, delta);
    const float cl = rootNearest(sq);
    const float ycl = recipNearest(cl);
    const float rest = Plastic ? original + plastic : original;
    const float raw = rsm + 2.0F * dot(edge, du) + dot(du, du);
    const float num = Plastic ? raw - plastic * (rest + original) : raw;
    const float den = cl + rest;
    const float alpha = quotient(compliance, S.dt_sq, S.dt_sq_recip);
    const float w = wa + wb + alpha;
    const float pull = -quotient(num, den, recipNearest(den)) - alpha * lambda;
    FloatStep s;
    s.dl = quotient(pull, w, recipNearest(w));
    s.dir = {quotient(delta.x, cl, ycl), quotient(delta.y, cl, ycl), quotient(delta.z, cl, ycl)};
    s.moves = true; // a square of 2^-78 or more: the length is above 1e-12
    const std::uint32_t least =
        __vimin3_u32(__vimin3_u32(dividendKey(delta.x), dividendKey(delta.y), dividendKey(delta.z)), dividendKey(num),
                     min(dividendKey(pull), dividendKey(compliance)));
    // An infinite or NaN operand leaves a NaN or an infinity in s.dl or w.
    if (!(rootOk(sq) && sq >= 0x1p-78F && divisorOk(den) && divisorOk(w) && least >= kDividendLeast && fabsf(s.dl) < 0x1p100F))
        s = floatStepAnywhere<Plastic>(ua, ub, edge, rsm, original, compliance, wa, wb, lambda, plastic, S.dt);
    return s;
}

// What the double lane's step needs and no kernel of the sweep writes, for a
// level to fetch and form before it waits for the level ahead of it: the rest
// positions and the compliance over dt^2 (the float lane works on differences
// and divides branch-free, and takes neither).
template <class R> struct BondAhead {
    V3<R> x0a, x0b;
    R alpha;
};
template <class R, bool Direct>
__device__ __forceinline__ BondAhead<R> bondAhead(const Dev<R> &L, const Settings<R> &S, const BondRec<R> &rec,
                                                  R compliance) {
    BondAhead<R> h{};
    if (Direct && !(rec.a & kDeadBit)) {
        h.x0a = xyz(L.x0[endA(rec)]);
        h.x0b = xyz(L.x0[endB(rec)]);
        h.alpha = compliance / (S.dt * S.dt);
    }
    return h;
}

// Where a sweep keeps its nodes' positions: the lattice's array in global
// memory (through L2, which every SM shares), or a CTA's shared memory
// (StagedNodes, below).
template <class R> struct GlobalNodes {
    Q4<R> *u;
    __device__ __forceinline__ Q4<R> load(std::uint32_t i) const { return ldShared(u + i); }
    __device__ __forceinline__ void store(std::uint32_t i, const Q4<R> &q) const { u[i] = q; }
};

// The support projection of a node after its last bond of the sweep.
template <class R, class Nodes>
__device__ __forceinline__ void supportLast(const Dev<R> &L, const Settings<R> &S, const Nodes &nodes, std::uint32_t i,
                                            bool have, Q4<R> &q, bool &write) {
    if (!have) q = nodes.load(i);
    V3<R> u = xyz(q);
    if (supportProject(L, S, i, u)) {
        q = Q4<R>{u.x, u.y, u.z, q.w};
        write = true;
    }
}
// A bond from its record, geometry, multiplier and plastic extension: its nodes
// gathered, the projection, then the support projection of the nodes whose
// last bond of the sweep it is, then the write-back of what moved. The
// multiplier is stored in every iteration: a bond that is degenerate in a
// substep's first one, which would start it from zero, goes on from the
// substep before (LatticePhysics.hpp:1133-1168). A degenerate bond leaves its
// nodes; a broken or degenerate last bond still carries their support
// projection.
template <class R, bool Direct, bool Plastic, bool Support, class Nodes>
__device__ __forceinline__ void solveBond(const Dev<R> &L, const Settings<R> &S, const Nodes &nodes, R *lambdas,
                                          std::uint32_t d, const BondRec<R> &rec, const Q4<R> &g, R lambda, R plastic,
                                          const BondAhead<R> &ahead) {
    const std::uint32_t a = endA(rec), b = endB(rec);
    const bool live = !(rec.a & kDeadBit);
    bool write_a = false, write_b = false;
    Q4<R> qa{}, qb{};
    if (live) {
        qa = nodes.load(a);
        qb = nodes.load(b);
        const V3<R> ua = xyz(qa), ub = xyz(qb), edge{g.x, g.y, g.z};
        const R wa = qa.w, wb = qb.w;
        V3<R> dir;
        R dl;
        bool moves;
        if constexpr (std::is_same<R, float>::value && !Direct) {
            const FloatStep s = floatStep<Plastic>(S, ua, ub, edge, rec.rsm, rec.rest, g.w, wa, wb, lambda, plastic);
            dir = s.dir;
            dl = s.dl;
            moves = s.moves;
        } else {
            moves = bondStep<R, Direct, Plastic>(ahead.x0a, ahead.x0b, ua, ub, edge, rec.rsm, rec.rest, ahead.alpha, wa,
                                                 wb, lambda, plastic, dir, dl);
        }
        if (moves) {
            __stcs(lambdas + d, lambda + dl);
            const V3<R> na = ua - (wa * dl) * dir;
            const V3<R> nb = ub + (wb * dl) * dir;
            qa = Q4<R>{na.x, na.y, na.z, wa};
            qb = Q4<R>{nb.x, nb.y, nb.z, wb};
            write_a = write_b = true;
        }
    }
    if (Support && ((rec.a & kLastABit) || (rec.b & kLastBBit))) {
        if (rec.a & kLastABit) supportLast(L, S, nodes, a, live, qa, write_a);
        if (rec.b & kLastBBit) supportLast(L, S, nodes, b, live, qb, write_b);
    }
    if (write_a) nodes.store(a, qa);
    if (write_b) nodes.store(b, qb);
}

template <class R, bool Many, bool Direct, bool First, bool Plastic, bool Support>
__global__ void __launch_bounds__(kSolveThreads<R>, kSolveBlocks<R>) kSolve(const Grid<R> launch, Settings<R> S) {
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    const std::uint32_t at = w.begin + threadIdx.x;
    BondRec<R> rec{};
    Q4<R> geo{};
    R lam = R(0), pl = R(0);
    // Everything that no kernel since the last end sample has written.
    if (at < w.end) {
        rec = ldStream(L.rec + at);
        geo = ldStream(L.geo + at);
        if (!First) lam = __ldcs(L.lambda + at);
        if (Plastic) pl = L.plastic[at].x;
    }
    const bool solve = at < w.end && endsInBounds(rec, L.N, kSiteSolve);
    BondAhead<R> ahead{};
    if (solve) ahead = bondAhead<R, Direct>(L, S, rec, geo.w);
    const unsigned stop = L.ctl->stop;
    waitPreviousGrid();
    allowNextGrid();
    if (stop) return;
    const GlobalNodes<R> nodes{L.u};
    if (solve) solveBond<R, Direct, Plastic, Support>(L, S, nodes, L.lambda, at, rec, geo, lam, pl, ahead);
}

// The whole sweep of one lattice in one CTA: every iteration, every level in
// order with a barrier between levels, then the isolated nodes' support. Its
// nodes stay in L2 (and the SM's L1) across all its levels instead of being
// streamed from HBM again at every level launch; the arithmetic and the
// per-node order are those of the level launches.
//
// What bounds it is one CTA's chain of L2 round trips, so it is for batches
// whose lattices outnumber the SMs several times, and only the autotuner
// chooses it (CTA size and reach). Sweep per substep, level launches and this
// (ms): 600 lattices of 8 to 48 a side 6.62 and 6.32, 2,000 22.6 and 21.9,
// 4,096 47.5 and 46.0 (1,024 threads, up to 2^18 bonds); 1,000 of 16 to 24 a
// side 4.24 and 4.02; of 8 to 12 a side, 300 0.24 and 0.26, 4,000 2.26 and 2.32
// (512 threads); 128 of 8 to 48 1.46 and 4.01.
constexpr unsigned kSweepThreads = 512; // the default shape
constexpr std::uint32_t kMaxFusedLevels = 1024;

template <class R, bool Support>
__device__ __forceinline__ void supportIsolatedInCta(const Dev<R> &L, const Settings<R> &S) {
    if (!Support || !L.isolated_count) return;
    __syncthreads();
    for (std::uint32_t t = threadIdx.x; t < L.isolated_count; t += blockDim.x) {
        const std::uint32_t i = L.isolated[t];
        if (!inBounds(i, L.N, kSiteIsolated)) continue;
        const Q4<R> uq = L.u[i];
        V3<R> u = xyz(uq);
        if (supportProject(L, S, i, u)) L.u[i] = Q4<R>{u.x, u.y, u.z, uq.w};
    }
}

template <class R, bool Direct, bool Plastic, bool Support, unsigned T>
__global__ void __launch_bounds__(T, T >= 1024 ? 1 : 2) kSweepLattice(const Grid<R> launch, Settings<R> S) {
    startAfterPrevious();
    // The lattice's descriptor, copied once into shared memory: its fields
    // are read throughout the sweep, and shared memory is never written by
    // the sweep's global stores, so the compiler may keep them as it likes.
    __shared__ __align__(16) unsigned char desc[sizeof(Dev<R>)];
    {
        const Work w = item<true>(launch);
        const unsigned *src = reinterpret_cast<const unsigned *>(launch.table + w.lattice);
        unsigned *dst = reinterpret_cast<unsigned *>(desc);
        for (unsigned k = threadIdx.x; k < sizeof(Dev<R>) / sizeof(unsigned); k += blockDim.x) dst[k] = src[k];
    }
    __syncthreads();
    const Dev<R> &L = *reinterpret_cast<const Dev<R> *>(desc);
    if (L.ctl->stop) return;
    const GlobalNodes<R> nodes{L.u};
    const unsigned I = S.iterations;
    // One bond per thread per round; the rounds of the whole sweep in order
    // (iteration, level, base). The next round's streamed data (record,
    // geometry, multiplier, plastic extension: nothing the node updates
    // touch) is loaded before the current round's node gathers, so two
    // rounds' memory traffic is in flight. A round's multipliers are written
    // one iteration before the round reads them, except in a sweep of one
    // round per iteration, whose next round is itself: there they are loaded
    // after the write.
    struct Round {
        unsigned it;
        std::uint32_t lv, base;
    };
    struct Streamed {
        BondRec<R> rec;
        Q4<R> geo;
        R lam, pl;
    };
    auto advance = [&](Round &r) {
        r.base += T;
        if (r.base < L.level_begin[r.lv + 1]) return true;
        if (++r.lv == L.level_count) {
            r.lv = 0;
            if (++r.it == I) return false;
        }
        r.base = L.level_begin[r.lv];
        return true;
    };
    const bool self_next = L.level_count == 1 && L.level_begin[1] - L.level_begin[0] <= T;
    auto load = [&](const Round &r, Streamed &x) {
        const std::uint32_t d = r.base + threadIdx.x;
        if (d < L.level_begin[r.lv + 1]) {
            x.rec = ldStream(L.rec + d);
            x.geo = ldStream(L.geo + d);
            x.lam = (r.it == 0 || self_next) ? R(0) : __ldcs(L.lambda + d);
            x.pl = Plastic ? L.plastic[d].x : R(0);
        }
    };
    Round cur{0, 0, L.level_begin[0]};
    Streamed now{}, next{};
    load(cur, now);
    for (;;) {
        Round nxt = cur;
        const bool more = advance(nxt);
        if (more) load(nxt, next);
        const std::uint32_t end = L.level_begin[cur.lv + 1];
        const std::uint32_t d = cur.base + threadIdx.x;
        if (d < end && endsInBounds(now.rec, L.N, kSiteSolve)) {
            if (self_next && cur.it != 0) now.lam = __ldcs(L.lambda + d);
            solveBond<R, Direct, Plastic, Support>(L, S, nodes, L.lambda, d, now.rec, now.geo, now.lam, now.pl,
                                                   bondAhead<R, Direct>(L, S, now.rec, now.geo.w));
        }
        if (!more) {
            supportIsolatedInCta<R, Support>(L, S);
            break;
        }
        if (nxt.lv != cur.lv || nxt.it != cur.it) {
            __syncthreads();
            if (nxt.it != cur.it) {
                supportIsolatedInCta<R, Support>(L, S);
                __syncthreads();
            }
        }
        cur = nxt;
        now = next;
    }
}

// The whole sweep of a small lattice in one CTA (float lane), its positions in
// shared memory for every iteration and level: one thread for every bond of
// the widest level, a CTA barrier between levels, the next level's records
// fetched while this one is solved (two buffers, used in turn: a register
// that a load is still filling is never copied, which would wait for the
// load). The arithmetic and the per-node order are those of the level launches.
//
// What bounds it: a level is one dependent chain (gather, solve, write,
// barrier), and its warps share one SM's issue slots. Spreading a lattice over
// a thread-block cluster was measured and is not kept: making a level's writes
// visible across the cluster costs 0.43 us (the fence 330 cycles of it), as
// much as the launch of a level saves.
constexpr std::uint32_t kStagedMaxNodes = 14336; // the launch shape's largest value; capped at kStagedNodes
constexpr std::uint32_t kStagedNodes = 14080;    // 220 KiB, the level table and the descriptor beside
constexpr std::uint32_t kStagedLevels = 512;
constexpr unsigned kStagedThreads = 1024;        // at most; 64 registers a thread

struct StagedNodes {
    Q4<float> *u; // shared memory
    __device__ __forceinline__ Q4<float> load(std::uint32_t i) const { return u[i]; }
    __device__ __forceinline__ void store(std::uint32_t i, const Q4<float> &q) const { u[i] = q; }
};

template <bool Plastic, bool Support>
__global__ void __launch_bounds__(kStagedThreads, 1)
kSweepStaged(const __grid_constant__ Grid<float> launch, const __grid_constant__ Settings<float> S) {
    extern __shared__ __align__(16) unsigned char staged_smem[];
    __shared__ SharedDesc<float> desc;
    const unsigned T = blockDim.x, t = threadIdx.x;
    // The lattice's descriptor in shared memory, read from there as needed:
    // one lattice's comes from the launch's own parameters.
    {
        const unsigned *src = reinterpret_cast<const unsigned *>(
            launch.list ? launch.table + launch.list[blockIdx.x].lattice : &launch.one);
        unsigned *dst = reinterpret_cast<unsigned *>(desc.bytes);
        for (unsigned k = t; k < sizeof(Dev<float>) / sizeof(unsigned); k += T) dst[k] = src[k];
        __syncthreads();
    }
    startAfterPrevious();
    const Dev<float> &L = *reinterpret_cast<const Dev<float> *>(desc.bytes);
    if (L.ctl->stop) return;
    const std::uint32_t N = L.N, levels = L.level_count, I = S.iterations;
    Q4<float> *own = reinterpret_cast<Q4<float> *>(staged_smem);
    std::uint32_t *begin = reinterpret_cast<std::uint32_t *>(staged_smem + sizeof(Q4<float>) * N);
    Q4<float> *const u = L.u;
#pragma unroll 4
    for (std::uint32_t k = t; k < N; k += T) own[k] = ldShared(u + k);
    for (std::uint32_t k = t; k <= levels; k += T) begin[k] = L.level_begin[k];
    const StagedNodes nodes{own};
    const BondRec<float> *const recs = L.rec;
    const Q4<float> *const geos = L.geo;
    float *const lambdas = L.lambda;
    __syncthreads();

    // A bond is one thread's for the whole sweep, which writes its multiplier
    // an iteration before reading it; with a single level that is the step
    // before, so it is then loaded after the write.
    const bool late_lambda = levels == 1;
    struct Streamed {
        BondRec<float> rec;
        Q4<float> geo;
        float lam, pl;
        std::uint32_t d; // the bond, or kNoBond
    };
    auto fetch = [&](std::uint32_t it, std::uint32_t lv, Streamed &x) {
        const std::uint32_t d = begin[lv] + t;
        const bool has = it < I && d < begin[lv + 1];
        x.d = has ? d : kNoBond;
        if (has) {
            x.rec = ldStream(recs + d);
            x.geo = ldStream(geos + d);
            x.lam = (it == 0 || late_lambda) ? 0.0F : __ldcs(lambdas + d);
            x.pl = Plastic ? L.plastic[d].x : 0.0F;
        }
    };
    std::uint32_t it = 0, lv = 0;
    // One level; false after the last one of the sweep.
    auto level = [&](Streamed &now, Streamed &next) {
        std::uint32_t next_it = it, next_lv = lv + 1;
        if (next_lv == levels) {
            next_lv = 0;
            ++next_it;
        }
        fetch(next_it, next_lv, next);
        if (now.d != kNoBond && endsInBounds(now.rec, N, kSiteSolve)) {
            if (late_lambda && it != 0) now.lam = __ldcs(lambdas + now.d);
            solveBond<float, false, Plastic, Support>(L, S, nodes, lambdas, now.d, now.rec, now.geo, now.lam, now.pl,
                                                      BondAhead<float>{});
        }
        if (Support && next_it != it) {
            // Nodes without bonds, each iteration by the same thread; no
            // bond's solve touches them.
            for (std::uint32_t k = t; k < L.isolated_count; k += T) {
                const std::uint32_t i = L.isolated[k];
                if (!inBounds(i, N, kSiteIsolated)) continue;
                const Q4<float> uq = nodes.load(i);
                V3<float> p = xyz(uq);
                if (supportProject(L, S, i, p)) nodes.store(i, Q4<float>{p.x, p.y, p.z, uq.w});
            }
        }
        __syncthreads();
        it = next_it;
        lv = next_lv;
        return it < I;
    };
    Streamed x0{}, x1{};
    fetch(0, 0, x0);
    while (level(x0, x1) && level(x1, x0)) {
    }
    for (std::uint32_t k = t; k < N; k += T) u[k] = own[k];
}

// Radial pair damping of one level (LatticePhysics.hpp:1170-1184).
template <class R, bool Many, bool Direct>
__global__ void __launch_bounds__(kThreads) kDamp(const Grid<R> launch, R fraction) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    if (L.ctl->stop) return;
    // Items are sweep levels' ranges: any length, strided over the CTA.
    for (std::uint32_t d = w.begin + threadIdx.x; d < w.end; d += blockDim.x) {
        const BondRec<R> rec = L.rec[d];
        if ((rec.a & kDeadBit) || !endsInBounds(rec, L.N, kSiteDamp)) continue;
        const std::uint32_t a = endA(rec), b = endB(rec);
        const Q4<R> va = L.v[a], vb = L.v[b];
        const R ma = va.w, mb = vb.w;
        if (ma <= R(0) || mb <= R(0)) continue;
        const Q4<R> g = L.geo[d];
        const V3<R> n = normalized(bondVector<R, Direct>(viewOf(L), a, b, V3<R>{g.x, g.y, g.z}));
        const R rel = dot(xyz(vb) - xyz(va), n);
        const R im = R(1) / ma + R(1) / mb;
        const R impulse = -fraction * rel / im;
        const V3<R> na = xyz(va) - (impulse / ma) * n;
        const V3<R> nb = xyz(vb) + (impulse / mb) * n;
        L.v[a] = Q4<R>{na.x, na.y, na.z, ma};
        L.v[b] = Q4<R>{nb.x, nb.y, nb.z, mb};
    }
}

// Support projection of the nodes that have no bond to carry it (isolated
// nodes), after a sweep (LatticePhysics.hpp:1255-1261).
template <class R, bool Many>
__global__ void __launch_bounds__(kThreads) kSupportIsolated(const Grid<R> launch, Settings<R> S) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    if (L.ctl->stop) return;
    const std::uint32_t t = w.begin + threadIdx.x;
    if (t >= w.end) return;
    const std::uint32_t i = L.isolated[t];
    if (!inBounds(i, L.N, kSiteIsolated)) return;
    const Q4<R> uq = L.u[i];
    V3<R> u = xyz(uq);
    // Written back whenever a projection ran, even by a zero distance, so the
    // sign of a zero component is whatever the projection made it.
    if (supportProject(L, S, i, u)) L.u[i] = Q4<R>{u.x, u.y, u.z, uq.w};
}

// Velocity from accepted positions, then the support response of
// non-candidates when no damping sweep follows (LatticePhysics.hpp:1725-1730).
template <class R, bool Many>
__global__ void __launch_bounds__(kThreads) kVelocity(const Grid<R> launch, Settings<R> S, int respond) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    __shared__ SharedDesc<R> desc;
    const Dev<R> &L = descriptorIn<R, Many>(launch, w, desc);
    if (L.ctl->stop) return;
    const std::uint32_t i = w.begin + threadIdx.x;
    if (i >= w.end) return;
    const Q4<R> vq = L.v[i];
    V3<R> vel = (xyz(L.u[i]) - xyz(L.up[i])) / S.dt;
    if (respond && !L.candidate[i])
        for (std::uint32_t p = 0; p < S.plane_count; ++p)
            if (L.engaged[p * L.N + i]) vel = supportVelocity(S.planes[p], vel, L.approach[p * L.N + i]);
    L.v[i] = Q4<R>{vel.x, vel.y, vel.z, vq.w};
}

// Support response of non-candidates after the damping sweep (CpuLatticeBackend.cpp:414-415).
template <class R, bool Many>
__global__ void __launch_bounds__(kThreads) kSupportVelocity(const Grid<R> launch, Settings<R> S) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    if (L.ctl->stop) return;
    const std::uint32_t i = w.begin + threadIdx.x;
    if (i >= w.end || L.candidate[i]) return;
    const Q4<R> vq = L.v[i];
    V3<R> vel = xyz(vq);
    for (std::uint32_t p = 0; p < S.plane_count; ++p)
        if (L.engaged[p * L.N + i]) vel = supportVelocity(S.planes[p], vel, L.approach[p * L.N + i]);
    L.v[i] = Q4<R>{vel.x, vel.y, vel.z, vq.w};
}

// ---------------------------------------------------------------------------
// End-of-substep sample, plastic return and failure (LatticePhysics.hpp:1018-1114).
// One thread per bond in schedule order; a CTA is one "tile" of 256 bonds.
// The reference folds its FP64 ledgers one bond at a time in bond order
// (CpuLatticeBackend.cpp:446-478). Here every reduction has a fixed order that
// depends on the bond order only, never on thread timing: plastic work is
// summed per tile by a fixed shuffle tree and the tiles in index order; broken
// bonds and damage-record candidates are flagged one bit per bond and listed
// in bond order by kTileCounts/kEventScan/kTopScan/kEmitEvents.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned floatBits(float x) { return __float_as_uint(x); }

// Sum over a warp in a fixed order (lane 0 holds the result).
__device__ __forceinline__ double warpSumFixed(double x) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffU, x, o);
    return x;
}

// One tile, by the whole CTA.
template <class R, bool Direct, bool Plastic>
__device__ __forceinline__ void endSampleTile(const Dev<R> &L, const Settings<R> &S, const Work &w, double *tile_work) {
    const std::uint32_t j = w.begin + threadIdx.x; // storage index; items start on multiples of 256
    double plastic_work = 0.0;
    unsigned peaks[4] = {0, 0, 0, 0};
    if (j < w.end) {
        // Every per-bond array is loaded at once, ahead of the liveness test
        // and of the node gathers that wait on the record: one trip to memory
        // for all of them rather than one after another (single-use data,
        // streamed past L2 so the node arrays stay there).
        const BondRec<R> rec = ldStream(L.rec + j);
        const Q4<R> g = ldStream(L.geo + j);
        Q4<R> pv = L.prev[j];
        const Q4<R> t4 = ldStream(L.thr4 + j);
        const Q2<R> t2 = L.thr2[j];
        Q2<R> pl = Plastic ? L.plastic[j] : Q2<R>{R(0), R(0)};
        if (!(rec.a & kDeadBit) && endsInBounds(rec, L.N, kSiteEndSample)) {
            const std::uint32_t a = endA(rec), b = endB(rec);
            const V3<R> edge{g.x, g.y, g.z};
            float plastic_stretch = 0.0F;
            R pext = R(0);
            // The bond's current length, used by the plastic return, the
            // sample and the stored energy of a failure alike.
            const BondSample<R> sample = sampleOf<R, Direct>(viewOf(L), a, b, rec, edge);
            const R len = sample.len, t = sample.t, c = sample.c, s = sample.s;
            if (Plastic) {
                pext = pl.x;
                if (S.yield_stretch > R(0)) {
                    const R elastic = len - rec.rest - pl.x;
                    const R magnitude = absR(elastic);
                    const R h = S.hardening;
                    const R yield = S.yield_stretch * rec.rest + h * pl.y;
                    if (magnitude > yield) {
                        const R inc = (magnitude - yield) / (R(1) + h);
                        pl.x = pl.x + (elastic < R(0) ? -inc : inc);
                        pl.y = pl.y + inc;
                        L.plastic[j] = pl;
                        pext = pl.x;
                        if (g.w > R(0)) {
                            const R yield_end = yield + h * inc;
                            plastic_work = static_cast<double>(R(0.5) * (yield + yield_end) * inc / g.w);
                        }
                    }
                    plastic_stretch = static_cast<float>(absR(pl.x) / rec.rest);
                }
            }
            const R pt = maxR(R(0), maxR(pv.x, t));
            const R pc = maxR(R(0), maxR(pv.y, c));
            const R ps = maxR(R(0), maxR(pv.z, s));
            pv.x = maxR(R(0), t);
            pv.y = maxR(R(0), c);
            pv.z = maxR(R(0), s);
            const R dtn = damageProgress(pt, t4.x, t4.y);
            const R dcp = damageProgress(pc, t4.z, t4.w);
            const R dsh = damageProgress(ps, t2.x, t2.y);
            R damage = dtn;
            std::uint8_t mode = 1;
            if (dcp > damage) { damage = dcp; mode = 2; }
            if (dsh > damage) { damage = dsh; mode = 3; }
            if (damage > pv.w) {
                pv.w = damage;
                L.mode[j] = mode;
            }
            L.prev[j] = pv;
            const float dmg = static_cast<float>(pv.w);
            if (pv.w >= R(1)) {
                const std::uint32_t js = L.dev2sched[j];
                const R cc = g.w;
                R energy = R(0);
                if (!(cc <= R(0))) {
                    const R ext = len - rec.rest - pext;
                    energy = R(0.5) * ext * ext / cc;
                }
                L.rec[j].a = rec.a | kDeadBit;
                // Both slots keep their weight, sign-flipped: dead for the
                // strain, still there for a sheet's rest geometry.
                L.nbr[L.slot_a[j]].w = -absR(L.nbr[L.slot_a[j]].w);
                L.nbr[L.slot_b[j]].w = -absR(L.nbr[L.slot_b[j]].w);
                L.ev_removed[js] = static_cast<double>(energy);
                L.ev_ends[js] = make_uint2(a, b);
                atomicOr(L.ev_bits + (js >> 5), 1U << (js & 31U));
            }
            // A bond can raise the run's damage maximum only if it exceeds the
            // maximum as the substep began (CpuLatticeBackend.cpp:462-465);
            // the bound is a float (kLedger), so no thread forms an FP64 one.
            if (dmg > L.ctl->damage_floor) {
                const std::uint32_t js = L.dev2sched[j];
                L.ev_damage[js] = dmg;
                atomicOr(L.dmg_bits + (js >> 5), 1U << (js & 31U));
            }
            // Peaks are non-negative, so their bit patterns order as the values do.
            peaks[0] = floatBits(static_cast<float>(pt));
            peaks[1] = floatBits(static_cast<float>(pc));
            peaks[2] = floatBits(static_cast<float>(ps));
            if (Plastic && S.yield_stretch > R(0)) peaks[3] = floatBits(plastic_stretch);
        }
    }
    // The run's peaks: a warp asks for the atomic only above what it reads
    // there (they only grow, so a stale read asks once too often at most).
    unsigned *const records[4] = {&L.ctl->max_t, &L.ctl->max_c, &L.ctl->max_s, &L.ctl->max_plastic};
    for (int q = 0; q < (Plastic ? 4 : 3); ++q) {
        const unsigned top = __reduce_max_sync(0xffffffffU, peaks[q]);
        if ((threadIdx.x & 31) == 0 && top > *records[q]) atomicMax(records[q], top);
    }
    if (!Plastic) return;
    // Fixed-order sums of the plastic work; a sum of zeros is +0 whichever
    // way it is formed, so all-zero tiles skip the FP64 adds.
    if (!__syncthreads_or(plastic_work != 0.0)) {
        if (threadIdx.x == 0) L.tile_plastic[w.begin / kThreads] = 0.0;
        return;
    }
    const double warp_work = warpSumFixed(plastic_work);
    if ((threadIdx.x & 31) == 0) tile_work[threadIdx.x / 32] = warp_work;
    __syncthreads();
    if (threadIdx.x == 0) {
        double wsum = 0.0;
        for (int q = 0; q < kThreads / 32; ++q) wsum += tile_work[q];
        L.tile_plastic[w.begin / kThreads] = wsum;
    }
}

// Whether a tile of the bonds touches the contact halo of this substep.
template <class R> __device__ __forceinline__ bool lateTile(const Dev<R> &L, const Work &w) {
    return L.late_tile_stamp[w.begin / kThreads] == substepStamp(L);
}

// Every tile (outside_halo 0), or those outside the contact halo (1). Bonds lie
// level after level, and every level covers the whole lattice, so tiles in
// storage order read each node's arrays again once per level, from HBM where
// the lattice's do not fit in L2 (256x128x128: 134 MB). The CTAs therefore
// start in stripes of the tiles in turn -- as many as the lattice has levels of
// the widest's size -- so that those running together sample one region of
// every level. 256x128x128: 1,107 us in storage order, 896 us in stripes. A
// batch's lattices, listed one after another, are each small.
template <class R, bool Many, bool Direct, bool Plastic>
__global__ void __launch_bounds__(kThreads) kEndSample(const Grid<R> launch, Settings<R> S, int outside_halo,
                                                       std::uint32_t each, std::uint32_t extra) {
    startAfterPrevious();
    Work w;
    if (Many) {
        w = launch.list[blockIdx.x];
    } else {
        // Stripe p (a column of the grid) holds `each` tiles, the first `extra`
        // stripes one more.
        const std::uint32_t p = blockIdx.x, q = blockIdx.y;
        if (q == each && p >= extra) return;
        const std::uint32_t b = launch.base + (p * each + (p < extra ? p : extra) + q) * kThreads;
        w = Work{0U, b, b + kThreads < launch.end ? b + kThreads : launch.end};
    }
    __shared__ SharedDesc<R> desc;
    const Dev<R> &L = descriptorIn<R, Many>(launch, w, desc);
    __shared__ double tile_work[kThreads / 32];
    if (L.ctl->stop || (outside_halo && lateTile(L, w))) return;
    endSampleTile<R, Direct, Plastic>(L, S, w, tile_work);
}

// The tiles inside the contact halo, few among many: a CTA looks at the stamps
// of up to kLateTiles of them, a lane a tile, and samples those that are. They
// lie together, so a CTA's are gridDim.x apart. One tile a CTA, 145,860 CTAs of
// 256x128x128 that mostly return took 153 us, this 28 us.
constexpr unsigned kLateTiles = 16;
template <class R, bool Many, bool Direct, bool Plastic>
__global__ void __launch_bounds__(kThreads) kEndSampleLate(const Grid<R> launch, Settings<R> S, std::uint32_t tiles) {
    startAfterPrevious();
    __shared__ SharedDesc<R> desc;
    __shared__ double tile_work[kThreads / 32];
    auto tileAt = [&](std::uint32_t k) {
        if (Many) return launch.list[k];
        const std::uint32_t b = launch.base + k * kThreads;
        return Work{0U, b, b + kThreads < launch.end ? b + kThreads : launch.end};
    };
    bool late = false;
    const std::uint32_t mine = blockIdx.x + (threadIdx.x & 31U) * gridDim.x;
    if ((threadIdx.x & 31U) < kLateTiles && mine < tiles) {
        const Work w = tileAt(mine);
        if (Many) {
            const Dev<R> &L = launch.table[w.lattice];
            late = !L.ctl->stop && lateTile(L, w);
        } else {
            late = !launch.one.ctl->stop && lateTile(launch.one, w);
        }
    }
    // The same in every warp: nothing that runs beside this writes stamps or stops.
    for (unsigned left = __ballot_sync(0xffffffffU, late); left; left &= left - 1) {
        const Work w = tileAt(blockIdx.x + static_cast<std::uint32_t>(__ffs(left) - 1) * gridDim.x);
        if (Many) __syncthreads(); // the descriptor of the tile before is read no more
        endSampleTile<R, Direct, Plastic>(descriptorIn<R, Many>(launch, w, desc), S, w, tile_work);
    }
}

// ---------------------------------------------------------------------------
// The substep ledger's ordered lists and FP64 sums, fully parallel and in a
// fixed order. A "tile" is 256 bonds of schedule order (8 bit words); a scan
// block is kScanBlock tiles. Every sum below is formed in an order fixed by the
// bond order alone: sequential inside a 32-bond word, a tree over the words of
// a tile, shuffle scans across the tiles of a block (warps, then their
// totals), the same across the blocks.
//
// These are small launches whose time is their own latency: barriers (a scan
// through shared memory took twenty of them per value, two now) and, where
// bonds break, the loads of their records, which therefore go word by word or
// bond by bond in parallel (one thread summing a whole tile's made the scan of
// 128 shattering trials, end sample included, 1.17 ms long against 0.62).
// ---------------------------------------------------------------------------
constexpr unsigned kScanBlock = 1024;
constexpr unsigned kTileWords = kThreads / 32;

__device__ __forceinline__ unsigned blockExclusiveScanU(unsigned x, unsigned *buf, unsigned &total) {
    buf[threadIdx.x] = x;
    __syncthreads();
    for (unsigned o = 1; o < blockDim.x; o <<= 1) {
        const unsigned y = threadIdx.x >= o ? buf[threadIdx.x - o] : 0U;
        __syncthreads();
        if (threadIdx.x >= o) buf[threadIdx.x] += y;
        __syncthreads();
    }
    const unsigned inclusive = buf[threadIdx.x];
    total = buf[blockDim.x - 1];
    __syncthreads();
    return inclusive - x;
}

// Inclusive scan over a warp in a fixed order.
template <class T> __device__ __forceinline__ T warpInclusive(T x) {
    const unsigned lane = threadIdx.x & 31;
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(0xffffffffU, x, o);
        if (lane >= static_cast<unsigned>(o)) x += y;
    }
    return x;
}

// What one thread of a 1024-thread CTA contributes to the ledger's scans, and
// what comes back: its exclusive prefixes, and the CTA's totals.
struct LedgerScan {
    unsigned broken, damaged;
    double removed, work; // work: total only
};
__device__ __forceinline__ LedgerScan ledgerScan(const LedgerScan &in, LedgerScan &total) {
    __shared__ unsigned wb[32], wd[32];
    __shared__ double wr[32], ww[32];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    const unsigned ib = warpInclusive(in.broken), id = warpInclusive(in.damaged);
    const double ir = warpInclusive(in.removed), work = warpSumFixed(in.work);
    if (lane == 31) {
        wb[warp] = ib;
        wd[warp] = id;
        wr[warp] = ir;
    }
    if (lane == 0) ww[warp] = work;
    __syncthreads();
    // Every warp scans the 32 totals itself: no second trip through memory.
    const unsigned tb = warpInclusive(wb[lane]), td = warpInclusive(wd[lane]);
    const double tr = warpInclusive(wr[lane]), tw = warpSumFixed(ww[lane]);
    total = {__shfl_sync(0xffffffffU, tb, 31), __shfl_sync(0xffffffffU, td, 31), __shfl_sync(0xffffffffU, tr, 31),
             __shfl_sync(0xffffffffU, tw, 0)};
    const int before = static_cast<int>(warp) - 1;
    const unsigned sb = __shfl_sync(0xffffffffU, tb, before < 0 ? 0 : before);
    const unsigned sd = __shfl_sync(0xffffffffU, td, before < 0 ? 0 : before);
    const double sr = __shfl_sync(0xffffffffU, tr, before < 0 ? 0 : before);
    const double er = __shfl_up_sync(0xffffffffU, ir, 1);
    LedgerScan out;
    out.broken = (before < 0 ? 0U : sb) + ib - in.broken;
    out.damaged = (before < 0 ? 0U : sd) + id - in.damaged;
    out.removed = (before < 0 ? 0.0 : sr) + (lane == 0 ? 0.0 : er);
    out.work = 0.0;
    __syncthreads(); // the totals may be overwritten by a next round
    return out;
}

// A word's removed energy, in bond order.
__device__ __forceinline__ double wordRemoved(const double *removed, std::uint32_t word, unsigned bits) {
    double sum = 0.0;
    for (; bits; bits &= bits - 1) sum += removed[word * 32 + static_cast<unsigned>(__ffs(bits) - 1)];
    return sum;
}

// The substep's totals, once every block's prefix is known.
__device__ __forceinline__ void ledgerTotals(Ctl &c, const LedgerScan &total) {
    c.event_count = total.broken;
    c.dmg_count = total.damaged;
    c.removed_substep = total.removed;
    c.plastic_substep = total.work;
    c.energy_gain = 0;
    c.dirty_count = 0; // the restart of this substep has consumed the list
}

// Eight lanes per tile, one per word: broken-bond and damage-candidate counts
// and the tile's removed energy.
constexpr unsigned kCountTiles = kThreads / kTileWords; // tiles per CTA
template <class R, bool Many>
__global__ void __launch_bounds__(kThreads) kTileCounts(const Grid<R> launch) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    __shared__ SharedDesc<R> desc;
    const Dev<R> &L = descriptorIn<R, Many>(launch, w, desc);
    if (L.ctl->stop) return;
    const unsigned tile = w.begin + threadIdx.x / kTileWords; // items: up to kCountTiles tiles of one lattice
    const bool in = tile < w.end;
    const std::uint32_t wd = tile * kTileWords + threadIdx.x % kTileWords;
    const unsigned bits = in ? L.ev_bits[wd] : 0U;
    unsigned broken = __popc(bits), damaged = in ? __popc(L.dmg_bits[wd]) : 0U;
    double removed = bits ? wordRemoved(L.ev_removed, wd, bits) : 0.0;
    for (int o = 1; o < static_cast<int>(kTileWords); o <<= 1) {
        broken += __shfl_xor_sync(0xffffffffU, broken, o);
        damaged += __shfl_xor_sync(0xffffffffU, damaged, o);
        removed += __shfl_xor_sync(0xffffffffU, removed, o);
    }
    if (in && threadIdx.x % kTileWords == 0) {
        L.ev_tile[tile] = broken;
        L.dmg_tile[tile] = damaged;
        L.tile_removed[tile] = removed;
    }
}

// One CTA per scan block, a thread per tile: the tiles' exclusive offsets
// inside the block, and the block's totals with its plastic work. A lattice
// of one block (up to 1,023 tiles, 261,888 bonds) is done; kTopScan follows for
// the others.
template <class R, bool Many>
__global__ void __launch_bounds__(kScanBlock) kEventScan(const Grid<R> launch, int plastic) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    __shared__ SharedDesc<R> desc;
    const Dev<R> &L = descriptorIn<R, Many>(launch, w, desc);
    Ctl &c = *L.ctl;
    if (c.stop) return;
    const unsigned blk = w.begin; // one item per (lattice, scan block)
    const unsigned t = blk * kScanBlock + threadIdx.x;
    const bool in = t < L.tiles_b;
    LedgerScan own{0U, 0U, 0.0, plastic && in ? L.tile_plastic[t] : 0.0};
    if (in) {
        own.broken = L.ev_tile[t];
        own.damaged = L.dmg_tile[t];
        own.removed = L.tile_removed[t];
    }
    LedgerScan total{};
    const LedgerScan before = ledgerScan(own, total);
    // Only a tile with events is looked at again.
    if (in && (own.broken || own.damaged)) {
        L.ev_tile[t] = before.broken;
        L.dmg_tile[t] = before.damaged;
        L.tile_removed[t] = before.removed;
    }
    if (threadIdx.x == 0) {
        const bool alone = L.tiles_b < kScanBlock;
        L.blk_ev[blk] = alone ? 0U : total.broken;
        L.blk_dmg[blk] = alone ? 0U : total.damaged;
        L.blk_removed[blk] = alone ? 0.0 : total.removed;
        L.blk_plastic[blk] = total.work;
        if (alone) ledgerTotals(c, total);
    }
}

// One CTA per lattice of several blocks: their exclusive offsets (rounds of
// 1024 blocks with a carry), and the substep's totals.
template <class R, bool Many>
__global__ void __launch_bounds__(kScanBlock) kTopScan(const Grid<R> launch) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    __shared__ SharedDesc<R> desc;
    const Dev<R> &L = descriptorIn<R, Many>(launch, w, desc);
    const unsigned blocks = L.tiles_b / kScanBlock + 1; // one item per lattice
    Ctl &c = *L.ctl;
    if (c.stop || blocks == 1) return;
    LedgerScan carry{0U, 0U, 0.0, 0.0};
    for (unsigned base = 0; base < blocks; base += kScanBlock) {
        const unsigned k = base + threadIdx.x;
        const bool in = k < blocks;
        LedgerScan own{0U, 0U, 0.0, 0.0}, total{};
        if (in) own = {L.blk_ev[k], L.blk_dmg[k], L.blk_removed[k], L.blk_plastic[k]};
        const LedgerScan before = ledgerScan(own, total);
        if (in) {
            L.blk_ev[k] = carry.broken + before.broken;
            L.blk_dmg[k] = carry.damaged + before.damaged;
            L.blk_removed[k] = carry.removed + before.removed;
        }
        carry.broken += total.broken;
        carry.damaged += total.damaged;
        carry.removed += total.removed;
        carry.work += total.work;
    }
    if (threadIdx.x == 0) ledgerTotals(c, carry);
}

// One warp per kEmitTiles tiles, the tiles with events one after another, in
// bond order. Broken bonds: the energy-gain test of each against the running
// removed energy it would see (CpuLatticeBackend.cpp:469-474; its prefix is
// block offset, tile offset and in-tile scan, the orders of the counts), the
// first-failure list, and the dirty marks and list of the next substep's
// restart (CpuLatticeBackend.cpp:476-477). Damage candidates: their values in
// order. The bit words are cleared for the next substep. A tile's bonds are
// listed in shared memory by the lane of their word, then taken one per lane,
// so that their records' loads and the dirty marks' atomics overlap.
constexpr unsigned kEmitTiles = 8;
constexpr unsigned kEmitThreads = 128;
template <class R, bool Many>
__global__ void __launch_bounds__(kEmitThreads) kEmitEvents(const Grid<R> launch) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    __shared__ SharedDesc<R> desc;
    __shared__ std::uint16_t lists[kEmitThreads / 32][kThreads];
    __shared__ double energies[kEmitThreads / 32][kThreads];
    const Dev<R> &L = descriptorIn<R, Many>(launch, w, desc);
    Ctl &c = *L.ctl;
    if (c.stop || (c.event_count == 0 && c.dmg_count == 0)) return;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    std::uint16_t *list = lists[warp];  // a tile's broken bonds in order, then its damage candidates
    double *energy = energies[warp];    // the removed energy of each, then its in-tile inclusive prefix
    const bool first_round = c.broken_bonds == 0;
    const double prior = c.removed_energy;
    const double fraction = c.energy_flat_fraction;
    const unsigned first = w.begin + warp * kEmitTiles; // items: up to kEmitTiles tiles per warp of one lattice
    for (unsigned tile = first; tile < first + kEmitTiles && tile < w.end; ++tile) {
        const unsigned wd = tile * kTileWords + lane;
        const unsigned blk = tile / kScanBlock;
        const unsigned bits = lane < kTileWords ? L.ev_bits[wd] : 0U;
        const unsigned dbits = lane < kTileWords ? L.dmg_bits[wd] : 0U;
        // The set bits of the lanes' words into `list`, in order.
        auto enlist = [&](unsigned set, unsigned from) {
            for (; set; set &= set - 1)
                list[from++] = static_cast<std::uint16_t>(lane * 32 + static_cast<unsigned>(__ffs(set) - 1));
        };
        if (__any_sync(0xffffffffU, bits != 0)) {
            const unsigned n = __popc(bits), upto = warpInclusive(n);
            const unsigned count = __shfl_sync(0xffffffffU, upto, 31);
            enlist(bits, upto - n);
            if (bits) L.ev_bits[wd] = 0; // the end sample sets bits with atomicOr
            __syncwarp();
            for (unsigned e = lane; e < count; e += 32) energy[e] = L.ev_removed[tile * kThreads + list[e]];
            __syncwarp();
            double own = 0.0;
            for (unsigned e = upto - n; e < upto; ++e) own += energy[e];
            double run = __shfl_up_sync(0xffffffffU, warpInclusive(own), 1);
            if (lane == 0) run = 0.0;
            __syncwarp();
            for (unsigned e = upto - n; e < upto; ++e) {
                run += energy[e];
                energy[e] = run;
            }
            __syncwarp();
            const unsigned at = L.blk_ev[blk] + L.ev_tile[tile];
            const double offset = L.blk_removed[blk] + L.tile_removed[tile];
            bool gain = false;
            for (unsigned e = lane; e < count; e += 32) {
                const std::uint32_t j = tile * kThreads + list[e];
                if (!inBounds(j, L.B, kSiteEvent)) continue;
                const double removed = L.ev_removed[j], running = prior + (offset + energy[e]);
                gain = gain || removed > fraction * (running < 1.0e-12 ? 1.0e-12 : running);
                if (first_round) L.ffb[at + e] = j;
                const uint2 e2 = L.ev_ends[j];
                const std::uint32_t ends[2] = {e2.x, e2.y};
                for (int q = 0; q < 2; ++q) {
                    const std::uint32_t node = ends[q];
                    if (!inBounds(node, L.N, kSiteEventEnd)) continue;
                    unsigned *word = reinterpret_cast<unsigned *>(L.dirty + (node & ~3U));
                    const unsigned bit = 1U << (8 * (node & 3U));
                    if (!(atomicOr(word, bit) & bit)) {
                        const unsigned slot = atomicAdd(&c.dirty_count, 1U);
                        if (inBounds(slot, L.N, kSiteDirty)) L.dirty_list[slot] = node;
                    }
                }
            }
            if (__any_sync(0xffffffffU, gain) && lane == 0) atomicOr(&c.energy_gain, 1U);
            __syncwarp();
        }
        if (__any_sync(0xffffffffU, dbits != 0)) {
            const unsigned n = __popc(dbits), upto = warpInclusive(n);
            const unsigned count = __shfl_sync(0xffffffffU, upto, 31);
            enlist(dbits, upto - n);
            if (dbits) L.dmg_bits[wd] = 0;
            __syncwarp();
            const unsigned at = L.blk_dmg[blk] + L.dmg_tile[tile];
            for (unsigned e = lane; e < count; e += 32) L.dmg_value[at + e] = L.ev_damage[tile * kThreads + list[e]];
            __syncwarp();
        }
    }
}

// ---------------------------------------------------------------------------
// The energy audit's measure (LatticePhysics.hpp:1676-1682): a lattice's
// kinetic energy, each node's term formed in backend precision and widened,
// folded serially in node order as the reference folds it, so the audit
// ledgers match the reference's bit for bit. The CTA forms the next chunk of
// terms in shared memory while warp 0 folds the current one (foldSerial).
// kAuditMark keeps the energy before a phase; the other modes charge the drop
// across the phase to the striker or the damping ledger.
// ---------------------------------------------------------------------------
constexpr unsigned kFoldThreads = 1024;
constexpr int kAuditMark = 0, kAuditStriker = 1, kAuditDamping = 2;

template <class R, bool Many>
__global__ void __launch_bounds__(kFoldThreads) kKineticFold(const Grid<R> launch, int mode) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    Ctl &c = *L.ctl;
    if (c.stop) return;
    __shared__ double terms[2][kFoldThreads];
    double total = 0.0;
    unsigned buf = 0;
    // Warp 0 reaches the barrier of chunk k+1 only after folding chunk k,
    // so chunk k+2 never overwrites a buffer still being read.
    for (std::uint32_t base = 0; base < L.N; base += kFoldThreads, buf ^= 1U) {
        const std::uint32_t i = base + threadIdx.x;
        if (i < L.N) {
            const Q4<R> q = L.v[i]; // w: the node's mass
            const V3<R> v = xyz(q);
            terms[buf][threadIdx.x] = static_cast<double>(R(0.5) * q.w * dot(v, v));
        }
        __syncthreads();
        if (threadIdx.x < 32)
            total = foldOneSign(total, terms[buf], L.N - base < kFoldThreads ? L.N - base : kFoldThreads);
    }
    if (threadIdx.x != 0) return;
    if (mode == kAuditMark) c.ke_mark = total;
    else if (mode == kAuditStriker) c.striker_dissipated += c.ke_mark - total;
    else c.damping_dissipated += c.ke_mark - total;
}

// ---------------------------------------------------------------------------
// The external-load ledger of a substep (ExternalLoads.hpp:126-140): thirteen
// independent serial folds over the loaded nodes in list order -- impulse,
// angular impulse, work, requested impulse and requested angular impulse, per
// component -- then added to the run's ledger. The wrench sources' node runs
// tile the list in source order, so the same pass folds each source's own
// change and hands it to its ledger when its run ends.
//
// Nothing in the substep reads the ledger before the exit rules at its end, so
// the kernel runs on a stream of its own from the kick, whose contributions it
// reads, beside the contact passes, the sweep and the end sample.
// ---------------------------------------------------------------------------
constexpr int kLedgerFolds = 13;
constexpr unsigned kLedgerThreads = 160;                   // a warp for the total, one for the sources, three staging ones
constexpr unsigned kLedgerStagers = kLedgerThreads - 64;
constexpr unsigned kLedgerChunk = 768;                      // entries staged per round

// Adds a source's folded change (component q) to its ledger.
__device__ __forceinline__ void addLoadComponent(LoadLedger &g, int q, double x) {
    if (q < 3) g.imp[q] = g.imp[q] + x;
    else if (q < 6) g.ang[q - 3] = g.ang[q - 3] + x;
    else if (q == 6) g.work = g.work + x;
    else if (q < 10) g.req_imp[q - 7] = g.req_imp[q - 7] + x;
    else g.req_ang[q - 10] = g.req_ang[q - 10] + x;
}

// One CTA per (lattice, component): blockIdx.y is the component q. Warp 0
// folds its total and warp 1 its sources' runs, beside one another (foldSerial);
// the other warps stage the next chunk of its node contributions.
template <class R, bool Many>
__global__ void __launch_bounds__(kLedgerThreads) kLoadLedger(const Grid<R> launch, Settings<R> S) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    Ctl &c = *L.ctl;
    // A lattice stopped, or whose kick failed this substep, folds nothing
    // (kLedger stops the latter).
    if (c.stop || c.error) return;
    if (!(c.ext_count && c.loads_remaining > 0)) return;
    __shared__ double stage[2][kLedgerChunk];
    const int q = static_cast<int>(blockIdx.y);
    const unsigned warp = threadIdx.x / 32;
    const bool stager = warp >= 2;
    const std::uint32_t n = c.ext_count;
    const unsigned sources = c.wrench_count;
    const auto fill = [&](std::uint32_t base, unsigned buf) {
        const std::uint32_t cnt = n - base < kLedgerChunk ? n - base : kLedgerChunk;
#pragma unroll 4
        for (unsigned e = threadIdx.x - 64; e < cnt; e += kLedgerStagers) {
            const std::uint32_t node = L.ext_nodes[base + e];
            stage[buf][e] = inBounds(node, L.N, kSiteLoad)
                ? L.ext_contrib[kLedgerFolds * static_cast<std::size_t>(node) + q] : 0.0;
        }
    };
    // Flushes every source whose run ends at `at`: the component's change to
    // the source's ledger; component 0 also keeps the step count, the elapsed
    // time and the source's place in the status order.
    unsigned k = 0;
    double run = 0.0;
    const auto flush = [&](std::uint32_t at) {
        while (k < sources && L.wrench[k].end == at) {
            if (threadIdx.x == 32) {
                SourceSlot &slot = L.sources[L.wrench[k].slot];
                addLoadComponent(slot.load, q, run);
                if (q == 0) {
                    if (slot.load.steps == 0) slot.order = c.source_seq++;
                    slot.load.steps += 1;
                    slot.load.elapsed = slot.load.elapsed + static_cast<double>(S.dt);
                }
            }
            run = 0.0;
            ++k;
        }
    };
    if (stager) fill(0, 0);
    else if (warp == 1) flush(0);
    __syncthreads();
    double total = 0.0;
    unsigned buf = 0;
    FoldPace pace;
    for (std::uint32_t base = 0; base < n; base += kLedgerChunk, buf ^= 1U) {
        if (stager) {
            if (base + kLedgerChunk < n) fill(base + kLedgerChunk, buf ^ 1U);
        } else {
            const std::uint32_t cnt = n - base < kLedgerChunk ? n - base : kLedgerChunk;
            const double *col = stage[buf];
            if (warp == 0) total = foldSerial(total, col, cnt, pace);
            for (std::uint32_t e = 0; warp == 1 && k < sources && e < cnt;) {
                const std::uint32_t end = L.wrench[k].end - base;
                const std::uint32_t upto = end < cnt ? end : cnt;
                run = foldSerial(run, col + e, upto - e, pace);
                e = upto;
                flush(base + e);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        LoadLedger &g = c.ext;
        addLoadComponent(g, q, total);
        if (q == 0) {
            g.steps += 1;
            g.elapsed += static_cast<double>(S.dt);
        }
    }
    // loads_remaining counts down in kLedger, after every component's CTA
    // has read it.
}

// ---------------------------------------------------------------------------
// The serial tail of a substep, one warp: the damage-record scan over its
// candidates in bond order; then one thread: the substep's FP64 sums into the
// run totals, the sphere drift and support contact, the failure-round
// bookkeeping and the exit rules (CpuLatticeBackend.cpp:279-298, 441-488),
// after the load ledger.
// ---------------------------------------------------------------------------
template <class R, bool Many>
__global__ void __launch_bounds__(32) kLedger(const Grid<R> launch, Settings<R> S) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    Ctl &c = *L.ctl;
    if (c.stop) return;
    // The damage record over its candidates in bond order: the warp looks for
    // the next one above the record as it stands, 32 at a time (a candidate
    // rarely is: the record only grows). One thread reading them one after
    // another took 162 us of a substep of 128 shattering trials.
    double record = c.max_damage;
    bool gained = false;
    if (!c.error) {
        const unsigned n = c.dmg_count;
        for (unsigned base = 0; base < n; base += 32) {
            const unsigned e = base + threadIdx.x;
            const double dmg = e < n ? static_cast<double>(L.dmg_value[e]) : -1.0;
            for (unsigned from = 0; from < 32;) {
                const unsigned above = __ballot_sync(0xffffffffU, threadIdx.x >= from && dmg > record + 1.0e-6);
                if (!above) break;
                const unsigned at = static_cast<unsigned>(__ffs(above) - 1);
                record = __shfl_sync(0xffffffffU, dmg, static_cast<int>(at));
                gained = true;
                from = at + 1;
            }
        }
    }
    if (threadIdx.x != 0) return;
    if (c.error) {
        c.stop = 1;
        atomicSub(L.running, 1U);
        return;
    }
    const unsigned long long step = c.total_steps;
    if (c.ext_count && c.loads_remaining > 0) c.loads_remaining -= 1; // the substep's load, folded by kLoadLedger
    c.full_restart = 0;
    c.plastic_work += c.plastic_substep;
    if (gained) {
        c.max_damage = record;
        c.damage_floor = __double2float_rd(record + 1.0e-6);
        c.last_damage_gain_step = step;
    }
    const unsigned broken = c.event_count;
    c.projections += (c.live_bonds - c.broken_bonds) * S.iterations;
    if (broken) {
        c.nc_rebuild = 1; // a failure changes which pairs no live bond holds
        if (c.broken_bonds == 0) c.ffb_count = broken;
        c.removed_energy += c.removed_substep;
        if (c.energy_gain) c.last_energy_gain_step = step;
        c.broken_bonds += broken;
    }
    Sphere<R> sp = *L.sphere;
    if (!S.sphere_enabled) sp.velocity = sp.velocity + S.dt * S.gravity;
    sp.center = sp.center + S.dt * sp.velocity;
    sphereSupport(S, sp, c.contact);
    *L.sphere = sp;
    c.total_steps = step + 1;
    if (broken) {
        if (c.first_failure_step == ~0ULL) c.first_failure_step = step;
        c.last_failure_step = step;
        ++c.failure_rounds;
    }
    const double available = c.removable_energy + c.ext.work;
    c.exit_reason = c.removable_energy > 0 && available <= 0
        ? 6U
        : exitReason(c.total_steps, c.broken_bonds, c.last_failure_step, c.quiet_steps, c.min_steps, c.no_failure_steps,
                     c.energy_flat_steps, c.last_energy_gain_step, c.calm_steps, c.last_damage_gain_step, c.max_damage,
                     c.calm_damage_margin, c.removed_energy, c.removable_energy > 0 ? available : 0.0);
    if (c.exit_reason == 0 && c.step_limit != 0 && c.total_steps >= c.step_limit) c.exit_reason = 3U;
    if (c.exit_reason != 0) {
        c.stop = 1;
        atomicSub(L.running, 1U);
    }
}

// ---------------------------------------------------------------------------
// Node-to-node contact (LatticePhysics.hpp:1441-1647; stage order
// CpuLatticeBackend.cpp:424-436), after the second sphere pass and before the
// end sample. The pair list holds, for every movable owner node, the movable
// nodes of higher index within 2 r + skin that no live bond holds, in the
// order of the 27 grid cells around the owner (z, then y, then x, from -1)
// and ascending within a cell, at most kPairsPerNode per owner. It is rebuilt
// when a bond failed in the previous substep or a node drifted more than
// skin / 2 since the last build. The grid is hashed into buckets whose
// members are kept ascending; every bucket scan keeps only the nodes of the
// cell it visits, so which cells share a bucket never changes the list, and
// each lattice sizes its own table. The narrow phase is the reference's
// serial chain in list order, run by one warp.
// ---------------------------------------------------------------------------
constexpr std::uint32_t kPairsPerNode = 24;
constexpr unsigned kContactScanThreads = 1024;

// Teschner et al., "Optimized Spatial Hashing for Collision Detection of
// Deformable Objects" (2003): three primes, exclusive-or, masked.
__device__ __forceinline__ std::uint32_t cellBucket(int x, int y, int z, std::uint32_t mask) {
    return ((static_cast<std::uint32_t>(x) * 73856093U) ^ (static_cast<std::uint32_t>(y) * 19349663U) ^
            (static_cast<std::uint32_t>(z) * 83492791U)) & mask;
}

template <class R> __device__ __forceinline__ R contactCutoff(const Settings<R> &S) {
    return R(2) * S.nc_radius + S.nc_skin;
}

// The drift test (nodeContactStale): any node farther than skin / 2 from where
// the list was built asks for a rebuild.
template <class R, bool Many>
__global__ void __launch_bounds__(kThreads) kContactStale(const Grid<R> launch, Settings<R> S) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    Ctl &c = *L.ctl;
    if (c.stop || *static_cast<volatile unsigned *>(&c.nc_rebuild)) return;
    const std::uint32_t i = w.begin + threadIdx.x;
    if (i >= w.end) return;
    const R half = R(0.5) * S.nc_skin;
    const R limit = half * half;
    const V3<R> d = xyz(L.u[i]) - xyz(L.nc_built[i]);
    if (dot(d, d) > limit) c.nc_rebuild = 1U;
}

// Rebuild, step 0 (bucket items): clear the bucket counts.
template <class R, bool Many>
__global__ void __launch_bounds__(kThreads) kContactClear(const Grid<R> launch) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    Ctl &c = *L.ctl;
    if (c.stop || !c.nc_rebuild) return;
    const std::uint32_t b = w.begin + threadIdx.x;
    if (b < w.end) L.nc_count[b] = 0U;
    if (w.begin == 0 && threadIdx.x == 0) c.nc_members = 0U;
}

// Rebuild, step 1 (nodeContactStoreCell, node items): the node's cell at the
// positions of this substep, the positions kept for the drift test, and the
// bucket counts of the movable nodes.
template <class R, bool Many>
__global__ void __launch_bounds__(kThreads) kContactCells(const Grid<R> launch, Settings<R> S) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    if (L.ctl->stop || !L.ctl->nc_rebuild) return;
    const std::uint32_t i = w.begin + threadIdx.x;
    if (i >= w.end) return;
    const R inverse_cell = R(1) / contactCutoff(S);
    const V3<R> p = pos(L, i);
    const int x = static_cast<int>(floor(p.x * inverse_cell));
    const int y = static_cast<int>(floor(p.y * inverse_cell));
    const int z = static_cast<int>(floor(p.z * inverse_cell));
    const std::uint32_t b = cellBucket(x, y, z, L.nc_mask);
    L.nc_cell[i] = make_int4(x, y, z, static_cast<int>(b));
    L.nc_built[i] = L.u[i];
    if (i % kThreads == 0) L.nc_tile[i / kThreads] = 0U; // the gather adds to it
    if (!(L.v[i].w <= R(0))) atomicAdd(&L.nc_count[b], 1U);
}

// Rebuild, step 2 (bucket items): each bucket's first member slot. Buckets of
// one CTA are contiguous; the CTAs' runs are placed in any order, which only
// moves whole buckets. The count becomes the scatter cursor.
template <class R, bool Many>
__global__ void __launch_bounds__(kThreads) kContactBuckets(const Grid<R> launch) {
    startAfterPrevious();
    __shared__ unsigned buf[kThreads];
    __shared__ unsigned base;
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    Ctl &c = *L.ctl;
    if (c.stop || !c.nc_rebuild) return;
    const std::uint32_t b = w.begin + threadIdx.x;
    const unsigned n = b < w.end ? L.nc_count[b] : 0U;
    unsigned total = 0;
    const unsigned ex = blockExclusiveScanU(n, buf, total);
    if (threadIdx.x == 0) base = atomicAdd(&c.nc_members, total);
    __syncthreads();
    if (b < w.end) {
        L.nc_start[b] = base + ex;
        L.nc_count[b] = 0U;
    }
}

// Rebuild, step 3 (node items): the movable nodes into their buckets.
template <class R, bool Many>
__global__ void __launch_bounds__(kThreads) kContactScatter(const Grid<R> launch) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    if (L.ctl->stop || !L.ctl->nc_rebuild) return;
    const std::uint32_t i = w.begin + threadIdx.x;
    if (i >= w.end || L.v[i].w <= R(0)) return;
    const std::uint32_t b = static_cast<std::uint32_t>(L.nc_cell[i].w);
    L.nc_members[L.nc_start[b] + atomicAdd(&L.nc_count[b], 1U)] = i;
}

// Rebuild, step 4 (bucket items): each bucket's members ascending (buckets
// hold half a node on average; an insertion sort in place).
template <class R, bool Many>
__global__ void __launch_bounds__(kThreads) kContactSort(const Grid<R> launch) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    if (L.ctl->stop || !L.ctl->nc_rebuild) return;
    const std::uint32_t b = w.begin + threadIdx.x;
    if (b >= w.end) return;
    const std::uint32_t n = L.nc_count[b];
    std::uint32_t *m = L.nc_members + L.nc_start[b];
    for (std::uint32_t k = 1; k < n; ++k) {
        const std::uint32_t v = m[k];
        std::uint32_t j = k;
        for (; j > 0 && m[j - 1] > v; --j) m[j] = m[j - 1];
        m[j] = v;
    }
}

// Rebuild, step 5 (nodeContactGather; a tile is 256 nodes). Count pass: each
// owner's pairs and the tile's total, and the pairs that did not fit. Write
// pass: the pairs at the owner's place in the list. One warp per owner, a lane
// per cell: the 27 cells' chains of loads (bucket, members, cell, position,
// the owner's bonds) run side by side, and a scan over the lanes puts the
// pairs in cell order; owners without pairs, most of a lattice whose bonds hold,
// are passed over by the write pass.
//
// Both passes are launched every substep and mostly return at once, so what
// bounds them then is starting CTAs: at most kGatherPerSm of them an SM, each
// over a run of owners, whose lists lie together. Broad phase without a rebuild
// and with one, us: 640,000 nodes 59 and 1,086 (a CTA per 8 owners 211 and
// 1,190; a thread per owner 57 and 1,313), 163,840 nodes 31 and 255 (64 and
// 280; 41 and 413), 4,320 nodes 14 and 37 (14 and 37; 39 and 197); at 16, 64 an
// SM 54 and 1,114, 67 and 1,068 with 640,000.
constexpr unsigned kGatherOwners = kThreads / 32; // a CTA's at a time
constexpr unsigned kGatherPerSm = 32;
constexpr unsigned kGatherSlots = 32;             // an owner's bonds kept in shared memory
template <class R, bool Many, bool Write>
__global__ void __launch_bounds__(kThreads) kContactGather(const Grid<R> launch, Settings<R> S) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    __shared__ SharedDesc<R> desc;
    __shared__ std::uint32_t others[kGatherOwners][kGatherSlots], bonds[kGatherOwners][kGatherSlots];
    __shared__ bool lives[kGatherOwners][kGatherSlots];
    {
        const Ctl *ctl = Many ? launch.table[w.lattice].ctl : launch.one.ctl;
        if (ctl->stop || !ctl->nc_rebuild) return;
    }
    const Dev<R> &L = descriptorIn<R, Many>(launch, w, desc);
    Ctl &c = *L.ctl;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    const std::size_t N = L.N;
    const R cutoff = contactCutoff(S);
    const R cutoff_sq = cutoff * cutoff;
    for (std::uint32_t i = w.begin + warp; i < w.end; i += kGatherOwners) {
        __syncwarp(); // the bonds of the owner before are read no more
        const std::uint32_t tile = i / kThreads;
        if (Write) {
            if (L.nc_fill[i] == 0U) continue;
        } else if (L.v[i].w <= R(0)) { // not movable: no pairs of its own
            if (lane == 0) L.nc_fill[i] = 0U;
            continue;
        }
        // The owner's bonds, in slot order up to the first padded slot.
        const std::uint32_t kept = L.D < kGatherSlots ? L.D : kGatherSlots;
        std::uint32_t bs = kNoBond;
        if (lane < kept) {
            const std::size_t slot = lane * N + i;
            bs = L.nbr_bond[slot];
            others[warp][lane] = L.nbr_other[slot];
            bonds[warp][lane] = bs;
            lives[warp][lane] = !signbit(L.nbr[slot].w);
        }
        const unsigned padded = __ballot_sync(0xffffffffU, bs == kNoBond);
        const std::uint32_t listed = padded ? static_cast<std::uint32_t>(__ffs(padded) - 1) : 32U;
        __syncwarp();
        // The owner's bond to j, if it lists one; whether that bond is alive.
        auto bondTo = [&](std::uint32_t j, std::uint32_t &bond) {
            for (std::uint32_t s = 0; s < listed; ++s)
                if (others[warp][s] == j) {
                    bond = bonds[warp][s];
                    return lives[warp][s];
                }
            for (std::uint32_t s = kGatherSlots; listed == kGatherSlots && s < L.D; ++s) {
                const std::size_t slot = s * N + i;
                const std::uint32_t far = L.nbr_bond[slot];
                if (far == kNoBond) break;
                if (L.nbr_other[slot] != j) continue;
                bond = far;
                return !signbit(L.nbr[slot].w);
            }
            return false;
        };
        const V3<R> p = pos(L, i);
        const int4 home = L.nc_cell[i];
        const int gx = home.x + static_cast<int>(lane % 3) - 1, gy = home.y + static_cast<int>(lane / 3 % 3) - 1,
                  gz = home.z + static_cast<int>(lane / 9) - 1;
        std::uint32_t first = 0, members = 0;
        if (lane < 27) {
            const std::uint32_t b = cellBucket(gx, gy, gz, L.nc_mask);
            first = L.nc_start[b];
            members = L.nc_count[b];
        }
        // The cell's pairs in member order: take(j, bond).
        auto pairs = [&](auto &&take) {
            for (std::uint32_t k = 0; k < members; ++k) {
                const std::uint32_t j = L.nc_members[first + k];
                if (j <= i) continue;
                const int4 cj = L.nc_cell[j];
                if (cj.x != gx || cj.y != gy || cj.z != gz) continue;
                const V3<R> r = pos(L, j) - p;
                if (dot(r, r) > cutoff_sq) continue;
                std::uint32_t bond = kNoBond;
                if (bondTo(j, bond)) continue; // a live bond holds the pair
                take(j, bond);
            }
        };
        std::uint32_t mine = 0;
        pairs([&](std::uint32_t, std::uint32_t) { ++mine; });
        const std::uint32_t upto = warpInclusive(mine);
        const std::uint32_t total = __shfl_sync(0xffffffffU, upto, 31);
        const std::uint32_t fill = total < kPairsPerNode ? total : kPairsPerNode;
        if (!Write) {
            if (lane == 0) {
                L.nc_fill[i] = fill;
                if (fill) atomicAdd(&L.nc_tile[tile], fill);
                if (total > fill) atomicAdd(&c.node.pair_overflow, static_cast<unsigned long long>(total - fill));
            }
            continue;
        }
        // The owner's place: its tile's first pair and the pairs of the tile's
        // nodes before it.
        std::uint32_t before = 0;
        for (std::uint32_t q = tile * kThreads + lane; q < i; q += 32) before += L.nc_fill[q];
        before = __reduce_add_sync(0xffffffffU, before);
        std::uint32_t rank = upto - mine;
        const std::uint32_t at = L.nc_tile[tile] + before;
        pairs([&](std::uint32_t j, std::uint32_t bond) {
            if (rank < kPairsPerNode) {
                L.nc_pa[at + rank] = i;
                L.nc_pb[at + rank] = j;
                L.nc_pbond[at + rank] = bond;
            }
            ++rank;
        });
    }
}

// Rebuild, step 6 (one CTA per lattice): the tiles' first pairs in node order,
// and the list's length (nodeContactActiveList).
template <class R, bool Many>
__global__ void __launch_bounds__(kContactScanThreads) kContactTiles(const Grid<R> launch) {
    startAfterPrevious();
    __shared__ unsigned buf[kContactScanThreads];
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    Ctl &c = *L.ctl;
    if (c.stop || !c.nc_rebuild) return;
    const std::uint32_t tiles = (L.N + kThreads - 1) / kThreads;
    unsigned carry = 0;
    for (std::uint32_t t0 = 0; t0 < tiles; t0 += kContactScanThreads) {
        const std::uint32_t t = t0 + threadIdx.x;
        unsigned total = 0;
        const unsigned ex = blockExclusiveScanU(t < tiles ? L.nc_tile[t] : 0U, buf, total);
        if (t < tiles) L.nc_tile[t] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) {
        c.nc_pairs = carry;
        c.node.pairs_listed += carry;
    }
}

// One pair against the current state (nodeContactPair, LatticePhysics.hpp:
// 1441-1647): its gap, whether it responds, and the velocities after it.
template <class R> struct PairResponse {
    bool acts, impulse_on;
    R gap, ia, ib; // 1 / mass of the two nodes, once past the contact gate
    V3<R> n, va, vb;
    R lost;            // kinetic energy before minus after
    V3<R> momentum;    // what rounding left of the pair's momentum change
};
template <class R, class M>
__device__ __forceinline__ PairResponse<R> pairResponse(M &m, const Settings<R> &S, bool respond, V3<R> r, const Q4<R> &qa,
                                                        const Q4<R> &qb) {
    PairResponse<R> o{};
    const R ma = qa.w, mb = qb.w;
    const R distance = m.root(dot(r, r));
    o.n = distance > R(1.0e-12) ? m.div(r, distance) : mk<R>(1, 0, 0); // normalized(r)
    o.gap = distance - R(2) * S.nc_radius;
    o.va = xyz(qa);
    o.vb = xyz(qb);
    if (!respond) return o;
    const R vn = dot(o.vb - o.va, o.n);
    if (o.gap > maxR(S.nc_margin, -vn * S.dt)) return o;
    o.ia = m.div(R(1), ma);
    o.ib = m.div(R(1), mb);
    const R pair_inverse = o.ia + o.ib;
    const R restitution = -vn > S.nc_threshold ? S.nc_restitution : R(0);
    const R desired = o.gap > S.nc_margin ? m.div(-o.gap, S.dt) : -restitution * minR(vn, R(0));
    const R impulse = maxR(R(0), m.div(desired - vn, pair_inverse));
    o.impulse_on = impulse > R(0);
    o.acts = o.impulse_on || o.gap < -S.nc_margin;
    if (!o.impulse_on) return o;
    const V3<R> va0 = o.va, vb0 = o.vb;
    const R before = R(0.5) * ma * dot(va0, va0) + R(0.5) * mb * dot(vb0, vb0);
    const V3<R> j = impulse * o.n;
    o.vb = o.vb + o.ib * j;
    o.va = o.va - o.ia * j;
    const V3<R> rel = o.vb - o.va;
    const V3<R> t = rel - dot(rel, o.n) * o.n;
    const R sq = dot(t, t);
    if (!(sq < R(0x1p-80))) { // below, the speed is under 1e-12 whatever its root's rounding
        const R speed = m.root(sq);
        if (speed > R(1.0e-12)) {
            const V3<R> dir = m.div(t, speed);
            const R stick = m.div(speed, pair_inverse);
            const R friction = stick <= S.nc_static * impulse ? stick : minR(stick, S.nc_dynamic * impulse);
            const V3<R> f = -friction * dir;
            o.vb = o.vb + o.ib * f;
            o.va = o.va - o.ia * f;
        }
    }
    o.lost = before - (R(0.5) * ma * dot(o.va, o.va) + R(0.5) * mb * dot(o.vb, o.vb));
    o.momentum = {ma * (o.va.x - va0.x) + mb * (o.vb.x - vb0.x), ma * (o.va.y - va0.y) + mb * (o.vb.y - vb0.y),
                  ma * (o.va.z - va0.z) + mb * (o.vb.z - vb0.z)};
    return o;
}

// A pair of the list in a lane's registers: its nodes' velocities, rest
// positions and displacements. A pair that a live bond holds or with a fixed
// node is not tested.
template <class R> struct PairState {
    std::uint32_t a, b;
    bool tested;
    Q4<R> va, vb, ua, ub;
    V3<R> xa, xb;

    __device__ __forceinline__ void load(const Dev<R> &L, std::uint32_t pa, std::uint32_t pb, std::uint32_t bond, bool has) {
        a = has ? pa : kNoBond;
        b = has ? pb : kNoBond;
        tested = false;
        if (!has) return;
        va = L.v[a];
        vb = L.v[b];
        ua = L.u[a];
        ub = L.u[b];
        xa = xyz(L.x0[a]);
        xb = xyz(L.x0[b]);
        const bool held = bond != kNoBond && !(L.rec[bond].a & kDeadBit);
        tested = !held && !(va.w <= R(0) || vb.w <= R(0));
    }
    // Nodes A and B after a response; whether this pair has one of them.
    __device__ __forceinline__ bool take(std::uint32_t A, std::uint32_t B, const V3<R> &nva, const V3<R> &nvb,
                                         const V3<R> &nua, const V3<R> &nub) {
        const bool a_is_a = a == A, a_is_b = a == B, b_is_a = b == A, b_is_b = b == B;
        if (a_is_a || a_is_b) {
            const V3<R> v = a_is_a ? nva : nvb, u = a_is_a ? nua : nub;
            va = Q4<R>{v.x, v.y, v.z, va.w};
            ua = Q4<R>{u.x, u.y, u.z, ua.w};
        }
        if (b_is_a || b_is_b) {
            const V3<R> v = b_is_a ? nva : nvb, u = b_is_a ? nua : nub;
            vb = Q4<R>{v.x, v.y, v.z, vb.w};
            ub = Q4<R>{u.x, u.y, u.z, ub.w};
        }
        return a_is_a || a_is_b || b_is_a || b_is_b;
    }
};
template <class R> __device__ __forceinline__ V3<R> shfl3(const V3<R> &v, int src) {
    constexpr unsigned kAll = 0xffffffffU;
    return {__shfl_sync(kAll, v.x, src), __shfl_sync(kAll, v.y, src), __shfl_sync(kAll, v.z, src)};
}

// The narrow phase (nodeContactPass and nodeContactPair), one warp per lattice:
// a serial chain over the list, 32 pairs at a time in the lanes' registers. The
// lanes evaluate their pairs against the current state at once; the first pair
// whose response changes a velocity or a position is applied and its two nodes'
// new state passed to every lane; the later pairs that share a node are
// evaluated again, the others' results stand. Pairs before it changed nothing,
// so each is tested against exactly the state the serial order shows it, and
// its test and overlap are counted as they are.
//
// What bounds it is the chain: a response is a ballot, the shuffles and, where
// a later pair shares a node, one evaluation; the next 32 pairs' nodes are
// loaded meanwhile and take the same updates. Reading every pair's nodes again
// from memory after each response, the window moved up to the next pair, took
// 305 us where this takes 173 (24x10x18 box), and the first
// 20 substeps of cracking 53.1 ms against 30.9.
template <class R, bool Many>
__global__ void __launch_bounds__(32) kContactNarrow(const Grid<R> launch, Settings<R> S) {
    startAfterPrevious();
    const Work w = item<Many>(launch);
    const Dev<R> L = descriptor<R, Many>(launch, w);
    Ctl &c = *L.ctl;
    if (c.stop) return;
    const unsigned lane = threadIdx.x;
    constexpr unsigned kAll = 0xffffffffU;
    if (lane == 0 && c.nc_rebuild) {
        ++c.node.rebuilds;
        c.nc_rebuild = 0U;
    }
    __syncwarp();
    const std::uint32_t count = c.nc_pairs;
    NodeAcc acc = c.node;
    const bool respond = S.nc_mode == 2U;
    // The records only ever hold a widened R; the four FP64 sums are lanes 0
    // to 3's, one each.
    R deepest = R(0), largest = R(0);
    double sum = lane == 0   ? acc.dissipated
                 : lane == 1 ? acc.momentum[0]
                 : lane == 2 ? acc.momentum[1]
                 : lane == 3 ? acc.momentum[2]
                             : 0.0;
    auto evaluate = [&](const PairState<R> &p) {
        const V3<R> r = (p.xb + xyz(p.ub)) - (p.xa + xyz(p.ua));
        PairResponse<R> o;
        if constexpr (std::is_same<R, float>::value) {
            QuickMath quick;
            o = pairResponse<R>(quick, S, respond, r, p.va, p.vb);
            if (!quick.good) {
                PlainMath<R> plain;
                o = pairResponse<R>(plain, S, respond, r, p.va, p.vb);
            }
        } else {
            PlainMath<R> plain;
            o = pairResponse<R>(plain, S, respond, r, p.va, p.vb);
        }
        return o;
    };
    struct Listed {
        std::uint32_t a, b, bond;
    };
    auto listed = [&](std::uint32_t q) {
        return q < count ? Listed{L.nc_pa[q], L.nc_pb[q], L.nc_pbond[q]} : Listed{0U, 0U, kNoBond};
    };
    PairState<R> cur{}, next{};
    {
        const Listed k = listed(lane);
        cur.load(L, k.a, k.b, k.bond, lane < count);
    }
    Listed ahead = listed(lane + 32U);
    for (std::uint32_t at = 0; at < count; at += 32) {
        // Every store so far is visible; a response from here on reaches the
        // next pairs through take().
        next.load(L, ahead.a, ahead.b, ahead.bond, at + 32U + lane < count);
        ahead = listed(at + 64U + lane);
        PairResponse<R> o{};
        if (cur.tested) o = evaluate(cur);
        for (unsigned from = 0; from < 32U;) {
            const unsigned acting = __ballot_sync(kAll, lane >= from && o.acts);
            const unsigned first = acting ? static_cast<unsigned>(__ffs(acting)) - 1U : 32U;
            const bool counted = cur.tested && lane >= from && lane <= first;
            acc.pair_tests += static_cast<unsigned long long>(__popc(__ballot_sync(kAll, counted)));
            if (counted && -o.gap > deepest) deepest = -o.gap;
            if (first == 32U) break;
            V3<R> nua = xyz(cur.ua), nub = xyz(cur.ub);
            if (lane == first) {
                if (o.impulse_on) {
                    L.v[cur.a] = Q4<R>{o.va.x, o.va.y, o.va.z, cur.va.w};
                    L.v[cur.b] = Q4<R>{o.vb.x, o.vb.y, o.vb.z, cur.vb.w};
                }
                if (o.gap < -S.nc_margin) {
                    const R correction = minR(-o.gap - S.nc_margin, R(0.2) * S.nc_radius);
                    const V3<R> shift = (correction / (o.ia + o.ib)) * o.n;
                    nua = nua - o.ia * shift;
                    nub = nub + o.ib * shift;
                    L.u[cur.a] = Q4<R>{nua.x, nua.y, nua.z, cur.ua.w};
                    L.u[cur.b] = Q4<R>{nub.x, nub.y, nub.z, cur.ub.w};
                    if (correction > largest) largest = correction;
                }
            }
            const int src = static_cast<int>(first);
            const std::uint32_t A = __shfl_sync(kAll, cur.a, src), B = __shfl_sync(kAll, cur.b, src);
            const V3<R> nva = shfl3(o.va, src), nvb = shfl3(o.vb, src);
            nua = shfl3(nua, src);
            nub = shfl3(nub, src);
            // The applied pair's sums, folded in list order.
            if (__ballot_sync(kAll, lane == first && o.impulse_on)) {
                const R x0 = __shfl_sync(kAll, o.lost, src);
                const V3<R> x = shfl3(o.momentum, src);
                if (lane < 4) sum += static_cast<double>(lane == 0 ? x0 : lane == 1 ? x.x : lane == 2 ? x.y : x.z);
                ++acc.contacts;
            }
            next.take(A, B, nva, nvb, nua, nub);
            const bool again = cur.take(A, B, nva, nvb, nua, nub) && cur.tested && lane > first;
            from = first + 1U;
            if (again) o = evaluate(cur);
        }
        __syncwarp(); // this window's stores, before loads further down the list
        cur = next;
    }
    for (int o = 16; o > 0; o >>= 1) {
        deepest = maxR(deepest, __shfl_xor_sync(kAll, deepest, o));
        largest = maxR(largest, __shfl_xor_sync(kAll, largest, o));
    }
    if (deepest > static_cast<R>(acc.max_overlap)) acc.max_overlap = static_cast<double>(deepest);
    if (largest > static_cast<R>(acc.max_correction)) acc.max_correction = static_cast<double>(largest);
    acc.dissipated = __shfl_sync(kAll, sum, 0);
    for (int q = 0; q < 3; ++q) acc.momentum[q] = __shfl_sync(kAll, sum, q + 1);
    if (lane == 0) c.node = acc;
}

// ---------------------------------------------------------------------------
// Bond order between the state (schedule order) and the device (storage,
// level-major order), moved on the device: upload writes the per-bond arrays
// in schedule order and download reads them in schedule order, so the host
// converts element by element in sequence and never gathers.
// ---------------------------------------------------------------------------
template <class R> struct BondSet {
    std::uint32_t *slot_a, *slot_b;
    BondRec<R> *rec;
    Q4<R> *geo, *prev, *thr4;
    Q2<R> *thr2, *plastic;
    std::uint8_t *mode;
};

__device__ __forceinline__ std::size_t gridStride() { return static_cast<std::size_t>(gridDim.x) * blockDim.x; }
__device__ __forceinline__ std::size_t gridFirst() {
    return static_cast<std::size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
}

// Upload: storage entry dd takes schedule entry dev2sched[dd].
template <class R>
__global__ void __launch_bounds__(kThreads) kBondsToStorage(BondSet<R> dst, BondSet<R> src,
                                                            const std::uint32_t *dev2sched, std::uint32_t B) {
    for (std::size_t dd = gridFirst(); dd < B; dd += gridStride()) {
        const std::uint32_t j = dev2sched[dd];
        dst.slot_a[dd] = src.slot_a[j];
        dst.slot_b[dd] = src.slot_b[j];
        dst.rec[dd] = src.rec[j];
        dst.geo[dd] = src.geo[j];
        dst.prev[dd] = src.prev[j];
        dst.thr4[dd] = src.thr4[j];
        dst.thr2[dd] = src.thr2[j];
        dst.plastic[dd] = src.plastic[j];
        dst.mode[dd] = src.mode[j];
    }
}

// The inverse permutation, schedule index -> storage index.
__global__ void __launch_bounds__(kThreads) kInvertOrder(std::uint32_t *sched2dev, const std::uint32_t *dev2sched,
                                                         std::uint32_t B) {
    for (std::size_t dd = gridFirst(); dd < B; dd += gridStride()) sched2dev[dev2sched[dd]] = static_cast<std::uint32_t>(dd);
}

// Neighbour slots name their bond by schedule index on upload; the device
// keeps storage indices.
__global__ void __launch_bounds__(kThreads) kSlotsToStorage(std::uint32_t *nbr_bond, const std::uint32_t *sched2dev,
                                                            std::size_t P) {
    for (std::size_t s = gridFirst(); s < P; s += gridStride()) {
        const std::uint32_t j = nbr_bond[s];
        if (j != kNoBond) nbr_bond[s] = sched2dev[j];
    }
}

// Download straight into the state's layout: doubles (exact widenings), bonds
// in schedule order, so the host copies each array as it is.
template <class R>
__global__ void __launch_bounds__(kThreads) kNodesOut(double *u, double *up, double *v, const Q4<R> *du,
                                                      const Q4<R> *dup, const Q4<R> *dv, std::uint32_t N) {
    for (std::size_t i = gridFirst(); i < N; i += gridStride()) {
        const Q4<R> a = du[i], b = dup[i], c = dv[i];
        u[3 * i] = a.x; u[3 * i + 1] = a.y; u[3 * i + 2] = a.z;
        up[3 * i] = b.x; up[3 * i + 1] = b.y; up[3 * i + 2] = b.z;
        v[3 * i] = c.x; v[3 * i + 1] = c.y; v[3 * i + 2] = c.z;
    }
}

struct BondsOut {
    std::uint8_t *alive, *mode;
    double *damage, *tensile, *compressive, *shear, *plastic_extension, *plastic_strain;
};

template <class R>
__global__ void __launch_bounds__(kThreads) kBondsOut(BondsOut o, BondSet<R> src, const std::uint32_t *dev2sched,
                                                      std::uint32_t B) {
    for (std::size_t dd = gridFirst(); dd < B; dd += gridStride()) {
        const std::uint32_t j = dev2sched[dd];
        const Q4<R> p = src.prev[dd];
        const Q2<R> pl = src.plastic[dd];
        o.alive[j] = (src.rec[dd].a & kDeadBit) ? 0 : 1;
        o.mode[j] = src.mode[dd];
        o.damage[j] = p.w;
        o.tensile[j] = p.x;
        o.compressive[j] = p.y;
        o.shear[j] = p.z;
        o.plastic_extension[j] = pl.x;
        o.plastic_strain[j] = pl.y;
    }
}

// Upload straight from the state's layout: a chunk of the caller's arrays
// (doubles, schedule order) staged on the device as it is, converted here to
// the device layout (WorkingLattice::fromState, LatticeWorking.hpp:53-124;
// each value rounded once, to nearest, as the host cast rounds it).
struct NodesIn {
    const double *u, *up, *v, *x0, *mass, *inv_mass;
};
template <class R>
__global__ void __launch_bounds__(kThreads) kNodesIn(Q4<R> *du, Q4<R> *dv, Q4<R> *dx0, Q4<R> *dup, NodesIn in,
                                                     std::size_t first, std::size_t n) {
    for (std::size_t k = gridFirst(); k < n; k += gridStride()) {
        const std::size_t i = first + k;
        du[i] = Q4<R>{R(in.u[3 * k]), R(in.u[3 * k + 1]), R(in.u[3 * k + 2]), R(in.inv_mass[k])};
        dv[i] = Q4<R>{R(in.v[3 * k]), R(in.v[3 * k + 1]), R(in.v[3 * k + 2]), R(in.mass[k])};
        dx0[i] = Q4<R>{R(in.x0[3 * k]), R(in.x0[3 * k + 1]), R(in.x0[3 * k + 2]), R(0)};
        dup[i] = Q4<R>{R(in.up[3 * k]), R(in.up[3 * k + 1]), R(in.up[3 * k + 2]), R(0)};
    }
}

// Neighbour slots: (rest, weight if alive), the other node (itself when
// padded), the bond by schedule index (kSlotsToStorage maps it).
struct SlotsIn {
    const double *rest, *weight;
    const std::uint8_t *alive;
    const std::uint32_t *other, *bond;
};
template <class R>
__global__ void __launch_bounds__(kThreads) kSlotsIn(Q4<R> *nbr, std::uint32_t *nbr_other, std::uint32_t *nbr_bond,
                                                     SlotsIn in, std::size_t first, std::size_t n, std::uint32_t N) {
    for (std::size_t k = gridFirst(); k < n; k += gridStride()) {
        const std::size_t s = first + k;
        const std::uint32_t bond = in.bond[k];
        const bool present = bond != kNoBond;
        const R w = R(in.weight[k]);
        nbr[s] = Q4<R>{R(in.rest[3 * k]), R(in.rest[3 * k + 1]), R(in.rest[3 * k + 2]),
                       present ? (in.alive[k] ? w : -absR(w)) : R(0)};
        nbr_other[s] = present ? in.other[k] : static_cast<std::uint32_t>(s % N);
        nbr_bond[s] = bond;
    }
}

// Bonds, in schedule order; `plastic` is set when any bond has flowed.
struct BondsIn {
    const std::uint32_t *a, *b, *slot_a, *slot_b;
    const std::uint8_t *alive, *mode, *last_a, *last_b;
    const double *rsm, *rest, *edge, *compliance, *tensile, *compressive, *shear, *damage, *threshold, *extension,
        *strain;
};
template <class R>
__global__ void __launch_bounds__(kThreads) kBondsIn(BondSet<R> out, BondsIn in, std::size_t first, std::size_t n,
                                                     unsigned *plastic) {
    bool flowed = false;
    for (std::size_t k = gridFirst(); k < n; k += gridStride()) {
        const std::size_t j = first + k;
        out.rec[j] = BondRec<R>{in.a[k] | (in.alive[k] ? 0U : kDeadBit) | (in.last_a[k] ? kLastABit : 0U),
                                in.b[k] | (in.last_b[k] ? kLastBBit : 0U), R(in.rsm[k]), R(in.rest[k])};
        out.geo[j] = Q4<R>{R(in.edge[3 * k]), R(in.edge[3 * k + 1]), R(in.edge[3 * k + 2]), R(in.compliance[k])};
        out.prev[j] = Q4<R>{R(in.tensile[k]), R(in.compressive[k]), R(in.shear[k]), R(in.damage[k])};
        const double *t = in.threshold + 6 * k;
        out.thr4[j] = Q4<R>{R(t[0]), R(t[1]), R(t[2]), R(t[3])};
        out.thr2[j] = Q2<R>{R(t[4]), R(t[5])};
        const Q2<R> pl{R(in.extension[k]), R(in.strain[k])};
        out.plastic[j] = pl;
        flowed = flowed || pl.x != R(0);
        out.slot_a[j] = in.slot_a[k];
        out.slot_b[j] = in.slot_b[k];
        out.mode[j] = in.mode[k];
    }
    if (__any_sync(0xffffffffU, flowed) && (threadIdx.x & 31) == 0) atomicOr(plastic, 1U);
}

// A frame (captureFrame, LatticeWorking.hpp:290-303): positions as float,
// aliveness and damage (as float) by schedule index.
template <class R>
__global__ void __launch_bounds__(kThreads) kFrameOut(float *u, std::uint8_t *alive, float *damage, const Q4<R> *du,
                                                      BondSet<R> src, const std::uint32_t *dev2sched, std::uint32_t N,
                                                      std::uint32_t B) {
    for (std::size_t i = gridFirst(); i < N; i += gridStride()) {
        const Q4<R> a = du[i];
        u[3 * i] = static_cast<float>(a.x);
        u[3 * i + 1] = static_cast<float>(a.y);
        u[3 * i + 2] = static_cast<float>(a.z);
    }
    for (std::size_t dd = gridFirst(); dd < B; dd += gridStride()) {
        const std::uint32_t j = dev2sched[dd];
        alive[j] = (src.rec[dd].a & kDeadBit) ? 0 : 1;
        damage[j] = static_cast<float>(src.prev[dd].w);
    }
}

// Words copied by the device from any memory it can read (host memory in
// place, where the device has coherent pageable access).
__global__ void __launch_bounds__(kThreads) kCopyWords(std::uint32_t *dst, const std::uint32_t *src, std::size_t n) {
    for (std::size_t k = gridFirst(); k < n; k += gridStride()) dst[k] = src[k];
}

} // namespace gbl
