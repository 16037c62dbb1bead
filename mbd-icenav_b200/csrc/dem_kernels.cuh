// dem_kernels.cuh — device code of the DPDEM frame step for sm_100a.
//
// One templated kernel (T = float or double) runs the phases of one or more
// frames.  Launched cooperatively with one CTA per resident slot, it runs every
// phase of every frame with bounded grid barriers in between (persistent mode);
// launched once per phase it needs no barrier (phased mode).  Both modes
// execute the same device functions, so they give identical results.
//
// Phases of a frame (reference: medea_ice_ship/jax_simulation.py:397-699)
//   P_CULL     elements near the hull, escapes from the neighbour lists' margins,
//              compaction of the grid's buckets
//   P_NEAR     ship contact of the near elements (jax_geometry.py:515-594); beside
//              it the escaped elements' new references
//   P_CFORCE   contact force, side push, submergence + buoyancy
//              (jax_simulation.py:431-496), floe collision flags, per-chunk partial
//              sums for the thrust cap; beside it the rebuild of marked lists
//   P_REDUCE   fixed-order reduction of the partials -> thrust scale, reaction
//              on the ship, vessel step (jax_vessel_dynamics.py:246-348),
//              floe activation (jax_simulation.py:498-524), crack-front flags and
//              bond slot records of the active elements
//   per substep s (jax_simulation.py:363-395, 527-532):
//     escape, build_all   neighbour lists of elements that left their margin within
//               the frame, or of all (skipped otherwise)
//     P_FORCE   fused bond forces + ice-ice contact + drag + rotational drag +
//               semi-implicit integration of the active elements, in gather form
//               (no atomics: each element sums its own bond and contact terms in
//               the reference's scatter order); all substeps in one go with the
//               elements in shared memory while it holds them, else by groups of
//               lanes or a thread per element
//   P_FRACTURE crack front, DPDEM damage, collision breaks (jax_simulation.py:534-653),
//              DPDEM eligibility and history rows
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "dem_b200.h"
#include "dem_math.cuh"

namespace dem {

constexpr int kThreads = 256;          // threads per CTA (chunk size of the fixed-order sums)
constexpr int kMaxNbLocal = 64;        // upper bound of DemParams.max_neighbors
constexpr int kMaxV = 32;              // upper bound of max_v (padded vertices per element)
constexpr int kMaxHull = 256;          // upper bound of hull outline points
constexpr int kMaxEdgeSamples = 16;
constexpr unsigned long long kBarrierLimitNs = 2000000000ull;  // 2 s per barrier wait
constexpr int kMaxPhaseTimes = 4096;

// Phases of one frame: cull, near contact, contact forces, reduce, then per
// substep escape round, all-lists rebuild and force, and last fracture.
__host__ __device__ constexpr int phases_per_frame(int k_sub) { return 5 + 3 * k_sub; }
#ifndef DEM_MIN_BLOCKS
#define DEM_MIN_BLOCKS 2  // resident CTAs per SM the register allocation targets
#endif

// Per-frame record of one bond slot (see phase_reduce): partner index with the
// slot's role in the sign bit, rest length, stiffness E*mean(h)*factor, and
// (1 - damage), or -1 when the bond adds no force this frame (broken, or its
// endpoints differ in active state; jax_simulation.py:86-96).
template <typename T> struct SlotRec;
template <> struct __align__(16) SlotRec<float> {
    int o;
    float rest, stiff, omd;
};
template <> struct __align__(16) SlotRec<double> {
    int o, pad;
    double rest, stiff, omd;
};

template <typename T>
struct IcePtrs {
    T *pos, *vel, *rot, *avel, *sub;
    uint8_t* intact;
    T *dmg, *dm0, *dmmax, *ds;
    uint8_t *active, *elig;
};

template <typename T>
struct ShipPtrs {
    T *eta, *nu, *na, *ei;
};

// Force-phase constants in the kernel's dtype, converted once on the host and
// read from the kernel parameter (constant bank) rather than held in registers.
template <typename T>
struct ForceConst {
    T hf, hexp, mu, fcap, c_drag, href, lin, c_rot, dti, damp, alo, ahi, vclip, pclip;
    int h15;  // hertz_exponent == 1.5: overlap * sqrt(overlap) instead of pow
};

template <typename T>
struct KArgs {
    DemParams P;
    int n, V, nb, nf, S, K, k_sub, nchunks;
    // independent systems (an ice window with its own ship) advanced together;
    // 1 for a plain field.  Elements of system s are [sys_start_s, sys_end[s]),
    // its force chunks [part_base[s], part_base[s + 1]).
    int nsys;
    const int* sys_of;        // (n) system of each element (read when nsys > 1)
    const int* floe_sys;      // (nf) system of each floe (read when nsys > 1)
    const int2* chunk_info;   // (nchunks) {system, first element} of each chunk of kThreads elements
    const int* sys_end;       // (nsys) one past each system's last element
    const int* part_base;     // (nsys + 1) first chunk of each system
    const T* u_ctrl;          // (K, nsys, 3) body-frame ship controls of planner rollouts, or NULL
    int n_buckets, bucket_cap, max_nb, mode;
    int force_split, mark_split;  // DEM_SPLIT_*: how substep work is split (tests and tuning)
    T k_n, k_s, min_bstr, cell, skin, hull_r;
    T hull_bx, hull_by;  // half sides of the box, in the ship's frame, that holds the hull and its outline
    T t_frame;     // frame duration k_sub * dt_ice, for the prediction at the frame's start
    T reach_max;   // largest reach radius (r_max + skin / 2): two reach at most a grid cell
    T margin_max;  // largest margin of a fast element
    T t_samp[kMaxEdgeSamples];
    // static data (caller-owned)
    const T* polys;
    const uint8_t* pmask;
    const T *mass, *inertia, *radii, *areas, *thick, *rest, *bstr, *sbar, *hull;
    const int *bi, *bj, *floe_of;
    // derived at create
    const int* boff;    // (n+1) CSR offsets of per-element bond slots
    const int2* bslot;  // (2 nb) {bond | role<<31, partner}; role 0: element is bond_i
    const T* slot_rest; // (2 nb) rest length of each slot's bond
    const T* slot_stiff;// (2 nb) E * mean(h) * factor of each slot's bond
    const T* vert_r;    // (n) max local vertex radius, rounded up
    // broad phase: grids, reference positions and lists persist across calls
    int* bcnt;          // (n_buckets) grid-hash bucket fill
    int* bitems;        // (n_buckets * bucket_cap) entries; stale ones are filtered by home cell
    int2* ecell;        // (n) home cell of each reference position
    int* ncnt;          // (n) neighbour count
    int* nbr;           // (max_nb * n) neighbour lists, slot-major
    T* pos_ref;         // (n,2) reference positions (NaN before the first build)
    T* reach;           // (n) reach radius of each reference: radius + margin
    unsigned* dirty;    // (n) stamp of the round whose list rebuild the element needs
    int* bflag;         // (n_buckets) bucket queued for compaction
    // buckets to compact at the next frame start: a ring of n_buckets (a power of
    // two) entries, at most one per bucket; comp_cnt = {end, start, end at the
    // last cull}, all running counts
    int* comp_list;
    int* comp_cnt;
    unsigned* esc_cnt;  // (k_sub + 2) escaped elements found before substep s
    // per-frame scratch
    int* near_list;     // (n) elements whose bounding circle reaches the hull
    int* near_cnt;      // (1)
    T *cpen, *cnx, *cny;  // (n) max penetration contact per element
    T* soi;             // (n,2) ship force on ice (with buoyancy), constant over substeps
    T* fraw;            // (n) contact force magnitude before the thrust cap
    uint8_t* crack;     // (n) element touches a broken bond
    int* fcoll;         // (nf) floe touched by the ship this frame
    unsigned long long* fmax;  // (nf) max force magnitude per floe (ordered bits)
    double* part;       // (nchunks * 3) per-chunk sums: soi_x, soi_y, moment
    // per force chunk, for phase_cforce in a call's later frames
    uint8_t* cwarm;     // (nchunks) an element in contact or submerged at the last cforce
    unsigned* cnear;    // (nchunks) frame stamp of the last frame with a near element
    T* kin[2];          // (n,4) {x, y, radius, radius^3} of the substep being read / written
    T* kvel[2];         // (n,2) {vx, vy} of the substep being read / written
    int* esc_list;      // (n) escaped elements of the current detection
    int* dirty_list;    // (n) elements whose list is rebuilt
    int* dirty_cnt;     // (k_sub + 2) lists to rebuild, per substep
    int* work_cnt;      // (k_sub + 2) element chunks handed out dynamically, per substep
    int* act_list;      // (n) elements active this frame (built by phase_reduce)
    unsigned* bstamp;   // (nb) frame stamp of the bonds with an active end (set by phase_reduce)
    int* fb_list;       // (nb) the frame's bonds with an active end, each once (phase_reduce)
    int* fb_cnt;        // (1) entries of fb_list
    int* act_cnt;       // its entries
    unsigned round_base;  // first dirty stamp of this call minus one (advanced by the host)
    int fail_phase;       // test hook: the last CTA skips the barrier after this phase (-1: off)
    ForceConst<T> fc;     // force-phase constants
    T *sp_rot[2], *sp_avel[2];  // substep ping-pong of own-element angles
    void* slotrec;      // (2 nb) SlotRec<T>: per-frame bond slot records
    const T* r3;        // (n) radius^3 (dtype pow, once at create)
    const T* econ;      // (n,4) {mass, inertia, thickness, area}, packed once at create
    double* fscal;      // (4) frame scalars: thrust scale, F_x, F_y, M
    unsigned long long* ptimes;  // (2 * kMaxPhaseTimes) [phase, globaltimer ns] or null
    // call arguments
    IcePtrs<T> in, out;  // frame 0 reads in; every frame writes out (in place after frame 0)
    ShipPtrs<T> ship_in, ship_out, ship_tmp[2];
    const T* setpoints;   // (K,6)
    const T* vw;          // (K,n,2)
    const T* vws;         // (K,2) or null
    const uint8_t* elig0; // dpdem_eligible argument of frame 0
    T *d_pen, *d_fmag, *d_F, *d_J;
    T *h_pos, *h_rot, *h_eta, *h_sub, *h_J, *h_F;
    uint8_t* h_intact;
    unsigned* bar;        // top arrival word of the grid barrier
    unsigned* bar_groups; // group arrival words, kBarGroupStride apart (kBarGroup > 0)
    unsigned long long* sub_bar;  // barrier word of the substeps' CTAs (sub_barrier)
    int sub_flags;                // its escape counts cannot overflow in this call
    // contact-set recording (parity aid, off when crec is null): every pair
    // whose contact term a force phase computes goes to crec as {e, o}, seen
    // from the active element e; crec_marks[f * k_sub + s] = pairs recorded
    // up to the end of substep s of frame f
    int2* crec;
    unsigned* crec_cnt;
    int crec_cap, crec_max_marks;
    int* crec_marks;
    int* status;
    volatile int* host_flag;  // in host memory: set with the status, so that a call without one costs no copy
    long long* stats;     // [rounds, max list, max bucket, re-referenced, lists rebuilt, overflow flags]
};

template <typename A> __device__ __forceinline__ void raise_status(const A& a, int v) {
    atomicMax(a.status, v);
    __threadfence();
    *a.host_flag = 1;
}

template <typename T> struct vec4_of;
template <> struct vec4_of<float> { typedef float4 type; };
template <> struct vec4_of<double> { typedef double4 type; };

template <typename T>
__device__ __forceinline__ typename vec4_of<T>::type ld4(const T* p, int i) {
    return reinterpret_cast<const typename vec4_of<T>::type*>(p)[i];
}

// ─── per-frame pointer bundle ───────────────────────────────────────────────
template <typename T>
struct Frame {
    int f;
    IcePtrs<T> src, dst;
    ShipPtrs<T> ship_src, ship_dst;
    const uint8_t* elig_in;
    const T* vw;
    const T* sp;   // (nsys, 6) [setpoint, setpoint_next] of this frame
    const T* vws;  // (nsys, 2) current at the ships, or NULL (none)
};

template <typename T>
__device__ __forceinline__ Frame<T> make_frame(const KArgs<T>& a, int f) {
    Frame<T> F;
    F.f = f;
    const int K = a.K;
    // frame 0 reads the call's input and writes all of `out`; later frames update
    // `out` in place (every phase reads and writes only its own element or bond,
    // or reads a partner's flag that only turns on), so state that does not
    // change (frozen elements, bonds between them) is not copied frame to frame
    F.dst = a.out;
    F.src = (f == 0) ? a.in : a.out;
    F.ship_dst = (f == K - 1) ? a.ship_out : a.ship_tmp[f & 1];
    F.ship_src = (f == 0) ? a.ship_in : a.ship_tmp[(f - 1) & 1];
    F.elig_in = (f == 0) ? a.elig0 : F.src.elig;
    F.vw = a.vw + (size_t)f * a.n * 2;
    F.sp = a.setpoints ? a.setpoints + (size_t)f * a.nsys * 6 : nullptr;
    F.vws = a.vws ? a.vws + (size_t)f * a.nsys * 2 : nullptr;
    return F;
}

// Stamp of frame f of this call: the dirty stamp of its first rebuild round,
// unique since the stamps were last cleared (never 0)
template <typename T>
__device__ __forceinline__ unsigned frame_stamp(const KArgs<T>& a, const Frame<T>& F) {
    return a.round_base + (unsigned)(F.f * a.k_sub) + 1u;
}

// ─── the words that steer a phase ────────────────────────────────────────────
// Every CTA takes the same branches from a few counters in global memory.  One
// warp per CTA reads them, each lane one word, right after the barrier, and the
// CTA takes them from shared memory: with every warp of the grid reading them
// (2,368 requests for one line, served one after another) four words cost
// 1.1 us per phase on top of a 1.47 us barrier (a barrier loop alone, 296 CTAs).
struct PhaseCtl {
    unsigned esc;    // escaped elements to process before this substep
    int dirty;       // lists to rebuild at this substep
    int act;         // the frame's active elements
    int comp_end;    // buckets to compact: the queue's end and start
    int comp_start;
    int near;        // elements within the hull's reach
    int fb;          // bonds with an active end
    int pad;
    double scale;    // thrust-cap scale of the (first) system
};

// All lanes of one warp call this with the phase that comes next; the caller
// synchronises the CTA afterwards.
template <typename T>
__device__ __forceinline__ void load_ctl(const KArgs<T>& a, int ph, PhaseCtl* c) {
    const int lane = threadIdx.x & 31;
    const int per_frame = phases_per_frame(a.k_sub);
    const int p = ph % per_frame;
    const int* w = nullptr;
    if (p >= 1 && p < per_frame - 1) {
        const int s = p < 4 ? 0 : (p - 4) / 3;
        if (lane == 0) w = reinterpret_cast<const int*>(&a.esc_cnt[s]);
        if (lane == 1) w = &a.dirty_cnt[s];
        if (lane == 2) w = a.act_cnt;
        if (lane == 5 && p == 1) w = a.near_cnt;
    } else if (p == 0) {
        if (lane == 3 || lane == 4) w = a.comp_cnt + (lane - 3);
    } else {
        if (lane == 6) w = a.fb_cnt;
        if (lane == 8) c->scale = *((volatile const double*)a.fscal);
    }
    if (w) reinterpret_cast<int*>(c)[lane] = *((volatile const int*)w);
}

// ─── grid barrier (bounded) ──────────────────────────────────────────────────
// Returns false (and records DEM_ERR_TIMEOUT) if the wait exceeds its limit;
// callers then return.
//
// Arrival counts use flip words: of the n arrivals at a word, the first CTA of
// the set adds 2^31 - (n - 1) and every other one adds 1, so the arrivals of
// one barrier sum to 2^31, bit 31 of the word flips exactly at the last
// arrival (the one whose add carries into bit 31), and no word needs a reset
// between barriers.  With DEM_BAR_GROUP = g > 0 the CTAs arrive in groups of g
// consecutive CTAs, each group on a word of its own 128-byte line
// (a.bar_groups); the last arrival of a group carries it to the top word
// a.bar, and every CTA polls a.bar.  The hottest word then takes
// ceil(grid / g) atomics per barrier instead of one per CTA.
#ifndef DEM_BAR_GROUP
#define DEM_BAR_GROUP 0
#endif
constexpr int kBarGroup = DEM_BAR_GROUP;
constexpr int kBarGroupStride = 32;  // words between group counters (128 bytes)

template <typename T>
__device__ bool grid_barrier(const KArgs<T>& a, int next_ph, PhaseCtl* ctl) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        // the arrivals are releases at GPU scope, cumulative over the CTA's
        // writes ordered before them by __syncthreads; a group arrival is an
        // acquire too, so that the group's last arrival, which reads every
        // earlier arrival of its group, carries their writes into its release
        // on the top word; the polls are acquires: the pattern orders every
        // CTA's phase writes before every CTA's next phase
        unsigned old;
        if (kBarGroup > 0) {
            const unsigned g = blockIdx.x / (unsigned)kBarGroup;
            const unsigned first = g * (unsigned)kBarGroup;
            const unsigned size = min((unsigned)kBarGroup, gridDim.x - first);
            const unsigned ginc = (blockIdx.x == first) ? 0x80000000u - (size - 1u) : 1u;
            const unsigned gold = atom_add_acqrel_u32(a.bar_groups + (size_t)g * kBarGroupStride, ginc);
            const unsigned n_groups = (gridDim.x + (unsigned)kBarGroup - 1u) / (unsigned)kBarGroup;
            if (((gold + ginc) ^ gold) & 0x80000000u) {
                // this group's last arrival: carry the group to the top word
                const unsigned tinc = (g == 0u) ? 0x80000000u - (n_groups - 1u) : 1u;
                atom_add_release_u32(a.bar, tinc);
            }
            // every word flips once per barrier, so the group word's bit 31
            // before this arrival is the top word's before the barrier
            old = gold;
        } else {
            const unsigned inc = (blockIdx.x == 0) ? 0x80000000u - (gridDim.x - 1u) : 1u;
            old = atom_add_release_u32(a.bar, inc);
        }
        int ok = 1;
        unsigned long long t0 = 0;
        for (unsigned it = 0; ((ld_acquire_u32(a.bar) ^ old) & 0x80000000u) == 0u; ++it) {
            if ((it & 63u) != 0u) continue;  // the time limit is read every 64 polls
            const unsigned long long t = globaltimer_ns();
            if (it == 0) {
                t0 = t;
            } else if (t - t0 > kBarrierLimitNs) {
                // a CTA that gives up returns; every other CTA's wait then ends
                // at its own limit, so the launch always finishes
                raise_status(a, DEM_ERR_TIMEOUT);
                ok = 0;
                break;
            }
        }
        s_ok = ok;
    }
    if (threadIdx.x < 32) {
        __syncwarp();  // the barrier's acquire, by lane 0, comes before the other lanes' reads
        load_ctl(a, next_ph, ctl);
    }
    __syncthreads();
    return s_ok != 0;
}

// Barrier of the substeps, among CTAs 0..n-1, that also carries "an element has
// escaped": bits 52..63 count arrivals as above (bit 63 flips at the last one
// and the carry falls off), bits 0..25 and 26..51 count CTAs with an escape at
// barriers of parity 0 and 1.  No CTA can be two barriers ahead, so a field
// stands still while its barrier's CTAs read it; base holds its last value.
// The word that ends the wait thus says whether the escape counters need
// reading at all: a load less on every substep's critical path (0.4 us).  In a
// call of so many substeps that a count could carry into the next bits (sub_flags
// is 0) none is added, and the counters are always read.
// Returns 0, 1 (read the counters) or -1 (the wait ran out).
struct SubSync {
    unsigned long long base[2];
    int flag, res;
};

// What a CTA of a barrier's n adds to the word.
__host__ __device__ __forceinline__ unsigned long long sub_arrival(bool first, unsigned n, int parity, bool escape,
                                                                   bool counted) {
    const unsigned long long add = (first ? 2048ull - (n - 1u) : 1ull) << 52;
    return add + (escape && counted ? 1ull << (parity ? 26 : 0) : 0ull);
}

template <typename T>
__device__ int sub_barrier(const KArgs<T>& a, unsigned n, int parity, SubSync* y) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const int sh = parity ? 26 : 0;
        const unsigned long long add = sub_arrival(blockIdx.x == 0, n, parity, y->flag != 0, a.sub_flags != 0);
        y->flag = 0;
        const unsigned long long old = atom_add_release_u64(a.sub_bar, add);
        unsigned long long now, t0 = 0;
        int res = 0;
        for (unsigned it = 0; (((now = ld_acquire_u64(a.sub_bar)) ^ old) >> 63) == 0ull; ++it) {
            if ((it & 63u) != 0u) continue;  // the time limit is read every 64 polls
            const unsigned long long t = globaltimer_ns();
            if (it == 0) {
                t0 = t;
            } else if (t - t0 > kBarrierLimitNs) {
                raise_status(a, DEM_ERR_TIMEOUT);
                res = -1;
                break;
            }
        }
        if (res == 0) {
            const unsigned long long f = (now >> sh) & 0x3ffffffull;
            res = (f != y->base[parity] || !a.sub_flags) ? 1 : 0;
            y->base[parity] = f;
        }
        y->res = res;
    }
    __syncthreads();
    return y->res;
}

// ─── grid hash ──────────────────────────────────────────────────────────────
template <typename T>
__device__ __forceinline__ int2 cell_of(const KArgs<T>& a, T x, T y) {
    const double lim = 1073741823.0;  // keep cell indices inside int range
    double cx = fmin(fmax(floor((double)x / (double)a.cell), -lim), lim);
    double cy = fmin(fmax(floor((double)y / (double)a.cell), -lim), lim);
    return make_int2((int)cx, (int)cy);
}
// The system id is part of the key: systems that occupy the same space (planner
// rollouts on overlapping windows) hash their cells to different buckets, so a
// neighbourhood scan reads its own system's entries only.
__device__ __forceinline__ int bucket_of(int2 c, int sys, int n_buckets) {
    unsigned h = (unsigned)c.x * 73856093u ^ (unsigned)c.y * 19349663u ^ (unsigned)sys * 83492791u;
    return (int)(h & (unsigned)(n_buckets - 1));
}
template <typename T>
__device__ __forceinline__ int sys_id(const KArgs<T>& a, int e) {
    return a.nsys > 1 ? a.sys_of[e] : 0;
}

// Neighbour lists are Verlet lists over reference positions: list(e) holds every
// o with |ref_e - ref_o| < R_e + R_o, where the reach R is an element's radius
// plus its margin m: skin / 2, and more for an element that moves fast, as far
// as R stays within reach_max (elements smaller than the largest have room for
// a wider margin in the same stencil of grid cells).  An element whose position
// leaves the ball of radius h = 0.891 m around its reference "escapes": it takes
// a new reference and reach, and every element within reach of it rebuilds its
// list.  With |p - ref| < m for every element at every use of the lists, any
// pair closer than r_e + r_o is in both lists, so the contact set equals the
// all-pairs one of the reference (jax_ice_state.py:212-214).
//
// Every substep tests each element it moved against its h, the limit of the
// very next use; an element past it is processed in an escape phase before the
// next substep, so every use of a list is valid.  Most lists are kept up once
// per frame instead, beside the ship contact, off the substeps' critical path:
// cull finds the elements that have moved past h, and the active ones that
// their velocity would carry past 0.9 h by the frame's end; the near phase
// marks their neighbourhoods and gives them a new reference, ahead of them
// along their velocity; the cforce phase rebuilds the marked lists.  Only an
// element that the ice accelerates hard within a frame then meets an escape
// phase.  (A reference is any point within m of the element at each use; it
// need not be a place the element has been.)
//
// What this is for: with the lists kept up inside the substeps (re-referencing
// at the even ones, rebuilding at the odd ones) a force phase was as long as a
// rebuild and the element's force after it, 10 us, and with one margin for all
// a frame of the 12k-element field had 1.7 escape phases.  With the upkeep beside
// the ship contact, and the elements' loads as they were, a force phase there took
// 7.8 us and one frame in five had an escape phase: 149 -> 122 us a frame; the
// 237k-element pack 205 -> 150 us, all of it active 842 -> 750 us.  (With the
// elements in shared memory a substep is 3.5 to 4.4 us and such a frame 81.)

template <typename T>
__device__ __forceinline__ bool escaped_from(T px, T py, T rx, T ry, T h) {
    const bool fp = jfinite(px) && jfinite(py);
    const bool fr = jfinite(rx) && jfinite(ry);
    if (fp != fr) return true;
    if (!fp) return false;
    // |p - ref| > h; h carries a 1 % margin so rounding of the test can only make
    // an element escape early, never late
    const T dx = px - rx, dy = py - ry;
    return dx * dx + dy * dy > h * h;
}

// one atomic per CTA: add the CTA's count of `v` to *ctr (all threads must call)
__device__ __forceinline__ void cta_count_add(unsigned* ctr, int v) {
    __shared__ int s_cnt;
    if (threadIdx.x == 0) s_cnt = 0;
    __syncthreads();
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&s_cnt, v);
    __syncthreads();
    if (threadIdx.x == 0 && s_cnt) atomicAdd(ctr, (unsigned)s_cnt);
    __syncthreads();
}

// Grid-hash buckets of fixed capacity.  An element that escapes is appended to
// the bucket of its new home cell; its old entry goes stale and is ignored
// (its home cell no longer matches) until the next compaction drops it.
template <typename T>
__device__ __forceinline__ void grid_put(const KArgs<T>& a, int e, T px, T py) {
    if (!(jfinite(px) && jfinite(py))) {
        a.ecell[e] = make_int2(INT_MIN, INT_MIN);
        return;
    }
    int2 c = cell_of(a, px, py);
    a.ecell[e] = c;
    int b = bucket_of(c, sys_id(a, e), a.n_buckets);
    int slot = atomicAdd(&a.bcnt[b], 1);
    if (slot < a.bucket_cap) {
        a.bitems[(size_t)b * a.bucket_cap + slot] = e;
    } else {
        raise_status(a, DEM_ERR_CAPACITY);
        atomicOr((unsigned long long*)&a.stats[5], 1ull);  // a grid bucket overflowed
    }
    if (slot + 1 > a.bucket_cap / 2) atomicMax((unsigned long long*)&a.stats[2], (unsigned long long)(slot + 1));
}

// Warp-cooperative neighbourhood scan: the 9 stencil buckets' entries are
// spread over the lanes; `fn(o)` runs on the lane that found o.  Every element
// within reach + R_o of (px, py) (double test with a margin) is visited; an
// element can be visited twice (stale + current entry in one bucket).
template <typename T, typename Fn>
__device__ __forceinline__ void warp_near_at(const KArgs<T>& a, int e, T px, T py, T reach, int2 c, Fn fn) {
    const int lane = threadIdx.x & 31;
    if (c.x == INT_MIN) return;
    // lanes 0..8 own one stencil bucket each; warp prefix of their fills
    const int se = sys_id(a, e);
    int b = 0, m = 0;
    if (lane < 9) {
        const int2 cc = make_int2(c.x + (lane % 3) - 1, c.y + (lane / 3) - 1);
        b = bucket_of(cc, se, a.n_buckets);
        m = min(a.bcnt[b], a.bucket_cap);
    }
    int incl = m;
    for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += v;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    const int excl = incl - m;
    // uniform trip count: every lane executes every shuffle
    for (int t0 = 0; t0 < total; t0 += 32) {
        const int t = t0 + lane;
        // bucket j holding entry t: the last stencil lane whose prefix start <= t
        int q = 0, qb = 0, qe = 0;
        for (int j = 0; j < 9; ++j) {
            const int ej = __shfl_sync(0xffffffffu, excl, j);
            const int bj = __shfl_sync(0xffffffffu, b, j);
            if (t >= ej) {
                q = j;
                qb = bj;
                qe = ej;
            }
        }
        if (t >= total) continue;
        // entries are written after their slot is claimed: a concurrent insertion
        // can show an old value (-1 or a valid stale index), never an invalid one
        const int o = ((volatile const int*)a.bitems)[(size_t)qb * a.bucket_cap + (t - qe)];
        if (o < 0 || o >= a.n || o == e) continue;
        if (a.nsys > 1 && a.sys_of[o] != se) continue;  // systems never interact
        const int2 cc = make_int2(c.x + (q % 3) - 1, c.y + (q / 3) - 1);
        const int2 oc = a.ecell[o];
        if (oc.x != cc.x || oc.y != cc.y) continue;  // stale entry or hash collision
        const double ddx = (double)a.pos_ref[2 * o] - (double)px, ddy = (double)a.pos_ref[2 * o + 1] - (double)py;
        const double lim = ((double)reach + (double)a.reach[o]) * (1.0 + 1e-5) + 1e-6;
        if (ddx * ddx + ddy * ddy < lim * lim) fn(o);
    }
}

// The same neighbourhood scan by a whole CTA (every thread must call it with
// the same e): the stencil entries are spread over all threads, so the scan
// takes one or two dependent load rounds instead of the warp's several.
template <typename T, typename Fn>
__device__ __forceinline__ void block_near_at(const KArgs<T>& a, int e, T px, T py, T reach, int2 c, Fn fn) {
    __shared__ int s_b[9];
    __shared__ int s_start[10];
    if (c.x == INT_MIN) return;  // depends on e only: uniform over the CTA
    if (threadIdx.x < 9) {
        const int2 cc = make_int2(c.x + ((int)threadIdx.x % 3) - 1, c.y + ((int)threadIdx.x / 3) - 1);
        const int b = bucket_of(cc, sys_id(a, e), a.n_buckets);
        s_b[threadIdx.x] = b;
        s_start[threadIdx.x + 1] = min(a.bcnt[b], a.bucket_cap);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        s_start[0] = 0;
        for (int j = 0; j < 9; ++j) s_start[j + 1] += s_start[j];
    }
    __syncthreads();
    const int total = s_start[9];
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int q = 0;
        while (q < 8 && t >= s_start[q + 1]) ++q;
        // entries are written after their slot is claimed: a concurrent insertion
        // can show an old value (-1 or a valid stale index), never an invalid one
        const int o = ((volatile const int*)a.bitems)[(size_t)s_b[q] * a.bucket_cap + (t - s_start[q])];
        if (o < 0 || o >= a.n || o == e) continue;
        if (a.nsys > 1 && a.sys_of[o] != a.sys_of[e]) continue;  // systems never interact
        const int2 cc = make_int2(c.x + (q % 3) - 1, c.y + (q / 3) - 1);
        const int2 oc = a.ecell[o];
        if (oc.x != cc.x || oc.y != cc.y) continue;  // stale entry or hash collision
        const double ddx = (double)a.pos_ref[2 * o] - (double)px, ddy = (double)a.pos_ref[2 * o + 1] - (double)py;
        const double lim = ((double)reach + (double)a.reach[o]) * (1.0 + 1e-5) + 1e-6;
        if (ddx * ddx + ddy * ddy < lim * lim) fn(o);
    }
    __syncthreads();  // s_b / s_start are reused by the next call
}

template <typename T, typename Fn>
__device__ __forceinline__ void warp_near(const KArgs<T>& a, int e, Fn fn) {
    warp_near_at(a, e, a.pos_ref[2 * e], a.pos_ref[2 * e + 1], a.reach[e], a.ecell[e], fn);
}

// Append `flag`-set lanes' values to list[atomicAdd(cnt)] with one atomic per warp.
__device__ __forceinline__ void warp_append(int* list, int* cnt, bool flag, int v) {
    const unsigned am = __activemask();
    const unsigned bal = __ballot_sync(am, flag);
    if (!bal) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(am) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(cnt, __popc(bal));
    base = __shfl_sync(am, base, leader);
    if (flag) list[base + __popc(bal & ((1u << lane) - 1u))] = v;
}

// Two flagged values per lane, appended with one atomic per warp (the
// frame's bond list: up to two slots per lane and step).
__device__ __forceinline__ void warp_append2(int* list, int* cnt, bool f0, int v0, bool f1, int v1) {
    const unsigned am = __activemask();
    const unsigned bal0 = __ballot_sync(am, f0), bal1 = __ballot_sync(am, f1);
    const int n0 = __popc(bal0), n = n0 + __popc(bal1);
    if (!n) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(am) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(cnt, n);
    base = __shfl_sync(am, base, leader);
    const unsigned lt = (1u << lane) - 1u;
    if (f0) list[base + __popc(bal0 & lt)] = v0;
    if (f1) list[base + n0 + __popc(bal1 & lt)] = v1;
}

// Build element e's list (one warp): candidates are gathered in shared memory,
// sorted and deduplicated, then stored so that indices above e come first
// (ascending), then indices below e (ascending) — the order in which the
// reference's scatter-adds reach e: pairs (e, j>e) through pair_i, then pairs
// (i<e, e) through pair_j (jax_simulation.py:152-162).
template <typename T>
__device__ void warp_build(const KArgs<T>& a, int e) {
    __shared__ int s_buf[kThreads / 32][2 * kMaxNbLocal];  // one slice per warp, for every caller
    __shared__ int s_cnt[kThreads / 32];
    int* sbuf = s_buf[threadIdx.x >> 5];
    int* scnt = &s_cnt[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    if (lane == 0) *scnt = 0;
    __syncwarp();
    const int cap = 2 * kMaxNbLocal;
    warp_near(a, e, [&](int o) {
        const int slot = atomicAdd(scnt, 1);
        if (slot < cap) sbuf[slot] = o;
    });
    __syncwarp();
    const int found = *scnt;
    const int cnt = min(found, cap);
    // drop repeats (a stale and a current entry of one element), in parallel:
    // entry i stays if no earlier entry holds the same index.  All lanes walk
    // the buffer together (broadcast reads, no early exit, so the reads
    // pipeline); a lane holds entries lane, lane + 32, ...
    constexpr int kPer = (2 * kMaxNbLocal + 31) / 32;
    int v[kPer];
    bool keep[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int i = lane + 32 * k;
        v[k] = (i < cnt) ? sbuf[i] : -1;
        keep[k] = i < cnt;
    }
    if (cnt <= 64) {
#pragma unroll 4
        for (int j = 0; j < cnt; ++j) {
            const int u = sbuf[j];
            keep[0] = keep[0] && !(j < lane && u == v[0]);
            keep[1] = keep[1] && !(j < lane + 32 && u == v[1]);
        }
    } else {
#pragma unroll 2
        for (int j = 0; j < cnt; ++j) {
            const int u = sbuf[j];
#pragma unroll
            for (int k = 0; k < kPer; ++k) keep[k] = keep[k] && !(j < lane + 32 * k && u == v[k]);
        }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kPer; ++k)
        if (lane + 32 * k < cnt && !keep[k]) sbuf[lane + 32 * k] = -1;
    __syncwarp();
    int nk = 0, nlow = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        nk += keep[k] ? 1 : 0;
        nlow += (keep[k] && v[k] < e) ? 1 : 0;
    }
    const int w = __reduce_add_sync(0xffffffffu, nk);
    const int split = __reduce_add_sync(0xffffffffu, nlow);  // kept indices below e
    if (lane == 0) {
        if (found > cap || w > a.max_nb) {
            raise_status(a, DEM_ERR_CAPACITY);
            atomicOr((unsigned long long*)&a.stats[5], 2ull);  // a neighbour list overflowed
        }
        if (w > 16) atomicMax((unsigned long long*)&a.stats[1], (unsigned long long)w);
    }
    const int m = min(w, a.max_nb);
    // slot of a kept index = its rank among the kept ones, indices above e first
    int r[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) r[k] = 0;
    if (cnt <= 64) {
#pragma unroll 4
        for (int j = 0; j < cnt; ++j) {
            const int u = sbuf[j];
            r[0] += (u >= 0 && u < v[0]) ? 1 : 0;
            r[1] += (u >= 0 && u < v[1]) ? 1 : 0;
        }
    } else {
#pragma unroll 2
        for (int j = 0; j < cnt; ++j) {
            const int u = sbuf[j];
#pragma unroll
            for (int k = 0; k < kPer; ++k) r[k] += (u >= 0 && u < v[k]) ? 1 : 0;
        }
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        if (!keep[k]) continue;
        const int pos = (v[k] > e) ? r[k] - split : (w - split) + r[k];
        if (pos < m) a.nbr[(size_t)pos * a.n + e] = v[k];
    }
    if (lane == 0) a.ncnt[e] = m;
    __syncwarp();
}

// The same list build by a whole CTA (every thread must call it with the same
// e): the stencil entries are scanned in one load round (block_near_at), and
// thread t checks gathered candidate t (at most 2 kMaxNbLocal <= kThreads).
// The list equals warp_build's: the same candidates, repeats dropped, the
// same order and the same capacity flags.
template <typename T>
__device__ void block_build(const KArgs<T>& a, int e) {
    constexpr int cap = 2 * kMaxNbLocal;
    static_assert(cap <= kThreads, "one candidate per thread");
    __shared__ int s_c[cap];
    __shared__ int s_n;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    block_near_at(a, e, a.pos_ref[2 * e], a.pos_ref[2 * e + 1], a.reach[e], a.ecell[e], [&](int o) {
        const int slot = atomicAdd(&s_n, 1);
        if (slot < cap) s_c[slot] = o;
    });  // ends with __syncthreads (or returns at once, before any, for an element without a cell)
    __syncthreads();
    const int found = s_n;
    const int cnt = min(found, cap);
    const int t = threadIdx.x;
    const int v = (t < cnt) ? s_c[t] : -1;
    bool keep = t < cnt;
    if ((t & ~31) < cnt) {  // warp-uniform: warps holding candidates
#pragma unroll 4
        for (int j = 0; j < cnt; ++j) {
            const int u = s_c[j];
            keep = keep && !(j < t && u == v);
        }
    }
    const int w = __syncthreads_count(keep);
    const int split = __syncthreads_count(keep && v < e);  // kept indices below e
    if (t < cnt && !keep) s_c[t] = -1;
    __syncthreads();
    if (t == 0) {
        if (found > cap || w > a.max_nb) {
            raise_status(a, DEM_ERR_CAPACITY);
            atomicOr((unsigned long long*)&a.stats[5], 2ull);  // a neighbour list overflowed
        }
        if (w > 16) atomicMax((unsigned long long*)&a.stats[1], (unsigned long long)w);
    }
    const int m = min(w, a.max_nb);
    if (keep) {
        int r = 0;
#pragma unroll 4
        for (int j = 0; j < cnt; ++j) {
            const int u = s_c[j];
            r += (u >= 0 && u < v) ? 1 : 0;
        }
        const int pos = (v > e) ? r - split : (w - split) + r;
        if (pos < m) a.nbr[(size_t)pos * a.n + e] = v;
    }
    if (t == 0) a.ncnt[e] = m;
    __syncthreads();  // the list is complete for the CTA; s_c / s_n are reused by the next call
}

// Stamp o dirty for this round; the first stamper lists it.
template <typename T>
__device__ __forceinline__ void mark_dirty(const KArgs<T>& a, int o, int s, unsigned round) {
    if (atomicExch(&a.dirty[o], round) != round) a.dirty_list[atomicAdd(&a.dirty_cnt[s], 1)] = o;
}

// Move escaped element e to its new reference (px, py) and home bucket; old and
// new buckets are queued for compaction at the next frame start, the
// independent atomics of each level issued together.
template <typename T>
__device__ __forceinline__ void rereference(const KArgs<T>& a, int e, T px, T py, T reach, int2 c) {
    const int2 old = a.ecell[e];
    a.reach[e] = reach;
    a.pos_ref[2 * e] = px;
    a.pos_ref[2 * e + 1] = py;
    a.ecell[e] = c;
    const int se = sys_id(a, e);
    const int bo = (old.x != INT_MIN) ? bucket_of(old, se, a.n_buckets) : -1;
    const int bn = (c.x != INT_MIN) ? bucket_of(c, se, a.n_buckets) : -1;
    const int slot = (bn >= 0) ? atomicAdd(&a.bcnt[bn], 1) : 0;
    const int fo = (bo >= 0) ? atomicExch(&a.bflag[bo], 1) : 1;
    const int fn = (bn >= 0 && bn != bo) ? atomicExch(&a.bflag[bn], 1) : 1;
    if (bn >= 0) {
        if (slot < a.bucket_cap) {
            a.bitems[(size_t)bn * a.bucket_cap + slot] = e;
        } else {
            raise_status(a, DEM_ERR_CAPACITY);
            atomicOr((unsigned long long*)&a.stats[5], 1ull);  // a grid bucket overflowed
        }
        if (slot + 1 > a.bucket_cap / 2) atomicMax((unsigned long long*)&a.stats[2], (unsigned long long)(slot + 1));
    }
    if (fo == 0) a.comp_list[atomicAdd(a.comp_cnt, 1) & (a.n_buckets - 1)] = bo;
    if (fn == 0) a.comp_list[atomicAdd(a.comp_cnt, 1) & (a.n_buckets - 1)] = bn;
}

// Whether o's list already holds e, whose reference was (rx, ry) with reach re:
// o's list was built with e's reference there, and it takes every element
// within (R_o + re)(1 + 1e-5) + 1e-6 of its own reference (warp_near_at, seen
// from o).  The test is made a little stricter than the builder's, so rounding
// can only send o to a needless rebuild.
template <typename T>
__device__ __forceinline__ bool list_holds(const KArgs<T>& a, int o, double rx, double ry, double re) {
    const double dx = rx - (double)a.pos_ref[2 * o], dy = ry - (double)a.pos_ref[2 * o + 1];
    const double lim = ((double)a.reach[o] + re) * (1.0 + 1e-5) + 1e-6;
    return dx * dx + dy * dy < lim * lim * (1.0 - 1e-9);
}

// The new reference of an escaped element: position, cell and reach.
template <typename T>
struct NewRef {
    T x, y, reach;
    int2 c;
};

// For element e at (px, py) moving at (vx, vy) (a frozen one: 0): a margin of
// skin / 2 plus two frames' movement, up to the skin and to what the grid's
// cells leave room for, and a reference ahead of the element by up to 0.53 of
// the margin and two frames.
template <typename T>
__device__ __forceinline__ NewRef<T> new_ref(const KArgs<T>& a, int e, T px, T py, T vx, T vy) {
    NewRef<T> q;
    q.x = px;
    q.y = py;
    const T r = a.radii[e];
    T m = T(0.5) * a.skin;
    const T d = jsqrt(vx * vx + vy * vy) * a.t_frame;
    if (d > T(0)) {  // not for NaN
        m = jmax(m, jmin(jmin(m + T(2) * d, a.margin_max), a.reach_max - r));
        const T lead = jmin(T(2), T(0.53) * m / d) * a.t_frame;
        const T qx = px + vx * lead, qy = py + vy * lead;
        if (jfinite(qx) && jfinite(qy)) {
            q.x = qx;
            q.y = qy;
        }
    }
    q.reach = r + m;
    q.c = (jfinite(q.x) && jfinite(q.y)) ? cell_of(a, q.x, q.y) : make_int2(INT_MIN, INT_MIN);
    return q;
}

// Escape distance of element e from its reference: 0.891 of its margin.
template <typename T>
__device__ __forceinline__ T esc_h_of(const KArgs<T>& a, int e, T r) {
    return T(0.891) * (a.reach[e] - r);
}

// Stamp dirty what escaped element e's new reference brings into reach, and e
// itself, for the rebuild at substep s; then re-reference e.  By a whole CTA,
// or by a warp.
template <typename T>
__device__ __forceinline__ void escape_block(const KArgs<T>& a, int e, const NewRef<T>& q, int s, unsigned round) {
    const double rx = (double)a.pos_ref[2 * e], ry = (double)a.pos_ref[2 * e + 1], re = (double)a.reach[e];
    const bool had = isfinite(rx) && isfinite(ry) && a.ecell[e].x != INT_MIN;
    block_near_at(a, e, q.x, q.y, q.reach, q.c, [&](int o) {
        if (!(had && list_holds(a, o, rx, ry, re))) mark_dirty(a, o, s, round);
    });
    __syncthreads();  // every thread is done with e's old reference
    if (threadIdx.x == 0) {
        mark_dirty(a, e, s, round);
        rereference(a, e, q.x, q.y, q.reach, q.c);
    }
}
template <typename T>
__device__ __forceinline__ void escape_warp(const KArgs<T>& a, int e, const NewRef<T>& q, int s, unsigned round) {
    const double rx = (double)a.pos_ref[2 * e], ry = (double)a.pos_ref[2 * e + 1], re = (double)a.reach[e];
    const bool had = isfinite(rx) && isfinite(ry) && a.ecell[e].x != INT_MIN;
    warp_near_at(a, e, q.x, q.y, q.reach, q.c, [&](int o) {
        if (!(had && list_holds(a, o, rx, ry, re))) mark_dirty(a, o, s, round);
    });
    __syncwarp();  // every lane is done with e's old reference
    if ((threadIdx.x & 31) == 0) {
        mark_dirty(a, e, s, round);
        rereference(a, e, q.x, q.y, q.reach, q.c);
    }
}

// One rebuild round before substep s.  For each escaped element e (a CTA each
// when they fit one per CTA, else a warp each): e is stamped dirty, and so is
// every element o within reach of e's new reference whose list does not hold e
// yet (e was out of o's reach at its old reference).  An o whose list holds e
// keeps it, and keeps an entry of an e that moved out of reach: such an entry is
// a candidate that does not touch, whose terms are exact zeros, and it goes at
// o's next rebuild.  The same unit then re-references e, after reading e's old
// reference.  Candidates' references are read concurrently with other escaped
// elements' re-referencing; those elements rebuild their own lists anyway.
// When most elements escaped, every list is rebuilt instead (no marking).
template <typename T>
__device__ void phase_escape(const KArgs<T>& a, const Frame<T>& F, unsigned cnt, int s, unsigned round, bool all,
                             int nblk) {
    // by CTAs 0..nblk-1
    const int n_esc = (int)cnt;
    const T *kin = a.kin[s & 1], *kvin = a.kvel[s & 1];
    auto ref_of = [&](int e) {
        const typename vec2_of<T>::type v = ld2(kvin, e);
        const bool on = F.dst.active[e] != 0;  // a frozen element stays, whatever its velocity
        return new_ref(a, e, kin[4 * (size_t)e], kin[4 * (size_t)e + 1], on ? v.x : T(0), on ? v.y : T(0));
    };
    if (all) {
        const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
        const int gsz = nblk * blockDim.x;
        for (int q = gtid; q < n_esc; q += gsz) {
            const int e = a.esc_list[q];
            const NewRef<T> q2 = ref_of(e);
            rereference(a, e, q2.x, q2.y, q2.reach, q2.c);
        }
    } else if (a.mark_split == DEM_SPLIT_CTA || (a.mark_split == DEM_SPLIT_AUTO && n_esc <= nblk)) {
        // few escapes: a CTA per element, its stencil entries in one load round
        for (int q = blockIdx.x; q < n_esc; q += nblk) {
            const int e = a.esc_list[q];
            escape_block(a, e, ref_of(e), s, round);
        }
    } else {
        // many escapes (batched windows): a warp per element
        const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        const int nwarps = (nblk * blockDim.x) >> 5;
        for (int q = warp; q < n_esc; q += nwarps) {
            const int e = a.esc_list[q];
            escape_warp(a, e, ref_of(e), s, round);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd((unsigned long long*)&a.stats[0], 1ull);
        atomicAdd((unsigned long long*)&a.stats[3], (unsigned long long)n_esc);
    }
}

// Whether so many elements escaped (a handle's first call, a call from another
// state) that every list is rebuilt, by the escape and build_all phases, instead
// of the marked ones.
template <typename T>
__device__ __forceinline__ bool rebuild_all(const KArgs<T>& a, unsigned cnt) {
    return (unsigned long long)cnt * 8ull > (unsigned long long)a.n;
}
// List upkeep at the frame's start (see the notes on the Verlet lists): whether
// this frame's escapes are processed beside the ship contact; when every list is
// rebuilt, that is done before substep 0.
template <typename T>
__device__ __forceinline__ bool upkeep_now(const KArgs<T>& a, unsigned cnt) {
    return cnt != 0u && !rebuild_all(a, cnt);
}

// Near phase: mark and re-reference the frame's escaped elements.  A few take
// a CTA each, from the grid's end (the near elements fill it from the front);
// many a warp each, after the warp's near elements.
template <typename T>
__device__ void upkeep_mark(const KArgs<T>& a, const Frame<T>& F, int n_esc, unsigned round) {
    const bool by_cta = a.mark_split == DEM_SPLIT_CTA || (a.mark_split == DEM_SPLIT_AUTO && n_esc <= (int)gridDim.x);
    const int last = by_cta ? gridDim.x - 1 - blockIdx.x : ((gridDim.x - blockIdx.x) * blockDim.x - 1 - threadIdx.x) >> 5;
    const int step = by_cta ? gridDim.x : (gridDim.x * blockDim.x) >> 5;
    for (int q = last; q < n_esc; q += step) {
        const int e = a.esc_list[q];
        const typename vec2_of<T>::type p = ld2(F.src.pos, e), v = ld2(F.src.vel, e);
        const bool on = F.src.active[e] != 0;
        const NewRef<T> ref = new_ref(a, e, p.x, p.y, on ? v.x : T(0), on ? v.y : T(0));
        if (by_cta)
            escape_block(a, e, ref, 0, round);
        else
            escape_warp(a, e, ref, 0, round);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd((unsigned long long*)&a.stats[0], 1ull);
        atomicAdd((unsigned long long*)&a.stats[3], (unsigned long long)n_esc);
    }
}

// Cforce phase: rebuild the marked lists, a CTA each from the grid's end, or a
// warp each when there are many.
template <typename T>
__device__ void upkeep_build(const KArgs<T>& a, int nd) {
    if (a.mark_split == DEM_SPLIT_CTA || (a.mark_split == DEM_SPLIT_AUTO && nd <= 2 * (int)gridDim.x)) {
        for (int q = gridDim.x - 1 - blockIdx.x; q < nd; q += gridDim.x) block_build(a, a.dirty_list[q]);
    } else {
        const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        const int nwarps = (gridDim.x * blockDim.x) >> 5;
        for (int q = warp; q < nd; q += nwarps) warp_build(a, a.dirty_list[q]);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd((unsigned long long*)&a.stats[4], (unsigned long long)nd);
}

// Rebuild every list (when most elements escaped at once).
template <typename T>
__device__ void phase_build_all(const KArgs<T>& a, int nblk) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (nblk * blockDim.x) >> 5;
    for (int e = warp; e < a.n; e += nwarps) warp_build(a, e);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd((unsigned long long*)&a.stats[4], (unsigned long long)a.n);
}

// Drop stale and duplicate entries of the queued buckets (run while nothing
// reads or writes the grid).
template <typename T>
__device__ void compact_buckets(const KArgs<T>& a, int start, int end) {
    // one warp per queued bucket: lanes test 32 entries at a time; an entry
    // stays if it is current (its home cell hashes here) and no earlier entry
    // holds the same element; kept entries move to the front in their order
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int nq = (int)((unsigned)end - (unsigned)start);
    for (int i = warp; i < nq; i += nwarps) {
        const int b = a.comp_list[(start + i) & (a.n_buckets - 1)];
        const int m = min(a.bcnt[b], a.bucket_cap);
        int* it = a.bitems + (size_t)b * a.bucket_cap;
        int w = 0;
        for (int k0 = 0; k0 < m; k0 += 32) {
            const int k = k0 + lane;
            const int o = (k < m) ? it[k] : -1;
            bool keep = false;
            if (o >= 0 && o < a.n) {
                const int2 c = a.ecell[o];
                keep = c.x != INT_MIN && bucket_of(c, sys_id(a, o), a.n_buckets) == b;
            }
            for (int q = 0; keep && q < w; ++q)  // kept in earlier chunks
                if (it[q] == o) keep = false;
            for (int j = 0; j < 32; ++j) {       // earlier lanes of this chunk
                const int oj = __shfl_sync(0xffffffffu, o, j);
                const bool kj = __shfl_sync(0xffffffffu, keep, j);
                if (j < lane && kj && oj == o) keep = false;
            }
            const unsigned bal = __ballot_sync(0xffffffffu, keep);
            __syncwarp();  // every lane has read its entry before any is overwritten
            if (keep) it[w + __popc(bal & ((1u << lane) - 1u))] = o;
            w += __popc(bal);
            __syncwarp();
        }
        for (int k = w + lane; k < m; k += 32) it[k] = -1;
        if (lane == 0) {
            a.bcnt[b] = w;
            a.bflag[b] = 0;
        }
    }
}

// ─── ship contact (jax_geometry.py) ─────────────────────────────────────────
// Analytic tapered hull test of one point (jax_geometry.py:42-134).
template <typename T>
struct HullPose {
    T sx, sy, c_neg, s_neg, c_h, s_h, hl, hb, hb005;
};

template <typename T>
__device__ __forceinline__ void hull_point(const HullPose<T>& H, T px, T py, T& pen, T& nx, T& ny) {
    const T bts = T(0.6);
    const T one_m_bts = T(1.0 - 0.6);
    T dx = px - H.sx;
    T dy = py - H.sy;
    T rel_x = H.c_neg * dx - H.s_neg * dy;
    T rel_y = H.s_neg * dx + H.c_neg * dy;
    T x_rel = rel_x / H.hl;
    bool in_bow = x_rel < -bts;
    T t_bow = jclip((-x_rel - bts) / one_m_bts, T(0), T(1));
    T hb_bow = H.hb * (T(1) - T(0.9) * jpow(t_bow, T(1.5)));
    hb_bow = jmax(hb_bow, H.hb005);
    T hb_loc = in_bow ? hb_bow : H.hb;
    T arel_y = fabs(rel_y);
    bool inside = (rel_x >= -H.hl) && (rel_x <= H.hl) && (arel_y <= hb_loc);
    if (!inside) {
        pen = T(0);
        nx = T(0);
        ny = T(0);
        return;
    }
    T d_bow = rel_x + H.hl;
    T d_side = hb_loc - arel_y;
    T nxb, nyb, praw;
    if (in_bow) {
        T ang = T(0.3) + T(0.5) * t_bow;
        nxb = -jcos(ang);
        nyb = jsign(rel_y) * jsin(ang);
        praw = jmin(d_bow, d_side) + T(0.5);
    } else {
        bool side = d_side <= d_bow;
        nxb = side ? T(0) : T(-1);
        nyb = side ? jsign(rel_y) : T(0);
        praw = side ? d_side : d_bow;
    }
    nx = H.c_h * nxb - H.s_h * nyb;
    ny = H.s_h * nxb + H.c_h * nyb;
    pen = jmax(praw, T(0));
}

// ─── fixed-order sums (deterministic, independent of the grid size) ─────────
// lane 0 receives the warp's sum (shuffle-down tree)
__device__ __forceinline__ double warp_sum_lane0(double v) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    return v;
}

// thread 0 receives the block's sums: a tree in each warp, then over the warps
template <int N>
__device__ __forceinline__ void block_sum3(double v0, double v1, double v2, double* out3) {
    constexpr int kW = N / 32;
    __shared__ double sh[3][kW];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    v0 = warp_sum_lane0(v0);
    v1 = warp_sum_lane0(v1);
    v2 = warp_sum_lane0(v2);
    if (lane == 0) {
        sh[0][w] = v0;
        sh[1][w] = v1;
        sh[2][w] = v2;
    }
    __syncthreads();
    if (w == 0) {
        double u0 = lane < kW ? sh[0][lane] : 0.0, u1 = lane < kW ? sh[1][lane] : 0.0;
        double u2 = lane < kW ? sh[2][lane] : 0.0;
        u0 = warp_sum_lane0(u0);
        u1 = warp_sum_lane0(u1);
        u2 = warp_sum_lane0(u2);
        if (lane == 0) {
            out3[0] = u0;
            out3[1] = u1;
            out3[2] = u2;
        }
    }
    __syncthreads();  // sh is reused by the next call
}

template <typename T>
__device__ __forceinline__ HullPose<T> hull_pose(const KArgs<T>& a, const T* eta) {
    HullPose<T> H;
    H.sx = eta[0];
    H.sy = eta[1];
    const T spsi = eta[2];
    jsincos(-spsi, &H.s_neg, &H.c_neg);
    jsincos(spsi, &H.s_h, &H.c_h);
    H.hl = T(a.P.half_len);
    H.hb = T(a.P.half_beam);
    H.hb005 = T(a.P.half_beam * 0.05);
    return H;
}

// Force chunk of element e: chunks of kThreads elements from each system's
// first element.
template <typename T>
__device__ __forceinline__ int chunk_of(const KArgs<T>& a, int e) {
    if (a.nsys == 1) return e / kThreads;
    const int s = a.sys_of[e];
    return a.part_base[s] + (e - (s > 0 ? a.sys_end[s - 1] : 0)) / kThreads;
}

// ─── P_CULL: elements whose bounding circle reaches the hull; escapes ───────
template <typename T>
__device__ void phase_cull(const KArgs<T>& a, const Frame<T>& F, int comp_start, int comp_end) {
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const int gsz = gridDim.x * blockDim.x;
    const T reach = a.hull_r * T(1.0001) + T(1e-3);
    // nothing reads the grid in this phase: drop stale entries queued last frame
    compact_buckets(a, comp_start, comp_end);
    if (gtid == 0) {
        a.act_cnt[0] = 0;  // read last by the previous frame's force phases
        *a.fb_cnt = 0;   // read last by the previous frame's fracture
        a.comp_cnt[2] = comp_end;  // the queue's start from the cforce phase on
    }
    // per-floe scratch of this frame (read last by the previous frame's fracture)
    for (int fl = gtid; fl < a.nf; fl += gsz) {
        a.fcoll[fl] = 0;
        a.fmax[fl] = 0ull;
    }
    const unsigned fstamp = frame_stamp(a, F);
    // What bounds it: the latency of a thread's few elements, so two elements' loads
    // go out together, ahead of the first store.  (One at a time, and half of the
    // loads behind the stores: 20 us with 236,640 active elements, now 17.)
    typedef typename vec2_of<T>::type V2;
    constexpr int kAhead = 2;
    for (int e0 = gtid; e0 < a.n; e0 += kAhead * gsz) {
        V2 pp[kAhead], rf[kAhead];
        T vr[kAhead], hh[kAhead], eta0[kAhead], eta1[kAhead], eta2[kAhead];
        bool act[kAhead];
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
            const int e = e0 + j * gsz;
            if (j > 0 && e >= a.n) break;
            const T* eta = F.ship_src.eta + 3 * (a.nsys > 1 ? a.sys_of[e] : 0);  // this element's ship
            pp[j] = ld2(F.src.pos, e);
            rf[j] = ld2(a.pos_ref, e);
            vr[j] = a.vert_r[e];
            hh[j] = esc_h_of(a, e, a.radii[e]);
            act[j] = F.src.active[e] != 0;
            eta0[j] = eta[0];
            eta1[j] = eta[1];
            eta2[j] = eta[2];
        }
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
            const int e = e0 + j * gsz;
            if (j > 0 && e >= a.n) break;
            const V2 p = pp[j], ref = rf[j];
            const T ddx = p.x - eta0[j], ddy = p.y - eta1[j];
            const T lim = reach + vr[j];
            // every query point of e lies within vert_r of its centroid and every hull
            // point within hull_r of the ship: farther elements get pen = 0, which is
            // what all of their point tests return (jax_geometry.py:104-134, :359-368);
            // the test keeps NaN positions (comparison false) on the exact path
            bool near = !(ddx * ddx + ddy * ddy > lim * lim * T(1.0001));
            if (near) {
                // the same against the hull's box in the ship's frame: on the 12 x 60 m
                // hull it keeps a third of what the circle keeps.  The slack covers the
                // rounding of the point tests at large coordinates.
                T sn, cs;
                jsincos(eta2[j], &sn, &cs);
                const T ax = fabs(cs * ddx + sn * ddy), ay = fabs(cs * ddy - sn * ddx);
                const T slack =
                    vr[j] + T(1e-2) + T(2e-6) * (fabs(p.x) + fabs(p.y) + fabs(eta0[j]) + fabs(eta1[j]));
                near = !(ax > a.hull_bx + slack) && !(ay > a.hull_by + slack);
            }
            warp_append(a.near_list, a.near_cnt, near, e);
            if (near) {
                a.cnear[chunk_of(a, e)] = fstamp;  // phase_cforce runs this chunk
            } else {
                a.cpen[e] = T(0);
                a.cnx[e] = T(0);
                a.cny[e] = T(0);
            }
            a.crack[e] = 0;  // set by phase_reduce for elements touching a broken bond
            const T h = hh[j];
            bool esc = escaped_from(p.x, p.y, ref.x, ref.y, h);
            if (!esc && act[j]) {
                const V2 v = ld2(F.src.vel, e);
                esc = escaped_from(p.x + v.x * a.t_frame, p.y + v.y * a.t_frame, ref.x, ref.y, T(0.9) * h);
            }
            warp_append(a.esc_list, (int*)&a.esc_cnt[0], esc, e);
        }
    }
}

// ─── P_NEAR: one warp per near element (jax_geometry.py:515-594) ────────────
// Pass 1: the element's vertices and edge samples vs the analytic hull; pass 2:
// the hull outline points inside the element's polygon; element-wise max.  Lanes
// split the points; argmax/argmin keep the reference's first-index ties.
template <typename T>
struct Best {
    T p, nx, ny;
    int i;
};

template <typename T>
__device__ __forceinline__ void better(Best<T>& b, T p, T nx, T ny, int i) {
    if (p > b.p || (p == b.p && i < b.i)) {
        b.p = p;
        b.nx = nx;
        b.ny = ny;
        b.i = i;
    }
}

template <typename T>
__device__ __forceinline__ Best<T> warp_best(Best<T> b) {
    for (int off = 16; off > 0; off >>= 1) {
        Best<T> o;
        o.p = __shfl_xor_sync(0xffffffffu, b.p, off);
        o.nx = __shfl_xor_sync(0xffffffffu, b.nx, off);
        o.ny = __shfl_xor_sync(0xffffffffu, b.ny, off);
        o.i = __shfl_xor_sync(0xffffffffu, b.i, off);
        better(b, o.p, o.nx, o.ny, o.i);
    }
    return b;
}

// NumPy's pairwise sum (np_pairwise_sum) of the values that lanes 0..n-1 hold;
// every lane gets it.
template <typename T>
__device__ __forceinline__ T warp_pairwise_sum(T v, int n) {
    const unsigned full = 0xffffffffu;
    if (n < 8) {
        T res = -T(0);
        for (int i = 0; i < n; ++i) res += __shfl_sync(full, v, i);
        return res;
    }
    const int lane = threadIdx.x & 31, m = n - (n % 8);
    T r = v;  // lane j < 8: partial sum j
    for (int i = 8; i < m; i += 8) r += __shfl_sync(full, v, i + (lane & 7));
    r += __shfl_down_sync(full, r, 1);
    r += __shfl_down_sync(full, r, 2);
    r += __shfl_down_sync(full, r, 4);
    T res = __shfl_sync(full, r, 0);
    for (int i = m; i < n; ++i) res += __shfl_sync(full, v, i);
    return res;
}

template <typename T>
__device__ void phase_near(const KArgs<T>& a, const Frame<T>& F, T* hullw, int nnear, int n_esc) {
    // hull outline in world frame: ship_hull_local @ R.T + [x, y] (jax_geometry.py:568-572),
    // staged once per CTA for a single ship; with several ships each element
    // transforms its own ship's outline point by point (the same expression)
    const bool one_ship = a.nsys == 1;
    HullPose<T> H1 = hull_pose(a, F.ship_src.eta);
    if (one_ship) {
        for (int i = threadIdx.x; i < a.S; i += blockDim.x) {
            T lx = a.hull[2 * i], ly = a.hull[2 * i + 1];
            hullw[2 * i] = lx * H1.c_h + ly * (-H1.s_h) + H1.sx;
            hullw[2 * i + 1] = lx * H1.s_h + ly * H1.c_h + H1.sy;
        }
    }
    __syncthreads();
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    // consecutive near elements go to different SMs
    const int warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int V = a.V;
    const int E = a.P.n_edge_samples;
    const int P1 = V * (1 + E);
    // Pass 2 takes a hull point by a group of 16 or 32 lanes, an edge each, or by
    // one lane that walks the edges, whichever has fewer steps: 4 against 11 for
    // the 7-point hull and 11 vertices, 31 against 22 for 62 points.
    const int W = V <= 16 ? 16 : 32;
    const bool by_edge = (a.S * W + 31) / 32 < ((a.S + 31) / 32) * V;
    for (int q = warp; q < nnear; q += nwarps) {
        const int e = a.near_list[q];
        const HullPose<T> H = one_ship ? H1 : hull_pose(a, F.ship_src.eta + 3 * a.sys_of[e]);
        typename vec2_of<T>::type pe = ld2(F.src.pos, e);
        T c, sn;
        jsincos(F.src.rot[e], &sn, &c);
        // lane k holds world vertex k (jax_geometry.py:176-180)
        const int kv = min(lane, V - 1);
        const typename vec2_of<T>::type lv = ld2(a.polys + (size_t)e * V * 2, kv);
        const bool mk = lane < V && a.pmask[(size_t)e * V + kv] != 0;
        const T wx = c * lv.x - sn * lv.y + pe.x;
        const T wy = sn * lv.x + c * lv.y + pe.y;
        const unsigned mkb = __ballot_sync(full, mk);
        // pass 1: point index = vertex * (1 + E) + sample (jax_geometry.py:190-211)
        Best<T> b1 = {T(0), T(0), T(0), INT_MAX};
        for (int p0 = 0; p0 < P1; p0 += 32) {
            const int pt = min(p0 + lane, P1 - 1);
            const int k = pt / (1 + E), j = pt % (1 + E);
            const int k1 = (k + 1 == V) ? 0 : k + 1;
            T qx = __shfl_sync(full, wx, k), qy = __shfl_sync(full, wy, k);
            const T x1 = __shfl_sync(full, wx, k1), y1 = __shfl_sync(full, wy, k1);
            if (p0 + lane >= P1) continue;
            if (j > 0) {
                T t = a.t_samp[j - 1];
                T omt = T(1) - t;
                qx = qx * omt + x1 * t;
                qy = qy * omt + y1 * t;
            }
            T p, nx, ny;
            hull_point(H, qx, qy, p, nx, ny);
            if (!((mkb >> k) & 1u)) p = T(0);
            better(b1, p, nx, ny, pt);
        }
        __syncwarp();
        // most near elements touch nothing: a warp without a point inside has its answer
        if (__any_sync(full, b1.p > T(0) || b1.nx != T(0) || b1.ny != T(0)))
            b1 = warp_best(b1);
        else
            b1 = {T(0), T(0), T(0), 0};
        // pass 2 (jax_geometry.py:300-510)
        auto hull_at = [&](int si, T& hx, T& hy) {
            if (one_ship) {
                hx = hullw[2 * si];
                hy = hullw[2 * si + 1];
            } else {
                const T lx = a.hull[2 * si], ly = a.hull[2 * si + 1];
                hx = lx * H.c_h + ly * (-H.s_h) + H.sx;
                hy = lx * H.s_h + ly * H.c_h + H.sy;
            }
        };
        // edge (xi, yi)-(xj, yj) seen from hull point (hx, hy): a crossing of the
        // point's ray, and the point's distance
        auto edge_test = [](T xi, T yi, T xj, T yj, T hx, T hy, T& d) -> bool {
            const bool cond_y = (yi > hy) != (yj > hy);
            const T x_int = (xj - xi) * (hy - yi) / (yj - yi + T(1e-10)) + xi;
            const T vx = xj - xi, vy = yj - yi;
            const T c1 = (hx - xi) * vx + (hy - yi) * vy;
            const T c2 = vx * vx + vy * vy + T(1e-20);
            const T t = jclip(c1 / c2, T(0), T(1));
            const T ddx = hx - (xi + t * vx), ddy = hy - (yi + t * vy);
            d = jsqrt(ddx * ddx + ddy * ddy + T(1e-20));
            return cond_y && (hx < x_int);
        };
        Best<T> b2 = {T(0), T(0), T(0), INT_MAX};
        // outward normal of the closest edge of a hull point that lies inside
        // (jax_geometry.py:389-405); every lane calls it, with its own candidate
        auto inside_point = [&](bool in, int si, T dmin, int k) {
            if (!__any_sync(full, in)) return;
            // masked vertex mean, in the reference's summation order
            const T n_real = jmax(warp_pairwise_sum(mk ? T(1) : T(0), V), T(1));
            const T cxc = warp_pairwise_sum(mk ? wx : T(0), V) / n_real;
            const T cyc = warp_pairwise_sum(mk ? wy : T(0), V) / n_real;
            const int k1 = (k + 1 == V) ? 0 : k + 1;
            const T xi = __shfl_sync(full, wx, k), yi = __shfl_sync(full, wy, k);
            const T xj = __shfl_sync(full, wx, k1), yj = __shfl_sync(full, wy, k1);
            if (!in) return;
            const T ex = xj - xi, ey = yj - yi;
            T nxe = ey, nye = -ex;
            const T nlen = jsqrt(nxe * nxe + nye * nye + T(1e-20));
            nxe = nxe / nlen;
            nye = nye / nlen;
            const T midx = (xi + xj) / T(2), midy = (yi + yj) / T(2);
            const T dotc = (midx - cxc) * nxe + (midy - cyc) * nye;
            if (dotc < T(0)) {
                nxe = -nxe;
                nye = -nye;
            }
            better(b2, dmin, nxe, nye, si);
        };
        if (by_edge) {
            const int k = lane & (W - 1), g = lane / W, ke = min(k, V - 1);
            const int k1 = (ke + 1 == V) ? 0 : ke + 1;
            const T xi = __shfl_sync(full, wx, ke), yi = __shfl_sync(full, wy, ke);
            const T xj = __shfl_sync(full, wx, k1), yj = __shfl_sync(full, wy, k1);
            const unsigned gm = (W == 32) ? full : (0xffffu << (16 * g));
            for (int s0 = 0; s0 < a.S; s0 += 32 / W) {
                const int si = min(s0 + g, a.S - 1);
                T hx, hy, d;
                hull_at(si, hx, hy);
                const bool cross = edge_test(xi, yi, xj, yj, hx, hy, d) && k < V;
                const bool odd = __popc(__ballot_sync(full, cross) & gm) & 1;
                const bool in = odd && s0 + g < a.S;
                if (!__any_sync(full, in)) continue;
                // argmin over the edges, first index wins; a NaN distance is less than none
                // and, at edge 0, greater than none: it stays, as in a walk from edge 0
                T dm = d;
                int km = k;
                const T d0 = __shfl_sync(full, d, g * W);
                if (k >= V || dm != dm) {
                    dm = d0;
                    km = 0;
                }
                for (int off = W / 2; off > 0; off >>= 1) {
                    const T od = __shfl_xor_sync(full, dm, off);
                    const int ok = __shfl_xor_sync(full, km, off);
                    if (od < dm || (od == dm && ok < km)) {
                        dm = od;
                        km = ok;
                    }
                }
                if (d0 != d0) {
                    dm = d0;
                    km = 0;
                }
                inside_point(in && k == 0, si, dm, km);
            }
        } else {
            for (int s0 = 0; s0 < a.S; s0 += 32) {
                const int si = min(s0 + lane, a.S - 1);
                T hx, hy;
                hull_at(si, hx, hy);
                int crossings = 0, kbest = 0;
                T dmin = T(0);
                for (int k = 0; k < V; ++k) {
                    const int k1 = (k + 1 == V) ? 0 : k + 1;
                    const T xi = __shfl_sync(full, wx, k), yi = __shfl_sync(full, wy, k);
                    const T xj = __shfl_sync(full, wx, k1), yj = __shfl_sync(full, wy, k1);
                    T d;
                    if (edge_test(xi, yi, xj, yj, hx, hy, d)) ++crossings;
                    if (k == 0 || d < dmin) {  // argmin, first index wins
                        dmin = d;
                        kbest = k;
                    }
                }
                inside_point((crossings % 2) == 1 && s0 + lane < a.S, si, dmin, kbest);
            }
        }
        __syncwarp();
        if (__any_sync(full, b2.p > T(0))) b2 = warp_best(b2);
        if (lane == 0) {
            // pass 2 replaces pass 1 only where strictly deeper (jax_geometry.py:585-590)
            const bool use2 = (b2.p > T(0)) && (b2.p > b1.p);
            a.cpen[e] = use2 ? b2.p : b1.p;
            a.cnx[e] = use2 ? b2.nx : b1.nx;
            a.cny[e] = use2 ? b2.ny : b1.ny;
        }
    }
    if (n_esc > 0) {
        __syncthreads();
        upkeep_mark(a, F, n_esc, frame_stamp(a, F));
    }
}

// ─── P_CFORCE: ship force on ice, submergence, reductions (jax_simulation.py:431-496)
template <typename T>
__device__ void phase_cforce(const KArgs<T>& a, const Frame<T>& F, int nd) {
    const DemParams& P = a.P;
    const T wcf = T(P.w_contact_radius_factor), wcap = T(P.w_contact_cap);
    const T flex = T(P.flexural_strength_base);
    const T pcr = T(P.pen_crit_ref), pct = T(P.pen_crit_thickness_ref);
    const T spf = T(P.side_push_factor);
    const T srate = T(P.submergence_rate), scap = T(P.submergence_pen_cap);
    const T inv_rise = T(1.0 / P.rise_time_const);
    const T dt = T(P.dt);
    const T rho_g = T(P.water_density * 9.81);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.near_cnt = 0;   // P_NEAR is done with it
        a.comp_cnt[1] = a.comp_cnt[2];  // P_CULL compacted the queue up to there
    }
    const unsigned fstamp = frame_stamp(a, F);
    for (int chunk = blockIdx.x; chunk < a.nchunks; chunk += gridDim.x) {
        // in a call's later frames (state in place) a chunk with no element
        // near the hull now and none in contact or submerged at the last
        // cforce is skipped: every one of its elements would store what it
        // holds (no ship force, no contact force, submergence 0) and its sums
        // are the zeros it holds
        if (F.f >= 1 && !a.cwarm[chunk] && a.cnear[chunk] != fstamp) continue;  // uniform over the CTA
        // chunks of kThreads elements start at each system's first element, so a
        // system's sums are grouped as they would be if it were simulated alone
        const int2 ci = a.chunk_info[chunk];
        const int e = ci.y + threadIdx.x;
        const T sx = F.ship_src.eta[3 * ci.x], sy = F.ship_src.eta[3 * ci.x + 1];
        double s0 = 0.0, s1 = 0.0, s2 = 0.0;
        bool warm = false;
        if (e < a.sys_end[ci.x]) {
            typename vec2_of<T>::type p = ld2(F.src.pos, e);
            const T pen = a.cpen[e], nx = a.cnx[e], ny = a.cny[e];
            const bool has = pen > T(0);
            const T h = a.thick[e];
            const T w_contact = jmin(wcf * a.radii[e], wcap);
            const T sigma_f = flex * jsqrt(h);
            const T f_break = sigma_f * w_contact * (h * h);
            const T pen_crit = pcr * (h / pct);
            const T fm = has ? f_break * jmin(pen / jmax(pen_crit, T(1e-10)), T(1)) : T(0);
            T so_x = fm * nx;
            T so_y = fm * ny;
            so_y = so_y + spf * fm * jsign(p.y - sy);
            // moment on the ship uses the force before the thrust cap (jax_simulation.py:474-477)
            const T rx = p.x - sx, ry = p.y - sy;
            const T mom = has ? (rx * (-so_y) - ry * (-so_x)) : T(0);
            s0 = (double)so_x;
            s1 = (double)so_y;
            s2 = (double)mom;
            // submergence and buoyancy (jax_simulation.py:480-496)
            const T sub = F.src.sub[e];
            const T pen_c = jmin(pen, scap);
            const T new_sub = has ? jmin(sub + srate * pen_c * dt, h) : jmax(T(0), sub - inv_rise * sub * dt);
            const T z_sub = jmin(new_sub, h);
            const T f_buoy = rho_g * a.areas[e] * z_sub;
            if (has) {
                so_x = so_x + f_buoy * nx;
                so_y = so_y + f_buoy * ny;
            }
            st2(a.soi, e, so_x, so_y);
            a.fraw[e] = fm;
            F.dst.sub[e] = new_sub;
            warm = has || new_sub != T(0);
            if (a.d_pen) a.d_pen[e] = pen;
            const int fl = a.floe_of[e];
            if (has) atomicMax(&a.fcoll[fl], 1);
            if (fm > T(0)) {
                if (sizeof(T) == 4)
                    atomicMax(&a.fmax[fl], (unsigned long long)f2ord((float)fm));
                else
                    atomicMax(&a.fmax[fl], d2ord((double)fm));
            }
        }
        // most chunks are far from the ship: their sums are of zeros
        double r3[3] = {0.0, 0.0, 0.0};
        if (__syncthreads_or(!(s0 == 0.0 && s1 == 0.0 && s2 == 0.0))) block_sum3<kThreads>(s0, s1, s2, r3);
        const int any_warm = __syncthreads_or(warm ? 1 : 0);
        if (threadIdx.x == 0) {
            a.part[3 * chunk + 0] = r3[0];
            a.part[3 * chunk + 1] = r3[1];
            a.part[3 * chunk + 2] = r3[2];
            a.cwarm[chunk] = any_warm ? 1 : 0;
        }
    }
    if (nd > 0) upkeep_build(a, nd);
}

// ─── vessel step (jax_vessel_dynamics.py:246-348) ───────────────────────────
template <typename T>
__device__ void ship_step(const DemParams& P, const T* eta, const T* nu, const T* na, const T* ei,
                          const T* sp, const T* spn, const T* tau_ice, const T* vws, T* eta_o,
                          T* nu_o, T* na_o, T* ei_o, const T* u_ctrl = nullptr) {
    const T pi = T(M_PI), two_pi = T(2.0 * M_PI);
    const T dtf = T(P.dt);
    T c = jcos(eta[2]), s = jsin(eta[2]);
    // R = [[c,-s,0],[s,c,0],[0,0,1]]; R^T v with the full 3x3 product of the
    // reference (the zero terms add exactly)
    T nu_c[3];
    nu_c[0] = (c * vws[0] + s * vws[1]) + T(0) * T(0);
    nu_c[1] = ((-s) * vws[0] + c * vws[1]) + T(0) * T(0);
    nu_c[2] = (T(0) * vws[0] + T(0) * vws[1]) + T(1) * T(0);
    T tib[3];
    tib[0] = (c * tau_ice[0] + s * tau_ice[1]) + T(0) * tau_ice[2];
    tib[1] = ((-s) * tau_ice[0] + c * tau_ice[1]) + T(0) * tau_ice[2];
    tib[2] = (T(0) * tau_ice[0] + T(0) * tau_ice[1]) + T(1) * tau_ice[2];
    T tau_act[3];
    if (u_ctrl) {
        // planner rollouts: the body-frame control replaces the DP controller
        // and the thrust allocation (RPMs and integral error stay as they are)
        for (int i = 0; i < 3; ++i) {
            tau_act[i] = u_ctrl[i];
            ei_o[i] = ei[i];
        }
        for (int i = 0; i < 6; ++i) na_o[i] = na[i];
    } else {
        T dpsi_d = pymod(spn[2] - sp[2] + pi, two_pi) - pi;
        T v_d[3] = {(spn[0] - sp[0]) / dtf, (spn[1] - sp[1]) / dtf, dpsi_d / dtf};
        T nu_d[3];
        nu_d[0] = (c * v_d[0] + s * v_d[1]) + T(0) * v_d[2];
        nu_d[1] = ((-s) * v_d[0] + c * v_d[1]) + T(0) * v_d[2];
        nu_d[2] = (T(0) * v_d[0] + T(0) * v_d[1]) + T(1) * v_d[2];
        T tau_ff[3];
        {
            T DKt[9];
            for (int i = 0; i < 9; ++i) DKt[i] = T(P.D3[i]) + T(P.Kd[i]);
            for (int i = 0; i < 3; ++i)
                tau_ff[i] = (DKt[3 * i] * nu_d[0] + DKt[3 * i + 1] * nu_d[1]) + DKt[3 * i + 2] * nu_d[2];
        }
        // dp_control (jax_vessel_dynamics.py:127-184): tau = -(R^T Kp) e - Kd nu - (R^T Ki) e_int
        T e[3];
        e[0] = eta[0] - sp[0];
        e[1] = eta[1] - sp[1];
        e[2] = pymod(eta[2] - sp[2] + pi, two_pi) - pi;
        T Rt[9] = {c, s, T(0), -s, c, T(0), T(0), T(0), T(1)};
        T RKp[9], RKi[9];
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) {
                RKp[3 * i + j] = (Rt[3 * i] * T(P.Kp[j]) + Rt[3 * i + 1] * T(P.Kp[3 + j])) + Rt[3 * i + 2] * T(P.Kp[6 + j]);
                RKi[3 * i + j] = (Rt[3 * i] * T(P.Ki[j]) + Rt[3 * i + 1] * T(P.Ki[3 + j])) + Rt[3 * i + 2] * T(P.Ki[6 + j]);
            }
        T a1[3], a2[3], a3[3];
        for (int i = 0; i < 3; ++i) {
            a1[i] = (RKp[3 * i] * e[0] + RKp[3 * i + 1] * e[1]) + RKp[3 * i + 2] * e[2];
            a2[i] = (T(P.Kd[3 * i]) * nu[0] + T(P.Kd[3 * i + 1]) * nu[1]) + T(P.Kd[3 * i + 2]) * nu[2];
            a3[i] = (RKi[3 * i] * ei[0] + RKi[3 * i + 1] * ei[1]) + RKi[3 * i + 2] * ei[2];
        }
        T tau_c[3];
        for (int i = 0; i < 3; ++i) {
            tau_c[i] = (-a1[i] - a2[i]) - a3[i];
            ei_o[i] = ei[i] + dtf * e[i];
        }
        if (P.use_auto_icenav) {
            T tc[3] = {tau_c[0] + tau_ff[0], tau_c[1] + tau_ff[1], tau_c[2] + tau_ff[2]};
            T ncmd[6];
            for (int i = 0; i < 6; ++i) {
                T u = (T(P.B_pinv[3 * i]) * tc[0] + T(P.B_pinv[3 * i + 1]) * tc[1]) + T(P.B_pinv[3 * i + 2]) * tc[2];
                T n_ = jsign(u) * jsqrt(fabs(u) + T(1e-12));
                ncmd[i] = jclip(n_, -T(P.n_max[i]), T(P.n_max[i]));
                na_o[i] = na[i] + dtf * (ncmd[i] - na[i]) / T(P.T_n);
            }
            T q[6];
            for (int i = 0; i < 6; ++i) q[i] = fabs(na_o[i]) * na_o[i];
            for (int i = 0; i < 3; ++i) {
                T acc = T(P.B_mat[6 * i]) * q[0];
                for (int j = 1; j < 6; ++j) acc = acc + T(P.B_mat[6 * i + j]) * q[j];
                tau_act[i] = acc;
            }
        } else {
            for (int i = 0; i < 3; ++i) tau_act[i] = tau_c[i] + tau_ff[i];
            for (int i = 0; i < 6; ++i) na_o[i] = na[i];
        }
    }
    T tau_tot[3] = {tau_act[0] + tib[0], tau_act[1] + tib[1], tau_act[2] + tib[2]};
    // ship_euler_step_jax (jax_vessel_dynamics.py:54-84)
    T nu_r[3] = {nu[0] - nu_c[0], nu[1] - nu_c[1], nu[2] - nu_c[2]};
    T dnr[3];
    for (int i = 0; i < 3; ++i) dnr[i] = (T(P.D3[3 * i]) * nu_r[0] + T(P.D3[3 * i + 1]) * nu_r[1]) + T(P.D3[3 * i + 2]) * nu_r[2];
    T rhs[3] = {tau_tot[0] - dnr[0], tau_tot[1] - dnr[1], tau_tot[2] - dnr[2]};
    T nu_new[3];
    for (int i = 0; i < 3; ++i) {
        T nd = (T(P.M3inv[3 * i]) * rhs[0] + T(P.M3inv[3 * i + 1]) * rhs[1]) + T(P.M3inv[3 * i + 2]) * rhs[2];
        nu_new[i] = nu[i] + dtf * nd;
    }
    T vx = c * nu_new[0] - s * nu_new[1];
    T vy = s * nu_new[0] + c * nu_new[1];
    T psi_new = pymod(eta[2] + dtf * nu_new[2] + pi, two_pi) - pi;
    eta_o[0] = eta[0] + dtf * vx;
    eta_o[1] = eta[1] + dtf * vy;
    eta_o[2] = psi_new;
    nu_o[0] = jclip(nu_new[0], -T(P.vc_surge), T(P.vc_surge));
    nu_o[1] = jclip(nu_new[1], -T(P.vc_sway), T(P.vc_sway));
    nu_o[2] = jclip(nu_new[2], -T(P.vc_yaw), T(P.vc_yaw));
}

// ─── P_REDUCE ───────────────────────────────────────────────────────────────
// A warp reduces one system's chunk partials in a fixed order (lane 0 gets them).
template <typename T>
__device__ void frame_totals(const KArgs<T>& a, int sys, double* tot3) {
    const int lane = threadIdx.x & 31;
    double v0 = 0.0, v1 = 0.0, v2 = 0.0;
    for (int i = a.part_base[sys] + lane; i < a.part_base[sys + 1]; i += 32) {
        v0 += a.part[3 * i];
        v1 += a.part[3 * i + 1];
        v2 += a.part[3 * i + 2];
    }
    tot3[0] = warp_sum_lane0(v0);
    tot3[1] = warp_sum_lane0(v1);
    tot3[2] = warp_sum_lane0(v2);
}

template <typename T>
__device__ __forceinline__ T thrust_scale_of(const KArgs<T>& a, const double* tot3) {
    if (!a.P.has_max_ship_ice_force) return T(1);
    T fx = T(tot3[0]), fy = T(tot3[1]);
    T mag = jsqrt(fx * fx + fy * fy);
    T mx = T(a.P.max_ship_ice_force);
    return (mag > mx) ? mx / jmax(mag, T(1e-6)) : T(1);
}

// The bond slot records of a warp's active elements (mask m; w0 + lane) for this
// frame (only active elements read them); crack front = the element touches a bond
// broken at frame start (read for bonds between two active elements).  A bond
// with an active end is listed once, by its active end of lower index.
//
// What bounds it: the chain slot -> partner -> floe flag of dependent loads, so the
// slots of all the elements are one sequence, two a lane and step: as few steps
// as there can be, and whole lines of slots and records.  (An element's slots by one
// lane, or by the warp one element after another: the phase took 10.3 us with 205
// active elements, now 7.7, and 24 with 12,032, now 20.)
template <typename T>
__device__ __forceinline__ void slot_records(const KArgs<T>& a, const Frame<T>& F, SlotRec<T>* rec, unsigned m, int w0,
                                             unsigned fstamp) {
    const int lane = threadIdx.x & 31;
    const bool mine = (m >> lane) & 1u;
    const int s0 = mine ? a.boff[w0 + lane] : 0, cnt = mine ? a.boff[w0 + lane + 1] - s0 : 0;
    int end = cnt;  // slots up to and with this lane's
    for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, end, d);
        if (lane >= d) end += v;
    }
    const int start = end - cnt, total = __shfl_sync(0xffffffffu, end, 31);
    for (int k0 = 0; k0 < total; k0 += 64) {
        int sl[2], ee[2];
        bool on[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            // the last lane whose slots start at or before the k-th
            const int k = k0 + 32 * j + lane;
            int own = 0;
            for (int d = 16; d > 0; d >>= 1)
                if (__shfl_sync(0xffffffffu, start, own + d) <= k) own += d;
            on[j] = k < total;
            sl[j] = __shfl_sync(0xffffffffu, s0, own) + k - __shfl_sync(0xffffffffu, start, own);
            ee[j] = w0 + own;
        }
        int2 ent[2];
        int fo[2];
        bool in[2], ao[2];
        T dm[2], rr[2], kk[2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (on[j]) ent[j] = a.bslot[sl[j]];
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (on[j]) {
                const int b = ent[j].x & 0x7fffffff;
                in[j] = F.src.intact[b] != 0;
                ao[j] = F.src.active[ent[j].y] != 0;
                fo[j] = a.floe_of[ent[j].y];
                dm[j] = F.src.dmg[b];
                rr[j] = a.slot_rest[sl[j]];
                kk[j] = a.slot_stiff[sl[j]];
            }
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (on[j]) ao[j] = ao[j] || a.fcoll[fo[j]];
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (on[j]) {
                a.bstamp[ent[j].x & 0x7fffffff] = fstamp;
                if (!in[j]) a.crack[ee[j]] = 1;
                SlotRec<T> q;
                q.o = (ent[j].x < 0) ? (int)((unsigned)ent[j].y | 0x80000000u) : ent[j].y;
                q.rest = rr[j];
                q.stiff = kk[j];
                q.omd = (in[j] && ao[j]) ? T(1) - dm[j] : T(-1);  // the element is active: both ends must be
                rec[sl[j]] = q;
            }
        warp_append2(a.fb_list, a.fb_cnt, on[0] && !(ao[0] && ent[0].y < ee[0]), ent[0].x & 0x7fffffff,
                     on[1] && !(ao[1] && ent[1].y < ee[1]), ent[1].x & 0x7fffffff);
    }
}

template <typename T>
__device__ void phase_reduce(const KArgs<T>& a, const Frame<T>& F, bool upkept) {
    if (upkept && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        // the near and cforce phases have processed these
        a.esc_cnt[0] = 0u;
        a.dirty_cnt[0] = 0;
    }
    typedef typename vec2_of<T>::type V2;
    // one warp per system: totals, thrust cap and the vessel step (warp 0 of
    // CTA 0 for a single system)
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int ngwarp = (gridDim.x * blockDim.x) >> 5;
    for (int sys = gwarp; sys < a.nsys; sys += ngwarp) {
        double tot3[3];
        frame_totals(a, sys, tot3);
        if ((threadIdx.x & 31) == 0) {
            const T scale = thrust_scale_of(a, tot3);
            // reaction on the ship (jax_simulation.py:470-478)
            T Fx = -(T(tot3[0]) * scale), Fy = -(T(tot3[1]) * scale), M = T(tot3[2]);
            double* fs = a.fscal + 4 * sys;
            fs[0] = (double)scale;
            fs[1] = (double)Fx;
            fs[2] = (double)Fy;
            fs[3] = (double)M;
            T tau[3] = {Fx, Fy, M};
            T J = jsqrt(Fx * Fx + Fy * Fy) * T(a.P.dt);
            // rollouts drive the ship by controls (no setpoints, no ice brake)
            const T* u = a.u_ctrl ? a.u_ctrl + ((size_t)F.f * a.nsys + sys) * 3 : nullptr;
            const T zero6[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
            const T* spf = u ? zero6 : F.sp + 6 * sys;
            T sp[3] = {spf[0], spf[1], spf[2]};
            const T* eta = F.ship_src.eta + 3 * sys;
            if (!u && a.P.ice_brake_threshold > 0.0) {  // jax_simulation.py:658-669
                T thr = T(a.P.ice_brake_threshold);
                T bf = jclip(thr / jmax(fabs(tau[0]), thr), T(0.1), T(1));
                sp[0] = eta[0] + bf * (spf[0] - eta[0]);
                sp[1] = eta[1] + bf * (spf[1] - eta[1]);
            }
            const T vzero[2] = {T(0), T(0)};
            const T* vws = F.vws ? F.vws + 2 * sys : vzero;
            T eta_o[3], nu_o[3], na_o[6], ei_o[3];
            ship_step<T>(a.P, eta, F.ship_src.nu + 3 * sys, F.ship_src.na + 6 * sys, F.ship_src.ei + 3 * sys, sp,
                         spf + 3, tau, vws, eta_o, nu_o, na_o, ei_o, u);
            for (int i = 0; i < 3; ++i) {
                F.ship_dst.eta[3 * sys + i] = eta_o[i];
                F.ship_dst.nu[3 * sys + i] = nu_o[i];
                F.ship_dst.ei[3 * sys + i] = ei_o[i];
            }
            for (int i = 0; i < 6; ++i) F.ship_dst.na[6 * sys + i] = na_o[i];
            if (a.d_F) {
                a.d_F[2 * sys] = Fx;
                a.d_F[2 * sys + 1] = Fy;
            }
            if (a.d_J) a.d_J[sys] = J;
            const size_t fs_i = (size_t)F.f * a.nsys + sys;
            if (a.h_eta)
                for (int i = 0; i < 3; ++i) a.h_eta[fs_i * 3 + i] = eta_o[i];
            if (a.h_J) a.h_J[fs_i] = J;
            if (a.h_F) {
                a.h_F[fs_i * 2] = Fx;
                a.h_F[fs_i * 2 + 1] = Fy;
            }
        }
    }
    // With one system, CTA 0 runs the vessel step above and the other CTAs share
    // the element and slot work (all CTAs when the grid has one); with several
    // systems every CTA takes part in both.
    const int c0 = (gridDim.x > 1 && a.nsys == 1) ? 1 : 0;
    if ((int)blockIdx.x < c0) return;
    const int gtid = (blockIdx.x - c0) * blockDim.x + threadIdx.x;
    const int gsz = (gridDim.x - c0) * blockDim.x;
    SlotRec<T>* rec = reinterpret_cast<SlotRec<T>*>(a.slotrec);
    typedef typename vec4_of<T>::type V4;
    const unsigned fstamp = frame_stamp(a, F);
    // lanes take consecutive elements, as many of a warp's lanes as share them out
    // evenly; the loop bound is uniform over the warp, so that it can share the slot
    // work of the active elements it finds
    const int lane = threadIdx.x & 31;
    const int nw = gsz >> 5, take = min(32, max(4, (a.n + nw - 1) / nw));
    const int w1 = (gtid >> 5) * take;
    bool was_next = false;
    int fl_next = 0;
    if (lane < take && w1 + lane < a.n) {
        was_next = F.src.active[w1 + lane] != 0;
        fl_next = a.floe_of[w1 + lane];
    }
    for (int w0 = w1; w0 < a.n; w0 += nw * take) {
        const int e = w0 + lane;
        bool ae = false;
        const bool was = was_next, own = lane < take && e < a.n;
        const int fl = fl_next;
        if (lane < take && e + nw * take < a.n) {  // the next step's, ahead of this one's stores
            was_next = F.src.active[e + nw * take] != 0;
            fl_next = a.floe_of[e + nw * take];
        }
        if (own) {
            // activation (jax_simulation.py:498-509)
            ae = was || a.fcoll[fl];
            // after the first frame of a call, an element frozen before and
            // after this frame's activation has its state, substep buffers and
            // frame output in place already (the previous frame wrote them)
            if (F.f == 0 || ae) {
                F.dst.active[e] = ae ? 1 : 0;
                // packed kinematics read by substep 0
                const V2 p = ld2(F.src.pos, e), v = ld2(F.src.vel, e);
                V4 k4;
                k4.x = p.x;
                k4.y = p.y;
                k4.z = a.radii[e];
                k4.w = a.r3[e];
                reinterpret_cast<V4*>(a.kin[0])[e] = k4;
                st2(a.kvel[0], e, v.x, v.y);
                if (!ae) {
                    // frozen for the whole frame, it keeps its state
                    // (jax_simulation.py:257-262): both substep buffers and the
                    // frame's output hold it now, and the substeps skip it
                    reinterpret_cast<V4*>(a.kin[1])[e] = k4;
                    st2(a.kvel[1], e, v.x, v.y);
                    st2(F.dst.pos, e, p.x, p.y);
                    st2(F.dst.vel, e, v.x, v.y);
                    F.dst.rot[e] = F.src.rot[e];
                    F.dst.avel[e] = F.src.avel[e];
                }
            }
        }
        warp_append(a.act_list, a.act_cnt, ae, e);  // the frame's active list
        const unsigned m = __ballot_sync(0xffffffffu, ae);
        if (m) slot_records(a, F, rec, m, w0, fstamp);
    }
}

// ─── P_FORCE: one substep (jax_simulation.py:63-268, 363-395) ───────────────
// Gather form: each element, a thread's or a group of lanes', sums its own bond
// and contact terms in the reference's scatter order, so no atomics are needed.
// Positions are packed with radii as {x, y, r, r^3} (one 16-byte load per
// neighbour) and bond slots are 16-byte records; the loads of a batch are issued
// before any of them is used.
// Every operation is unfused (-fmad=false) and in the reference's order, with
// divisions where it divides, so that fp32 forces round as NumPy's fp32
// evaluation of the same expressions does.
#ifndef DEM_KBATCH
#define DEM_KBATCH 3
#endif
constexpr int kBatch = DEM_KBATCH;  // bond slots / contact candidates whose loads are issued together


// overlap^1.5 of the Hertz law, as the reference's power of an fp32 array: in
// float the product o * sqrt(o) is formed in double and rounded once, which
// gives the correctly rounded power (the value the C library's powf returns
// but for its rare last-place misses); in double as is
__device__ __forceinline__ float hertz15(float o) {
    const double od = (double)o;
    return (float)(od * sqrt(od));
}
__device__ __forceinline__ double hertz15(double o) { return o * sqrt(o); }

// The same without branches or doubles, for o in the fast range: o * sqrt(o) as
// a sum of two floats, good to 2^-44 (s the root rounded, o - s^2 exact, the
// product's own rounding error exact).  ok is cleared where that error could
// change the rounding (one case in 2^18 for full significands).
__device__ __forceinline__ float hertz15_nr(float o, bool& ok) {
    float h;
    const float s = sqrt_nr(o, h);
    const float p = o * s;
    const float c = fmaf(o, fmaf(-s, s, o) * h, fmaf(o, s, -p));
    const float d = p * 5.6843419e-14f;  // 2^-44
    const float lo = p + (c - d);
    ok = ok && lo == p + (c + d);
    return lo;
}
__device__ __forceinline__ double hertz15_nr(double o, bool&) {
    double h;
    return o * sqrt_nr(o, h);
}

// Constants and substep buffers of one force phase.
template <typename T>
struct ForceCtx {
    const T *kin, *kvin, *rin, *ain;
    T *kout, *kvout, *rout, *aout;
    const uint8_t* act;
    const SlotRec<T>* rec;
    bool last;
};

template <typename T>
__device__ __forceinline__ ForceCtx<T> force_ctx(const KArgs<T>& a, const Frame<T>& F, int s) {
    ForceCtx<T> c;
    const int k = a.k_sub;
    c.kin = a.kin[s & 1];
    c.kout = a.kin[(s + 1) & 1];
    c.kvin = a.kvel[s & 1];
    c.kvout = a.kvel[(s + 1) & 1];
    c.rin = (s == 0) ? F.src.rot : a.sp_rot[(s - 1) & 1];
    c.ain = (s == 0) ? F.src.avel : a.sp_avel[(s - 1) & 1];
    c.last = (s == k - 1);
    c.rout = c.last ? F.dst.rot : a.sp_rot[s & 1];
    c.aout = c.last ? F.dst.avel : a.sp_avel[s & 1];
    c.act = F.dst.active;
    c.rec = reinterpret_cast<const SlotRec<T>*>(a.slotrec);
    return c;
}

// Bond slot term (jax_simulation.py:63-108) of a slot record with omd >= 0:
// the force and half-moment that the slot's role adds to (role i) or
// subtracts from (role j) the element's bond sums.
template <typename T>
__device__ __forceinline__ void bond_term(const SlotRec<T>& r, typename vec2_of<T>::type kb, T ex, T ey, T& fx,
                                          T& fy, T& cr) {
    const bool role_j = r.o < 0;
    const T dx = role_j ? ex - kb.x : kb.x - ex;
    const T dy = role_j ? ey - kb.y : kb.y - ey;
    const T dist = jsqrt(dx * dx + dy * dy);
    const T dsafe = jmax(dist, T(1e-10));
    const T fmag = r.stiff * (dist - r.rest) * r.omd;
    fx = (dx / dsafe) * fmag;  // bond_dir * f_mag (jax_simulation.py:76-96)
    fy = (dy / dsafe) * fmag;
    cr = T(0.5) * (dx * fy - dy * fx);
}

// False for a candidate that does not touch: d2 > (min_dist (1 + 1e-5))^2, all
// roundings included, puts the rounded square root above min_dist, where the
// reference's overlap is exactly 0 (NaN gives true).
template <typename V4>
__device__ __forceinline__ bool may_touch(V4 ke, V4 ko, bool e_is_i) {
    const auto dx = e_is_i ? ko.x - ke.x : ke.x - ko.x;
    const auto dy = e_is_i ? ko.y - ke.y : ke.y - ko.y;
    const auto d2 = dx * dx + dy * dy;
    const auto min_dist = e_is_i ? ke.z + ko.z : ko.z + ke.z;
    const auto mdm = min_dist * decltype(d2)(1.00001);
    return !(d2 > mdm * mdm);
}

// Ice-ice contact term (jax_simulation.py:111-164) of element e (kinematics
// ke, ve) with candidate o (ko, vo); e_is_i = e < o.  Returns false when the
// pair does not touch; else e adds (tx, ty) to its contact force and adds
// (e_is_i) or subtracts hm from its contact moment.
template <typename T>
__device__ __forceinline__ bool contact_term(const ForceConst<T>& fc, bool h15, typename vec4_of<T>::type ke,
                                             typename vec2_of<T>::type ve, typename vec4_of<T>::type ko,
                                             typename vec2_of<T>::type vo, bool e_is_i, T& tx, T& ty, T& hm) {
    if (!may_touch(ke, ko, e_is_i)) return false;
    const T dx = e_is_i ? ko.x - ke.x : ke.x - ko.x;
    const T dy = e_is_i ? ko.y - ke.y : ke.y - ko.y;
    const T d2 = dx * dx + dy * dy;
    const T min_dist = e_is_i ? ke.z + ko.z : ko.z + ke.z;
    // the contact predicate, unfused as in the reference (jax_simulation.py:127-131)
    const T dist = jsqrt(d2);
    const T overlap = jmax(min_dist - dist, T(0));
    if (!((dist > T(1e-6)) && (overlap > T(0)))) return false;
    // direction = d / max(dist, 1e-10); here dist > 1e-6 (jax_simulation.py:133-136)
    const T ux = dx / dist, uy = dy / dist;
    const T fn = fc.hf * (h15 ? hertz15(overlap) : jpow(overlap, fc.hexp));
    const T fnx = ux * fn, fny = uy * fn;
    const T vrx = e_is_i ? vo.x - ve.x : ve.x - vo.x;
    const T vry = e_is_i ? vo.y - ve.y : ve.y - vo.y;
    // tangential relative velocity and kinetic friction (jax_simulation.py:139-149)
    const T vdot = vrx * ux + vry * uy;
    const T vtx = vrx - vdot * ux, vty = vry - vdot * uy;
    const T vtm = jsqrt(vtx * vtx + vty * vty);
    T ftx = T(0), fty = T(0);
    if (vtm > T(1e-6)) {
        const T ftm = jmin(fc.mu * fn, fc.fcap);
        ftx = (-vtx / vtm) * ftm;  // t_hat * f_t_mag
        fty = (-vty / vtm) * ftm;
    }
    const T oix = -fnx - ftx, oiy = -fny - fty;
    const T cr = -(dx * oiy - dy * oix);
    tx = e_is_i ? ftx - fnx : fnx - ftx;
    ty = e_is_i ? fty - fny : fny - fty;
    hm = T(0.5) * cr;
    return true;
}

// The same two terms without branches, for code that computes them for every
// lane and selects afterwards.  Each returns the same bits as the form above (but
// for the sign of a zero, which the sums take no notice of) when it leaves `ok`
// set; with `ok` cleared (an operand outside the fast range, or an undecided
// rounding) the caller takes the form above.
template <typename T>
__device__ __forceinline__ void bond_term_nr(const SlotRec<T>& r, typename vec2_of<T>::type kb, T ex, T ey, T& fx,
                                             T& fy, T& cr, bool& ok) {
    const bool role_j = r.o < 0;
    const T dx = role_j ? ex - kb.x : kb.x - ex;
    const T dy = role_j ? ey - kb.y : kb.y - ey;
    const T d2 = dx * dx + dy * dy;
    T h;
    const T dist = sqrt_nr(d2, h);
    const T dsafe = jmax(dist, T(1e-10));
    const T fmag = r.stiff * (dist - r.rest) * r.omd;
    const T y = rcp_nr(dsafe);
    fx = div_nr(dx, dsafe, y) * fmag;
    fy = div_nr(dy, dsafe, y) * fmag;
    cr = T(0.5) * (dx * fy - dy * fx);
    ok = ok && fast_ok(d2) && fast_num(dx) && fast_num(dy);
}

// Returns whether the pair touches (also when ok is cleared).
template <typename T>
__device__ __forceinline__ bool contact_term_nr(const ForceConst<T>& fc, typename vec4_of<T>::type ke,
                                                typename vec2_of<T>::type ve, typename vec4_of<T>::type ko,
                                                typename vec2_of<T>::type vo, bool e_is_i, T& tx, T& ty, T& hm,
                                                bool& ok) {
    const T sg = e_is_i ? T(1) : T(-1);
    const T dx = sg * (ko.x - ke.x), dy = sg * (ko.y - ke.y);  // exact sign changes
    const T d2 = dx * dx + dy * dy;
    T h;
    const T dist = sqrt_nr(d2, h);
    const T overlap = jmax((ke.z + ko.z) - dist, T(0));
    const bool touch = (dist > T(1e-6)) && (overlap > T(0));
    const T y = rcp_nr(dist);
    const T ux = div_nr(dx, dist, y), uy = div_nr(dy, dist, y);
    bool fine = fast_ok(d2) && fast_num(dx) && fast_num(dy) && fast_ok(overlap);
    const T fn = fc.hf * hertz15_nr(overlap, fine);
    const T fnx = ux * fn, fny = uy * fn;
    const T vrx = sg * (vo.x - ve.x), vry = sg * (vo.y - ve.y);
    const T vdot = vrx * ux + vry * uy;
    const T vtx = vrx - vdot * ux, vty = vry - vdot * uy;
    const T v2 = vtx * vtx + vty * vty;
    const T vtm = sqrt_nr(v2, h);
    const bool slips = v2 >= FastRange<T>::lo() && vtm > T(1e-6);
    const T yt = rcp_nr(vtm);
    const T ftm = jmin(fc.mu * fn, fc.fcap);
    const T ftx = slips ? div_nr(-vtx, vtm, yt) * ftm : T(0);
    const T fty = slips ? div_nr(-vty, vtm, yt) * ftm : T(0);
    fine = fine && v2 <= FastRange<T>::hi() && (!slips || (fast_num(vtx) && fast_num(vty)));
    const T oix = -fnx - ftx, oiy = -fny - fty;
    const T cr = -(dx * oiy - dy * oix);
    tx = sg * (ftx - fnx);
    ty = sg * (fty - fny);
    hm = T(0.5) * cr;
    // below the fast range a distance is no contact, above it the exact form decides
    ok = ok && (fine || !(touch || d2 > FastRange<T>::hi()));
    return touch;
}

// Contact-set recording (only when a.crec is set): one pair {e, o} whose
// contact term element e's force computation added.
template <typename T>
__device__ __forceinline__ void record_contact(const KArgs<T>& a, int e, int o) {
    const unsigned i = atomicAdd(a.crec_cnt, 1u);
    if (i < (unsigned)a.crec_cap) a.crec[i] = make_int2(e, o);
}

// Whether element e has escaped at its new position (processed before the next substep).
template <typename T>
__device__ __forceinline__ bool escapes(const KArgs<T>& a, const ForceCtx<T>& cx, int e, T px, T py, T r) {
    if (cx.last) return false;
    return escaped_from(px, py, a.pos_ref[2 * e], a.pos_ref[2 * e + 1], esc_h_of(a, e, r));
}

// Drag, rotational drag and the semi-implicit update of an active element
// from its bond and contact sums; stores the substep's output and returns
// whether the element has escaped.
template <typename T>
__device__ __forceinline__ bool integrate_element(const KArgs<T>& a, const Frame<T>& F, const ForceCtx<T>& cx, int e,
                                                  typename vec4_of<T>::type ke, typename vec2_of<T>::type ve,
                                                  typename vec4_of<T>::type ec, typename vec2_of<T>::type w, T sub,
                                                  typename vec2_of<T>::type so, T av, T rot, T fbx, T fby, T mb,
                                                  T fix, T fiy, T mi) {
    typedef typename vec4_of<T>::type V4;
    // drag (jax_simulation.py:167-192)
    const T m = ec.x, inertia = ec.y, h = ec.z, A = ec.w;
    const T a_drag = A * (h / a.fc.href);
    const T vrx = ve.x - w.x, vry = ve.y - w.y;
    const T vm = jsqrt(vrx * vrx + vry * vry);
    T fdx, fdy;
    if (vm > T(1e-6)) {
        // (v / |v|) * (c A |v|^2), evaluated as the reference writes it
        const T q = (a.fc.c_drag * a_drag) * (vm * vm);
        fdx = (vrx / vm) * q;
        fdy = (vry / vm) * q;
    } else {
        const T cl = a.fc.c_drag * a_drag * a.fc.lin;
        fdx = cl * vrx;
        fdy = cl * vry;
    }
    // rotational drag (jax_simulation.py:195-212)
    const T a_sub = A * jmin(sub / jmax(h, T(1e-10)), T(1));
    const T md = a.fc.c_rot * ke.w * av * fabs(av) * a_sub;
    const T Fx = ((fbx + fix) - fdx) + so.x;
    const T Fy = ((fby + fiy) - fdy) + so.y;
    const T Mz = (mb + mi) + md;
    // semi-implicit Euler (jax_simulation.py:215-268)
    const T dti = a.fc.dti, vclip = a.fc.vclip, pclip = a.fc.pclip;
    T nvx = jclip(ve.x + (Fx / m) * dti, -vclip, vclip);
    T nvy = jclip(ve.y + (Fy / m) * dti, -vclip, vclip);
    T npx = ke.x + nvx * dti, npy = ke.y + nvy * dti;
    const T alpha = Mz / inertia;
    const T nav = jclip(av * a.fc.damp + alpha * dti, a.fc.alo, a.fc.ahi);
    const T nrot = rot + nav * dti;
    if (!jfinite(nvx)) nvx = T(0);
    if (!jfinite(nvy)) nvy = T(0);
    if (!jfinite(npx)) npx = ke.x;
    if (!jfinite(npy)) npy = ke.y;
    npx = jclip(npx, -pclip, pclip);
    npy = jclip(npy, -pclip, pclip);
    if (cx.last) {
        st2(F.dst.pos, e, npx, npy);
        st2(F.dst.vel, e, nvx, nvy);
    } else {
        V4 v4;
        v4.x = npx;
        v4.y = npy;
        v4.z = ke.z;
        v4.w = ke.w;
        reinterpret_cast<V4*>(cx.kout)[e] = v4;
        st2(cx.kvout, e, nvx, nvy);
    }
    cx.rout[e] = nrot;
    cx.aout[e] = nav;
    return escapes(a, cx, e, npx, npy, ke.z);
}

// Forces, torque and the semi-implicit update of active element e for one
// substep, one thread per element; returns whether e has escaped.  For many
// active elements, where the instruction count decides: the bond slots first,
// kBatch at a time (records, then all partner gathers, then the terms); then the
// candidates' distances, which leave a bit for each that touches; then the
// contact terms of those alone.  Walking the candidates once, term and all, a
// warp went through the contact term at nearly every candidate, since one of its
// lanes touched there.  Each sum keeps the reference's order (bond slots with
// e == bond_i first, then e == bond_j; candidates above e ascending, then below
// e ascending).
template <typename T>
__device__ __forceinline__ bool force_element(const KArgs<T>& a, const Frame<T>& F, const ForceCtx<T>& cx, int e) {
    typedef typename vec2_of<T>::type V2;
    typedef typename vec4_of<T>::type V4;
    const T *kin = cx.kin, *kvin = cx.kvin;
    const SlotRec<T>* rec = cx.rec;
    const bool h15 = a.fc.h15 != 0;
    const V4 ke = ld4(kin, e);  // x, y, radius, radius^3
    const int s0 = a.boff[e], s1 = a.boff[e + 1];
    const int nc = a.ncnt[e];
    // bonds (jax_simulation.py:63-108)
    T fbx = T(0), fby = T(0), mb = T(0);
    for (int b = s0; b < s1; b += kBatch) {
        SlotRec<T> r[kBatch];
        V2 kb[kBatch];
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
            r[j].o = 0;
            r[j].omd = T(-1);
            if (b + j < s1) r[j] = rec[b + j];
        }
#pragma unroll
        for (int j = 0; j < kBatch; ++j)
            if (r[j].omd >= T(0)) kb[j] = reinterpret_cast<const V2*>(kin)[2 * (r[j].o & 0x7fffffff)];
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
            if (r[j].omd < T(0)) continue;  // no slot, broken, or active/frozen endpoints
            T fx, fy, cr;
            bond_term(r[j], kb[j], ke.x, ke.y, fx, fy, cr);
            const bool neg = r[j].o < 0;
            fbx += neg ? -fx : fx;
            fby += neg ? -fy : fy;
            mb += neg ? -cr : cr;
        }
    }
    // ice-ice contacts (:111-164): which candidates touch
    unsigned long long touch = 0ull;
    const int* nb = a.nbr + e;
    for (int c = 0; c < nc; c += kBatch) {
        int o[kBatch];
        V4 ko[kBatch];
#pragma unroll
        for (int j = 0; j < kBatch; ++j) o[j] = (c + j < nc) ? nb[(size_t)(c + j) * a.n] : -1;
#pragma unroll
        for (int j = 0; j < kBatch; ++j)
            if (o[j] >= 0) ko[j] = ld4(kin, o[j]);
#pragma unroll
        for (int j = 0; j < kBatch; ++j)
            if (o[j] >= 0 && may_touch(ke, ko[j], e < o[j])) touch |= 1ull << (c + j);
    }
    const V2 ve = ld2(kvin, e);
    T fix = T(0), fiy = T(0), mi = T(0);
    while (touch) {
        // two at a time: their loads go out together
        const int c0 = __ffsll((long long)touch) - 1;
        touch &= touch - 1ull;
        const int c1 = touch ? __ffsll((long long)touch) - 1 : -1;
        if (touch) touch &= touch - 1ull;
        const int o0 = nb[(size_t)c0 * a.n], o1 = c1 >= 0 ? nb[(size_t)c1 * a.n] : -1;
        const V4 k0 = ld4(kin, o0);
        const V2 v0 = ld2(kvin, o0);
        V4 k1;
        V2 v1;
        if (o1 >= 0) {
            k1 = ld4(kin, o1);
            v1 = ld2(kvin, o1);
        }
        T tx, ty, hm;
        if (contact_term(a.fc, h15, ke, ve, k0, v0, e < o0, tx, ty, hm)) {
            if (a.crec) record_contact(a, e, o0);
            fix += tx;
            fiy += ty;
            mi += (e < o0) ? hm : -hm;
        }
        if (o1 >= 0 && contact_term(a.fc, h15, ke, ve, k1, v1, e < o1, tx, ty, hm)) {
            if (a.crec) record_contact(a, e, o1);
            fix += tx;
            fiy += ty;
            mi += (e < o1) ? hm : -hm;
        }
    }
    const V4 ec = ld4(a.econ, e);  // mass, inertia, thickness, area
    return integrate_element(a, F, cx, e, ke, ve, ec, ld2(F.vw, e), F.dst.sub[e], ld2(a.soi, e), cx.ain[e], cx.rin[e],
                             fbx, fby, mb, fix, fiy, mi);
}

// The same substep by groups of kGroup lanes, four active elements to a warp
// (every lane calls it; lanes of one group with the same e, or -1): lane j of a
// group takes slots and candidates j, j + 8, ..., so all gathers of a round are
// in flight at once; the terms that exist go side by side through the warp's
// slice of shared memory and six lanes of the group take one sum each, in
// order.  For a middling number of active elements, where one element's chain
// of dependent loads decides the phase's length: 12,032 active elements of a
// batch took 17.5 us a substep with a thread each.  Lane 0 of a group returns
// whether its element has escaped.
constexpr int kGroup = 8;

// The warp's slice of shared memory for the terms of its elements: 6 x 32, or 4
// groups of 3 x 8 + 3 x 16 and a queue of 16 indices.
template <typename T>
constexpr int kGroupTerms = 9 * kGroup + 16 * 4 / (int)sizeof(T);

template <typename T>
__device__ __forceinline__ T* warp_terms() {
    __shared__ __align__(16) T s_terms[kThreads / 32][32 / kGroup * kGroupTerms<T>];
    return s_terms[threadIdx.x >> 5];
}

template <typename T>
__device__ __forceinline__ bool force_group(const KArgs<T>& a, const Frame<T>& F, const ForceCtx<T>& cx, int e) {
    typedef typename vec2_of<T>::type V2;
    typedef typename vec4_of<T>::type V4;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, gl = lane & (kGroup - 1), g0 = lane - gl;
    T* wt = warp_terms<T>() + g0;
    const T *kin = cx.kin, *kvin = cx.kvin;
    const bool h15 = a.fc.h15 != 0;
    const bool on = e >= 0;
    const int ee = on ? e : 0;
    const V4 ke = ld4(kin, ee);
    const V2 ve = ld2(kvin, ee);
    const int s0 = a.boff[ee];
    const int nbe = on ? a.boff[ee + 1] - s0 : 0, nc = on ? a.ncnt[ee] : 0;
    // the integration's own loads, beside the gathers
    const V4 ec = ld4(a.econ, ee);
    const V2 w = ld2(F.vw, ee);
    const T sub = F.dst.sub[ee];
    const V2 so = ld2(a.soi, ee);
    const T av = cx.ain[ee], rot = cx.rin[ee];
    const int m = __reduce_max_sync(full, max(nbe, nc));
    T acc = T(0);  // lanes 0..5 of a group: bond force x, y, moment, contact force x, y, moment
    for (int j0 = 0; j0 < m; j0 += kGroup) {
        const int j = j0 + gl;
        SlotRec<T> r;
        r.o = 0;
        r.omd = T(-1);
        if (j < nbe) r = cx.rec[s0 + j];
        const int o = (j < nc) ? a.nbr[(size_t)j * a.n + ee] : -1;
        const bool bv = r.omd >= T(0);
        V2 kb;
        V4 ko;
        V2 vo;
        if (bv) kb = reinterpret_cast<const V2*>(kin)[2 * (r.o & 0x7fffffff)];
        if (o >= 0) {
            ko = ld4(kin, o);
            vo = ld2(kvin, o);
        }
        T bfx = T(0), bfy = T(0), bcr = T(0);
        if (bv) bond_term(r, kb, ke.x, ke.y, bfx, bfy, bcr);
        T tx = T(0), ty = T(0), hm = T(0);
        const bool eis = ee < o;
        const bool cv = (o >= 0) && contact_term(a.fc, h15, ke, ve, ko, vo, eis, tx, ty, hm);
        if (cv && a.crec) record_contact(a, e, o);
        const unsigned gm = 0xffu << g0, lt = (1u << lane) - 1u;
        const unsigned bm = __ballot_sync(full, bv) & gm, cm = __ballot_sync(full, cv) & gm;
        if (bv) {
            const bool neg = r.o < 0;
            const int i = __popc(bm & lt);
            wt[i] = neg ? -bfx : bfx;
            wt[32 + i] = neg ? -bfy : bfy;
            wt[64 + i] = neg ? -bcr : bcr;
        }
        if (cv) {
            const int i = __popc(cm & lt);
            wt[96 + i] = tx;
            wt[128 + i] = ty;
            wt[160 + i] = eis ? hm : -hm;
        }
        __syncwarp();
        const int nt = gl < 3 ? __popc(bm) : (gl < 6 ? __popc(cm) : 0);
        const T* mt = wt + 32 * min(gl, 5);
        T x[kGroup];
#pragma unroll
        for (int i = 0; i < kGroup; ++i) x[i] = mt[i];
#pragma unroll
        for (int i = 0; i < kGroup; ++i)
            if (i < nt) acc += x[i];
        __syncwarp();  // the next round overwrites the terms
    }
    T f[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) f[i] = __shfl_sync(full, acc, g0 + i);
    bool esc = false;
    if (gl == 0 && on) esc = integrate_element(a, F, cx, e, ke, ve, ec, w, sub, so, av, rot, f[0], f[1], f[2], f[3], f[4], f[5]);
    __syncwarp();
    return esc;
}

// Out of place (a frame that writes the caller's separate output), the state of
// every bond is copied to the output during the substeps, a slice of the bond
// groups of four per substep, by warps that have no element work there (the
// substeps of a frame with few active elements leave most warps idle).  A
// bond keeps its state unless it has an active end (jax_simulation.py:534-653:
// with both ends frozen no gate opens and no collision breaks it), and the
// fracture phase overwrites the copies of the bonds that have one.  The shear
// displacement is copied as x + 0 and the intact flag as 0/1, as the update
// itself would write them.  Warp `cw` of `ncw` copiers takes its share.
template <typename T>
__device__ __forceinline__ void copy_bond_slice(const KArgs<T>& a, const Frame<T>& F, int s, int cw, int ncw) {
    const int ng = (a.nb + 3) >> 2;
    const int per = (ng + a.k_sub - 1) / a.k_sub;  // groups of a slice
    const int g_lo = (int)min((long long)per * s, (long long)ng), g_hi = min(g_lo + per, ng);
    auto al16 = [](const void* p) { return ((size_t)p & 15u) == 0; };
    const bool vec = al16(F.src.ds) && al16(F.dst.ds) && al16(F.src.dmg) && al16(F.dst.dmg) && al16(F.src.dm0) &&
                     al16(F.dst.dm0) && al16(F.src.dmmax) && al16(F.dst.dmmax) &&
                     ((size_t)F.src.intact & 3u) == 0 && ((size_t)F.dst.intact & 3u) == 0;
    typedef typename vec4_of<T>::type V4;
    for (int g = g_lo + cw * 32 + (threadIdx.x & 31); g < g_hi; g += ncw * 32) {
        const int b0 = 4 * g;
        const int cnt = min(4, a.nb - b0);
        if (vec && cnt == 4) {
            // every load before the first store, which the compiler could not
            // move them across: one memory round per group instead of five
            V4 d = ld4(F.src.ds, g);
            const V4 m = ld4(F.src.dmg, g), m0 = ld4(F.src.dm0, g), mx = ld4(F.src.dmmax, g);
            const unsigned raw = reinterpret_cast<const unsigned*>(F.src.intact)[g];
            d.x = d.x + T(0);
            d.y = d.y + T(0);
            d.z = d.z + T(0);
            d.w = d.w + T(0);
            unsigned in4 = 0u;
            for (int k = 0; k < 4; ++k)
                if ((raw >> (8 * k)) & 0xffu) in4 |= 1u << (8 * k);
            reinterpret_cast<V4*>(F.dst.ds)[g] = d;
            reinterpret_cast<V4*>(F.dst.dmg)[g] = m;
            reinterpret_cast<V4*>(F.dst.dm0)[g] = m0;
            reinterpret_cast<V4*>(F.dst.dmmax)[g] = mx;
            reinterpret_cast<unsigned*>(F.dst.intact)[g] = in4;
        } else {
            for (int k = 0; k < cnt; ++k) {
                const int b = b0 + k;
                F.dst.ds[b] = F.src.ds[b] + T(0);
                F.dst.dmg[b] = F.src.dmg[b];
                F.dst.dm0[b] = F.src.dm0[b];
                F.dst.dmmax[b] = F.src.dmmax[b];
                F.dst.intact[b] = F.src.intact[b] != 0 ? 1 : 0;
            }
        }
    }
}

constexpr int kPerWarp = 32 / kGroup;  // elements of a warp in force_group
constexpr int kGroupRounds = 3;        // groups of lanes take the elements while that many rounds suffice
// And the last, partial round of chunks of 32 while that many suffice: 236,640
// elements are 3.12 chunks a warp, and with groups for the 0.12 a substep takes 55
// us against 60 (a frame 728 against 781).
constexpr int kTailRounds = 2;

template <typename T>
__device__ void phase_force(const KArgs<T>& a, const Frame<T>& F, int s, unsigned round, int nd, int na) {
    const ForceCtx<T> cx = force_ctx(a, F, s);
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const int gsz = gridDim.x * blockDim.x;
    int* esc_ctr = (int*)&a.esc_cnt[s + 1];
    const int warp = gtid >> 5, nwarps = gsz >> 5, lane = threadIdx.x & 31;
    const bool has_dirty = nd > 0;
    if (has_dirty && gtid == 0) atomicAdd((unsigned long long*)&a.stats[4], (unsigned long long)nd);
    // Elements whose list this round's escapes invalidated are rebuilt, then
    // computed, here; the element loop below skips them.  A few take a CTA
    // each, so that a stencil scan is one load round, on CTAs that then take no
    // element work; many take a warp each.
    const bool cta_items = has_dirty && a.mark_split != DEM_SPLIT_WARP &&
                           nd <= (int)gridDim.x / (a.mark_split == DEM_SPLIT_CTA ? 2 : 4);
    if (cta_items) {
        if ((int)blockIdx.x < nd) {  // uniform over the CTA
            const int e = a.dirty_list[blockIdx.x];
            block_build(a, e);
            // a frozen element's substep buffers and output are written for the frame
            if (threadIdx.x < 32 && cx.act[e]) {
                const bool esc = force_group(a, F, cx, lane < kGroup ? e : -1);
                if (esc) a.esc_list[atomicAdd(esc_ctr, 1)] = e;
            }
            return;
        }
    } else if (has_dirty) {
        // one warp rebuilds the list, then computes the element
        for (int q = warp; q < nd; q += nwarps) {
            const int e = a.dirty_list[q];
            warp_build(a, e);
            // a frozen element's substep buffers and output are written for the frame
            const bool esc = cx.act[e] && force_group(a, F, cx, lane < kGroup ? e : -1);
            if (esc) a.esc_list[atomicAdd(esc_ctr, 1)] = e;
            __syncwarp();
        }
    }
    // The warps that rebuilt a list above take no share of the element loop
    // (while enough warps remain), so they do not finish the phase last; with a
    // CTA per item, those CTAs' warps.
    const int skip = cta_items ? nd * (kThreads / 32) : ((nd < nwarps / 2) ? nd : 0);
    if (warp < skip) return;
    // Only active elements move (frozen ones were carried over by phase_reduce).
    // Few of them go to groups of lanes, four to a warp.  Many go in chunks of 32, a
    // thread each: every warp starts with one chunk of its own, then takes further
    // ones from a counter (the next grab is issued before the current chunk is
    // computed), so uneven chunks do not leave warps idle.  The chunks of a last
    // round that only a quarter of the warps would have go to groups of lanes too,
    // in items of four elements: a third of a chunk's time, on all warps.
    const int nw2 = nwarps - skip;
    const bool copy_bonds = a.nb > 0 && F.src.ds != F.dst.ds;
    const bool lanes = a.force_split == DEM_SPLIT_WARP ||
                       (a.force_split == DEM_SPLIT_AUTO && na <= kGroupRounds * kPerWarp * nw2);
    const int chunks = (na + 31) >> 5, tail = chunks % nw2;
    const int nthr = lanes ? 0
                     : (a.force_split == DEM_SPLIT_AUTO && 32 * tail <= kTailRounds * kPerWarp * nw2) ? chunks - tail
                                                                                                      : chunks;
    const int items = nthr + max(0, (na - 32 * nthr + kPerWarp - 1) / kPerWarp);
    int c = warp - skip;
    int* ctr = &a.work_cnt[s];
    for (; c < nthr;) {
        int next = 0;
        if (lane == 0) next = nw2 + atomicAdd(ctr, 1);
        const int i = c * 32 + lane;
        const int e = i < na ? a.act_list[i] : -1;
        if (e >= 0 && !(has_dirty && a.dirty[e] == round)) {
            const bool esc = force_element(a, F, cx, e);
            if (!cx.last) warp_append(a.esc_list, esc_ctr, esc, e);
        }
        c = __shfl_sync(0xffffffffu, next, 0);
    }
    while (c < items) {
        int next = 0;
        if (nthr > 0 && lane == 0) next = nw2 + atomicAdd(ctr, 1);
        const int i = 32 * nthr + (c - nthr) * kPerWarp + lane / kGroup;
        int e = i < na ? a.act_list[i] : -1;
        if (e >= 0 && has_dirty && a.dirty[e] == round) e = -1;
        const bool esc = force_group(a, F, cx, e);
        if (!cx.last) warp_append(a.esc_list, esc_ctr, esc, e);
        c = nthr > 0 ? __shfl_sync(0xffffffffu, next, 0) : c + nw2;
    }
    if (copy_bonds) {
        // the warps without an element copy this substep's slice; when every
        // warp has one, all of them copy after it
        const int busy = nthr > 0 ? nw2 : min(items, nw2);
        if (busy < nw2) {
            if (warp - skip >= busy) copy_bond_slice(a, F, s, warp - skip - busy, nw2 - busy);
        } else {
            copy_bond_slice(a, F, s, warp - skip, nw2);
        }
    }
}

// ─── all substeps of a frame, the active elements held in shared memory ──────
// While the CTAs' shared memory holds every active element (its state, its
// constants, its reference, its bond slots and candidates), each stays with one
// group of lanes for the whole frame, and a substep loads its partners'
// positions and velocities and nothing else.  The group is a warp, a slot and a
// candidate per lane, while no CTA has more elements than warps; beyond that it
// is 8 lanes, a slot and two candidates per lane.  The terms that exist go side
// by side through shared memory, and six lanes of a group each take one of the
// sums (bond and contact force and moment) in slot or candidate order.
//
// What bounds it: the chain of one substep, a barrier (1.1 to 1.5 us), one gather
// from L2 and some 700 instructions of one warp, most of them waiting for the one
// before (4,100 cycles in all).  With the list, slot and constant loads in front
// of the gather (a phase at a time) the 205 active elements of the 12k field took
// 7.8 us a substep, now 3.5; the 12,032 of a batch of 256 rollouts 12.1 us with
// force_group, now 7.3 (two rounds of groups; bound by issue, 16 warps an SM).
template <typename T>
struct __align__(16) ResElem {
    // x, y, angle | radius;  vx, vy, angular velocity | escape distance;
    // mass, mass, inertia | drag factor;  ship force x, y, 0 | submerged area;
    // water velocity x, y | rotational drag factor, -;  reference x, y
    T p[4], v[4], m[4], so[4], w[4], ref[2];
    int e, nbe, nc, s0;
    int slots, cands, room, ref_ok;  // offsets of its slots and candidates in the pool (-1: in global memory)
};
constexpr int kResMaxElems = kThreads / 2;  // per CTA

// Bytes of one CTA's pool: the host adds them to the kernel's dynamic shared memory.
template <typename T>
__host__ __device__ constexpr int res_pool_bytes() { return sizeof(T) == 4 ? 32768 : 49152; }

// Elements a CTA can hold: half of the pool for their records, the rest for
// slots and candidates (those that find no room are read from global memory).
template <typename T>
__host__ __device__ constexpr int res_elems() {
    return res_pool_bytes<T>() / 2 / (int)sizeof(ResElem<T>) < kResMaxElems
               ? res_pool_bytes<T>() / 2 / (int)sizeof(ResElem<T>) : kResMaxElems;
}

// One substep of a group's element (el < 0: none; every lane of the warp calls it).
// wt: the group's terms, bond force x, y and moment [3][G] and contact force x,
// y and moment [3][kC * G].  After the sums, lanes 0, 1 and 2 of the group take
// x, y and the rotation through the same instructions.
template <typename T, int G>
__device__ __forceinline__ void resident_step(const KArgs<T>& a, const Frame<T>& F, unsigned char* pool, int el, T* wt,
                                              int s, bool last, int* flag) {
    typedef typename vec2_of<T>::type V2;
    typedef typename vec4_of<T>::type V4;
    constexpr int kC = G == 32 ? 1 : 2;  // candidates per lane and round
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, gl = lane & (G - 1), g0 = lane - gl;
    const T *kin = a.kin[s & 1], *kvin = a.kvel[s & 1];
    const bool h15 = a.fc.h15 != 0, on = el >= 0;
    ResElem<T>* E = reinterpret_cast<ResElem<T>*>(pool) + (on ? el : 0);
    const int e = E->e, nbe = on ? E->nbe : 0, nc = on ? E->nc : 0;
    const SlotRec<T>* rp = E->slots >= 0 ? reinterpret_cast<const SlotRec<T>*>(pool + E->slots)
                                         : reinterpret_cast<const SlotRec<T>*>(a.slotrec) + E->s0;
    const int* cp = E->cands >= 0 ? reinterpret_cast<const int*>(pool + E->cands) : a.nbr + e;
    const int cstep = E->cands >= 0 ? 1 : a.n;
    V4 ke;
    ke.x = E->p[0];
    ke.y = E->p[1];
    ke.z = E->p[3];
    ke.w = T(0);
    V2 ve;
    ve.x = E->v[0];
    ve.y = E->v[1];
    const int c3 = min(gl, 2);  // x, y or rotation
    T acc = T(0);  // lanes 0..5 of a group: bond force x, y, moment, contact force x, y, moment
    T fd = T(0);   // lanes 0..2: what the drag takes from the force (adds to the moment, negated)
    int m = max((nbe + G - 1) / G, (nc + G * kC - 1) / (G * kC));
    if (G < 32) m = __reduce_max_sync(full, m);
    for (int r0 = 0; r0 == 0 || r0 < m; ++r0) {
        SlotRec<T> r;
        r.o = 0;
        r.omd = T(-1);
        const int j = r0 * G + gl;
        if (j < nbe) r = rp[j];
        int o[kC];
#pragma unroll
        for (int c = 0; c < kC; ++c) {
            const int i = (r0 * kC + c) * G + gl;
            o[c] = i < nc ? cp[(size_t)i * cstep] : -1;
        }
        // lanes without a slot or candidate compute on stand-ins that add nothing
        const bool bv = r.omd >= T(0);
        V2 kb;
        kb.x = ke.x + T(1);
        kb.y = ke.y;
        V4 ko[kC];
        V2 vo[kC];
        if (bv) kb = reinterpret_cast<const V2*>(kin)[2 * (r.o & 0x7fffffff)];
#pragma unroll
        for (int c = 0; c < kC; ++c) {
            ko[c] = ke;
            ko[c].z = -ke.z;
            vo[c] = ve;
            if (o[c] >= 0) {
                ko[c] = ld4(kin, o[c]);
                vo[c] = ld2(kvin, o[c]);
            }
        }
        // while the gathers are in flight: no contact terms yet, and the drag
#pragma unroll
        for (int i = 0; i < 3 * kC; ++i) wt[3 * G + i * G + gl] = T(0);
        if (r0 == 0) {
            // drag (jax_simulation.py:167-192) and rotational drag (:195-212)
            const T q_drag = E->m[3], vrx = ve.x - E->w[0], vry = ve.y - E->w[1], vr = gl == 0 ? vrx : vry;
            const T v2 = vrx * vrx + vry * vry;
            T h;
            const T vm = sqrt_nr(v2, h);
            const T vq = q_drag * (vm * vm);
            fd = div_nr(vr, vm, rcp_nr(vm)) * vq;
            // beyond the fast range, where sqrt_nr has no value, the operators decide
            const bool over = v2 > FastRange<T>::hi(), quad = over || (v2 >= FastRange<T>::lo() && vm > T(1e-6));
            if (!quad) fd = (q_drag * a.fc.lin) * vr;  // too slow (or NaN): linear
            if (quad && (over || !fast_num(vr))) {
                const T ve_m = jsqrt(v2);
                fd = (vr / ve_m) * (q_drag * (ve_m * ve_m));
            }
            const T av = E->v[2];
            if (gl >= 2) fd = -(E->w[2] * av * fabs(av) * E->so[3]);
        }
        const unsigned gm = G == 32 ? full : (((1u << (G & 31)) - 1u) << g0), lt = (1u << lane) - 1u;
        T bfx, bfy, bcr;
        bool okb = true;
        bond_term_nr(r, kb, ke.x, ke.y, bfx, bfy, bcr, okb);
        if (__any_sync(full, bv && !okb)) {  // rare: an operand outside the fast range
            if (bv && !okb) bond_term(r, kb, ke.x, ke.y, bfx, bfy, bcr);
            __syncwarp();
        }
        const bool neg = r.o < 0;  // subtracted: an exact sum with the sign turned
        wt[gl] = bv ? (neg ? -bfx : bfx) : T(0);
        wt[G + gl] = bv ? (neg ? -bfy : bfy) : T(0);
        wt[2 * G + gl] = bv ? (neg ? -bcr : bcr) : T(0);
        // contact term of one candidate per lane (oc < 0: none); the terms that
        // exist follow those before
        int nct = 0;
        auto contact = [&](int oc, V4 kc, V2 vc) {
            T tx, ty, hm;
            bool okc = h15;
            bool cv = contact_term_nr(a.fc, ke, ve, kc, vc, e < oc, tx, ty, hm, okc) && oc >= 0;
            if (__any_sync(full, oc >= 0 && !okc)) {  // rare, and an undecided rounding
                if (oc >= 0 && !okc) cv = contact_term(a.fc, h15, ke, ve, kc, vc, e < oc, tx, ty, hm);
                __syncwarp();
            }
            if (cv && a.crec) record_contact(a, e, oc);
            const unsigned cm = __ballot_sync(full, cv) & gm;
            if (cv) {
                T* ct = wt + 3 * G + nct + __popc(cm & lt);
                ct[0] = tx;
                ct[kC * G] = ty;
                ct[2 * kC * G] = e < oc ? hm : -hm;
            }
            nct += __popc(cm);
        };
        __syncwarp();  // the zeros are in place
        if (kC == 1) {
            contact(o[0], ko[0], vo[0]);
        } else {
            // a group's touching candidates, some 4 of 16, move together first
            unsigned tm[2];
#pragma unroll
            for (int c = 0; c < 2; ++c)
                tm[c] = __ballot_sync(full, o[c % kC] >= 0 && may_touch(ke, ko[c % kC], e < o[c % kC])) & gm;
            const int n0 = __popc(tm[0]), n = n0 + __popc(tm[1]);
            int* cq = reinterpret_cast<int*>(wt + 9 * G);
            if ((tm[0] >> lane) & 1u) cq[__popc(tm[0] & lt)] = lane;
            if ((tm[1] >> lane) & 1u) cq[n0 + __popc(tm[1] & lt)] = 32 + lane;
            __syncwarp();
            for (int q0 = 0; __any_sync(full, q0 < n); q0 += G) {
                const bool has = q0 + gl < n;
                const int src = has ? cq[q0 + gl] : lane;
                const bool second = src >= 32;
                auto from = [&](T x0, T x1) {
                    const T y0 = __shfl_sync(full, x0, src), y1 = __shfl_sync(full, x1, src);
                    return second ? y1 : y0;
                };
                V4 kc;
                V2 vc;
                kc.x = from(ko[0].x, ko[kC - 1].x);
                kc.y = from(ko[0].y, ko[kC - 1].y);
                kc.z = from(ko[0].z, ko[kC - 1].z);
                kc.w = T(0);
                vc.x = from(vo[0].x, vo[kC - 1].x);
                vc.y = from(vo[0].y, vo[kC - 1].y);
                const int oa = __shfl_sync(full, o[0], src), ob = __shfl_sync(full, o[kC - 1], src);
                contact(has ? (second ? ob : oa) : -1, kc, vc);
            }
        }
        __syncwarp();
        // four terms a step; the zeros past a sum's last term leave it as it is
        const V4* mt = reinterpret_cast<const V4*>(wt + (gl < 3 ? gl * G : (gl < 6 ? 3 * G + (gl - 3) * kC * G : 0)));
        auto add4 = [&](int i) {
            const V4 x = mt[i];
            acc += x.x;
            acc += x.y;
            acc += x.z;
            acc += x.w;
        };
        if (G == 32) {
            const int n4 = max((min(nbe - r0 * G, G) + 3) / 4, (nct + 3) / 4);
            for (int i = 0; i < n4; ++i) add4(i);
        } else {
            add4(0);
            add4(1);
            if (gl >= 3 && nct > 8) {
                add4(2);
                add4(3);
            }
        }
        __syncwarp();  // the next round overwrites the terms
    }
    // semi-implicit Euler (jax_simulation.py:215-268): force sum ((bonds +
    // contacts) - drag) + ship, moment (bonds + contacts) + drag
    const T f = ((acc + __shfl_down_sync(full, acc, 3)) - fd) + E->so[c3];
    const T p0 = E->p[c3], v0 = E->v[c3];
    const T dti = a.fc.dti;
    const bool lin = c3 < 2;
    const T mass = E->m[c3];
    T acn = div_nr(f, mass, rcp_nr(mass));
    if (!(fast_num(f) && fast_ok(mass))) acn = f / mass;
    T nv = (lin ? v0 : v0 * a.fc.damp) + acn * dti;
    nv = jclip(nv, lin ? -a.fc.vclip : a.fc.alo, lin ? a.fc.vclip : a.fc.ahi);
    T np = p0 + nv * dti;
    if (lin) {
        if (!jfinite(nv)) nv = T(0);
        if (!jfinite(np)) np = p0;
        np = jclip(np, -a.fc.pclip, a.fc.pclip);
    }
    if (gl < 3 && on) {
        if (last) {
            if (lin) {
                F.dst.pos[2 * (size_t)e + gl] = np;
                F.dst.vel[2 * (size_t)e + gl] = nv;
            } else {
                F.dst.rot[e] = np;
                F.dst.avel[e] = nv;
            }
        } else {
            if (lin) {
                a.kin[(s + 1) & 1][4 * (size_t)e + gl] = np;
                a.kvel[(s + 1) & 1][2 * (size_t)e + gl] = nv;
            }
            E->p[gl] = np;
            E->v[gl] = nv;
        }
    }
    if (!last) {
        const T d = lin ? np - E->ref[c3] : T(0);
        const T dd = d * d;
        const T d2 = dd + __shfl_down_sync(full, dd, 1);
        const unsigned fin = __ballot_sync(full, jfinite(np));
        if (gl == 0 && on) {
            const bool fp = ((fin >> g0) & 3u) == 3u, fr = E->ref_ok != 0;
            const T h = E->v[3];
            if (fp != fr || (fp && d2 > h * h)) {
                a.esc_list[atomicAdd((int*)&a.esc_cnt[s + 1], 1)] = e;
                *flag = 1;
            }
        }
    }
    __syncwarp();
}

// Stage the candidates and the reference of element el (one warp).
template <typename T>
__device__ __forceinline__ void resident_list(const KArgs<T>& a, unsigned char* pool, int el) {
    ResElem<T>* E = reinterpret_cast<ResElem<T>*>(pool) + el;
    const int lane = threadIdx.x & 31;
    const int e = E->e, nc = a.ncnt[e];
    const bool fits = nc <= E->room;
    const int at = E->cands;
    __syncwarp();
    if (fits && at >= 0)
        for (int i = lane; i < nc; i += 32) reinterpret_cast<int*>(pool + at)[i] = a.nbr[(size_t)i * a.n + e];
    if (lane == 0) {
        E->nc = nc;
        if (!fits) E->cands = -1;
        const typename vec2_of<T>::type q = ld2(a.pos_ref, e);
        E->ref[0] = q.x;
        E->ref[1] = q.y;
        E->ref_ok = jfinite(q.x) && jfinite(q.y);
        E->v[3] = esc_h_of(a, e, E->p[3]);
    }
    __syncwarp();
}

// DPDEM floe eligibility after this frame's contact (jax_simulation.py:511-524):
// max(force * scale) == max(force) * scale because rounding is monotone.
template <typename T>
__device__ __forceinline__ bool new_elig(const KArgs<T>& a, const Frame<T>& F, int fl, T scale) {
    if (F.elig_in[fl]) return true;
    if (a.nb == 0 || !a.fcoll[fl]) return false;
    const unsigned long long bits = a.fmax[fl];
    const T fmx = (sizeof(T) == 4) ? T(__uint_as_float((unsigned)bits)) : T(__longlong_as_double((long long)bits));
    return fmx * scale > a.min_bstr * T(a.P.effective_strength_collision);
}

// thrust-cap scale of system `sys` for this frame (one value when nsys == 1)
template <typename T>
__device__ __forceinline__ T sys_scale(const KArgs<T>& a, T scale1, int sys) {
    return a.nsys == 1 ? scale1 : T(*((volatile double*)&a.fscal[4 * sys]));
}

// The history rows of an element's position and angle.
template <typename T>
__device__ __forceinline__ void element_rows(const KArgs<T>& a, const Frame<T>& F, int e) {
    if (a.h_pos) {
        const typename vec2_of<T>::type p = ld2(F.dst.pos, e);
        st2(a.h_pos + (size_t)F.f * a.n * 2, e, p.x, p.y);
    }
    if (a.h_rot) a.h_rot[(size_t)F.f * a.n + e] = F.dst.rot[e];
}

// What a frame writes beside its substeps and its bonds with an active end: the
// floes' eligibility, the diagnostics' contact force, and the history rows of bonds
// without an active end and of elements (frozen ones only with `frozen`).  All of
// it stands once phase_reduce has ended, so CTAs that hold no element write it while
// the others run the substeps: on the pack the fracture phase, which wrote it
// before, takes 8.9 us instead of 17.
template <typename T>
__device__ __forceinline__ void frame_outputs(const KArgs<T>& a, const Frame<T>& F, T scale, int gtid, int gsz,
                                              bool frozen) {
    if (a.h_intact) {
        const unsigned fstamp = frame_stamp(a, F);
        for (int b = gtid; b < a.nb; b += gsz)
            if (a.bstamp[b] != fstamp) a.h_intact[(size_t)F.f * a.nb + b] = F.src.intact[b] != 0 ? 1 : 0;
    }
    if (a.h_pos || a.h_rot || a.h_sub)
        for (int e = gtid; e < a.n; e += gsz) {
            if (a.h_sub) a.h_sub[(size_t)F.f * a.n + e] = F.dst.sub[e];
            if (frozen && F.dst.active[e]) continue;
            element_rows(a, F, e);
        }
    for (int fl = gtid; fl < a.nf; fl += gsz)
        F.dst.elig[fl] = new_elig(a, F, fl, sys_scale(a, scale, a.nsys > 1 ? a.floe_sys[fl] : 0)) ? 1 : 0;
    if (a.d_fmag)
        for (int e = gtid; e < a.n; e += gsz)
            a.d_fmag[e] = a.fraw[e] * sys_scale(a, scale, a.nsys > 1 ? a.sys_of[e] : 0);
}

// CTAs that hold `na` active elements in shared memory.  The elements go to few, a
// warp each: four to a CTA while that fills no more than half of the grid (a CTA per
// SM), then up to eight.  The substeps' barriers are among those CTAs alone (26
// arrivals take 1.1 us, 296 1.5 us).  (Eight to a CTA measured 3 % slower a frame than
// four on the 12k field; on the pack, 1,186 active, four leave no CTA for the
// frame's other writes: 123 against 114 us.)
__device__ __forceinline__ int resident_ctas(int na) {
    constexpr int kWarps = kThreads / 32;
    return min((int)gridDim.x, max(min((na + 3) / 4, (int)gridDim.x / 2), (na + kWarps - 1) / kWarps));
}
// Whether those CTAs are enough to rebuild every list too, where that comes first;
// with no active element there is none of them.  A one-frame call that rebuilds
// 12,127 lists takes 210 to 236 us with 100 to 296 such CTAs against 235 to 247
// phase by phase on the whole grid, 298 against 246 with 50 and 5.8 ms against 0.24
// with one; 236,640 lists take 770 us with 296 CTAs against 730, 33 ms with four.
constexpr int kBuildPerCta = 128;
template <typename T>
__device__ __forceinline__ bool enough_to_build(const KArgs<T>& a, int na) {
    return a.n <= kBuildPerCta * resident_ctas(na);
}
// Whether the CTAs without one are enough to take those writes: a quarter of the grid.
__device__ __forceinline__ bool others_write(int na) { return 4 * ((int)gridDim.x - resident_ctas(na)) >= (int)gridDim.x; }

template <typename T, typename End, typename Mark>
__device__ __forceinline__ bool resident_substeps(const KArgs<T>& a, const Frame<T>& F, int ph0, PhaseCtl& ctl,
                                                  unsigned char* pool, SubSync* sync, End end_phase, Mark mark) {
    typedef typename vec4_of<T>::type V4;
    constexpr int kWarps = kThreads / 32;
    __shared__ int s_used;
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const int na = ctl.act;
    // Element i belongs to CTA i mod n_cta; the other CTAs wait for the frame's next
    // phase, after writing what the frame writes beside its substeps.
    const int n_cta = resident_ctas(na);
    const int last_ph = ph0 + 3 * a.k_sub - 1;
    const bool copy_bonds = a.nb > 0 && F.src.ds != F.dst.ds;
    const bool others_copy = others_write(na);
    const bool test_fault = a.fail_phase >= ph0 && a.fail_phase <= last_ph;
    if ((int)blockIdx.x >= n_cta) {
        if (others_copy) {
            const int cw = (blockIdx.x - n_cta) * kWarps + wl, ncw = (gridDim.x - n_cta) * kWarps;
            for (int s = 0; copy_bonds && s < a.k_sub; ++s) copy_bond_slice(a, F, s, cw, ncw);
            const T scale = T(*((volatile const double*)a.fscal));
            frame_outputs(a, F, scale, cw * 32 + lane, ncw * 32, true);
        }
        if (test_fault && n_cta < 2 && blockIdx.x == gridDim.x - 1) return false;
        return end_phase(last_ph);
    }
    int parity = 0;
    // end of a substep's phase: 0, or 1 with the phase words read, or -1
    auto sub_end = [&](int ph) -> int {
        if (ph == a.fail_phase && n_cta > 1 && (int)blockIdx.x == n_cta - 1) return -1;
        const int res = sub_barrier(a, n_cta, parity, sync);
        parity ^= 1;
        mark(ph);
        if (res > 0) {
            if (threadIdx.x < 32) load_ctl(a, ph + 1, &ctl);
            __syncthreads();
        }
        return res;
    };
    const int per_cta = (na + n_cta - 1) / n_cta;  // at most
    const int mine = (na - 1 - (int)blockIdx.x) / n_cta + 1;
    const bool wide = per_cta <= kWarps;
    // stage the CTA's elements: a thread each for the records, then a warp each
    // for slots and candidates
    if (threadIdx.x == 0) s_used = per_cta * (int)sizeof(ResElem<T>);
    __syncthreads();
    if ((int)threadIdx.x < mine) {
        ResElem<T>* E = reinterpret_cast<ResElem<T>*>(pool) + threadIdx.x;
        const int e = a.act_list[blockIdx.x + threadIdx.x * n_cta];
        const V4 k = ld4(a.kin[0], e), ec = ld4(a.econ, e);  // ec: mass, inertia, thickness, area
        const int s0 = a.boff[e], nbe = a.boff[e + 1] - s0, nc = a.ncnt[e];
        const T sub = F.dst.sub[e];
        const typename vec2_of<T>::type v = ld2(a.kvel[0], e), w = ld2(F.vw, e), so = ld2(a.soi, e);
        E->p[0] = k.x;
        E->p[1] = k.y;
        E->p[2] = F.src.rot[e];
        E->p[3] = k.z;
        E->v[0] = v.x;
        E->v[1] = v.y;
        E->v[2] = F.src.avel[e];
        // the factors of the drag that do not change in a frame (integrate_element's, in its order)
        E->m[0] = E->m[1] = ec.x;
        E->m[2] = ec.y;
        E->m[3] = a.fc.c_drag * (ec.w * (ec.z / a.fc.href));
        E->so[0] = so.x;
        E->so[1] = so.y;
        E->so[2] = T(0);
        E->so[3] = ec.w * jmin(sub / jmax(ec.z, T(1e-10)), T(1));
        E->w[0] = w.x;
        E->w[1] = w.y;
        E->w[2] = a.fc.c_rot * k.w;
        reinterpret_cast<V4*>(a.kin[1])[e] = k;  // the radii of the other buffer; substeps write positions only
        E->e = e;
        E->nbe = nbe;
        E->s0 = s0;
        const int room = nc + 4;  // a rebuilt list may be a little longer
        const int bytes = nbe * (int)sizeof(SlotRec<T>) + ((room * 4 + 15) & ~15);
        const int at = atomicAdd(&s_used, bytes);
        const bool fits = at + bytes <= res_pool_bytes<T>();
        E->slots = fits ? at : -1;
        E->cands = fits ? at + nbe * (int)sizeof(SlotRec<T>) : -1;
        E->room = ((room * 4 + 15) & ~15) / 4;
    }
    __syncthreads();
    for (int el = wl; el < mine; el += kWarps) {
        const ResElem<T>* E = reinterpret_cast<const ResElem<T>*>(pool) + el;
        if (E->slots >= 0 && lane < E->nbe)
            for (int i = lane; i < E->nbe; i += 32)
                reinterpret_cast<SlotRec<T>*>(pool + E->slots)[i] = reinterpret_cast<const SlotRec<T>*>(a.slotrec)[E->s0 + i];
        resident_list(a, pool, el);
    }
    __syncthreads();
    unsigned cnt = ctl.esc;
    for (int s = 0; s < a.k_sub; ++s) {
        const unsigned round = a.round_base + (unsigned)(F.f * a.k_sub + s) + 1u;
        const bool all = rebuild_all(a, cnt);
        if (cnt != 0u) {  // uniform over the CTAs
            phase_escape(a, F, cnt, s, round, all, n_cta);
            __syncthreads();
            if (threadIdx.x == 0) sync->flag = 1;  // the marks' counter has to be read
            if (sub_end(ph0 + 3 * s) < 0) return false;
            if (all) {
                phase_build_all(a, n_cta);
                if (sub_end(ph0 + 3 * s + 1) < 0) return false;
            }
            const int nd = all ? 0 : ctl.dirty;
            if (nd > 0) {
                // an active element's warp rebuilds its list; any warp those of frozen elements
                if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd((unsigned long long*)&a.stats[4], (unsigned long long)nd);
                for (int q = wl * n_cta + blockIdx.x; q < nd; q += kWarps * n_cta) {
                    const int d = a.dirty_list[q];
                    if (!F.dst.active[d]) warp_build(a, d);
                }
            }
            if (nd > 0 || all)
                for (int el = wl; el < mine; el += kWarps) {
                    const int e = reinterpret_cast<const ResElem<T>*>(pool)[el].e;
                    const bool dirty = !all && a.dirty[e] == round;
                    if (dirty) warp_build(a, e);
                    if (dirty || all) resident_list(a, pool, el);
                }
        }
        const bool last = s == a.k_sub - 1;
        if (wide) {
            if (wl < mine) resident_step<T, 32>(a, F, pool, wl, warp_terms<T>(), s, last, &sync->flag);
        } else {
            const int g = lane / kGroup;
            T* wt = warp_terms<T>() + g * kGroupTerms<T>;
            for (int e0 = 0; e0 < mine; e0 += kThreads / kGroup) {
                const int el = e0 + g * kWarps + wl;
                if (e0 + wl < mine) resident_step<T, kGroup>(a, F, pool, el < mine ? el : -1, wt, s, last, &sync->flag);
            }
        }
        if (copy_bonds && !others_copy) copy_bond_slice(a, F, s, blockIdx.x * kWarps + wl, n_cta * kWarps);
        if (last) break;
        const int res = sub_end(ph0 + 3 * s + 2);
        if (res < 0) return false;
        cnt = res > 0 ? ctl.esc : 0u;
        if (a.crec && blockIdx.x == 0 && threadIdx.x == 0) {
            const int m = F.f * a.k_sub + s;
            if (m < a.crec_max_marks) a.crec_marks[m] = (int)*((volatile unsigned*)a.crec_cnt);
        }
    }
    if (test_fault && n_cta < 2 && blockIdx.x == gridDim.x - 1) return false;
    return end_phase(last_ph);
}

// ─── bond damage (jax_bond_fracture.py:133-208) ─────────────────────────────
template <typename T>
__device__ void bond_damage(const DemParams& P, T delta_n, T delta_s, T sigma_n, T sigma_t, T sigma_bar,
                            T cur_d, T cur_max, T cur_0, bool intact, T& nd, T& nmax, T& n0, bool& nint) {
    const T SC = T(1e12);
    delta_n = jclip(delta_n, T(-1e3), T(1e3));
    delta_s = jclip(delta_s, T(-1e3), T(1e3));
    sigma_bar = jclip(sigma_bar, T(1e-10), SC);
    // equivalent deformation (:69-77)
    T dn = jclip(delta_n, T(-1e3), T(1e3));
    T dsa = jclip(fabs(delta_s), T(0), T(1e3));
    T dnp = jmax(dn, T(0));
    T delta_m = jsqrt(jclip(dnp * dnp + dsa * dsa + T(1e-20), T(0), T(1e12)));
    nmax = jmax(cur_max, delta_m);
    // Mohr-Coulomb shear strength (:60-66)
    T tau_bar = jmax(T(P.bond_cohesion) - T(P.bond_internal_friction) * sigma_n, T(1e-6));
    // strength criterion (:35-57)
    T s_pos = jmax(jclip(sigma_n, -SC, SC), T(0));
    T tau = jclip(sigma_t, -SC, SC);
    T sb = jmax(jclip(sigma_bar, T(1e-10), SC), T(1e-10));
    T tb = jmax(jclip(tau_bar, T(1e-10), SC), T(1e-10));
    T q1 = s_pos / sb, q2 = tau / tb;
    T crit = jclip(q1 * q1 + q2 * q2, T(0), T(1e10));
    bool initiating = (crit >= T(1)) && (cur_0 <= T(0)) && (delta_m > T(1e-5));
    n0 = initiating ? delta_m : cur_0;
    // fracture-energy ratio and Benzeggagh-Kenane energy (:103-121)
    T dnp2 = jmax(delta_n, T(0));
    T g_ratio = (delta_s * delta_s) / (dnp2 * dnp2 + T(1e-10));
    T g_I = T(1) / (T(1) + g_ratio + T(1e-10));
    T g_II = g_ratio / (T(1) + g_ratio + T(1e-10));
    T g_tot = g_I + g_II + T(1e-10);
    T ratio = g_II / g_tot;
    const T dG = T(P.bond_G_c_II - P.bond_G_c_I);
    // (G_c^II - G_c^I) * ratio^eta with ratio in [0, 1]: exactly 0 when the energies are equal
    T g_c = T(P.bond_G_c_I) + ((dG != T(0)) ? dG * jpow(ratio, T(P.bond_eta_bk)) : dG * T(0));
    T snc = jclip(sigma_n, -SC, SC), stc = jclip(sigma_t, -SC, SC);
    T snp = jmax(snc, T(0));
    T sm0_raw = jsqrt(jclip(snp * snp + stc * stc + T(1e-20), T(0), T(1e24)));
    T sm0 = jmax(sm0_raw, T(1e-10));
    T dm_f = (T(2) * g_c) / (fabs(sm0) + T(1e-10));
    bool meaningful = sm0_raw >= T(1e4);
    bool has_dmg = (n0 > T(0)) && meaningful;
    // damage variable (:80-100)
    T comp = cur_d;
    if (has_dmg) {
        T d0c = jclip(n0, T(0), T(1e6));
        T dfc = jmax(jclip(dm_f, T(1e-10), T(1e6)), T(1e-10));
        T dmaxc = jmax(jclip(nmax, T(0), T(1e6)), d0c + T(1e-10));
        T denom = jmax(dmaxc * (dfc - d0c + T(1e-10)), T(1e-20));
        comp = jclip(dfc * (dmaxc - d0c) / denom, T(0), T(1));
    }
    T d = meaningful ? jmax(comp, cur_d) : cur_d;
    nd = jmin(d, cur_d + T(0.15));
    nint = intact && (nd < T(1));
}

// ─── P_FRACTURE (jax_simulation.py:534-653) + history ───────────────────────
// The full fracture update of bond b (jax_simulation.py:534-653), for a bond
// with an active end.
template <typename T>
__device__ __forceinline__ void fracture_bond(const KArgs<T>& a, const Frame<T>& F, T scale, int b) {
    typedef typename vec2_of<T>::type V2;
    const DemParams& P = a.P;
    const T mft = T(P.max_fracture_thickness);
    const T esc = T(P.effective_strength_collision);
    const T dti = T(P.dt_ice);
    const T kn = a.k_n, ks = a.k_s;
    const int i = a.bi[b], j = a.bj[b];
    const T ds0 = F.src.ds[b], cur_d = F.src.dmg[b], dmmax0 = F.src.dmmax[b], dm00 = F.src.dm0[b];
    const bool intact = F.src.intact[b] != 0;
    const T rest = a.rest[b], sbar = a.sbar[b], bstr = a.bstr[b];
    const V2 pi = ld2(F.dst.pos, i), pj = ld2(F.dst.pos, j);
    const V2 vi = ld2(F.dst.vel, i), vj = ld2(F.dst.vel, j);
    const bool both_act = F.dst.active[i] && F.dst.active[j];
    const int fli = a.floe_of[i], flj = a.floe_of[j];
    const bool breakable = (a.thick[i] <= mft) && (a.thick[j] <= mft);
    const T sc = sys_scale(a, scale, a.nsys > 1 ? a.sys_of[i] : 0);  // i and j share a system
    const T fmi = a.fraw[i] * sc, fmj = a.fraw[j] * sc;
    const bool at_crack = a.crack[i] || a.crack[j];
    const T scf = sys_scale(a, scale, a.nsys > 1 ? a.floe_sys[fli] : 0);
    const bool floe_ok = new_elig(a, F, fli, scf) && new_elig(a, F, flj, scf);
    T dx = pj.x - pi.x, dy = pj.y - pi.y;
    T dist = jsqrt(dx * dx + dy * dy);
    T dsafe = jmax(dist, T(1e-10));
    T bx = dx / dsafe, by = dy / dsafe;
    bool near = (fmi > T(0)) || (fmj > T(0));
    bool dpdem_ok = both_act && floe_ok && (near || at_crack) && breakable;
    T vrx = vj.x - vi.x, vry = vj.y - vi.y;
    T vn = vrx * bx + vry * by;
    T vtx = vrx - vn * bx, vty = vry - vn * by;
    T ds_incr = jsqrt(vtx * vtx + vty * vty) * dti;
    bool ds_gate = near && both_act && floe_ok && breakable;
    T new_ds = ds0 + (ds_gate ? ds_incr : T(0));
    T L0 = jmax(rest, T(1e-10));
    T delta_n = dist - rest;
    T dn_d = near ? delta_n : T(0);
    T sn = (kn * (dn_d / L0)) * (T(1) - cur_d);
    T st = (ks * (new_ds / L0)) * (T(1) - cur_d);
    T od = cur_d, omax = dmmax0, o0 = dm00;
    bool fin = intact;
    if (dpdem_ok) {
        // the damage law's result is only selected for DPDEM-eligible bonds
        // (jnp.where at jax_simulation.py:620-623); elsewhere the old state stays
        T nd, nmax, n0;
        bool nint;
        bond_damage<T>(P, delta_n, new_ds, sn, st, sbar, cur_d, omax, o0, intact, nd, nmax, n0, nint);
        od = nd;
        omax = nmax;
        o0 = n0;
        if (breakable) fin = nint;
    }
    // direct collision breaking (jax_simulation.py:629-637)
    bool coll_on = (fmi > T(0)) || (fmj > T(0));
    T coll_f = jmax(fmi, fmj);
    bool brk = intact && coll_on && (coll_f > bstr * esc) && breakable;
    fin = fin && !brk;
    F.dst.dmg[b] = od;
    F.dst.dmmax[b] = omax;
    F.dst.dm0[b] = o0;
    F.dst.ds[b] = new_ds;
    F.dst.intact[b] = fin ? 1 : 0;
    if (a.h_intact) a.h_intact[(size_t)F.f * a.nb + b] = fin ? 1 : 0;
}

template <typename T>
__device__ void phase_fracture(const KArgs<T>& a, const Frame<T>& F, T scale, int nfb, int na, bool written) {
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const int gsz = gridDim.x * blockDim.x;
    const unsigned fstamp = frame_stamp(a, F);
    // the bonds with an active end (listed by phase_reduce) take the full
    // update; every other bond keeps its state, which the force phases have
    // copied already when the frame writes a separate output, or which is in
    // place; its history row is that state
    if ((long long)nfb * 4 > (long long)a.nb) {
        // most bonds are listed: visit them in index order by their stamps,
        // with coalesced bond loads (the list's order is the append order)
        for (int b = gtid; b < a.nb; b += gsz)
            if (a.bstamp[b] == fstamp) fracture_bond(a, F, scale, b);
    } else {
        for (int i = gtid; i < nfb; i += gsz) fracture_bond(a, F, scale, a.fb_list[i]);
    }
    if (!written) {
        frame_outputs(a, F, scale, gtid, gsz, false);
    } else if (a.h_pos || a.h_rot) {
        for (int i = gtid; i < na; i += gsz) element_rows(a, F, a.act_list[i]);
    }
    for (int i = gtid; i < a.k_sub + 2; i += gsz) {
        a.esc_cnt[i] = 0u;
        a.dirty_cnt[i] = 0;
        a.work_cnt[i] = 0;
    }
}

// ─── the kernel ─────────────────────────────────────────────────────────────
// Phase numbering inside a frame: 0 cull (+ grid compaction), 1 near-element
// contact, 2 contact forces, 3 reduce + vessel, then for substep s: 4+3s
// escape round (re-reference + mark), 5+3s rebuild of every list (only when
// most elements escaped), 6+3s force (rebuilding marked lists first); last:
// 4+3k fracture.  Whether a list phase runs is decided by every CTA from the
// same word after a barrier, so skipped phases skip their barrier too.
template <typename T>
__global__ void __launch_bounds__(kThreads, DEM_MIN_BLOCKS) dem_frames_kernel(const __grid_constant__ KArgs<T> a, int ph_lo, int ph_hi) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* hullw = reinterpret_cast<T*>(smem_raw);  // the near phase's; the substeps' pool of elements takes the same bytes
    const int k = a.k_sub;
    const int per_frame = phases_per_frame(k);
    if (ph_hi > a.K * per_frame) ph_hi = a.K * per_frame;  // uniform over the grid
    const bool persistent = (a.mode == DEM_LAUNCH_PERSISTENT);
    if (persistent && a.ptimes && blockIdx.x == 0 && threadIdx.x == 0) a.ptimes[1] = globaltimer_ns();
    __shared__ SubSync sync;
    __shared__ PhaseCtl ctl;  // the words of the phase about to run, in every CTA
    if (threadIdx.x < 32) load_ctl(a, ph_lo, &ctl);
    __syncthreads();
    // phase end times (debug/profiling): entry i = [phase, globaltimer]
    auto mark = [&](int ph) {
        if (a.ptimes && blockIdx.x == 0 && threadIdx.x == 0) {
            const unsigned long long i = atomicAdd(a.ptimes, 1ull);
            if (i < (unsigned long long)kMaxPhaseTimes) {
                a.ptimes[2 + 2 * i] = (unsigned long long)ph;
                a.ptimes[3 + 2 * i] = globaltimer_ns();
            }
        }
    };
    // a barrier after every phase but the last; with profiling on, after the
    // last one too, so that its end time is recorded
    auto end_phase = [&](int ph) -> bool {
        if (!persistent || !(ph + 1 < ph_hi || a.ptimes)) return true;
        // failure-detection test: one CTA leaves, every other CTA's barrier
        // wait ends at its time limit with DEM_ERR_TIMEOUT
        if (ph == a.fail_phase && blockIdx.x == gridDim.x - 1) return false;
        if (ph % per_frame == 3 && threadIdx.x == 0) {
            // no substep barrier is under way: the escape counts stand still
            const unsigned long long v = ld_acquire_u64(a.sub_bar);
            sync.base[0] = v & 0x3ffffffull;
            sync.base[1] = (v >> 26) & 0x3ffffffull;
            sync.flag = 0;
        }
        if (!grid_barrier(a, ph + 1, &ctl)) return false;
        mark(ph);
        return true;
    };
    bool resident = false;  // this frame's substeps held their elements in shared memory
    for (int ph = ph_lo; ph < ph_hi; ++ph) {
        const int f = ph / per_frame;
        const int p = ph % per_frame;
        if (a.crec && p >= 7 && (p - 7) % 3 == 0 && blockIdx.x == 0 && threadIdx.x == 0) {
            // the force phase of substep (p - 7) / 3 has ended (barrier or launch boundary)
            const int m = f * k + (p - 7) / 3;
            if (m < a.crec_max_marks) a.crec_marks[m] = (int)*((volatile unsigned*)a.crec_cnt);
        }
        Frame<T> F = make_frame(a, f);
        if (p == 0) {
            resident = false;
            phase_cull(a, F, ctl.comp_start, ctl.comp_end);
        } else if (p == 1) {
            phase_near(a, F, hullw, ctl.near, upkeep_now(a, ctl.esc) ? (int)ctl.esc : 0);
        } else if (p == 2) {
            phase_cforce(a, F, upkeep_now(a, ctl.esc) ? ctl.dirty : 0);
        } else if (p == 3) {
            phase_reduce(a, F, upkeep_now(a, ctl.esc));
        } else if (p == per_frame - 1) {
            phase_fracture(a, F, T(ctl.scale), ctl.fb, ctl.act, resident && others_write(ctl.act));
        } else if (p == 4 && persistent && a.force_split != DEM_SPLIT_THREAD &&
                   ctl.act <= (int)gridDim.x * res_elems<T>() &&
                   (!rebuild_all(a, ctl.esc) || enough_to_build(a, ctl.act))) {
            // the CTAs' shared memory holds every active element: all substeps in one go
            if (!resident_substeps(a, F, ph, ctl, smem_raw, &sync, end_phase, mark)) return;
            ph += 3 * k - 1;  // the last force phase has ended
            resident = true;
            continue;
        } else {
            const int s = (p - 4) / 3;
            const int sub = (p - 4) % 3;
            const unsigned cnt = ctl.esc;
            const bool all = rebuild_all(a, cnt);
            // stamp of this rebuild round, unique since the dirty stamps were last cleared
            const unsigned round = a.round_base + (unsigned)(f * k + s) + 1u;
            if (sub == 0) {
                if (cnt == 0u) continue;  // uniform: no barrier either
                phase_escape(a, F, cnt, s, round, all, gridDim.x);
            } else if (sub == 1) {
                if (cnt == 0u || !all) continue;
                phase_build_all(a, gridDim.x);
            } else {
                phase_force(a, F, s, round, all ? 0 : ctl.dirty, ctl.act);
            }
        }
        if (!end_phase(ph)) return;
    }
}

// per-element constants packed for one vector load per substep
template <typename T>
__global__ void econ_kernel(const T* mass, const T* inertia, const T* thick, const T* area, int n, T* out) {
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    out[4 * (size_t)e + 0] = mass[e];
    out[4 * (size_t)e + 1] = inertia[e];
    out[4 * (size_t)e + 2] = thick[e];
    out[4 * (size_t)e + 3] = area[e];
}

// r^3 per element in the dtype (radii ** 3, jax_simulation.py:205)
template <typename T>
__global__ void cube_kernel(const T* r, int n, T* out) {
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n) out[e] = jpow(r[e], T(3));
}

// per-slot bond constants: rest length and E * ((h_i + h_j) * 0.5) * factor in
// the dtype (jax_simulation.py:81-82)
template <typename T>
__global__ void slot_setup_kernel(const T* thick, const T* rest, const int* bi, const int* bj,
                                  const int2* slots, int n_slots, double E, double factor, T* slot_rest,
                                  T* slot_stiff) {
    int sl = blockIdx.x * blockDim.x + threadIdx.x;
    if (sl >= n_slots) return;
    int b = slots[sl].x & 0x7fffffff;
    T avg = (thick[bi[b]] + thick[bj[b]]) * T(0.5);
    slot_stiff[sl] = T(E) * avg * T(factor);
    slot_rest[sl] = rest[b];
}

}  // namespace dem
