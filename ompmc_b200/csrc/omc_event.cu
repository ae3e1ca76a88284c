// Event-based FP32 transport: structure-of-arrays particle queues, one
// transport event per queued particle per launch, outputs appended with
// warp-aggregated atomics, FP64 tallies per batch slot.
//
// A transport cycle is five launches on one stream:
//   k_plan      how many new histories fit (in-flight target - occupancy),
//               the electron budget of this cycle, output queues emptied
//   k_source    primaries of those histories into the input queues
//   k_photon    one photon event per queued photon
//   k_electron  one electron event per queued e-/e+; electrons that reach a
//               discrete interaction are queued for
//   k_electron_interact  which samples those interactions (a kernel of its
//               own keeps the samplers' code out of the transport kernel's
//               instruction cache: 8 % faster on slab64)
// Queues are double-buffered (A -> B, then B -> A), so two cycles form an
// idempotent CUDA graph that the host replays until every history is
// injected (after that, one without k_source) and few particles are left;
// k_drain then runs those to the end.
//
// An event transports its particle until the next interaction, death or,
// for electrons, the end of the cycle's budget of tstep-loop iterations.
// The budget is small while the queues fill the GPU (lanes of a warp then do
// similar work) and grows as they drain, so the drain tail takes few
// cycles.  Each particle carries its own Philox stream (key, position) and
// secondaries get keys from the parent's key and stream position at their
// creation, so a particle's trajectory does not depend on where events are
// cut nor on scheduling: any budget gives the same result up to the
// summation order of the FP64 tallies.
#include <algorithm>
#include <cstdio>
#include <type_traits>

#include "omc_event.h"
#include "omc_ring.cuh"
#include "omc_rng.cuh"
#include "omc_source.cuh"

namespace omc {

constexpr int EV_BUDGET = 200000;  // transport steps one event may take
constexpr int EV_MAXOUT = 1;       // secondaries an event emits: every interaction sampler pushes one
constexpr int EV_MAXOUT_SPLIT = 2; // products of a split photon's sub-photon (pair: two)
constexpr int EV_MAX_BLOCK = 256;  // launch bound of the transport kernels
// Resident 256-thread blocks per SM the electron kernel is compiled for:
// four (64 registers) in FP32, two (128 registers) in FP64.  Measured on the
// served beamlet load and the slab beam with the step's state in
// registers: 3 blocks (80 registers) 50.6 and 70.3 M hist/s, 4 blocks 52.6
// and 71.8, 5 blocks (48 registers) 52.1 and 70.3.
template <typename R>
constexpr int electron_minb() {
    return sizeof(R) == 4 ? 4 : 2;
}

template <typename R>
using TransportKernelT = void (*)(DevData<R>, QueueT<R>, QueueT<R>, QueueT<R>, double *, long, Ctl *, uint32_t,
                                  ServeDev *, int, QueueT<R>);
using TransportKernel = TransportKernelT<float>;

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

template <int MAXOUT, typename R = float, typename Rng = Philox<R>, bool STATS = true>
struct EvEnv {
    static constexpr bool kBuffered = IsRing<Rng>::value;
    Rng rng;
    double *tally;   // the tallies of all slots, nvox apart
    long nvox;
    int slot;        // the particle's
    int pend_ir;
    double pend_e;
    Part<R> out[MAXOUT];
    uint32_t out_pos[MAXOUT];     // parent's stream position at each push
    int nout;
    unsigned flags;
    int work;
    int tleft;                    // tstep-loop iterations left in this event
    int ncross, ndep, natom;
    __device__ R uni() { return rng.uni(); }
    // Consecutive deposits into one voxel are summed before the atomic.
    __device__ void deposit(int ir, R e) {
        if (STATS) ndep++;
        if (ir != pend_ir) {
            flush();
            pend_ir = ir;
        }
        pend_e += (double)e;
    }
    __device__ void flush() {
        if (pend_ir > 0 && pend_e != 0.0) {
            // the lanes of the warp that flush here together into the same
            // tally element (same voxel and tally slot) add once: the
            // group's sum, by its lowest lane (+4-5 % on the served beamlet
            // load and the slab beam over one atomic per lane)
            double *dst = tally + ((long)slot * nvox + (pend_ir - 1));
            const unsigned act = __activemask();
            const unsigned grp = __match_any_sync(act, (unsigned long long)dst);
            const int lane = threadIdx.x & 31;
            double tot = pend_e;
            if (grp != (1u << lane)) {
                tot = 0.0;
                for (unsigned m = grp; m; m &= m - 1) tot += __shfl_sync(grp, pend_e, __ffs(m) - 1);
            }
            if (lane == __ffs(grp) - 1) {
                atomicAdd(dst, tot);
                if (STATS) natom++;
            }
        }
        pend_e = 0.0;
        pend_ir = -1;
    }
    __device__ void cross() {
        if (STATS) ncross++;
    }
    __device__ bool tstep_take() { return tleft-- > 0; }
    __device__ bool push(const Part<R> &q) { return push_at(q, rng.position()); }
    // A push made at stream position `pos` (an event run out of line).
    __device__ bool push_at(const Part<R> &q, uint32_t pos) {
        if (nout >= MAXOUT) {
            flags |= ERR_STACK;
            return false;
        }
        // static indices keep the outputs in registers
#pragma unroll
        for (int k = 0; k < MAXOUT; k++)
            if (k == nout) {
                out_pos[k] = pos;
                out[k] = q;
            }
        nout++;
        return true;
    }
    __device__ void err(unsigned f) { flags |= f; }
    // (the electron step bounds its own iterations far below the budget)
    __device__ bool tick() { return kBuffered && !STATS ? true : ++work < EV_BUDGET; }
};

// A photon event through the out-of-line photon_event_outline: its results
// folded back into the event environment in the order the photon step
// itself would have made them (stream, counters, deposit, pushed product).
template <int MAXOUT, typename R>
__device__ __forceinline__ bool photon_event(const DevData<R> &D, EvEnv<MAXOUT, R> &g, Part<R> &p) {
    const PhotonEventOut<R> o = photon_event_outline<R>(D, p, g.rng, g.work, EV_BUDGET);
    p = o.p;
    g.rng = o.e.rng;
    g.work = o.e.work;
    g.ncross += o.e.ncross;
    g.flags |= o.e.flags;
    if (o.e.dep_ir >= 0) g.deposit(o.e.dep_ir, o.e.dep_e);
    if (o.e.nq) g.push_at(o.e.q, o.e.qpos);
    return o.alive != 0;
}

template <typename R = float>
struct SrcEnv {
    Philox<R> rng;
    __device__ R uni() { return rng.uni(); }
};

// A queued particle is read once and written once per event, so its loads
// and stores bypass L1 and are marked streaming (evict first) in L2, which
// keeps the caches for the tables, the tallies and the kernels' local frames.
// SHARED: an entry that another block of the same launch wrote (read in L2).
template <bool SHARED, typename T>
__device__ __forceinline__ T qread(const T *p) {
    return SHARED ? __ldcg(p) : __ldcs(p);
}
template <bool SHARED = false>
__device__ __forceinline__ void qload(const Queue &q, int i, Part<float> &p, int &tag, uint32_t &k0, uint32_t &k1,
                                      uint32_t &ctr) {
    const float4 a = qread<SHARED>(&q.pos[i]);
    const float4 b = qread<SHARED>(&q.dir[i]);
    const uint4 c = qread<SHARED>(&q.id[i]);
    ctr = qread<SHARED>(&q.ctr[i]);
    p.x = a.x; p.y = a.y; p.z = a.z; p.u = a.w;
    p.v = b.x; p.w = b.y; p.e = b.z; p.wt = b.w;
    p.ir = (int)c.x;
    tag = (int)c.y;
    p.iq = (tag & 3) - 1;
    k0 = c.z; k1 = c.w;
}

__device__ __forceinline__ void qload(const QueueT<double> &q, int i, Part<double> &p, int &tag, uint32_t &k0,
                                      uint32_t &k1, uint32_t &ctr) {
    const double2 *pa = (const double2 *)&q.pos[i], *pb = (const double2 *)&q.dir[i];
    const double2 a0 = __ldcs(pa), a1 = __ldcs(pa + 1), b0 = __ldcs(pb), b1 = __ldcs(pb + 1);
    const uint4 c = __ldcs(&q.id[i]);
    ctr = __ldcs(&q.ctr[i]);
    p.x = a0.x; p.y = a0.y; p.z = a1.x; p.u = a1.y;
    p.v = b0.x; p.w = b0.y; p.e = b1.x; p.wt = b1.y;
    p.ir = (int)c.x;
    tag = (int)c.y;
    p.iq = (tag & 3) - 1;
    k0 = c.z; k1 = c.w;
}

// sp/sr: splitting state, stored where the queue has it (photon queues of
// splitting engines); -1 = a photon not yet split.
__device__ __forceinline__ void qstore(const Queue &q, int i, const Part<float> &p, int slot, uint32_t k0, uint32_t k1,
                                       uint32_t ctr, int sp = -1, float sr = 0.f) {
    __stcs(&q.pos[i], make_float4(p.x, p.y, p.z, p.u));
    __stcs(&q.dir[i], make_float4(p.v, p.w, p.e, p.wt));
    __stcs(&q.id[i], make_uint4((uint32_t)p.ir, (uint32_t)((p.iq + 1) | (slot << 2)), k0, k1));
    __stcs(&q.ctr[i], ctr);
    if (q.sp) {
        q.sp[i] = sp;
        q.sr[i] = sr;
    }
}

__device__ __forceinline__ void qstore(const QueueT<double> &q, int i, const Part<double> &p, int slot, uint32_t k0,
                                       uint32_t k1, uint32_t ctr, int sp = -1, float sr = 0.f) {
    double2 *pa = (double2 *)&q.pos[i], *pb = (double2 *)&q.dir[i];
    __stcs(pa, make_double2(p.x, p.y));
    __stcs(pa + 1, make_double2(p.z, p.u));
    __stcs(pb, make_double2(p.v, p.w));
    __stcs(pb + 1, make_double2(p.e, p.wt));
    __stcs(&q.id[i], make_uint4((uint32_t)p.ir, (uint32_t)((p.iq + 1) | (slot << 2)), k0, k1));
    __stcs(&q.ctr[i], ctr);
    if (q.sp) {
        q.sp[i] = sp;
        q.sr[i] = sr;
    }
}

// Slot of a warp-aggregated append to `q` for the lanes with `want`: from
// the bottom, or from the top for lanes with `hi`; -1 for the other lanes
// (or on overflow, flagged).
template <typename Q>
__device__ __forceinline__ int warp_append(const Q &q, bool want, bool hi, unsigned active, unsigned &flags) {
    const int lane = threadIdx.x & 31;
    const unsigned mlo = __ballot_sync(active, want && !hi);
    const unsigned mhi = __ballot_sync(active, want && hi);
    int blo = 0, bhi = 0;
    if (mlo) {
        int leader = __ffs(mlo) - 1;
        if (lane == leader) blo = atomicAdd(q.count, __popc(mlo));
        blo = __shfl_sync(active, blo, leader);
    }
    if (mhi) {
        int leader = __ffs(mhi) - 1;
        if (lane == leader) bhi = atomicAdd(q.count_hi, __popc(mhi));
        bhi = __shfl_sync(active, bhi, leader);
    }
    if (!want) return -1;
    int k = hi ? bhi + __popc(mhi & lanemask_lt()) : blo + __popc(mlo & lanemask_lt());
    if (k >= q.cap) {
        flags |= ERR_QUEUE;
        return -1;
    }
    return hi ? q.cap - 1 - k : k;
}

// Entries of a queue (both ends) and the index of the f-th, top end first.
template <typename Q>
__device__ __forceinline__ int queue_size(const Q &q) {
    return min(min(*q.count, q.cap) + min(*q.count_hi, q.cap), q.cap);
}
template <typename Q>
__device__ __forceinline__ int queue_index(const Q &q, int f) {
    int nhi = min(*q.count_hi, q.cap);
    return f < nhi ? q.cap - 1 - f : f - nhi;
}

// Route the event's surviving particle and its secondaries to the output
// queues.  A secondary's stream key is derived from its parent's key, the
// parent's stream position when it was created and its index among the
// event's secondaries.  All 32 lanes of the warp take part (lanes without a
// particle pass alive = false, nout = 0).  The survivor keeps its splitting
// state (sp, sr); secondaries start unsplit.  Photons of zero weight (lost
// a Russian roulette) would deposit nothing and are not queued, and an
// electron at or below its region's cut-off is not queued either: its
// first event would only deposit its kinetic energy where it stands (the
// entry test of electron_step, which the drain applies to the same
// particle), so that deposit is made here.  It draws no random number, so
// trajectories do not change.  Returns the particles this lane queued.
template <int MAXOUT, bool DEFER = false, typename R = float, typename Env>
__device__ __forceinline__ int emit(const DevData<R> &D, const QueueT<R> &outP, const QueueT<R> &outE, bool alive,
                                    const Part<R> &p, Env &g, int slot, uint32_t k0, uint32_t k1,
                                    float esplit, int sp = -1, float sr = 0.f, const QueueT<R> *outI = nullptr,
                                    bool defer = false) {
    const unsigned full = 0xffffffffu;
    uint64_t pkey = ((uint64_t)k1 << 32) | k0;
    int queued = 0;
#pragma unroll
    for (int k = 0; k < 1 + MAXOUT; k++) {
        bool has;
        Part<R> q;
        uint32_t a0 = k0, a1 = k1, ac;
        if (k == 0) {
            has = alive;
            q = p;
            ac = g.rng.position();
        } else {
            has = k - 1 < g.nout;
            q = g.out[k - 1];
            uint64_t ck = mix64(pkey * 0x9E3779B97F4A7C15ull + ((uint64_t)g.out_pos[k - 1] << 1) + 1u +
                                ((uint64_t)(k - 1) << 40));
            a0 = (uint32_t)ck;
            a1 = (uint32_t)(ck >> 32);
            ac = 0;
        }
        if (__ballot_sync(full, has) == 0) continue;
        if (has && !(q.e == q.e && q.x == q.x && q.u == q.u)) {
            g.flags |= ERR_NAN;
            has = false;
        }
        if (has && q.iq == 0 && q.wt == R(0)) has = false;
        // an electron left at its discrete interaction goes to the
        // interaction queue
        const bool toi = DEFER && k == 0 && defer;
        bool isph = has && q.iq == 0 && !toi;
        bool isel = has && q.iq != 0 && !toi;
        if (isel && q.iq < 0 && q.e <= ecut_of(D, q.ir)) {
            g.deposit(q.ir, q.wt * (q.e - R(D_RM)));
            isel = false;
        }
        int ip = warp_append(outP, isph, false, full, g.flags);
        int ie = warp_append(outE, isel, esplit > 0.f && q.e > (R)esplit, full, g.flags);
        if (ip >= 0) qstore(outP, ip, q, slot, a0, a1, ac, k == 0 ? sp : -1, k == 0 ? sr : 0.f);
        if (ie >= 0) qstore(outE, ie, q, slot, a0, a1, ac);
        queued += (ip >= 0) + (ie >= 0);
        if (DEFER && k == 0) {
            int ii = warp_append(*outI, has && toi, false, full, g.flags);
            if (ii >= 0) qstore(*outI, ii, q, slot, a0, a1, ac);
            queued += ii >= 0;
        }
    }
    g.flush();
    return queued;
}

__device__ __forceinline__ void report_flags(Ctl *ctl, unsigned flags, unsigned active) {
    unsigned f = __reduce_or_sync(active, flags);
    if (f && (threadIdx.x & 31) == __ffs(active) - 1) atomicOr(&ctl->flags, f);
}

__device__ __forceinline__ void report_count(unsigned long long *dst, unsigned v, unsigned active) {
    unsigned t = __reduce_add_sync(active, v);
    if (t && (threadIdx.x & 31) == __ffs(active) - 1) atomicAdd(dst, (unsigned long long)t);
}

// Live-particle count of a serving request: +delta for the request whose
// tally slots start at req*nbmax, aggregated over the lanes of the warp that
// hold particles of the same request.
__device__ __forceinline__ void add_live(int *live, int nbmax, int slot, int delta, unsigned active) {
    int req = slot / nbmax;
    unsigned grp = __match_any_sync(active, req);
    int tot = __reduce_add_sync(grp, delta);
    if (tot != 0 && (threadIdx.x & 31) == __ffs(grp) - 1) atomicAdd(&live[req], tot);
}

// One event of a split photon (photon splitting, ompmc.c:1867-2139 with
// nsplit > 1).  A queued photon is a ray of nsplit sub-photons of weight
// wt/nsplit whose interaction sites are stratified along it.  Its first
// event checks the cut-off, draws the stratification offset r and the
// surviving sub-photon, and sets the ray's weight; every event then moves
// one sub-photon, k, from the previous site by its share of mean free
// paths, ln(eta_{k-1} / eta_k) with eta_k = (nsplit - k - r) / nsplit
// (eta_{-1} = 1), and samples its interaction.  The charged products are
// pushed with the sub-photon's weight; the scattered photon of the
// surviving sub-photon is pushed with the full weight (as a new, unsplit
// photon) and the others' are dropped.  p becomes the ray at the site;
// returns true while it has sub-photons left.  The draws differ from the
// plain form's order (one stream per ray), the sampled distribution is the
// same.
template <typename R, typename Env>
__device__ __forceinline__ bool split_event(const DevData<R> &D, Env &g, Part<R> &p, int &sp, float &sr) {
    const int ns = D.nsplit;
    if (sp < 0) {
        if (p.e <= pcut_of(D, p.ir) || p.wt == 0.f) {
            g.deposit(p.ir, p.wt * p.e);
            return false;
        }
        sr = g.uni();
        int isurv = (int)(g.uni() * (float)ns);
        sp = min(isurv, ns - 1);
        p.wt = p.wt / (float)ns;
    }
    const int isplit = sp >> 16, isurv = sp & 0xffff;
    const float den = (float)(ns - isplit) - sr;
    if (den <= 0.f) return false;
    const float num = isplit == 0 ? (float)ns : den + 1.f;
    const float dpmfp = m_log(num / den);
    const float gle = m_log(p.e);
    Part<float> q = p;
    q.iq = 0;
    int imed, lgle;
    float cohfac;
    if (!photon_walk(D, g, q, gle, dpmfp, imed, lgle, cohfac)) return false;
    p.x = q.x; p.y = q.y; p.z = q.z;
    p.ir = q.ir;
    const bool surv = isplit == isurv;
    if (g.uni() <= 1.f - cohfac) {
        if (surv) {
            q.wt *= (float)ns;
            rayleigh(D, g, q, imed, gle, lgle);
            g.push(q);
        }
    } else {
        photon_interact(D, g, q, p.e, gle, imed, lgle);
        // the interaction pushed at most one product; keep it and q as the
        // splitting rules say
        if (g.nout == 1 && g.out[0].iq == 0) {
            if (surv) g.out[0].wt *= (float)ns;
            else g.nout = 0;
        }
        if (q.iq != 0 || surv) {
            if (q.iq == 0) q.wt *= (float)ns;
            g.push(q);
        }
    }
    sp = ((isplit + 1) << 16) | isurv;
    return isplit + 1 < ns;
}

// Events of one queue.  Warps take 32 particles at a time from a counter,
// so work is balanced between warps however long their events run.
// KIND: EV_PHOTON, EV_ELECTRON, EV_SPLIT (photons of a splitting engine)
// or EV_INTERACT (electrons at their discrete interaction, with
// D.defer_interact).  `qi`: the interaction queue (EV_ELECTRON with
// D.defer_interact appends there).
enum { EV_PHOTON = 0, EV_ELECTRON = 1, EV_SPLIT = 2, EV_INTERACT = 3, EV_ELECTRON_DEFER = 4 };
template <int KIND, typename R = float, bool STATS = true>
__device__ __forceinline__ void transport_events(const DevData<R> &D, const QueueT<R> &in, const QueueT<R> &outP,
                                                 const QueueT<R> &outE, double *tallies, long nvox, Ctl *ctl,
                                                 uint32_t seedw, ServeDev *sd, int nbmax, const QueueT<R> &qi) {
    constexpr int MAXOUT = KIND == EV_SPLIT ? EV_MAXOUT_SPLIT : EV_MAXOUT;
    const unsigned full = 0xffffffffu;
    constexpr bool ELECTRON = KIND == EV_ELECTRON || KIND == EV_ELECTRON_DEFER;
    using Rng = typename std::conditional<KIND == EV_ELECTRON_DEFER && sizeof(R) == 4, RingStream<EV_MAX_BLOCK>, Philox<R>>::type;
    using Env = EvEnv<MAXOUT, R, Rng, STATS>;
    const int kq = ELECTRON ? 1 : (KIND == EV_INTERACT ? 2 : 0);
    const int ks = KIND == EV_PHOTON || KIND == EV_SPLIT ? 0 : 1;   // counters: photon or electron
    const int lane = threadIdx.x & 31;
    unsigned c_ev = 0, c_steps = 0, c_cross = 0, c_dep = 0, c_atom = 0;
    for (int guard = 0; guard < (1 << 26); guard++) {
        int base = 0;
        if (lane == 0) base = atomicAdd(&ctl->fetch[kq], 32);
        base = __shfl_sync(full, base, 0);
        const int n = queue_size(in);
        if (base >= n) break;
        const bool valid = base + lane < n;
        const int i = valid ? queue_index(in, base + lane) : 0;
        Part<R> p;
        int tag = 0;
        uint32_t k0 = 0, k1 = 0, pos = 0;
        if (valid) qload(in, i, p, tag, k0, k1, pos);
        int sp = -1;
        float sr = 0.f;
        if (KIND == EV_SPLIT && valid) {
            sp = in.sp[i];
            sr = in.sr[i];
        }
        const int slot = tag >> 2;
        Env g;
        g.rng.init(((uint64_t)k1 << 32) | k0, seedw, pos);
        g.tally = tallies;
        g.nvox = nvox;
        g.slot = slot;
        g.pend_ir = -1;
        g.pend_e = 0.0;
        g.nout = 0;
        g.flags = 0;
        g.work = 0;
        g.tleft = ctl->tsteps;
        g.ncross = g.ndep = g.natom = 0;
        bool alive = false, defer = false;
        if (valid) {
            if constexpr (KIND == EV_PHOTON) {
                alive = photon_event(D, g, p);
            } else if constexpr (ELECTRON) {
                int r = electron_step<R, Env, KIND == EV_ELECTRON_DEFER>(D, g, p);
                alive = r != E_DEAD;
                defer = r == E_INTERACT;
            } else if constexpr (KIND == EV_SPLIT) {
                alive = split_event(D, g, p, sp, sr);
            } else {
                electron_interact(D, g, p);
                alive = true;
            }
            g.flush();
        }
        if constexpr (Env::kBuffered) {
            const uint64_t key = g.rng.key();
            k0 = (uint32_t)key;
            k1 = (uint32_t)(key >> 32);
        }
        const float esplit = ctl->esplit;
        int emitted = KIND == EV_ELECTRON_DEFER
                          ? emit<MAXOUT, true, R>(D, outP, outE, alive, p, g, slot, k0, k1, esplit, sp, sr, &qi, defer)
                          : emit<MAXOUT, false, R>(D, outP, outE, alive, p, g, slot, k0, k1, esplit, sp, sr);
        if (sd) add_live(sd->live, nbmax, valid ? slot : 0, valid ? emitted - 1 : 0, full);
        report_flags(ctl, g.flags, full);
        if (STATS) {
            c_ev += valid;
            c_steps += g.work;
            c_cross += g.ncross;
            c_dep += g.ndep;
            c_atom += g.natom;
        }
    }
    if (!STATS) return;
    if (KIND != EV_INTERACT) report_count(&ctl->st_events[ks], c_ev, full);
    report_count(&ctl->st_steps[ks], c_steps, full);
    report_count(&ctl->st_cross[ks], c_cross, full);
    report_count(&ctl->st_dep[ks], c_dep, full);
    report_count(&ctl->st_atom[ks], c_atom, full);
}

// Photon events of the queued photons.  `live` (may be null) receives the
// change of each serving request's live-particle count.
template <typename R>
__global__ void __launch_bounds__(EV_MAX_BLOCK) k_photon_step(DevData<R> D, QueueT<R> in, QueueT<R> outP,
                                                     QueueT<R> outE, double *tallies, long nvox, Ctl *ctl,
                                                     uint32_t seedw, ServeDev *sd, int nbmax, QueueT<R> qi) {
    transport_events<EV_PHOTON, R>(D, in, outP, outE, tallies, nvox, ctl, seedw, sd, nbmax, qi);
}

// Photon events of a splitting engine (nsplit > 1): one sub-photon each.
__global__ void __launch_bounds__(EV_MAX_BLOCK) k_photon_split_step(DevData<float> D, Queue in, Queue outP,
                                                           Queue outE, double *tallies, long nvox, Ctl *ctl,
                                                           uint32_t seedw, ServeDev *sd, int nbmax, Queue qi) {
    transport_events<EV_SPLIT>(D, in, outP, outE, tallies, nvox, ctl, seedw, sd, nbmax, qi);
}

// Electron/positron events of the queued charged particles: at most the
// cycle's budget of tstep-loop iterations each, then the particle is
// re-queued.  The step is latency bound; the occupancy it is compiled for
// (electron_minb) trades resident warps against spilled local frames.
template <bool DEFER, typename R = float, bool STATS = true>
__global__ void __launch_bounds__(EV_MAX_BLOCK, electron_minb<R>())
    k_electron_step(DevData<R> D, QueueT<R> in, QueueT<R> outP, QueueT<R> outE, double *tallies, long nvox, Ctl *ctl,
                    uint32_t seedw, ServeDev *sd, int nbmax, QueueT<R> qi) {
    transport_events<DEFER ? EV_ELECTRON_DEFER : EV_ELECTRON, R, STATS>(D, in, outP, outE, tallies, nvox, ctl, seedw, sd,
                                                                  nbmax, qi);
}

// The electron kernel of the engine: interactions in a kernel of their own
// (D.defer_interact) or in place.
template <typename R = float>
static TransportKernelT<R> electron_kernel(const omc_engine *e) {
    if (!e->d32.d.defer_interact) return k_electron_step<false, R>;
    return e->opt.profile ? k_electron_step<true, R> : k_electron_step<true, R, false>;
}

// Discrete interactions of the electrons the electron kernel left at their
// interaction sites (D.defer_interact): the samplers run in a kernel of
// their own, so the transport kernel's code stays small.
template <typename R = float>
__global__ void __launch_bounds__(EV_MAX_BLOCK) k_electron_interact(DevData<R> D, QueueT<R> in, QueueT<R> outP,
                                                           QueueT<R> outE, double *tallies, long nvox, Ctl *ctl,
                                                           uint32_t seedw, ServeDev *sd, int nbmax, QueueT<R> qi) {
    transport_events<EV_INTERACT, R>(D, in, outP, outE, tallies, nvox, ctl, seedw, sd, nbmax, qi);
}

// ------------------------------------------------------------ drain
// Once every history is injected and few particles remain, transport
// cycles launch mostly idle kernels whose duration is the latency of their
// longest events, and each particle waits a whole cycle between events.
// The drain runs the remaining particles to the end of their sub-histories
// in one launch instead.  Every particle keeps its own random stream and its
// secondaries get the keys emit() gives them, and interactions are sampled
// in place (the same draws as the interaction kernel), so the dose is the
// one the cycles would have produced, up to the summation order of the FP64
// tallies.
//
// A task is a particle with everything it gives rise to; a lane runs one
// task at a time, its secondaries on a local stack.  Electrons run one
// tstep-loop iteration at a time (budgets do not change trajectories), so
// that the lanes of a warp meet again soon.  A lane's electron step costs the
// instructions of every branch that any lane of its warp takes (a warp of one
// particle takes 4.3 us a step where nothing else runs), so the particles
// are spread over all resident warps, and a warp that has run out of work is
// given another's oldest pending particle, or one that a crowded warp has in
// hand, through a pool in global memory: the launch ends with the longest
// track, not with the longest sub-history.
//
// The warps of an SM are bound by the instructions they fetch: fifteen
// warps of one particle each took 50 us an iteration where three took 15
// and one 11.5 (a miss of the instruction cache is served every 23 cycles
// or so).  So the one block of an SM runs its iterations, and the
// transport, interactions and photons of an iteration, in step: its warps
// share what they fetch.  37 k particles on the slab phantom, ms a launch:
// one particle a thread in order 20.0; spread, donating, numbers from shared
// memory 16.5; blocks of 256 in step 16.0; of 512, in step by phase 14.8.
//
// The pool needs no lock: a warp without work draws a ticket (drain_head);
// tickets below the number of queued particles are those, the others wait
// for the pool entry of their number to be marked ready, or for the end.
// A lane donates only while tickets outnumber entries (compare and swap), so
// an entry has a taker at once; one that a full stack puts there waits for the
// next warp without work.  The launch is over when as many tasks are
// done as were made.  Lanes wait only when no particle is left unclaimed, so
// blocks that are not resident yet hold nobody up, and the wait has a limit:
// a block that finds nothing while no task ends anywhere gives up (ERR_DRAIN),
// and as its tickets may be given more, the run fails.
// SPLIT: photons are split rays (nsplit > 1) whose state (next sub-photon,
// survivor, offset) rides along with them, as in the photon queues.
constexpr int DRAIN_STACK = 48;
// One block of 512 per SM: up to 128 registers, which keep the step's state
// out of memory.
constexpr int DRAIN_BLOCK = 512;
// The ring of a drain lane, filled by the warp before a turn where few lanes
// are at work: a lone lane spent 23 % of its step in the generator, one block
// of four numbers after the other.  A turn draws some 45 numbers.  Water 1e4
// 4.02 -> 3.65 ms, slab 1e6 24.1 -> 23.3; rings of 64 gave the same, with
// less L1 left (18 MV on 200^3: 75.3 for 73.1 ms), helping up to 4 lanes a warp less.
constexpr int DRAIN_RING = 32;
constexpr int DRAIN_HELPED = 8;
constexpr size_t DRAIN_SHARED = sizeof(RingStore<DRAIN_BLOCK, DRAIN_RING>);
constexpr int DRAIN_TSTEPS = 1;               // tstep-loop iterations a turn
constexpr int DRAIN_POOL = 1 << 18;           // donations per launch; beyond them lanes keep their work
constexpr int DRAIN_POLLS = 1 << 24;          // looks of an idle block (1 us each) while no task ends before it gives up

template <typename R>
struct DrainPart {
    Part<R> p;
    uint32_t k0, k1, pos;
    int sp;       // splitting state (-1: not yet split)
    float sr;
};

__device__ __forceinline__ int ld_volatile(const int *p) { return *(const volatile int *)p; }

// The environment of a sampler run on copies: g's stream, with nothing
// pending, and back into g with what the sampler did.
template <typename Env, typename Host>
__device__ __forceinline__ void sampler_env(Env &h, const Host &g) {
    h.rng.init(g.rng.key(), g.rng.seedw, g.rng.position());
    h.tally = g.tally;
    h.nvox = g.nvox;
    h.slot = g.slot;
    h.pend_ir = g.pend_ir;
    h.pend_e = g.pend_e;
    h.nout = 0;
    h.flags = 0;
    h.work = g.work;
    h.tleft = 0;
    h.ncross = h.ndep = h.natom = 0;
}
template <int MAXOUT, typename Host, typename Env>
__device__ __forceinline__ void sampled(Host &g, const Env &h) {
    if constexpr (Host::kBuffered) g.rng.seek(h.rng.position());
    else g.rng = h.rng;
    g.pend_ir = h.pend_ir;
    g.pend_e = h.pend_e;
    g.nout = h.nout;
#pragma unroll
    for (int k = 0; k < MAXOUT; k++) {
        g.out[k] = h.out[k];
        g.out_pos[k] = h.out_pos[k];
    }
    g.flags |= h.flags;
    g.work = h.work;
    g.ncross += h.ncross;
    g.ndep += h.ndep;
    g.natom += h.natom;
}

// An electron's turn in the drain, out of line and by value, as a photon's
// is: its registers are then its own, not the drain's (inlined, the served
// load took 10 % longer).
template <typename R, typename Rng, bool STATS>
struct ElectronEventOut {
    Part<R> p, q;
    Rng rng;
    int pend_ir;
    double pend_e;
    uint32_t qpos;
    int r, nq, work, ncross, ndep, natom;
    unsigned flags;
};
template <typename R, typename Rng, bool STATS>
__device__ __noinline__ ElectronEventOut<R, Rng, STATS> electron_event_outline(const DevData<R> &D, Part<R> p, Rng rng,
                                                                               double *tally, long nvox, int slot,
                                                                               int pend_ir, double pend_e) {
    EvEnv<1, R, Rng, STATS> g;
    g.rng = rng;
    g.tally = tally;
    g.nvox = nvox;
    g.slot = slot;
    g.pend_ir = pend_ir;
    g.pend_e = pend_e;
    g.nout = 0;
    g.flags = 0;
    g.work = 0;
    g.tleft = DRAIN_TSTEPS;
    g.ncross = g.ndep = g.natom = 0;
    ElectronEventOut<R, Rng, STATS> o;
    o.r = electron_step<R, EvEnv<1, R, Rng, STATS>, true>(D, g, p);
    o.p = p;
    o.q = g.out[0];
    o.qpos = g.out_pos[0];
    o.nq = g.nout;
    o.rng = g.rng;
    o.pend_ir = g.pend_ir;
    o.pend_e = g.pend_e;
    o.work = g.work;
    o.ncross = g.ncross;
    o.ndep = g.ndep;
    o.natom = g.natom;
    o.flags = g.flags;
    return o;
}

// STATS (profiled runs): count, and record the largest sub-history a lane ran.
template <bool SPLIT, bool STATS = false>
__global__ void __launch_bounds__(DRAIN_BLOCK, 1)
    k_drain(DevData<float> D, Queue qP, Queue qE, Queue pool, int *ready, double *tallies, long nvox, Ctl *ctl,
            uint32_t seedw, int polls) {
    constexpr int MAXOUT = SPLIT ? EV_MAXOUT_SPLIT : EV_MAXOUT;
    using R = float;
    using Rng = RingStream<DRAIN_BLOCK, DRAIN_RING>;
    using Env = EvEnv<MAXOUT, R, Rng, STATS>;
    const unsigned full = 0xffffffffu;
    const int np = queue_size(qP), ne = queue_size(qE);
    const int n = np + ne;
    const int pool_cap = min(DRAIN_POOL, pool.cap);
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (DRAIN_BLOCK / 32);
    const bool takes = lane < (n + warps - 1) / warps;
    DrainPart<R> st[DRAIN_STACK];   // the task's pending particles
    int depth = 0;
    Part<R> p;                      // the particle in hand
    p.iq = 0;
    int sp = -1;
    float sr = 0.f;
    bool busy = false, alone = false;
    int ticket = -1;
    Env g;
    g.tally = tallies;
    g.nvox = nvox;
    unsigned c_ev[2] = {0, 0}, c_steps[2] = {0, 0}, c_cross[2] = {0, 0}, c_dep[2] = {0, 0}, c_atom = 0;
    int x_ev = 0, x_chain = 0, x_steps = 0;   // this task: events, events of its first particle, steps
    int first_at = 0;                         // where the first particle is: stack entry, -1 in hand, -2 gone
    // the oldest pending particle into pool entry k
    auto give = [&](int k) {
        const DrainPart<R> &e = st[0];
        qstore(pool, k, e.p, g.slot, e.k0, e.k1, e.pos, e.sp, e.sr);
        depth--;
        for (int i = 0; i < depth; i++) st[i] = st[i + 1];
        first_at = first_at == 0 ? -2 : (first_at > 0 ? first_at - 1 : first_at);
        __threadfence();
        *(volatile int *)&ready[k] = 1;
    };
    int idle = 0, seen = -1;                  // thread 0: looks since a task ended, tasks done then
    for (;;) {
        // the warps of a block take their iterations, and the phases of an
        // iteration, together, so that they share the instructions they fetch
        const bool block_busy = __syncthreads_or(busy);
        if (!busy && ticket < 0 && takes && ((lane == 0 && alone) || ld_volatile(&ctl->drain_head) < n))
            ticket = atomicAdd(&ctl->drain_head, 1);
        if (!busy && ticket >= 0) {
            const int k = ticket - n;
            int tag = 0;
            uint32_t k0 = 0, k1 = 0, pos = 0;
            if (k < 0) {
                const QueueT<R> &q = ticket < np ? qP : qE;
                const int qi = queue_index(q, ticket < np ? ticket : ticket - np);
                qload(q, qi, p, tag, k0, k1, pos);
                sp = (SPLIT && q.sp) ? q.sp[qi] : -1;
                sr = (SPLIT && q.sr) ? q.sr[qi] : 0.f;
                busy = true;
            } else if (k < pool_cap && ld_volatile(&ready[k])) {
                __threadfence();
                qload<true>(pool, k, p, tag, k0, k1, pos);
                sp = SPLIT ? __ldcg(&pool.sp[k]) : -1;
                sr = SPLIT ? __ldcg(&pool.sr[k]) : 0.f;
                busy = true;
            }
            if (busy) {
                ticket = -1;
                g.slot = tag >> 2;
                g.rng.init(((uint64_t)k1 << 32) | k0, seedw, pos);
                g.pend_ir = -1;
                g.pend_e = 0.0;
                g.flags = 0;
                g.natom = 0;
                x_ev = x_chain = x_steps = 0;
                first_at = -1;
            }
        }
        alone = !__any_sync(full, busy);
        if (!block_busy) {
            // nothing in hand in this block: over, or wait for a donation.
            // Tasks done are read before tasks made: when they agree nobody
            // is left who could make more.
            int over = 0;
            if (threadIdx.x == 0) {
                const int done = ld_volatile(&ctl->drain_done);
                __threadfence();
                over = done >= n + min(ld_volatile(&ctl->drain_tail), pool_cap);
                idle = done == seen ? idle + 1 : 0;
                seen = done;
                if (!over && idle > polls) {
                    // its tickets may still be given particles: the run fails
                    atomicOr(&ctl->flags, (unsigned)ERR_DRAIN);
                    over = 1;
                }
            }
            if (__syncthreads_or(over)) break;
            if (alone) __nanosleep(1000);
        } else {
            idle = 0;
        }
        {
            // few lanes at work: the others fill their rings
            const unsigned charged = __ballot_sync(full, busy && p.iq != 0);
            if (charged && __popc(charged) <= DRAIN_HELPED) {
                g.rng.seedw = seedw;
                g.rng.assist(charged);
            }
        }
        const uint64_t pkey = g.rng.key();
        g.nout = 0;
        g.work = 0;
        g.ncross = g.ndep = 0;
        const int kind = p.iq == 0 ? 0 : 1;
        bool alive = false;
        int r = E_DEAD;
        if (busy && kind == 1) {
            const ElectronEventOut<R, Rng, STATS> o = electron_event_outline<R, Rng, STATS>(
                D, p, g.rng, tallies, nvox, g.slot, g.pend_ir, g.pend_e);
            r = o.r;
            p = o.p;
            g.rng = o.rng;
            g.pend_ir = o.pend_ir;
            g.pend_e = o.pend_e;
            g.flags |= o.flags;
            g.work = o.work;
            g.ncross = o.ncross;
            g.ndep = o.ndep;
            g.natom += o.natom;
            if (o.nq) g.push_at(o.q, o.qpos);
            alive = r != E_DEAD;
        }
        __syncthreads();
        if (r == E_INTERACT) {
            // the samplers run out of line on copies, so that the lane's
            // own particle and environment stay in registers
            EvEnv<MAXOUT, R> h;
            Part<R> q = p;
            sampler_env(h, g);
            electron_interact(D, h, q);
            p = q;
            sampled<MAXOUT>(g, h);
        }
        __syncthreads();
        if (!busy) continue;
        if (kind == 0) {
            EvEnv<MAXOUT, R> h;
            sampler_env(h, g);
            if constexpr (SPLIT) {
                Part<R> q = p;
                int hsp = sp;
                float hsr = sr;
                alive = split_event(D, h, q, hsp, hsr);
                sp = hsp;
                sr = hsr;
                p = q;
            } else {
                alive = photon_event(D, h, p);
            }
            sampled<MAXOUT>(g, h);
        }
        if (STATS) {
            c_ev[kind]++;
            c_steps[kind] += g.work;
            c_cross[kind] += g.ncross;
            c_dep[kind] += g.ndep;
            x_chain += first_at == -1;
            x_steps += g.work;
        }
        x_ev++;
        if (alive && !(p.e == p.e && p.x == p.x && p.u == p.u)) {
            g.flags |= ERR_NAN;
            alive = false;
        }
        if (alive && p.iq == 0 && p.wt == R(0)) alive = false;
        if (!alive && first_at == -1) first_at = -2;
        // children first: the parent waits on the stack, which then holds
        // one particle a generation (split rays: a few)
        for (int k = 0; k < g.nout; k++) {
            const Part<R> &s2 = g.out[k];
            if (!(s2.e == s2.e && s2.x == s2.x && s2.u == s2.u)) {
                g.flags |= ERR_NAN;
                continue;
            }
            if (s2.iq == 0 && s2.wt == R(0)) continue;
            const uint64_t ck = mix64(pkey * 0x9E3779B97F4A7C15ull + ((uint64_t)g.out_pos[k] << 1) + 1u +
                                      ((uint64_t)k << 40));
            if (alive) {
                if (depth >= DRAIN_STACK) {
                    // a full stack hands its oldest particle over, asked or
                    // not (deep cascades of split rays)
                    const int k2 = atomicAdd(&ctl->drain_tail, 1);
                    if (k2 >= pool_cap) {
                        g.flags |= ERR_STACK;
                        continue;
                    }
                    give(k2);
                }
                const uint64_t key = g.rng.key();
                st[depth].p = p;
                st[depth].k0 = (uint32_t)key;
                st[depth].k1 = (uint32_t)(key >> 32);
                st[depth].pos = g.rng.position();
                st[depth].sp = sp;
                st[depth].sr = sr;
                if (first_at == -1) first_at = depth;
                depth++;
            }
            p = s2;
            g.rng.init(ck, seedw);
            sp = -1;
            sr = 0.f;
            alive = true;
        }
        if (x_ev > (1 << 22)) {
            g.flags |= ERR_LOOP;
            alive = false;
            depth = 0;
        }
        if (!alive && depth > 0) {
            depth--;
            p = st[depth].p;
            g.rng.init(((uint64_t)st[depth].k1 << 32) | st[depth].k0, seedw, st[depth].pos);
            sp = st[depth].sp;
            sr = st[depth].sr;
            if (first_at == depth) first_at = -1;
            alive = true;
        }
        // warps without work wait for some: the oldest pending particle of a
        // lane, which has the most of its track left, or, where the warp has
        // other lanes at work, the particle in hand becomes a task of its own
        const unsigned working = __activemask();
        if (depth > 0 || (alive && lane != __ffs(working) - 1)) {
            const int tail = ld_volatile(&ctl->drain_tail);
            if (tail < pool_cap && ld_volatile(&ctl->drain_head) > n + tail &&
                atomicCAS(&ctl->drain_tail, tail, tail + 1) == tail) {
                if (depth > 0) {
                    give(tail);
                } else {
                    const uint64_t key = g.rng.key();
                    qstore(pool, tail, p, g.slot, (uint32_t)key, (uint32_t)(key >> 32), g.rng.position(), sp, sr);
                    alive = false;
                    __threadfence();
                    *(volatile int *)&ready[tail] = 1;
                }
            }
        }
        if (!alive) {
            g.flush();
            if (STATS) c_atom += g.natom;     // tally atomics of the whole task
            if (g.flags) atomicOr(&ctl->flags, g.flags);
            busy = false;
            if (STATS) {
                atomicMax(&ctl->drain_max_events, x_ev);
                atomicMax(&ctl->drain_max_chain, x_chain);
                atomicMax(&ctl->drain_max_steps, x_steps);
            }
            __threadfence();
            atomicAdd(&ctl->drain_done, 1);
        }
    }
    if (!STATS) return;
    __syncwarp();
    for (int k = 0; k < 2; k++) {
        report_count(&ctl->st_events[k], c_ev[k], full);
        report_count(&ctl->st_steps[k], c_steps[k], full);
        report_count(&ctl->st_cross[k], c_cross[k], full);
        report_count(&ctl->st_dep[k], c_dep[k], full);
    }
    report_count(&ctl->st_atom[1], c_atom, full);
}

// The FP64 event form's drain: one thread per queued particle in order, with
// its secondaries on the local stack.  FP64 rounding is the compiler's choice
// kernel by kernel, and the accuracy study's results rest on this one's.
constexpr int DRAIN64_BLOCK = 128;
template <typename R = double>
__global__ void __launch_bounds__(DRAIN64_BLOCK, 4) k_drain64(DevData<R> D, QueueT<R> qP, QueueT<R> qE, double *tallies,
                                                          long nvox, Ctl *ctl, uint32_t seedw) {
    constexpr int MAXOUT = EV_MAXOUT;
    const int np = queue_size(qP), ne = queue_size(qE);
    const int n = np + ne;
    DrainPart<R> st[DRAIN_STACK];
    unsigned flags = 0;
    unsigned long long c_ev[2] = {0, 0}, c_steps[2] = {0, 0}, c_cross[2] = {0, 0}, c_dep[2] = {0, 0},
                       c_atom[2] = {0, 0};
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const QueueT<R> &q = t < np ? qP : qE;
        int tag = 0;
        const int qi = queue_index(q, t < np ? t : t - np);
        qload(q, qi, st[0].p, tag, st[0].k0, st[0].k1, st[0].pos);
        EvEnv<MAXOUT, R> g;
        g.tally = tallies;
        g.nvox = nvox;
        g.slot = tag >> 2;
        g.pend_ir = -1;
        g.pend_e = 0.0;
        g.flags = 0;
        g.natom = 0;
        int top = 0;
        for (int guard = 0; top >= 0; guard++) {
            if (guard > (1 << 22)) {
                g.flags |= ERR_LOOP;
                break;
            }
            DrainPart<R> &e = st[top];
            Part<R> p = e.p;
            const uint64_t pkey = ((uint64_t)e.k1 << 32) | e.k0;
            g.rng.init(pkey, seedw, e.pos);
            g.nout = 0;
            g.work = 0;
            g.tleft = 1 << 30;
            g.ncross = g.ndep = 0;
            const int kind = p.iq == 0 ? 0 : 1;
            bool alive;
            if (kind == 1) alive = electron_step<R, EvEnv<MAXOUT, R>, false>(D, g, p) == E_ALIVE;
            else alive = photon_event(D, g, p);
            c_ev[kind]++;
            c_steps[kind] += g.work;
            c_cross[kind] += g.ncross;
            c_dep[kind] += g.ndep;
            if (alive && !(p.e == p.e && p.x == p.x && p.u == p.u)) {
                g.flags |= ERR_NAN;
                alive = false;
            }
            if (alive && p.iq == 0 && p.wt == R(0)) alive = false;
            if (alive) {
                e.p = p;
                e.pos = g.rng.position();
            } else {
                top--;
            }
            for (int k = 0; k < g.nout; k++) {
                const Part<R> &s2 = g.out[k];
                if (!(s2.e == s2.e && s2.x == s2.x && s2.u == s2.u)) {
                    g.flags |= ERR_NAN;
                    continue;
                }
                if (s2.iq == 0 && s2.wt == R(0)) continue;
                if (top + 1 >= DRAIN_STACK) {
                    g.flags |= ERR_STACK;
                    continue;
                }
                uint64_t ck = mix64(pkey * 0x9E3779B97F4A7C15ull + ((uint64_t)g.out_pos[k] << 1) + 1u +
                                    ((uint64_t)k << 40));
                top++;
                st[top].p = s2;
                st[top].k0 = (uint32_t)ck;
                st[top].k1 = (uint32_t)(ck >> 32);
                st[top].pos = 0;
            }
        }
        g.flush();
        c_atom[1] += g.natom;     // tally atomics of the whole sub-history
        flags |= g.flags;
    }
    if (flags) atomicOr(&ctl->flags, flags);
    for (int k = 0; k < 2; k++) {
        if (c_ev[k]) atomicAdd(&ctl->st_events[k], c_ev[k]);
        if (c_steps[k]) atomicAdd(&ctl->st_steps[k], c_steps[k]);
        if (c_cross[k]) atomicAdd(&ctl->st_cross[k], c_cross[k]);
        if (c_dep[k]) atomicAdd(&ctl->st_dep[k], c_dep[k]);
        if (c_atom[k]) atomicAdd(&ctl->st_atom[k], c_atom[k]);
    }
}

template <typename R = float>
__global__ void k_source(DevData<R> D, BeamSrc<R> S, QueueT<R> qP, QueueT<R> qE, Ctl *ctl, long long nper,
                         uint64_t seed, uint32_t seedw) {
    int n = ctl->inject;
    long long base = ctl->hist_base;
    double es = 0;
    unsigned flags = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        unsigned active = __activemask();
        long long h = base + i;
        SrcEnv<R> g;
        uint64_t key = mix64(seed ^ (uint64_t)h * 0x9E3779B97F4A7C15ull);
        g.rng.init(key, seedw);
        R ein;
        Part<R> p = beam_primary(D, S, g, ein);
        es += ein;
        int slot = (int)(h / nper);
        int ip = warp_append(qP, p.iq == 0, false, active, flags);
        int ie = warp_append(qE, p.iq != 0, ctl->esplit > 0.f && p.e > (R)ctl->esplit, active, flags);
        if (ip >= 0) qstore(qP, ip, p, slot, (uint32_t)key, (uint32_t)(key >> 32), g.rng.position());
        if (ie >= 0) qstore(qE, ie, p, slot, (uint32_t)key, (uint32_t)(key >> 32), g.rng.position());
    }
    for (int o = 16; o > 0; o >>= 1) es += __shfl_down_sync(0xffffffffu, es, o);
    if ((threadIdx.x & 31) == 0 && es != 0.0) atomicAdd(&ctl->src_energy, es);
    unsigned active = __activemask();
    report_flags(ctl, flags, active);
}

// Electron budget of a cycle whose electron queue holds nE particles on a
// GPU with `lanes` resident threads: the base budget while the queue fills
// the GPU, multiplied by up to `boost` as it drains (the drain tail then
// takes few cycles; a lane's events of any length give the same result).
__device__ __forceinline__ void plan_budget(Ctl *ctl, long long nE, const PlanCfg &c) {
    long long me = 1;
    if (c.boost > 1 && nE < c.lanes) {
        me = c.lanes / (nE > 0 ? nE : 1);
        me = me > c.boost ? c.boost : me;
    }
    ctl->tsteps = (int)(c.tsteps * me);
    ctl->esplit = c.esplit;
    ctl->fetch[0] = 0;
    ctl->fetch[1] = 0;
    ctl->fetch[2] = 0;
    ctl->cnt_int = 0;
    ctl->cnt_int_hi = 0;
}

// Particles in the cycle's input queues; an overflow of either (the two
// ends met) is flagged.  The output queues (the previous cycle's inputs,
// all consumed) are emptied.
__device__ __forceinline__ void plan_queues(Ctl *ctl, int iph, int iel, int cap, long long &np, long long &ne) {
    np = (long long)ctl->cnt[iph] + ctl->cnt_hi[iph];
    ne = (long long)ctl->cnt[iel] + ctl->cnt_hi[iel];
    if (np > cap || ne > cap) ctl->flags |= ERR_QUEUE;
    np = np > cap ? cap : np;
    ne = ne > cap ? cap : ne;
    ctl->cnt[iph ^ 2] = 0;
    ctl->cnt[iel ^ 2] = 0;
    ctl->cnt_hi[iph ^ 2] = 0;
    ctl->cnt_hi[iel ^ 2] = 0;
}

// Histories to inject this cycle: keep `target` particles in flight (a
// photon of a splitting engine counts nsplit times).  Also
// sets the cycle's electron budget and empties the output queues (the
// previous cycle's inputs, all consumed).
__global__ void k_plan(Ctl *ctl, int iph, int iel, PlanCfg c) {
    long long np, ne;
    plan_queues(ctl, iph, iel, c.cap, np, ne);
    long long rem = ctl->hist_total - ctl->hist_next;
    long long inj = (c.target - (np * c.pweight + ne)) / c.pweight;
    if (inj < 0) inj = 0;
    if (inj > rem) inj = rem;
    long long room = (long long)c.cap - (np > ne ? np : ne);
    if (inj > room) inj = room > 0 ? room : 0;
    ctl->inject = (int)inj;
    ctl->hist_base = ctl->hist_next;
    ctl->hist_next += inj;
    plan_budget(ctl, ne, c);
}

// ------------------------------------------------------------------ host
// The event state of precision R: the FP32 form's or the FP64 form's.
template <typename R>
EventStateT<R> *&state_of(omc_engine *e);
template <>
EventStateT<float> *&state_of<float>(omc_engine *e) {
    return e->ev;
}
template <>
EventStateT<double> *&state_of<double>(omc_engine *e) {
    return e->ev64;
}
template <typename R>
const EventStateT<R> &state(const omc_engine *e) {
    return *state_of<R>(const_cast<omc_engine *>(e));
}

// Tables and flags the event kernels of precision R run with.  The FP64
// event form uses the FP64 tables with the event form's options (re-drawn
// interaction distance, deferred interactions, delta tracking) instead of
// the plain form's.
template <typename R>
DevData<R> event_data(const omc_engine *e);
template <>
DevData<float> event_data<float>(const omc_engine *e) {
    return e->d32.d;
}
template <>
DevData<double> event_data<double>(const omc_engine *e) {
    DevData<double> d = e->d64.d;
    d.chsteps = e->d32.d.chsteps;
    d.defer_interact = e->d32.d.defer_interact;
    d.woodcock = d.uniform && e->d32.d.woodcock ? 1 : 0;
    d.nsplit = 1;
    return d;
}

template <typename R>
static int alloc_queue(omc_engine *e, DBuf &b, QueueT<R> &q, int cap, int *count, int *count_hi) {
    // pos and dir: 4 values of R each; id: 16 bytes; ctr: 4 bytes (every
    // array starts on a 16-byte boundary for any cap)
    const size_t v4 = (size_t)cap * 4 * sizeof(R), per = (size_t)cap * 4;
    int rc = b.alloc(2 * v4 + 5 * per);
    if (rc) return set_err(e, rc, "event queue allocation failed");
    char *p = (char *)b.p;
    q.pos = (typename QVec<R>::T *)p;
    q.dir = (typename QVec<R>::T *)(p + v4);
    q.id = (uint4 *)(p + 2 * v4);
    q.ctr = (uint32_t *)(p + 2 * v4 + 4 * per);
    q.count = count;
    q.count_hi = count_hi;
    q.cap = cap;
    q.sp = nullptr;
    q.sr = nullptr;
    return OMC_OK;
}

// The photon kernel of the engine: split photons when nsplit > 1 (FP32
// form only).
template <typename R = float>
static TransportKernelT<R> photon_kernel(const omc_engine *e);
template <>
TransportKernelT<float> photon_kernel<float>(const omc_engine *e) {
    return e->d32.d.nsplit > 1 ? k_photon_split_step : k_photon_step<float>;
}
template <>
TransportKernelT<double> photon_kernel<double>(const omc_engine *) {
    return k_photon_step<double>;
}

// Resident blocks per SM of the transport kernels -> one-wave grids.
template <typename R>
static void size_grids(omc_engine *e, EventStateT<R> &S) {
    int bp = 0, be = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bp, photon_kernel<R>(e), S.block, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&be, electron_kernel<R>(e), S.block, 0);
    S.grid_p = e->sm_count * std::max(1, bp);
    S.grid_e = e->sm_count * std::max(1, be);
    int bi = 0, bd = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bi, k_electron_interact<R>, S.block, 0);
    S.grid_i = e->sm_count * std::max(1, bi);
    if constexpr (sizeof(R) == 4) {
        for (auto k : {k_drain<false, false>, k_drain<false, true>, k_drain<true, false>, k_drain<true, true>})
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DRAIN_SHARED);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bd, k_drain<false, false>, DRAIN_BLOCK, DRAIN_SHARED);
        S.drain_lanes = e->sm_count * std::max(1, bd) * DRAIN_BLOCK;
    } else {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bd, k_drain64<double>, DRAIN64_BLOCK, 0);
        S.drain_lanes = e->sm_count * std::max(1, bd) * DRAIN64_BLOCK;
    }
    S.lanes = S.grid_e * S.block;
}

// The interaction queue, allocated when the engine first needs it.
template <typename R>
static int event_interact_queue_t(omc_engine *e) {
    EventStateT<R> &S = *state_of<R>(e);
    if (!e->d32.d.defer_interact || S.int_buf.p) return OMC_OK;
    return alloc_queue(e, S.int_buf, S.qi, S.cap, &S.ctl_d->cnt_int, &S.ctl_d->cnt_int_hi);
}
int event_interact_queue(omc_engine *e) { return event_interact_queue_t<float>(e); }

// Electron budget of an event: tstep-loop iterations, of electron_chsteps
// condensed-history steps each, while the queue fills the GPU.  Lanes of a
// warp that go on together do similar work, but every event costs a round
// trip through the queue.  FP32: 1 / 2 / 3 iterations 100.3 / 98.4 / 108.1 ms
// on the slab beam (1e7 histories), 103.8 / 94.4 / 92.9 ms on the 200^3-class
// 18 MV beam (1e6); a server whose queues stay full (343 columns of 1.5e5
// histories) 62.9 / 65.9 M hist/s.  Splitting engines run one: their electron
// queues are full for most of a run, and the longer events of a warp cost
// more there than the round trips (1 / 2 iterations: 58.3 / 76.0 ms at nsplit
// 20 on 69^3 water voxels, 23.9 / 25.3 at 20 on 67^3, 31.0 / 32.0 at 10 on a
// 84^3 CT; 32.0 / 31.7 on the slab phantom).
template <typename R>
static int default_tsteps(int nsplit) {
    return sizeof(R) == 4 && nsplit <= 1 ? 2 : 1;
}

template <typename R>
static int event_prepare_t(omc_engine *e) {
    EventStateT<R> *&sp = state_of<R>(e);
    if (sp && sp->ready) return OMC_OK;
    if (!sp) sp = new EventStateT<R>();
    EventStateT<R> &S = *sp;
    long cap = e->opt.queue_capacity > 0 ? e->opt.queue_capacity : (1L << 22);
    S.cap = (int)std::min(cap, (long)(1L << 30));
    // warps fetch work 32 particles at a time: whole warps per block, at
    // most the transport kernels' launch bound
    S.block = e->opt.block > 0 ? std::min(EV_MAX_BLOCK, (e->opt.block + 31) / 32 * 32) : 256;
    S.grid = e->sm_count * std::max(1, 2048 / S.block);
    size_grids(e, S);
    S.tsteps = e->opt.electron_tsteps > 0 ? e->opt.electron_tsteps : default_tsteps<R>(e->opt.nsplit);
    S.boost = e->opt.tail_boost > 0 ? e->opt.tail_boost : 32;
    S.inflight = e->opt.inflight > 0 ? e->opt.inflight : (1LL << 20);
    S.esplit = e->opt.electron_split > 0 ? e->opt.electron_split + D_RM : 0.0;
    int rc = S.ctl.alloc(sizeof(Ctl));
    if (rc) return set_err(e, rc, "control block allocation failed");
    S.ctl_d = S.ctl.template as<Ctl>();
    for (int i = 0; i < 4; i++)
        if ((rc = alloc_queue(e, S.buf[i], S.q[i], S.cap, &S.ctl_d->cnt[i], &S.ctl_d->cnt_hi[i]))) return rc;
    if (sizeof(R) == 4 && (rc = S.drain_ready.alloc(DRAIN_POOL * sizeof(int)))) return set_err(e, rc, "drain pool allocation failed");
    if (e->d32.d.nsplit > 1 && sizeof(R) == 4) {
        // splitting state of the two photon queues (A and B)
        for (int k = 0; k < 2; k++) {
            size_t per = (size_t)S.cap * 4;
            if ((rc = S.split_buf[k].alloc(per * 2))) return set_err(e, rc, "splitting state allocation failed");
            QueueT<R> &q = S.q[2 * k];
            q.sp = S.split_buf[k].template as<int>();
            q.sr = (float *)((char *)S.split_buf[k].p + per);
        }
    }
    if (cudaHostAlloc((void **)&S.snap, 2 * sizeof(Ctl), cudaHostAllocDefault) != cudaSuccess ||
        cudaEventCreateWithFlags(&S.snap_ev[0], cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&S.snap_ev[1], cudaEventDisableTiming) != cudaSuccess)
        return set_err(e, OMC_E_DEVICE, "control block snapshots");
    if (cudaStreamCreateWithFlags(&S.side, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&S.fork, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&S.join, cudaEventDisableTiming) != cudaSuccess)
        return set_err(e, OMC_E_DEVICE, "side stream creation failed");
    S.ready = true;
    return OMC_OK;
}
int event_prepare(omc_engine *e) { return event_prepare_t<float>(e); }

// The transport kernels of one cycle after its source kernel.  Profiled
// (`ev`): one after the other on the engine's stream, an event after each.
// Otherwise (captured into the cycle graphs) the photon kernel runs on the
// side stream beside the electron kernels: they read different input
// queues and append to the output queues, the tallies and the counters
// with atomics only.  Launched after the electron kernel, its blocks take
// the SMs that the electron kernel's last blocks leave (4-5 % faster on
// slab64; same dose).  The side stream joins the engine's stream before the
// next cycle.
template <typename R = float>
static void launch_transport(omc_engine *e, int iph, int iel, int oph, int oel, double *tallies, uint32_t seedw,
                             ServeDev *sd, int nbmax, cudaEvent_t *ev) {
    EventStateT<R> &S = *state_of<R>(e);
    const long nvox = e->ph.nvox();
    const DevData<R> D = event_data<R>(e);
    auto photons = [&](cudaStream_t st) {
        photon_kernel<R>(e)<<<S.grid_p, S.block, 0, st>>>(D, S.q[iph], S.q[oph], S.q[oel], tallies, nvox, S.ctl_d,
                                                          seedw, sd, nbmax, S.qi);
    };
    auto electrons = [&]() {
        electron_kernel<R>(e)<<<S.grid_e, S.block, 0, e->stream>>>(D, S.q[iel], S.q[oph], S.q[oel], tallies, nvox,
                                                                    S.ctl_d, seedw, sd, nbmax, S.qi);
        if (D.defer_interact)
            k_electron_interact<R><<<S.grid_i, S.block, 0, e->stream>>>(D, S.qi, S.q[oph], S.q[oel], tallies, nvox,
                                                                        S.ctl_d, seedw, sd, nbmax, S.qi);
    };
    if (ev || !S.side) {
        photons(e->stream);
        if (ev) cudaEventRecord(ev[3], e->stream);
        electrons();
        return;
    }
    cudaEventRecord(S.fork, e->stream);
    cudaStreamWaitEvent(S.side, S.fork, 0);
    electrons();
    photons(S.side);
    cudaEventRecord(S.join, S.side);
    cudaStreamWaitEvent(e->stream, S.join, 0);
}

// Event-form tuning parameters of an engine (values <= 0 keep the current
// one); the queues are not reallocated.
int event_set_params(omc_engine *e, int tsteps, int boost, long long inflight, int block, double split_kinetic) {
    if (tsteps > 0) e->opt.electron_tsteps = tsteps;
    if (boost > 0) e->opt.tail_boost = boost;
    if (inflight > 0) e->opt.inflight = inflight;
    if (split_kinetic >= 0) e->opt.electron_split = split_kinetic;
    if (block > 0) {
        if (block % 32 || block > EV_MAX_BLOCK)
            return set_err(e, OMC_E_ARG, "block must be a multiple of 32, at most 256");
        e->opt.block = block;
    }
    auto apply = [&](auto &S) {
        using R = decltype(S.q[0].pos->x);
        S.tsteps = e->opt.electron_tsteps > 0 ? e->opt.electron_tsteps : default_tsteps<R>(e->opt.nsplit);
        S.boost = e->opt.tail_boost > 0 ? e->opt.tail_boost : 32;
        S.inflight = e->opt.inflight > 0 ? e->opt.inflight : (1LL << 20);
        S.esplit = e->opt.electron_split > 0 ? e->opt.electron_split + D_RM : 0.0;
        S.block = e->opt.block > 0 ? std::min(EV_MAX_BLOCK, e->opt.block) : 256;
        S.grid = e->sm_count * std::max(1, 2048 / S.block);
        size_grids(e, S);
    };
    if (e->ev && e->ev->ready) apply(*e->ev);
    if (e->ev64 && e->ev64->ready) apply(*e->ev64);
    return OMC_OK;
}

template <typename R>
static PlanCfg plan_cfg_t(const omc_engine *e, long long target) {
    const EventStateT<R> &S = state<R>(e);
    PlanCfg c;
    c.target = target;
    c.cap = S.cap;
    c.lanes = S.lanes;
    c.boost = S.boost;
    c.tsteps = S.tsteps;
    c.esplit = (float)S.esplit;
    c.pweight = sizeof(R) == 4 ? std::max(1, e->d32.d.nsplit) : 1;
    return c;
}
PlanCfg plan_cfg(const omc_engine *e, long long target) { return plan_cfg_t<float>(e, target); }

void event_release(omc_engine *e) {
    delete e->ev;
    e->ev = nullptr;
    delete e->ev64;
    e->ev64 = nullptr;
}

// One transport cycle with input buffers `in` (0 = A, 1 = B).  With `ev`
// (profiling) the launches are sequential and an event is recorded before
// each and after the last.  source = false: a cycle after the last injection.
template <typename R = float>
static void launch_cycle(omc_engine *e, int in, const BeamSrc<R> &src, double *tallies, long nper, uint64_t seed,
                         long long target, cudaEvent_t *ev = nullptr, bool source = true) {
    EventStateT<R> &S = *state_of<R>(e);
    int iph = in == 0 ? 0 : 2, iel = iph + 1;
    int oph = in == 0 ? 2 : 0, oel = oph + 1;
    uint32_t seedw = (uint32_t)(seed >> 32);
    if (ev) cudaEventRecord(ev[0], e->stream);
    k_plan<<<1, 1, 0, e->stream>>>(S.ctl_d, iph, iel, plan_cfg_t<R>(e, target));
    if (ev) cudaEventRecord(ev[1], e->stream);
    if (source)
        k_source<R><<<S.grid, S.block, 0, e->stream>>>(event_data<R>(e), src, S.q[iph], S.q[iel], S.ctl_d, nper, seed,
                                                       seedw);
    if (ev) cudaEventRecord(ev[2], e->stream);
    launch_transport<R>(e, iph, iel, oph, oel, tallies, seedw, nullptr, 1, ev);
    if (ev) cudaEventRecord(ev[4], e->stream);
}

// Particles left in the queues at or below which the transport switches
// from cycles to the drain (0: never).  The drain spreads its particles over the GPU, so it takes
// over once a cycle is shorter than one wave of the electron kernel: one and
// a half times its resident threads (114 k; the slab beam of 1e6 histories
// took 26.1 / 25.4 / 25.0 / 25.0 / 25.2 ms from 38 / 75 / 110 / 200 / 300 k
// on); with photon splitting, whose rays a lane works off one sub-photon
// after the other, once them (water phantom, 124 k histories split in 20:
// 63.5 / 61.6 / 75.4 ms from 38 / 75 / 113 k on).  The FP64 form's runs one
// particle a thread: half of them.
template <typename R>
static long long drain_threshold_t(const omc_engine *e) {
    const EventStateT<R> &S = state<R>(e);
    if (e->opt.drain_particles < 0) return 0;
    if (e->opt.drain_particles > 0) return e->opt.drain_particles;
    if (sizeof(R) == 8) return S.drain_lanes / 2;
    return e->d32.d.nsplit > 1 ? S.drain_lanes : (long long)S.drain_lanes * 3 / 2;
}
long long drain_threshold(const omc_engine *e) { return drain_threshold_t<float>(e); }

// Cycles to wait with the drain after the last of `histories` is injected.  A
// cycle works off one sub-photon of a split ray, a drain lane all that are
// left of it one after the other: rays just injected go to the drain only if
// its warps hold their sub-photons at once, others once they have been worked
// off.  18 MeV photons in water, ms with and without the wait: 1000 histories
// split in 64 37 / 83, 3000 44 / 168, 3000 split in 20 30 / 60; 1000 split in 20,
// which need not wait, 31 (48 in cycles).
long split_cycles(const omc_engine *e, long long histories) {
    const int nsplit = e->d32.d.nsplit;
    return nsplit > 1 && histories * nsplit > state<float>(e).drain_lanes / 2 ? nsplit : 0;
}

// The drain over the queues `iph`/`iph + 1` holding `left` particles, on
// the streams of the cycles that filled them (seed word `seedw`); `stats`
// records its largest sub-history.
template <typename R = float>
static void launch_drain(omc_engine *e, int iph, long long left, double *tallies, uint32_t seedw,
                         bool stats = false) {
    EventStateT<R> &S = *state_of<R>(e);
    const DevData<R> D = event_data<R>(e);
    if constexpr (sizeof(R) == 8) {
        const long long g = std::max(1LL, std::min((left + DRAIN64_BLOCK - 1) / DRAIN64_BLOCK,
                                                   (long long)S.drain_lanes / DRAIN64_BLOCK * 4));
        k_drain64<double><<<(int)g, DRAIN64_BLOCK, 0, e->stream>>>(D, S.q[iph], S.q[iph + 1], tallies, e->ph.nvox(), S.ctl_d, seedw);
    } else {
        // a warp per particle, up to one wave of resident blocks
        const long long warps = DRAIN_BLOCK / 32;
        const long long g = std::max(1LL, std::min((left + warps - 1) / warps, (long long)S.drain_lanes / DRAIN_BLOCK));
        auto kd = D.nsplit > 1 ? (stats ? k_drain<true, true> : k_drain<true, false>)
                               : (stats ? k_drain<false, true> : k_drain<false, false>);
        // the pool: the photon output queue, empty between cycles, and its flags
        int *ready = S.drain_ready.template as<int>();
        cudaMemsetAsync(ready, 0, DRAIN_POOL * sizeof(int), e->stream);
        cudaMemsetAsync(&S.ctl_d->drain_head, 0, 3 * sizeof(int), e->stream);
        kd<<<(int)g, DRAIN_BLOCK, DRAIN_SHARED, e->stream>>>(D, S.q[iph], S.q[iph + 1], S.q[iph ^ 2], ready, tallies, e->ph.nvox(),
                                                  S.ctl_d, seedw, e->drain_polls > 0 ? e->drain_polls : DRAIN_POLLS);
    }
}

// Profiled transport: cycles launched one by one with events around each
// kernel; per-kernel device time accumulated into S.prof, one trace row per
// cycle.
static int run_profiled(omc_engine *e, const BeamSrc<float> &src, double *tallies, long nper, uint64_t seed,
                        long long target, Ctl &h, long &cycles) {
    EventState &S = *e->ev;
    for (auto &p : S.prof) p = KernelProfile();
    S.trace.clear();
    for (double &v : S.drain_stats) v = 0;
    cudaEvent_t ev[5];
    for (auto &x : ev) cudaEventCreate(&x);
    int rc = OMC_OK;
    cycles = 0;
    int cnt_in[2] = {0, 0};   // queue sizes the cycle starts with (before injection)
    long injected = 0;        // cycles up to the last injection
    for (;;) {
        int in = (int)(cycles & 1);
        launch_cycle(e, in, src, tallies, nper, seed, target, ev);
        cycles++;
        if ((rc = cuda_check(e, cudaEventSynchronize(ev[4]), "profiled cycle"))) break;
        float t[4];
        for (int k = 0; k < 4; k++) cudaEventElapsedTime(&t[k], ev[k], ev[k + 1]);
        cudaMemcpy(&h, S.ctl_d, sizeof(Ctl), cudaMemcpyDeviceToHost);
        int oph = in == 0 ? 2 : 0;
        if (h.inject > 0) injected = cycles;
        double row[6] = {(double)h.inject, (double)cnt_in[0] + h.inject, (double)cnt_in[1], t[1], t[2], t[3]};
        S.trace.insert(S.trace.end(), row, row + 6);
        cnt_in[0] = std::min(h.cnt[oph] + h.cnt_hi[oph], S.cap);
        cnt_in[1] = std::min(h.cnt[oph + 1] + h.cnt_hi[oph + 1], S.cap);
        S.prof[3].seconds += t[0] * 1e-3;
        S.prof[3].launches += 1;
        S.prof[0].seconds += t[1] * 1e-3;
        S.prof[0].launches += 1;
        S.prof[1].seconds += t[2] * 1e-3;
        S.prof[1].launches += 1;
        S.prof[2].seconds += t[3] * 1e-3;
        S.prof[2].launches += 1;
        if (h.hist_next >= h.hist_total && cnt_in[0] == 0 && cnt_in[1] == 0) break;
        if (h.flags & ERR_QUEUE) break;
        long long dthr = drain_threshold(e);
        if (dthr > 0 && h.hist_next >= h.hist_total && cnt_in[0] + cnt_in[1] <= dthr &&
            cycles - injected >= split_cycles(e, h.hist_total)) {
            cudaEventRecord(ev[0], e->stream);
            launch_drain(e, oph, (long long)cnt_in[0] + cnt_in[1], tallies, (uint32_t)(seed >> 32), true);
            cudaEventRecord(ev[1], e->stream);
            if ((rc = cuda_check(e, cudaEventSynchronize(ev[1]), "drain"))) break;
            float td = 0;
            cudaEventElapsedTime(&td, ev[0], ev[1]);
            double row2[6] = {0.0, (double)cnt_in[0], (double)cnt_in[1], 0.0, 0.0, (double)td};
            S.trace.insert(S.trace.end(), row2, row2 + 6);
            S.prof[2].seconds += td * 1e-3;
            S.prof[2].launches += 1;
            cudaMemcpy(&h, S.ctl_d, sizeof(Ctl), cudaMemcpyDeviceToHost);
            double ds[5] = {(double)td, (double)cnt_in[0] + cnt_in[1], (double)h.drain_max_events,
                            (double)h.drain_max_chain, (double)h.drain_max_steps};
            std::copy(ds, ds + 5, S.drain_stats);
            break;
        }
        if (cycles > 200000) {
            rc = set_err(e, OMC_E_DEVICE, "event transport did not drain");
            break;
        }
    }
    for (auto &x : ev) cudaEventDestroy(x);
    return rc;
}

template <typename R>
int event_run_beam(omc_engine *e, const omc_beam *b, long nper, int nbatch, uint64_t seed, double *sum, double *sum2,
                   double *src_energy, KernelStats &ks) {
    if (sizeof(R) == 8 && e->d32.d.nsplit > 1)
        return set_err(e, OMC_E_RANGE, "the FP64 event form has no photon splitting (nsplit > 1)");
    int rc = event_prepare_t<R>(e);
    if (!rc) rc = event_interact_queue_t<R>(e);
    if (rc) return rc;
    EventStateT<R> &S = *state_of<R>(e);
    long nvox = e->ph.nvox();
    DBuf &tal = e->run_tal, &cdf = e->run_cdf32;
    if ((rc = tal.reserve((size_t)nbatch * nvox * 8))) return set_err(e, rc, "batch tallies allocation failed");
    cudaMemsetAsync(tal.p, 0, (size_t)nbatch * nvox * 8, e->stream);
    int ncdf = b->energy.n;
    BeamSrc<R> src = beam_setup<R>(e, b);
    if (ncdf > 0) {
        std::vector<R> c(b->energy.cdf1, b->energy.cdf1 + ncdf);
        c.insert(c.end(), b->energy.cdf2, b->energy.cdf2 + ncdf);
        if ((rc = cdf.reserve(c.size() * sizeof(R)))) return set_err(e, rc, "alloc");
        cudaMemcpyAsync(cdf.p, c.data(), c.size() * sizeof(R), cudaMemcpyHostToDevice, e->stream);
        src.cdf1 = cdf.as<R>();
        src.cdf2 = cdf.as<R>() + ncdf;
    }
    Ctl c0{};
    c0.hist_total = (long long)nper * nbatch;
    cudaMemcpyAsync(S.ctl_d, &c0, sizeof(Ctl), cudaMemcpyHostToDevice, e->stream);
    long long target = std::min<long long>((long long)S.cap / 2, S.inflight);

    if (e->opt.profile && sizeof(R) == 4) {
        Ctl h{};
        long cycles = 0;
        cudaEvent_t t0, t1;
        cudaEventCreate(&t0);
        cudaEventCreate(&t1);
        cudaEventRecord(t0, e->stream);
        if constexpr (sizeof(R) == 4) rc = run_profiled(e, src, tal.as<double>(), nper, seed, target, h, cycles);
        if (!rc) rc = fold(e, tal.as<double>(), nbatch, sum, sum2, nvox, 1.0);
        cudaEventRecord(t1, e->stream);
        cudaEventSynchronize(t1);
        float ms = 0;
        cudaEventElapsedTime(&ms, t0, t1);
        cudaEventDestroy(t0);
        cudaEventDestroy(t1);
        ks.seconds = ms * 1e-3;
        ks.launches = cycles * (e->d32.d.defer_interact ? 5 : 4) + 1 + (drain_threshold(e) > 0 ? 1 : 0);
        ks.flags |= h.flags;
        for (int k = 0; k < 2; k++) {
            KernelProfile &P = S.prof[1 + k];
            P.particles = (double)h.st_events[k];
            P.steps = (double)h.st_steps[k];
            P.cross = (double)h.st_cross[k];
            P.dep = (double)h.st_dep[k];
            P.atom = (double)h.st_atom[k];
        }
        S.prof[0].particles = (double)h.hist_total;
        if (rc) return rc;
        cudaMemcpyAsync(src_energy, &S.ctl_d->src_energy, 8, cudaMemcpyDeviceToDevice, e->stream);
        return OMC_OK;
    }

    cudaEvent_t t0, t1;
    cudaEventCreate(&t0);
    cudaEventCreate(&t1);
    Ctl h{};
    long launches = 0;
    const uint32_t seedw = (uint32_t)(seed >> 32);
    const int cycle_launches = e->d32.d.defer_interact ? 5 : 4;
    const long long dthr = drain_threshold_t<R>(e);
    const int pweight = plan_cfg_t<R>(e, target).pweight;
    // A run whose histories the drain's warps hold at once goes to the drain
    // as it is (10^4 histories on the water phantom 8.4 -> 4.1 ms, 3 10^4
    // 8.9 -> 5.4, 10^5 no gain).
    const bool direct = sizeof(R) == 4 && pweight == 1 &&
                        c0.hist_total <= std::min({dthr, (long long)S.drain_lanes / 2, target});
    // two cycles (A -> B, B -> A) as one graph, and two without injection
    cudaGraph_t graph[2] = {nullptr, nullptr};
    cudaGraphExec_t exec[2] = {nullptr, nullptr};
    auto capture = [&](int k) {
        int r = cuda_check(e, cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal), "capture");
        if (r) return r;
        for (int in = 0; in < 2; in++)
            launch_cycle<R>(e, in, src, tal.as<double>(), nper, seed, target, nullptr, k == 0);
        if ((r = cuda_check(e, cudaStreamEndCapture(e->stream, &graph[k]), "end capture"))) return r;
        return cuda_check(e, cudaGraphInstantiate(&exec[k], graph[k], 0), "graph instantiate");
    };
    auto queued = [&](const Ctl &c) {   // a graph ends with a B -> A cycle: its outputs are queues A
        return (long long)std::min(c.cnt[0] + c.cnt_hi[0], S.cap) + std::min(c.cnt[1] + c.cnt_hi[1], S.cap);
    };
    cudaEventRecord(t0, e->stream);
    long long left = 0;   // particles for the drain, at most
    if (direct) {
        k_plan<<<1, 1, 0, e->stream>>>(S.ctl_d, 0, 1, plan_cfg_t<R>(e, target));
        k_source<R><<<S.grid, S.block, 0, e->stream>>>(event_data<R>(e), src, S.q[0], S.q[1], S.ctl_d, nper, seed,
                                                       seedw);
        launches += 2;
        left = c0.hist_total;
    } else if (!(rc = capture(0))) {
        // Checked after every graph where the end is near: from the start on
        // when one cycle injects all (with splitting, where the drain's lanes
        // hold all sub-photons: 10^3 histories split in 20 15.7 -> 11.1 ms).
        const long long few = pweight == 1 ? target : S.drain_lanes;
        int per_check = sizeof(R) == 4 && c0.hist_total * pweight <= few ? 1 : 4;
        for (long graphs = 0;;) {
            for (int k = 0; k < per_check; k++) cudaGraphLaunch(exec[0], e->stream);
            graphs += per_check;
            launches += per_check * 2 * cycle_launches;
            cudaMemcpyAsync(S.snap, S.ctl_d, sizeof(Ctl), cudaMemcpyDeviceToHost, e->stream);
            if ((rc = cuda_check(e, cudaStreamSynchronize(e->stream), "event transport"))) break;
            h = S.snap[0];
            left = queued(h);
            if ((h.hist_next >= h.hist_total && left == 0) || (h.flags & ERR_QUEUE)) break;
            if (dthr > 0 && h.hist_next >= h.hist_total) {
                if (sizeof(R) == 4 || left <= dthr) break;
                per_check = 1;
                continue;
            }
            // every cycle advances each queued particle by one event, so a run
            // needs (histories / injection rate) + (longest history) cycles
            if (graphs > 50000 + h.hist_total / 1000) {
                rc = set_err(e, OMC_E_DEVICE, "event transport did not drain");
                break;
            }
            per_check = std::min(per_check * 2, 64);
            if (sizeof(R) == 4 && h.hist_next < h.hist_total)
                per_check = (int)std::max(1.0, std::min<double>(per_check, 0.5 * graphs * (h.hist_total - h.hist_next) /
                                                                               std::max<long long>(h.hist_next, 1)));
        }
        // FP32, every history injected: cycles without the source kernel, the
        // next pair queued before the last one's state is looked at
        const long ripe = sizeof(R) == 4 ? split_cycles(e, c0.hist_total) : 0;
        if (sizeof(R) == 4 && !rc && dthr > 0 && left > 0 && (left > dthr || ripe > 0) && !(h.flags & ERR_QUEUE) &&
            !(rc = capture(1))) {
            for (long graphs = 0;; graphs++) {
                cudaGraphLaunch(exec[1], e->stream);
                launches += 2 * (cycle_launches - 1);
                const int k = graphs & 1;
                cudaMemcpyAsync(&S.snap[k], S.ctl_d, sizeof(Ctl), cudaMemcpyDeviceToHost, e->stream);
                cudaEventRecord(S.snap_ev[k], e->stream);
                if (graphs == 0) continue;
                if ((rc = cuda_check(e, cudaEventSynchronize(S.snap_ev[k ^ 1]), "event transport"))) break;
                h = S.snap[k ^ 1];
                left = queued(h);
                if (left == 0 || (left <= dthr && 2 * graphs >= ripe) || (h.flags & ERR_QUEUE)) break;
                if (graphs > 100000) {
                    rc = set_err(e, OMC_E_DEVICE, "event transport did not drain");
                    break;
                }
            }
        }
    }
    if (!rc && left > 0 && dthr > 0 && !(h.flags & ERR_QUEUE)) {
        launch_drain<R>(e, 0, left, tal.as<double>(), seedw);
        launches++;
    }
    // fold the batch tallies into the sums (accumEndep per batch)
    if (!rc) rc = fold(e, tal.as<double>(), nbatch, sum, sum2, nvox, 1.0);
    cudaEventRecord(t1, e->stream);
    // source energy, and the error flags of all that ran
    cudaMemcpyAsync(src_energy, &S.ctl_d->src_energy, 8, cudaMemcpyDeviceToDevice, e->stream);
    cudaMemcpyAsync(S.snap, S.ctl_d, sizeof(Ctl), cudaMemcpyDeviceToHost, e->stream);
    const int sync = cuda_check(e, cudaStreamSynchronize(e->stream), "event transport");
    if (!rc) rc = sync;
    if (!rc) {
        float ms = 0;
        cudaEventElapsedTime(&ms, t0, t1);
        ks.seconds = ms * 1e-3;
        ks.launches = launches + 1;
        ks.flags |= S.snap[0].flags;
    }
    for (int k = 0; k < 2; k++) {
        if (exec[k]) cudaGraphExecDestroy(exec[k]);
        if (graph[k]) cudaGraphDestroy(graph[k]);
    }
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    return rc;
}
template int event_run_beam<float>(omc_engine *, const omc_beam *, long, int, uint64_t, double *, double *, double *,
                                   KernelStats &);
template int event_run_beam<double>(omc_engine *, const omc_beam *, long, int, uint64_t, double *, double *, double *,
                                    KernelStats &);

// ============================================================== serving
// Inclusive prefix sum over the block (blockDim.x a multiple of 32, at most
// 1024) of one value per thread.
template <typename T>
__device__ __forceinline__ T block_inclusive_scan(T v, T *warp_tot) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        T t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) warp_tot[wid] = v;
    __syncthreads();
    if (wid == 0) {
        T w = lane < nw ? warp_tot[lane] : T(0);
        for (int o = 1; o < 32; o <<= 1) {
            T t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        if (lane < nw) warp_tot[lane] = w;
    }
    __syncthreads();
    if (wid > 0) v += warp_tot[wid - 1];
    __syncthreads();
    return v;
}

// Histories to inject this cycle across the admitted requests, first come
// first served, keeping `target` particles in flight.  One block of
// SERVE_MAX threads, one per position in the admission order: request k
// takes min(its remaining histories, room left after requests 0..k-1),
// found by a prefix sum of the remaining histories.
__global__ void __launch_bounds__(SERVE_MAX) k_serve_plan(ServeDev *sd, Ctl *ctl, int iph, int iel, PlanCfg c) {
    __shared__ long long s_room;
    __shared__ long long warp_ll[SERVE_MAX / 32];
    __shared__ int warp_i[SERVE_MAX / 32];
    const int cap = c.cap;
    if (threadIdx.x == 0) {
        long long np, ne;
        plan_queues(ctl, iph, iel, cap, np, ne);
        long long room = (c.target - (np * c.pweight + ne)) / c.pweight;
        long long qroom = (long long)cap - (np > ne ? np : ne);
        if (room > qroom) room = qroom;
        s_room = room;
        plan_budget(ctl, ne, c);
    }
    __syncthreads();
    const long long room = s_room;
    const int k = threadIdx.x;
    int slot = -1;
    long long rem = 0, next = 0;
    if (k < sd->norder) {
        slot = sd->order[k];
        const ServeReq &r = sd->req[slot];
        if (r.kind >= 0 && r.nhist > r.next) {
            rem = r.nhist - r.next;
            next = r.next;
        }
    }
    const long long before = block_inclusive_scan(rem, warp_ll) - rem;
    long long take = room - before;
    take = take < 0 ? 0 : (take > rem ? rem : take);
    const int planned = take > 0;
    const int pos = block_inclusive_scan(planned, warp_i) - planned;
    if (planned) {
        // every request before this one got all it asked for: `before` is
        // the injections planned ahead of it
        sd->plan_slot[pos] = slot;
        sd->plan_first[pos] = next;
        sd->plan_cum[pos] = (int)before;
        sd->req[slot].next = next + take;
    }
    // the last thread sees the totals
    if (k == blockDim.x - 1) {
        const long long total_rem = before + rem;
        const long long total = total_rem < room ? total_rem : (room > 0 ? room : 0);
        const int nplan = pos + planned;
        sd->plan_cum[nplan] = (int)total;
        sd->nplan = nplan;
        sd->inject_total = (int)total;
    }
}

// Primaries of the planned histories; each history's stream key is derived
// from its request's seed and its index within the request.
__global__ void k_serve_source(DevData<float> D, ServeDev *sd, Queue qP, Queue qE, Ctl *ctl, int nbmax,
                               uint32_t seedw) {
    int n = sd->inject_total, np = sd->nplan;
    unsigned flags = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        unsigned active = __activemask();
        int lo = 0, hi = np - 1;
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (sd->plan_cum[mid] <= i) lo = mid;
            else hi = mid - 1;
        }
        int s = sd->plan_slot[lo];
        const ServeReq &r = sd->req[s];
        long long local = sd->plan_first[lo] + (i - sd->plan_cum[lo]);
        uint64_t key = mix64(r.seed ^ (uint64_t)local * 0x9E3779B97F4A7C15ull);
        SrcEnv<float> g;
        g.rng.init(key, seedw);
        float ein;
        Part<float> p = r.kind == 0 ? beam_primary(D, sd->beam[s], g, ein) : beamlet_primary(D, sd->bl[s], r.bixel, g, ein);
        int slot = s * nbmax + (int)(local / r.nper);
        int ip = warp_append(qP, p.iq == 0, false, active, flags);
        int ie = warp_append(qE, p.iq != 0, ctl->esplit > 0.f && p.e > ctl->esplit, active, flags);
        if (ip >= 0) qstore(qP, ip, p, slot, (uint32_t)key, (uint32_t)(key >> 32), g.rng.position());
        if (ie >= 0) qstore(qE, ie, p, slot, (uint32_t)key, (uint32_t)(key >> 32), g.rng.position());
        add_live(sd->live, nbmax, slot, (ip >= 0) + (ie >= 0), active);
    }
    unsigned active = __activemask();
    report_flags(ctl, flags, active);
}

void serve_launch_cycle(omc_engine *e, int in, ServeDev *sd, double *tallies, int nbmax, long long target) {
    EventState &S = *e->ev;
    int iph = in == 0 ? 0 : 2, iel = iph + 1;
    int oph = in == 0 ? 2 : 0, oel = oph + 1;
    const uint32_t seedw = SERVE_SEEDW;
    k_serve_plan<<<1, SERVE_MAX, 0, e->stream>>>(sd, S.ctl_d, iph, iel, plan_cfg(e, target));
    k_serve_source<<<S.grid, S.block, 0, e->stream>>>(e->d32.d, sd, S.q[iph], S.q[iel], S.ctl_d, nbmax, seedw);
    launch_transport(e, iph, iel, oph, oel, tallies, seedw, sd, nbmax, nullptr);
}

// A serving cycle launched on its own with an event around each kernel
// (engines created with options.profile): the per-kernel device time is
// added to the engine's profile; the transport counters are those the
// control block has accumulated since the server was created.
int serve_profiled_cycle(omc_engine *e, int in, ServeDev *sd, double *tallies, int nbmax, long long target) {
    EventState &S = *e->ev;
    int iph = in == 0 ? 0 : 2, iel = iph + 1;
    int oph = in == 0 ? 2 : 0, oel = oph + 1;
    const uint32_t seedw = SERVE_SEEDW;
    cudaEvent_t ev[5];
    for (auto &x : ev) cudaEventCreate(&x);
    cudaEventRecord(ev[0], e->stream);
    k_serve_plan<<<1, SERVE_MAX, 0, e->stream>>>(sd, S.ctl_d, iph, iel, plan_cfg(e, target));
    cudaEventRecord(ev[1], e->stream);
    k_serve_source<<<S.grid, S.block, 0, e->stream>>>(e->d32.d, sd, S.q[iph], S.q[iel], S.ctl_d, nbmax, seedw);
    cudaEventRecord(ev[2], e->stream);
    launch_transport(e, iph, iel, oph, oel, tallies, seedw, sd, nbmax, ev);
    cudaEventRecord(ev[4], e->stream);
    int rc = cuda_check(e, cudaEventSynchronize(ev[4]), "profiled serving cycle");
    if (!rc) {
        float t[4];
        for (int k = 0; k < 4; k++) cudaEventElapsedTime(&t[k], ev[k], ev[k + 1]);
        const int map[4] = {3, 0, 1, 2};   // plan, source, photon, electron (+ interactions)
        for (int k = 0; k < 4; k++) {
            S.prof[map[k]].seconds += t[k] * 1e-3;
            S.prof[map[k]].launches += 1;
        }
        Ctl h{};
        cudaMemcpy(&h, S.ctl_d, sizeof(Ctl), cudaMemcpyDeviceToHost);
        for (int k = 0; k < 2; k++) {
            KernelProfile &P = S.prof[1 + k];
            P.particles = (double)h.st_events[k];
            P.steps = (double)h.st_steps[k];
            P.cross = (double)h.st_cross[k];
            P.dep = (double)h.st_dep[k];
            P.atom = (double)h.st_atom[k];
        }
    }
    for (auto &x : ev) cudaEventDestroy(x);
    return rc;
}

void serve_profile_reset(omc_engine *e) {
    for (auto &p : e->ev->prof) p = KernelProfile();
}

// The drain in serving: the particles left in queues A (where a graph of
// two cycles leaves them) run to the end on the serving streams; then the
// queues are emptied and every request's live count is zero.
void serve_drain(omc_engine *e, ServeDev *sd, long long left, double *tallies) {
    EventState &S = *e->ev;
    launch_drain(e, 0, left, tallies, SERVE_SEEDW, e->opt.profile != 0);
    cudaMemsetAsync(sd->live, 0, sizeof(sd->live), e->stream);
    cudaMemsetAsync(S.ctl_d->cnt, 0, 2 * sizeof(int), e->stream);
    cudaMemsetAsync(S.ctl_d->cnt_hi, 0, 2 * sizeof(int), e->stream);
}

}  // namespace omc
