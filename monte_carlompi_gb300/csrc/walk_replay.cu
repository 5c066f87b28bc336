// FP64 replay walk: the reference's arithmetic order, uniforms from the photon-indexed
// Philox replay stream.  Compiled with --fmad=false so every product and sum is rounded on
// its own, as NumPy does.
//
// Restates MonteCarlo.monte_carlo3D (monte_carloMPI/monte_carlo3D.py:1111-1490) with the draws
// of populate_pdfs (:905-1025) and initial_pdfs (:1027-1044), and the wavelength draw of
// MonteCarlo.run (:1515-1520): walk_replay_kernel the HG branch, walk_replay_pol_kernel the
// polarised branch of aspherical grains, one thread per photon (the rejection sampler of
// populate_pdfs, :922-1004, and the Stokes-vector update of monte_carlo3D, :1282-1342).
//
// What bounds the HG walk: an FP64 instruction takes a warp 64 cycles of its sub-core's FP64
// pipe, however many of its lanes are active and whether or not it waits for the one before.  A
// walk of one thread's own took about 170 of them per event, 5.6 us, and the longest walk of
// 10,000 photons has 25,000 events.  So the work is laid out across lanes and warps:
//  * a block of four warps holds up to sixteen photons and walks them in rounds of 32 steps (all of
//    one photon's, or two each of sixteen), its warps a round apart: the first draws the steps
//    (angles, optical path, path increment, absorption; none of them depends on where the photon
//    is), the second walks mu_z, which depends on mu_z alone, the third mu_x and mu_y, the fourth
//    depth and path, where a walk ends.  So a lone photon's step costs what the longest of the
//    three chains costs, mu_z's twelve FP64 instructions one after the other;
//  * in those chains every FP64 instruction takes its operands from another FP64 instruction or
//    from memory: a result that a select, a shuffle or a test takes first costs 110 to 290 cycles
//    on its way to the next instead of 66.  Directions about the vertical, which need one, are
//    walked again with it when the chain turns out to have met one;
//  * sqrt(1 - mu_z^2) and its reciprocal come from one Newton step and a residual correction
//    (Markstein, IBM J. Res. Dev. 34, 1990), six operations, and the two divisions by it take
//    three each (rounded.cuh).
// The draws assume that a step does nothing but scatter: a photon that ends, is reflected or is
// replaced sits out the two rounds under way.  Every value is the one-thread walk's, in
// its order of operations, every square root and quotient correctly rounded: the third warp looks
// at the residuals of all steps of a round side by side, and a step whose rounding they leave open (some
// five in a million) is walked again with sqrt() and /, its photon's draws ahead dropped as at an
// event.  10,000 photons of the reference's default run 14.4 to 16.3 ms without the look, 14.6 to 15.8
// with it; 100,000 of a thin layer, which fill the FP64 pipe, 1.00 and 1.09.
// 10,000 photons of the reference's default run: 193.7 ms on one thread each; 30.5 ms (0.94 us an
// event of the longest walk) with one warp drawing and one walking, four lanes a photon, each
// FP64 instruction serving all four through selects and shuffles; 16.0 ms now (0.47 us, 970
// cycles an event, of which mu_z's chain is 880).
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "mcw_internal.cuh"
#include "rounded.cuh"
#include "ssp_device.cuh"
#include "tally.cuh"

namespace mcw {

namespace {

__device__ double replay_uniform(uint64_t seed, uint32_t tag, uint64_t photon, uint64_t k) {
    uint4 x = philox10_seed(make_uint4((uint32_t)(k >> 1), tag, (uint32_t)photon,
                                       (uint32_t)(photon >> 32)), seed);
    uint64_t w = (k & 1) ? (((uint64_t)x.w << 32) | x.z) : (((uint64_t)x.y << 32) | x.x);
    return u01_f64(w);
}

// Photon wavelength [um]: sigma = FWHM / 2.355, Box-Muller normal from the
// wavelength stream, np.around(x, 2) = rint(x * 100) / 100.
__device__ double replay_wavelength(const DevConfig &c, uint64_t seed, uint64_t gid) {
    double u0 = replay_uniform(seed, kTagWvl, gid, 0);
    double u1 = replay_uniform(seed, kTagWvl, gid, 1);
    double z = sqrt(-2.0 * log(u0)) * cos(kTwoPi * u1);
    double x = c.wvl0 + c.scale * z;
    return rint(x * 100.0) / 100.0;
}

// Record and tallies of a photon that ended with `condition` (0: stopped early) after i steps.
template <bool kPol>
__device__ void finish_photon(const ReplayArgs &a, int64_t gid, int ci, int condition, int64_t i, double wvl_um,
                              double mux_0, double muy_0, double muz_0, double path_length, double snow_depth,
                              const double *st) {
    mcw_record64p r;
    r.condition = condition;
    r.n_scat = (int32_t)(i - 1);                                      // :1487
    r.wvn = 1. / wvl_um;                                              // :1468
    r.theta_n = acos(muz_0);                                          // :1469
    r.flags = 0;
    if (i == 1) r.phi_n = 0.;                                         // :1472-1485
    else if (mux_0 > 0 && muy_0 > 0) r.phi_n = atan(muy_0 / mux_0);
    else if (mux_0 < 0 && muy_0 > 0) r.phi_n = atan(muy_0 / mux_0) + kPi;
    else if (mux_0 < 0 && muy_0 < 0) r.phi_n = atan(muy_0 / mux_0) + kPi;
    else if (mux_0 > 0 && muy_0 < 0) r.phi_n = atan(muy_0 / mux_0) + kTwoPi;
    else { r.phi_n = __longlong_as_double(0x7ff8000000000000LL); r.flags = 1u; }
    r.path_length = path_length;
    r.snow_depth = snow_depth;
    r.config = (uint32_t)ci;
    if (a.records) {
        if (kPol) {
            r.stokes_q = st[1];
            r.stokes_u = st[2];
            r.stokes_v = st[3];
            static_cast<mcw_record64p *>(a.records)[gid] = r;
        } else {
            mcw_record64 &d = static_cast<mcw_record64 *>(a.records)[gid];
            d.condition = r.condition;
            d.n_scat = r.n_scat;
            d.wvn = r.wvn;
            d.theta_n = r.theta_n;
            d.phi_n = r.phi_n;
            d.path_length = r.path_length;
            d.snow_depth = r.snow_depth;
            d.config = r.config;
            d.flags = r.flags;
        }
    }
    if (a.tallies && condition > 0) {
        const unsigned long long wfx = (unsigned long long)llrint(r.wvn * 4294967296.0);
        float th = (float)r.theta_n, ph = (r.flags ? 0.f : (float)r.phi_n);
        tally_global(a.tallies + ci, condition, r.n_scat, wfx, th, ph);
    }
}

// ---------------------------------------------------------------- the HG walk

constexpr int kSlots = 16;                   // photons a block walks at once
constexpr uint64_t kMaxUniforms = 1ull << 33;    // of a photon's stream
constexpr uint32_t kRefl = 1u, kSurface = 2u, kBottom = 4u, kIso = 8u, kActive = 16u;

// A photon in flight (shared memory).
struct Slot {
    double mux, muy, muz, z, path;
    double hg_b, hg_c, hg_d, hg_e, hg_a;     // 1-g^2, 1-g, 2g, 1/(2g), 1+g^2
    double ext, rext;                        // ext_cff * rho_snw and its reciprocal
    double ssa_ice, ssa_imp, p_imp, tau, R;
    double wvl_um, depth;
    uint64_t rid, k;                         // stream id, next uniform
    int64_t gid;
    int64_t i;                               // steps walked
    int32_t ci, row;                         // config, ice-table row
    uint32_t flags;
    __device__ __forceinline__ bool lambertian() const { return (flags & (kRefl | kSurface)) != 0; }
};

// A finished photon waiting for its record.
struct Finished {
    double mux, muy, muz, path, wvl_um, depth;
    int64_t gid, i;
    int32_t ci, cond;
};

// 32 steps drawn ahead, S of each of n photons: entry rank * S + t is step t of photon `rank`.
// Each warp of the block adds its part, a round after the warp before it.
struct Ahead {
    double ct[32], st[32], cp[32], sp[32], dtau[32], inc[32];
    uint32_t fl[32];                         // 1 absorbed here, 2 by ice
    int32_t n, S, pole;                      // pole: a step about the vertical among them
    uint32_t uncertain;                      // XY: steps to be walked again (uncertain_steps)
    int32_t slot[kSlots], steps[kSlots], lamb[kSlots], first[kSlots], shift[kSlots];
    uint32_t gen[kSlots];                    // the slot's count of events that the draws assume
    uint64_t k0[kSlots];                     // the photon's stream before the steps
    double mzb[32], sq[32], h2[32], mz[32];  // Z: mu_z before, sqrt(1 - mu_z^2), 1 / that, mu_z after
    double x[32], y[32], z[32], path[32];    // XY and M: the state after the step
    double numx[32], quox[32], numy[32], quoy[32];   // XY: the quotients by sqrt(1 - mu_z^2) in them
};

struct ReplayBlock {
    Ahead ahead[3];
    Slot slots[kSlots], born[32];
    Finished fin[32];
    uint32_t gen[kSlots];                    // events of the slot's photons so far
    uint32_t drawn_gen[kSlots];              // producer: the count at its last draw,
    uint64_t next_k[kSlots];                 // and the stream after it
    double mz[kSlots];                       // Z: mu_z after its last steps
    int32_t stop;
};

__device__ __forceinline__ double from_bits(uint64_t b) { return __longlong_as_double((long long)b); }

// u01_f64 by its bits: 1.m - (1 - 2^-53), exact, one FP64 operation.
__device__ __forceinline__ double u01_bits(uint64_t w) {
    return from_bits(0x3ff0000000000000ull | (w >> 12)) - 0x1.fffffffffffffp-1;
}

__device__ __forceinline__ uint4 stream_block(uint64_t seed, uint64_t rid, uint64_t block) {
    return philox10_seed(make_uint4((uint32_t)block, kTagWalk, (uint32_t)rid, (uint32_t)(rid >> 32)), seed);
}

__device__ __forceinline__ uint64_t word(const uint4 x, bool second) {
    return second ? (((uint64_t)x.w << 32) | x.z) : (((uint64_t)x.y << 32) | x.x);
}

// Uniform k of a photon's stream.
__device__ __forceinline__ double uniform_at(uint64_t seed, uint64_t rid, uint64_t k) {
    return u01_bits(word(stream_block(seed, rid, k >> 1), k & 1));
}

// x > 0 and x < -t (t >= 0) by their bits, false for NaN: no FP64 operation.
__device__ __forceinline__ bool is_pos(double x) {
    const uint64_t b = to_bits(x);
    return b > 0 && b <= 0x7ff0000000000000ull;
}
__device__ __forceinline__ bool below_minus(double x, double t) {
    const uint64_t b = to_bits(x), m = b & 0x7fffffffffffffffull;
    return (b >> 63) && m > to_bits(t) && m <= 0x7ff0000000000000ull;
}
__device__ __forceinline__ bool is_nan(double x) { return (to_bits(x) & 0x7fffffffffffffffull) > 0x7ff0000000000000ull; }
__device__ __forceinline__ bool is_unit(double x) { return (to_bits(x) & 0x7fffffffffffffffull) == 0x3ff0000000000000ull; }

__device__ __forceinline__ double shfl_d(double x, int src) { return __shfl_sync(0xffffffffu, x, src); }

// The end of a step (:1390-1466) at depth z (z_prev before it): the path's exit correction, the
// bottom's reflectance draw (uniform *k, taken when drawn), the end condition (0: walking on, or
// reflected, kRefl set in *flags).
__device__ int step_end(const Slot &s, uint64_t seed, double &z, double z_prev, double dtau, double muz, double &path,
                        bool first, bool absorbed, bool ice, uint64_t *k, uint32_t *flags) {
    if (z > 0) {                                                      // :1390-1397
        path += -((z * dtau) / ((z - z_prev) * s.ext));
        return 1;
    }
    if (z < -s.tau) {                                                 // :1399-1459
        path += -(((z + s.tau) * dtau) / ((z - z_prev) * s.ext));
        const double corr = -(((z + s.tau) / (z_prev - z)) * dtau);
        z = z - (muz * corr);
        if (s.flags & kBottom) {
            const double u = uniform_at(seed, s.rid, *k);
            *k += 1;
            if (u <= s.R) {
                *flags |= kRefl;
                return 0;
            }
        }
        return first ? 3 : 2;
    }
    return absorbed ? (ice ? 4 : 5) : 0;                              // :1461-1466
}

// Photon gid at its birth and after its first step (:1215-1237: the direction is the beam's), into
// a slot; returns its end condition.
__device__ int replay_birth(const ReplayArgs &a, int64_t gid, Slot &out) {
    const int ci = find_config(a.prefix, a.n_cfg, gid);
    const DevConfig &c = a.cfgs[ci];
    Slot s;
    s.gid = gid;
    s.ci = ci;
    s.rid = c.rng_base + (uint64_t)(gid - c.offset);
    const double wvl = replay_wavelength(c, a.seed, s.rid);
    const Optics o = photon_optics(c, a.ice[c.ice_table], a.imp, wvl);
    const double g = o.g;
    s.flags = kActive | ((c.flags & kFlagLamSurface) ? kSurface : 0u) | ((c.flags & kFlagLamBottom) ? kBottom : 0u) |
              (g == 0 ? kIso : 0u);
    s.hg_b = 1 - g * g;
    s.hg_c = 1 - g;
    s.hg_d = 2 * g;
    s.hg_e = 1. / (2. * g);
    s.hg_a = 1 + g * g;
    s.ext = o.ext_cff_mss * c.rho_snw;                                // :1355-1356
    s.rext = 1.0 / s.ext;
    s.tau = c.tau_tot_d;
    s.R = c.R_d;
    s.ssa_ice = (s.flags & kSurface) ? s.R : o.ssa_ice;               // :1385-1387
    s.ssa_imp = (s.flags & kSurface) ? s.R : o.ssa_imp;
    s.p_imp = o.p_imp;
    s.wvl_um = o.wvl_um;
    s.depth = o.snow_depth;
    s.row = o.row;
    s.mux = c.mux0_d;                                                 // :1121-1124
    s.muy = 0;
    s.muz = c.muz0_d;
    s.i = 1;
    s.k = 3;
    const double dtau = (s.flags & kSurface) ? 0 : -log(uniform_at(a.seed, s.rid, 0));   // :1035-1038, :1227-1229
    const double ssa_rand = uniform_at(a.seed, s.rid, 1);
    const bool ice = uniform_at(a.seed, s.rid, 2) > s.p_imp;          // :1375-1383
    s.path = 0 + dtau / s.ext;                                        // :1372
    s.z = 0 + dtau * s.muz;                                           // :1352
    const int cond = step_end(s, a.seed, s.z, 0, dtau, s.muz, s.path, true, ssa_rand >= (ice ? s.ssa_ice : s.ssa_imp),
                              ice, &s.k, &s.flags);
    out = s;
    return cond;
}

// The photons that no block has claimed when the time is out, 32 a warp at a time.  Warp-collective.
template <bool kPol>
__device__ __noinline__ void leave_unwalked(const ReplayArgs &a, int lane) {
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(a.work, 32ull);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= (unsigned long long)a.total) return;
        if (base + lane < (unsigned long long)a.total) {
            Slot s;
            const int cond = replay_birth(a, (int64_t)(base + lane), s);
            finish_photon<kPol>(a, s.gid, s.ci, cond, s.i, s.wvl_um, s.mux, s.muy, s.muz, s.path, s.depth,
                                kPol ? a.cfgs[s.ci].stokes0 : nullptr);
        }
    }
}

// The producer's round: the next steps of the block's photons into `next`, assuming that those
// drawn before and not yet walked end in nothing.
__device__ void draw_ahead(const ReplayArgs &a, ReplayBlock &B, Ahead &next, int lane) {
    const unsigned act = __ballot_sync(0xffffffffu, lane < kSlots && (B.slots[lane & (kSlots - 1)].flags & kActive));
    const int n = __popc(act);
    const int S = n <= 1 ? 32 : 1 << (5 - (32 - __clz(n - 1)));       // 32 / n, a power of two
    const int rank = lane / S, t = lane % S;
    const bool mine = rank < n;
    const int si = mine ? __fns(act, 0, rank + 1) : 0;
    const uint32_t gen = B.gen[si];
    const bool first = B.drawn_gen[si] != gen;
    Slot s = B.slots[si];
    if (!first) s.k = B.next_k[si];
    const bool lamb = first ? s.lambertian() : (s.flags & kSurface) != 0;
    __syncwarp();
    // a Lambertian direction first (:1238-1250): its photon's lanes test pairs of uniforms past the
    // step's five, and the first that passes is taken
    int shift = 0;
    double ct_l = 1.0;
    bool look = mine && lamb;
    const unsigned group = S == 32 ? 0xffffffffu : ((1u << S) - 1u) << (rank * S);
    for (int round = 0; __any_sync(0xffffffffu, look); ++round) {
        bool pass = false;
        double c = 1.0;
        const int j = round * S + t;
        if (look) {
            const double theta = 0 + (kPi / 2 - 0) * uniform_at(a.seed, s.rid, s.k + 5 + 2 * (uint64_t)j);
            const double r1 = uniform_at(a.seed, s.rid, s.k + 6 + 2 * (uint64_t)j);
            double sn;
            sincos(theta, &sn, &c);
            pass = r1 < 2 * sn * c;
            if (round >= 4096) pass = true;                           // no stream needs as many
        }
        const unsigned hit = __ballot_sync(0xffffffffu, pass) & group;
        const int src = hit ? __ffs(hit) - 1 : lane;
        const double cs = shfl_d(c, src);
        if (look && hit) {
            ct_l = cs;
            shift = 2 * (round * S + (src - rank * S) + 1);
            look = false;
        }
    }
    if (mine) {
        const int steps = (s.flags & kSurface) ? 1 : S;               // on a surface every step's stream shifts
        const uint64_t k = s.k + 5 * (uint64_t)t + (t > 0 ? shift : 0);
        const uint4 x0 = stream_block(a.seed, s.rid, k >> 1), x1 = stream_block(a.seed, s.rid, (k >> 1) + 1),
                    x2 = stream_block(a.seed, s.rid, (k >> 1) + 2);
        const bool odd = k & 1;
        const double u0 = u01_bits(word(x0, odd)), u1 = u01_bits(odd ? word(x1, false) : word(x0, true)),
                     u2 = u01_bits(word(x1, odd)), u3 = u01_bits(odd ? word(x2, false) : word(x1, true)),
                     u4 = u01_bits(word(x2, odd));
        double sp, cp;
        sincos(u1 * kTwoPi, &sp, &cp);
        const double dtau = -log(u2);
        // the step's cosine, sine (sqrt(1 - ct^2) as the reference writes it) and path, their roundings
        // looked at together
        const bool given = t == 0 && lamb, iso = (s.flags & kIso) != 0;
        const double den = s.hg_c + s.hg_d * u0, q = quotient_res(s.hg_b, den, rcp_res(den));
        double ct = given ? ct_l : (iso ? 1 - 2 * u0 : s.hg_e * (s.hg_a - q * q));   // Henyey_Greenstein2 (:790-800)
        double h, inc = quotient_res(dtau, s.ext, s.rext);            // :1372
        const double x = 1 - ct * ct;
        double st = sqrt_res(x, h);
        if (!((given | iso | quotient_sure(q, s.hg_b, den)) & sqrt_sure(st, x) & quotient_sure(inc, dtau, s.ext))) {
            if (!(given | iso)) {
                const double e = s.hg_b / den;
                ct = s.hg_e * (s.hg_a - e * e);
            }
            st = sqrt(1 - ct * ct);
            inc = dtau / s.ext;
        }
        const bool ice = u4 > s.p_imp;                                // :1375-1383
        next.ct[lane] = ct;
        next.st[lane] = st;
        next.cp[lane] = cp;
        next.sp[lane] = sp;
        next.dtau[lane] = dtau;
        next.inc[lane] = inc;
        next.fl[lane] = (u3 >= (ice ? s.ssa_ice : s.ssa_imp) ? 1u : 0u) | (ice ? 2u : 0u);
        if (t == 0) {
            next.slot[rank] = si;
            next.steps[rank] = steps;
            next.lamb[rank] = lamb ? 1 : 0;
            next.first[rank] = first ? 1 : 0;
            next.shift[rank] = shift;
            next.gen[rank] = gen;
            next.k0[rank] = s.k;
            const uint64_t k1 = s.k + 5 * (uint64_t)steps + shift;
            B.drawn_gen[si] = gen;
            B.next_k[si] = k1;
        }
    }
    if (lane == 0) {
        next.n = n;
        next.S = S;
    }
}

// Whether rank r's steps are those that its slot's photon takes: nothing has happened to it since.
__device__ __forceinline__ bool holds(const ReplayBlock &B, const Ahead &A, int r) {
    return r < A.n && A.gen[r] == B.gen[A.slot[r]];
}

// Z: the chain of mu_z over the steps drawn in the round before, a lane per photon:
// mu_z' = mu_z ct - sqrt(1 - mu_z^2) st cp (:1277), which depends on mu_z alone.  kPole: with the
// directions about the vertical (:1262-1269): mu_z = +-1, or a Lambertian direction.
template <bool kPole>
__device__ __forceinline__ double z_chain(Ahead &A, double mz, const int base, const int steps, const int S) {
    double ct = A.ct[base], st = A.st[base], cp = A.cp[base];
    for (int it = 0; it < S; ++it) {
        const int e = base + it, e1 = base + min(it + 1, S - 1);
        const double ct1 = A.ct[e1], st1 = A.st[e1], cp1 = A.cp[e1];
        const double u = mz * ct;
        double h1;
        const double sq = sqrt_res(1.0 - mz * mz, h1);
        double nz = (sq * -st) * cp + u;
        if (kPole && is_unit(mz)) nz = to_bits(mz) >> 63 ? -ct : ct;
        if (it < steps) {
            A.mzb[e] = mz;
            A.sq[e] = sq;
            A.h2[e] = doubled(h1);
            A.mz[e] = nz;
        }
        mz = nz;
        ct = ct1, st = st1, cp = cp1;
    }
    return mz;
}

// A test of mu_z inside the chain costs 210 cycles a step beside its 880.  So it is walked without
// one: past the vertical it is all NaN (0 times infinity), and then walked again with it.
__device__ void walk_z(ReplayBlock &B, Ahead &A, int lane) {
    const bool held = lane < kSlots && holds(B, A, lane & (kSlots - 1));
    if (!__any_sync(0xffffffffu, held)) return;
    const int S = A.S, base = held ? lane * S : 0, steps = held ? A.steps[lane] : 0, si = held ? A.slot[lane] : 0;
    const double mz0 = !held ? 0.5 : (A.lamb[lane] ? 1.0 : (A.first[lane] ? B.slots[si].muz : B.mz[si]));
    double mz = mz0;
    bool pole = __any_sync(0xffffffffu, is_unit(mz0));
    if (!pole) {
        mz = z_chain<false>(A, mz0, base, steps, S);
        // (a photon on a surface, of fewer steps, starts every one from the vertical)
        pole = __any_sync(0xffffffffu, held && steps == S && is_nan(mz));
    }
    if (pole) mz = z_chain<true>(A, mz0, base, steps, S);
    if (held) B.mz[si] = mz;
    if (lane == 0) A.pole = pole ? 1 : 0;
}

// XY: mu_x and mu_y over the steps that Z walked in the round before, two lanes a photon:
// mu_x' = st (mu_x mu_z cp - mu_y sp) / sqrt(1 - mu_z^2) + mu_x ct, mu_y' alike (:1270-1276).
template <bool kPole>
__device__ __forceinline__ void xy_chain(Ahead &A, double va, double vb, const int base, const int steps, const int S,
                                         const bool isX, const int lane) {
    double *out = isX ? A.x : A.y, *nums = isX ? A.numx : A.numy, *quos = isX ? A.quox : A.quoy;
    double mzb = A.mzb[base], ct = A.ct[base], st = A.st[base], cp = A.cp[base], sp = A.sp[base], sq = A.sq[base],
           h2 = A.h2[base];
    for (int it = 0; it < S; ++it) {
        const int e = base + it, e1 = base + min(it + 1, S - 1);
        const double mzb1 = A.mzb[e1], ct1 = A.ct[e1], st1 = A.st[e1], cp1 = A.cp[e1], sp1 = A.sp[e1], sq1 = A.sq[e1],
                     h21 = A.h2[e1];
        const double p = va * mzb, w = va * ct;
        const double num = st * (p * cp + vb * (isX ? -sp : sp));
        const double q = quotient_res(num, sq, h2);
        double nv = q + w;
        if (kPole) {
            const double v = st * (isX ? cp : sp);
            if (is_unit(mzb)) nv = isX || !(to_bits(mzb) >> 63) ? v : -v;
        }
        if (it < steps) {
            out[e] = nv;
            nums[e] = num;
            quos[e] = q;
        }
        va = nv;
        vb = shfl_d(nv, lane ^ 1);
        mzb = mzb1, ct = ct1, st = st1, cp = cp1, sp = sp1, sq = sq1, h2 = h21;
    }
}

// The steps of A, a bit each, whose square root or quotients the chains may have rounded otherwise than
// sqrt() and / do (rounded.cuh).  A lane a step: six FP64 instructions for all of them, where a test in
// the chains would take as many a step; in XY's warp, whose chain is shorter than Z's (between the
// rounds, where the other warps wait for the states' commit, 14.4 -> 16.3 ms of 10,000 photons).
__device__ unsigned uncertain_steps(const Ahead &A, int lane) {
    const double mz = A.mzb[lane], sq = A.sq[lane];
    // (about the vertical there is neither; past it, by rounding, all is NaN either way)
    const bool sure = is_unit(mz) || is_nan(sq) ||
                      (sqrt_certain(sq, 1.0 - mz * mz) && quotient_certain(A.quox[lane], A.numx[lane], sq) &&
                       quotient_certain(A.quoy[lane], A.numy[lane], sq));
    return __ballot_sync(0xffffffffu, !sure);
}

__device__ void walk_xy(ReplayBlock &B, Ahead &A, int lane) {
    const int rk = lane >> 1;
    const bool isX = !(lane & 1), held = holds(B, A, rk);
    if (!__any_sync(0xffffffffu, held)) return;
    const int S = A.S, base = held ? rk * S : 0, steps = held ? A.steps[rk] : 0;
    const Slot &slot = B.slots[held ? A.slot[rk] : 0];
    const bool lamb = !held || A.lamb[rk];
    const double va = lamb ? 0.0 : (isX ? slot.mux : slot.muy), vb = lamb ? 0.0 : (isX ? slot.muy : slot.mux);
    if (A.pole) xy_chain<true>(A, va, vb, base, steps, S, isX, lane);
    else xy_chain<false>(A, va, vb, base, steps, S, isX, lane);
    __syncwarp();
    const unsigned uncertain = uncertain_steps(A, lane);
    if (lane == 0) A.uncertain = uncertain;
}

// M: depth and path over the same steps, two lanes a photon, and the first step with an end
// condition (:1390-1466).  Returns, on the depth's lane, the steps walked, negative if the last is
// such a step.
__device__ int walk_m(ReplayBlock &B, Ahead &A, int lane) {
    const int rk = lane >> 1;
    const bool isz = !(lane & 1), held = holds(B, A, rk);
    if (!__any_sync(0xffffffffu, held)) return 0;
    A.z[lane] = A.dtau[lane] * A.mz[lane];
    __syncwarp();
    const int S = A.S, base = held ? rk * S : 0, steps = held ? A.steps[rk] : 0;
    const Slot &slot = B.slots[held ? A.slot[rk] : 0];
    const double tau = slot.tau;
    double acc = isz ? slot.z : slot.path;
    const double *in = isz ? A.z : A.inc;
    double *out = isz ? A.z : A.path;
    int done = steps;
    bool event = false;
    double d = in[base];
    uint32_t fl = A.fl[base];
    for (int it = 0; it < S; ++it) {
        const int e = base + it, e1 = base + min(it + 1, S - 1);
        const double d1 = in[e1];
        const uint32_t fl1 = A.fl[e1];
        acc = acc + d;
        if (it < steps) {
            out[e] = acc;
            if (!event && (is_pos(acc) || below_minus(acc, tau) || (fl & 1u))) {
                event = true;
                done = it + 1;
            }
        }
        d = d1, fl = fl1;
    }
    return event ? -done : done;
}

// Step e, the `t`-th of its photon's, again with sqrt() and /, from the state before it.
__device__ __noinline__ void step_again(const Slot &slot, Ahead &A, int e, int t) {
    const double mux = t > 0 ? A.x[e - 1] : slot.mux, muy = t > 0 ? A.y[e - 1] : slot.muy, muz = A.mzb[e];
    const double ct = A.ct[e], st = A.st[e], cp = A.cp[e], sp = A.sp[e];
    const double sq = sqrt(1 - muz * muz);
    A.x[e] = (st * (mux * muz * cp - muy * sp)) / sq + mux * ct;
    A.y[e] = (st * (muy * muz * cp + mux * sp)) / sq + muy * ct;
    A.mz[e] = -sq * st * cp + muz * ct;
    A.z[e] = (t > 0 ? A.z[e - 1] : slot.z) + A.dtau[e] * A.mz[e];
    A.path[e] = (t > 0 ? A.path[e - 1] : slot.path) + A.inc[e];
}

// The photons' states after the steps that XY and M walked: lane `rank` its photon's.  `walked`:
// walk_m's result for it.  At the first uncertain step, walked again, the photon's draws ahead end as
// at an event.  Returns its end condition (-1: out of its stream).
__device__ int commit(const ReplayArgs &a, ReplayBlock &B, Ahead &A, int rank, int walked) {
    bool event = walked < 0;
    int done = event ? -walked : walked;
    const int si = A.slot[rank];
    Slot &slot = B.slots[si];
    const unsigned mine = (A.uncertain >> (rank * A.S)) & (0xffffffffu >> (32 - done));
    if (mine) {
        event = true;
        done = __ffs(mine);
        step_again(slot, A, rank * A.S + done - 1, done - 1);
    }
    const int e = rank * A.S + done - 1;
    uint32_t flags = slot.flags & ~kRefl;
    uint64_t k = A.k0[rank] + 5 * (uint64_t)done + A.shift[rank];
    double z = A.z[e], path = A.path[e];
    const double zp = done > 1 ? A.z[e - 1] : slot.z, mz = A.mz[e];
    slot.mux = A.x[e];
    slot.muy = A.y[e];
    slot.muz = mz;
    slot.i += done;
    int cond = 0;
    if (event) {
        const uint32_t f = A.fl[e];
        cond = step_end(slot, a.seed, z, zp, A.dtau[e], mz, path, false, f & 1u, f & 2u, &k, &flags);
    }
    if (k > kMaxUniforms) {
        atomicOr(a.status, kStatusStream);
        if (cond == 0) cond = -1;
    }
    if (event || cond) B.gen[si] += 1;
    slot.z = z;
    slot.path = path;
    slot.k = k;
    slot.flags = flags;
    return cond;
}

__global__ void __launch_bounds__(128, 4) walk_replay_kernel(const ReplayArgs a) {
    __shared__ ReplayBlock B;
    const int lane = threadIdx.x & 31;
    // the warps' parts, turned by a warp from one block of an SM to the next, so that each of its
    // four FP64 pipes gets one of each part
    enum { kDraw, kZ, kXY, kM };
    const int part = ((int)(threadIdx.x >> 5) + (int)((4ull * blockIdx.x) / gridDim.x)) & 3;
    const unsigned lt_mask = (1u << lane) - 1u;
    if (threadIdx.x < kSlots) {
        B.slots[threadIdx.x].flags = 0;
        B.gen[threadIdx.x] = 1;
        B.drawn_gen[threadIdx.x] = 0;
    }
    if (threadIdx.x < 3) {
        B.ahead[threadIdx.x].n = 0;
        B.ahead[threadIdx.x].S = 32;
    }
    if (threadIdx.x == 0) B.stop = 0;
    __syncthreads();
    bool exhausted = false;
    int n_born = 0, n_fin = 0, walked = 0;
    const unsigned long long t0 = global_ns();
    auto flush = [&]() {                             // the queued records, one per lane
        if (lane < n_fin) {
            const Finished &f = B.fin[lane];
            finish_photon<false>(a, f.gid, f.ci, f.cond, f.i, f.wvl_um, f.mux, f.muy, f.muz, f.path, f.depth, nullptr);
        }
        n_fin = 0;
        __syncwarp();
    };
    auto queue = [&](bool ended, const Slot &s, int cond) {
        const unsigned m = __ballot_sync(0xffffffffu, ended);
        if (ended) B.fin[n_fin + __popc(m & lt_mask)] =
            Finished{s.mux, s.muy, s.muz, s.path, s.wvl_um, s.depth, s.gid, s.i, s.ci, cond};
        n_fin += __popc(m);
        __syncwarp();
    };
    int drawn = 0;                                   // the buffer drawn into this round
    for (uint32_t round = 0;; ++round) {
        Ahead &now = B.ahead[drawn], &before = B.ahead[drawn == 0 ? 2 : drawn - 1],
              &last = B.ahead[drawn == 2 ? 0 : drawn + 1];
        if (part == kM) {
            // ---- the steps of `now`, walked in the round before: states, ends
            // (the buffer is the one that is drawn into next)
            const bool mine = lane < kSlots && holds(B, now, lane & (kSlots - 1));
            const int w = __shfl_sync(0xffffffffu, walked, (2 * lane) & 31);
            const int si = mine ? now.slot[lane] : 0;
            const int cond = mine ? commit(a, B, now, lane, w) : 0;
            __syncwarp();
            // ---- finished photons leave their slots
            if (__any_sync(0xffffffffu, cond != 0)) {
                Slot &s = B.slots[si];
                if (n_fin > 32 - kSlots) flush();
                queue(cond != 0, s, max(cond, 0));
                if (cond) s.flags = 0;
                __syncwarp();
            }
            // ---- free slots take photons already born; 32 at most are born at once
            unsigned idle = ~__ballot_sync(0xffffffffu, lane < kSlots && (B.slots[lane & (kSlots - 1)].flags & kActive)) &
                            ((1u << a.slots) - 1u);
            for (int tries = 0; tries < 4 && idle && n_born == 0 && !exhausted; ++tries) {
                if (n_fin > 0) flush();
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(a.work, (unsigned long long)a.claim);
                base = __shfl_sync(0xffffffffu, base, 0);
                const int64_t left = a.total - (int64_t)base;
                const int valid = (int)max((int64_t)0, min((int64_t)a.claim, left));
                exhausted = left <= a.claim;
                int c1 = 0;
                Slot s;
                if (lane < valid) c1 = replay_birth(a, (int64_t)base + lane, s);
                queue(lane < valid && c1 != 0, s, c1);
                const unsigned m = __ballot_sync(0xffffffffu, lane < valid && c1 == 0);
                if (lane < valid && c1 == 0) B.born[__popc(m & lt_mask)] = s;
                n_born = __popc(m);
                __syncwarp();
            }
            const int take = min(__popc(idle), n_born);
            if (lane < take) {
                const int f = __fns(idle, 0, lane + 1);
                B.slots[f] = B.born[n_born - 1 - lane];
                B.gen[f] += 1;
            }
            n_born -= take;
            __syncwarp();
            const bool any = __any_sync(0xffffffffu, lane < kSlots && (B.slots[lane & (kSlots - 1)].flags & kActive));
            int stop = !any && exhausted && n_born == 0;
            if ((round & 63u) == 63u && lane == 0) { // time budget (watchdog)
                if (global_ns() - t0 > a.budget_ns) atomicOr(a.status, kStatusBudget);
                if (*(volatile unsigned int *)a.status & kStatusBudget) stop = 1;
            }
            if (lane == 0 && stop) B.stop = 1;
        }
        __syncthreads();
        if (B.stop) break;
        if (part == kDraw) draw_ahead(a, B, now, lane);
        else if (part == kZ) walk_z(B, before, lane);
        else if (part == kXY) walk_xy(B, last, lane);
        else walked = walk_m(B, last, lane);
        __syncthreads();
        drawn = drawn == 2 ? 0 : drawn + 1;
    }
    if (part != kM) return;
    if (n_fin > 0) flush();
    // out of time: the photons in flight leave their records as they stand, those not begun yet after
    // their first step, with condition 0 unless that step is their last
    queue(lane < kSlots && (B.slots[lane & (kSlots - 1)].flags & kActive), B.slots[lane & (kSlots - 1)], 0);
    if (n_fin > 0) flush();
    queue(lane < n_born, B.born[lane], 0);
    if (n_fin > 0) flush();
    if (!exhausted) leave_unwalked<false>(a, lane);
}

// ---------------------------------------------------------------- the polarised walk

// Order of doubles as integers (no FP64 operation), -0 with 0.
__device__ __forceinline__ int64_t order_of(double x) {
    const int64_t b = (int64_t)to_bits(x);
    return b >= 0 ? b : ((int64_t)0x8000000000000000ull - b);
}

// sqrt(x) and a / b (rb: 1 / b nearly): by the corrections, `sure` kept where they are certain, or kExact
// by CUDA's.  A test of a result costs its step the 110 to 290 cycles to the integer side; so what goes
// into one decision is worked out by the corrections, looked at once, late, and, when not sure, worked
// out again exactly.
template <bool kExact>
__device__ __forceinline__ double root(double x, bool &sure) {
    if (kExact) return sqrt(x);
    double h;
    const double g = sqrt_res(x, h);
    sure = sure & sqrt_sure(g, x);
    return g;
}
template <bool kExact>
__device__ __forceinline__ double quotient(double a, double b, double rb, bool &sure) {
    if (kExact) return a / b;
    const double q = quotient_res(a, b, rb);
    sure = sure & quotient_sure(q, a, b);
    return q;
}

// scipy interp1d (linear) on an ascending grid: searchsorted (left) clipped to [1, n - 1], then the
// two-term form of interp1d._call_linear: the upper end's index and both weights.
struct Segment {
    int k;
    double lo, hi;
};
template <bool kExact>
__device__ __forceinline__ Segment segment_of(const DevPhase &ph, int e, double xn, bool &sure) {
    const double *x = ph.cos_asc[e];
    const int n = ph.n_angle[e];
    const int64_t key = order_of(xn);
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (order_of(__ldg(x + mid)) < key) lo = mid + 1; else hi = mid;
    }
    Segment s;
    s.k = lo < 1 ? 1 : (lo > n - 1 ? n - 1 : lo);
    const double xl = __ldg(x + s.k - 1), xh = __ldg(x + s.k), w = xh - xl;
    const double rw = kExact ? 0.0 : rcp_res(w);
    s.hi = quotient<kExact>(xn - xl, w, rw, sure);
    s.lo = quotient<kExact>(xh - xn, w, rw, sure);
    return s;
}
__device__ __forceinline__ double element(const DevPhase &ph, int e, int row, const Segment &s) {
    const double *y = ph.p_asc[e] + (size_t)row * ph.n_angle[e] + s.k;
    return s.hi * __ldg(y) + s.lo * __ldg(y - 1);
}

// rotate_stokes_vector (monte_carlo3D.py:1090-1109)
__device__ __forceinline__ void rotate_stokes(double angle, const double in[4], double out[4]) {
    const double d = 2 * angle;
    double sd, cd;
    sincos(d, &sd, &cd);
    out[0] = in[0];
    out[1] = in[1] * cd + in[2] * sd;
    out[2] = -in[1] * sd + in[2] * cd;
    out[3] = in[3];
}

// The envelope of the rejection sampler for a Stokes vector (populate_pdfs, :905-951).
struct PolEnvelope {
    double max1, max2, part1;
};
__device__ PolEnvelope pol_envelope(const DevPhase &ph, int row, const double st[4]) {
    const double I = st[0], Q = st[1], U = st[2];
    const double two_beta = (Q == 0) ? atan(U / 1e-15) : atan(U / Q);  // :908-911
    double sb, cb;
    sincos(two_beta, &sb, &cb);
    const double C = fabs(Q * cb + U * sb);                           // :935
    PolEnvelope v;
    v.max1 = fabs(I) * ph.a1[row] + ph.b1[row] * C;                   // :931-937
    v.max2 = fabs(I) * ph.a2[row] + ph.b2[row] * C;                   // :940-947
    const double area1 = (ph.cos_max - ph.cos_cutoff) * v.max1;       // :949-951
    const double area2 = (ph.cos_cutoff - ph.cos_min) * v.max2;
    v.part1 = area1 / (area1 + area2);
    return v;
}

// The sampler's candidate whose four uniforms begin at k (:953-1001): its cosine and doubled azimuth,
// and whether it passes.
__device__ __forceinline__ bool pol_candidate(const DevPhase &ph, const Slot &s, uint64_t seed, uint64_t k, const double st[4],
                                              const PolEnvelope &v, double &cos_theta, double &two_phi) {
    const uint4 x0 = stream_block(seed, s.rid, k >> 1), x1 = stream_block(seed, s.rid, (k >> 1) + 1),
                x2 = stream_block(seed, s.rid, (k >> 1) + 2);
    const bool odd = k & 1;
    const double u0 = u01_bits(word(x0, odd)), u1 = u01_bits(odd ? word(x1, false) : word(x0, true)),
                 u2 = u01_bits(word(x1, odd)), u3 = u01_bits(odd ? word(x2, false) : word(x1, true));
    const bool one = u0 < v.part1;                                    // :963-973
    cos_theta = one ? u1 * (ph.cos_max - ph.cos_cutoff) + ph.cos_cutoff
                    : -u1 * (ph.cos_cutoff - ph.cos_min) + ph.cos_cutoff;
    two_phi = 2 * (u2 * kTwoPi);
    const double r3 = 1.000001 * u3 * (one ? v.max1 : v.max2);        // :976-1001
    double sp, cp;
    sincos(two_phi, &sp, &cp);
    const double turn = st[1] * cp + st[2] * sp;
    bool sure = true;
    auto weight = [&](auto exact) {
        const Segment g0 = segment_of<decltype(exact)::value>(ph, 0, cos_theta, sure);
        const Segment g1 = ph.shared_grid ? g0 : segment_of<decltype(exact)::value>(ph, 1, cos_theta, sure);
        return st[0] * element(ph, 0, s.row, g0) + element(ph, 1, s.row, g1) * turn;
    };
    double pf = weight(std::false_type{});
    if (!sure) pf = weight(std::true_type{});
    return !(r3 > pf);
}

// Where a step of scattering cosine ct and azimuth phi takes a photon's direction and Stokes vector
// (:1251-1342), and its path increment.
struct PolMove {
    double nx, ny, nz, st[4], inc;
    bool sure;
};
template <bool kExact>
__device__ __forceinline__ PolMove pol_move(const DevPhase &ph, int row, double mux, double muy, double muz, double ct,
                                            double phi, double s0, double s1, double s2, double s3, bool reflected,
                                            double dtau, double ext, double rext) {
    PolMove m;
    bool sure = true;
    const double sint = root<kExact>(1 - ct * ct, sure);              // :1251-1253
    double sinphi, cosphi;
    sincos(phi, &sinphi, &cosphi);
    if (is_unit(muz)) {                                               // :1262-1269
        const bool up = !(to_bits(muz) >> 63);
        m.nx = sint * cosphi;
        m.ny = up ? sint * sinphi : -sint * sinphi;
        m.nz = up ? ct : -ct;
    } else {                                                          // :1270-1281
        const double sq = root<kExact>(1 - muz * muz, sure), rq = kExact ? 0.0 : rcp_res(sq);
        m.nx = quotient<kExact>(sint * (mux * muz * cosphi - muy * sinphi), sq, rq, sure) + mux * ct;
        m.ny = quotient<kExact>(sint * (muy * muz * cosphi + mux * sinphi), sq, rq, sure) + muy * ct;
        m.nz = -sq * sint * cosphi + muz * ct;
    }
    m.inc = quotient<kExact>(dtau, ext, rext, sure);                  // :1372
    m.st[0] = 1, m.st[1] = m.st[2] = m.st[3] = 0;
    if (!reflected) {                                                 // :1287-1342
        const double phi_sca = acos(cosphi);
        const double st[4] = {s0, s1, s2, s3};
        double sp[4], sc[4], sm[4], P[6];
        rotate_stokes(phi_sca, st, sp);
        const Segment g = segment_of<kExact>(ph, 0, ct, sure);
#pragma unroll
        for (int e = 0; e < 6; ++e)
            P[e] = element(ph, e, row, e == 0 || ph.shared_grid ? g : segment_of<kExact>(ph, e, ct, sure));
        const double P11 = P[0], P12 = P[1], P22 = P[2], P33 = P[3], P43 = P[4], P44 = P[5];
        sc[0] = sp[0] * P11 + sp[1] * P12;
        sc[1] = sp[0] * P12 + sp[1] * P22;
        sc[2] = sp[2] * P33 - sp[3] * P43;
        sc[3] = sp[2] * P43 + sp[3] * P44;
        // (by the corrections den is 0 or NaN only where it is not sure)
        const double den = root<kExact>((1 - ct * ct) * (1 - m.nz * m.nz), sure), d = phi_sca >= kPi ? den : -den;
        const double num = m.nz * ct - muz;
        double cos_i = kExact && den == 0 ? 0 : quotient<kExact>(num, d, kExact ? 0.0 : rcp_res(d), sure);
        if (cos_i < -1) cos_i = -1;
        else if (cos_i > 1) cos_i = 1;
        rotate_stokes(-acos(cos_i), sc, sm);
        const double ri = kExact ? 0.0 : rcp_res(sm[0]);
        if (kExact) m.st[0] = sm[0] / sm[0];
        else sure = sure & moderate(sm[0]);
#pragma unroll
        for (int k = 1; k < 4; ++k) {
            // (the scattering after a reflection leaves V at 0, of either sign)
            const bool zero = !kExact && to_bits(sm[k]) << 1 == 0;
            bool fine = true;
            m.st[k] = quotient<kExact>(sm[k], sm[0], ri, fine);
            if (zero) m.st[k] = sm[k] * ri;
            sure = sure & (zero | fine);
        }
    }
    m.sure = sure;
    return m;
}
__device__ __noinline__ PolMove pol_move_exact(const DevPhase &ph, int row, double mux, double muy, double muz, double ct,
                                               double phi, double s0, double s1, double s2, double s3, bool reflected,
                                               double dtau, double ext) {
    return pol_move<true>(ph, row, mux, muy, muz, ct, phi, s0, s1, s2, s3, reflected, dtau, ext, 0.0);
}

// A step of photon s past its first with its scattering angles (:1227-1466); returns its end
// condition.  Its uniforms begin at s.k.
__device__ int pol_step(const DevPhase &ph, Slot &s, uint64_t seed, double st[4], double p_rand, double two_phi) {
    const double dtau = -log(uniform_at(seed, s.rid, s.k));
    const double ssa_rand = uniform_at(seed, s.rid, s.k + 1);
    const bool ice = uniform_at(seed, s.rid, s.k + 2) > s.p_imp;      // :1375-1383
    s.k += 3;
    const bool reflected = (s.flags & kRefl) != 0;
    double mux = s.mux, muy = s.muy, muz = s.muz, ct = p_rand;
    if (s.lambertian()) {                                             // :1238-1250
        mux = muy = 0.;
        muz = 1.;
        for (int tries = 0;; ++tries) {
            const double theta = 0 + (kPi / 2 - 0) * uniform_at(seed, s.rid, s.k);
            const double r1 = uniform_at(seed, s.rid, s.k + 1);
            double sn;
            sincos(theta, &sn, &ct);
            s.k += 2;
            if (r1 < 2 * sn * ct || tries >= 131072) break;           // no stream needs as many
        }
    }
    // (the reference's phi; a reflected photon starts again unpolarised, :1283-1285)
    PolMove m = pol_move<false>(ph, s.row, mux, muy, muz, ct, two_phi / 2., st[0], st[1], st[2], st[3], reflected, dtau, s.ext,
                                s.rext);
    if (!m.sure) m = pol_move_exact(ph, s.row, mux, muy, muz, ct, two_phi / 2., st[0], st[1], st[2], st[3], reflected, dtau, s.ext);
#pragma unroll
    for (int k = 0; k < 4; ++k) st[k] = m.st[k];
    s.flags &= ~kRefl;
    const double zp = s.z;
    s.z = zp + dtau * m.nz;                                           // :1352
    s.mux = m.nx, s.muy = m.ny, s.muz = m.nz;                         // :1364-1369
    s.path += m.inc;                                                  // :1372
    s.i += 1;
    return step_end(s, seed, s.z, zp, dtau, m.nz, s.path, false, ssa_rand >= (ice ? s.ssa_ice : s.ssa_imp), ice, &s.k, &s.flags);
}

// 2^glog lanes a photon, the same state in each: they test candidates of the sampler side by side
// (a candidate takes four uniforms of the photon's stream, so candidate j's are known; the first that
// passes is the sampler's), and walk the rest of the step alike.  A group whose photon ends takes the
// next.  Bound by FP64 instructions, 64 cycles a warp each however many lanes take part.  So searches
// compare bits, the six elements share one segment's weights where they share a grid, quotients by
// one divisor its reciprocal, and sine and cosine come together: about 60 a candidate and 430 a
// step's rest (145 and 650 with one thread a photon, whose warp also waited for the slowest of 32
// samplers).  Hexagonal plates, 100 um, tau as below 40: 50 photons 40.4 -> 9.4 ms, 1,000
// 80.8 -> 20.3, 10,000 95.6 -> 34.9, 40,000 153 -> 87; a lone photon's step 17 us; with the look at the
// roots' and quotients' roundings 7% more for 50, 1 to 2% for 10,000 and up.
__global__ void __launch_bounds__(128, 3) walk_replay_pol_kernel(const ReplayArgs a, const int glog) {
    const int lane = threadIdx.x & 31, G = 1 << glog, gl = lane & (G - 1), g0 = lane - gl;
    const unsigned group = (G == 32 ? 0xffffffffu : ((1u << G) - 1u)) << g0;
    Slot s{};
    double st[4] = {1, 0, 0, 0};
    bool have = false, exhausted = false, stop = false;
    const unsigned long long t0 = global_ns();
    for (uint32_t it = 0; !stop; ++it) {
        int cond = 0;
        const unsigned need = __ballot_sync(0xffffffffu, !have && !exhausted && gl == 0);
        bool born = false;
        if (need) {
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(a.work, (unsigned long long)__popc(need));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (!have && !exhausted) {
                const unsigned long long n = base + __popc(need & ((1u << g0) - 1u));
                if (n < (unsigned long long)a.total) {
                    cond = replay_birth(a, (int64_t)n, s);
                    const DevConfig &c = a.cfgs[s.ci];
#pragma unroll
                    for (int k = 0; k < 4; ++k) st[k] = c.stokes0[k];
                    have = born = true;
                } else {
                    exhausted = true;
                }
            }
        }
        if (!__any_sync(0xffffffffu, have)) break;
        // ---- the scattering angles of the photons walking on
        const DevPhase &ph = a.phase[have ? a.cfgs[s.ci].ice_table : 0];
        bool pending = have && !born;
        PolEnvelope env{0, 0, 0};
        if (pending) env = pol_envelope(ph, s.row, st);
        double p_rand = 1, two_phi = 0;
        uint32_t j0 = 0;
        for (uint32_t round = 0; __any_sync(0xffffffffu, pending); ++round) {
            bool pass = false;
            double c = 1, t = 0;
            if (pending) pass = pol_candidate(ph, s, a.seed, s.k + 4 * (uint64_t)(j0 + gl), st, env, c, t);
            const unsigned hit = __ballot_sync(0xffffffffu, pass) & group;
            const int src = hit ? __ffs(hit) - 1 : lane;
            c = shfl_d(c, src);
            t = shfl_d(t, src);
            if (pending && hit) {
                p_rand = c;
                two_phi = t;
                s.k += 4 * (uint64_t)(j0 + (uint32_t)(src - g0) + 1);
                pending = false;
            }
            j0 += (uint32_t)G;
            if ((round & 255u) == 255u) {
                int over = 0;
                if (lane == 0) over = global_ns() - t0 > a.budget_ns;
                stop = __shfl_sync(0xffffffffu, over, 0) != 0;
                if (stop) break;
            }
        }
        if (stop && lane == 0) atomicOr(a.status, kStatusBudget);
        bool over = false;                                            // out of its stream
        if (have && !born && !stop) {
            cond = pol_step(ph, s, a.seed, st, p_rand, two_phi);
            over = s.k > kMaxUniforms;
            if (over && gl == 0) atomicOr(a.status, kStatusStream);
        }
        if (cond > 0 || over) {
            if (gl == 0) finish_photon<true>(a, s.gid, s.ci, cond, s.i, s.wvl_um, s.mux, s.muy, s.muz, s.path, s.depth, st);
            have = false;
        }
        if ((it & 63u) == 63u && !stop) {                             // time budget (watchdog)
            int late = 0;
            if (lane == 0) {
                if (global_ns() - t0 > a.budget_ns) atomicOr(a.status, kStatusBudget);
                late = *(volatile unsigned int *)a.status & kStatusBudget;
            }
            stop = __shfl_sync(0xffffffffu, late, 0) != 0;
        }
    }
    if (!stop) return;
    // as the HG walk's photons do (walk_replay_kernel)
    if (have && gl == 0) finish_photon<true>(a, s.gid, s.ci, 0, s.i, s.wvl_um, s.mux, s.muy, s.muz, s.path, s.depth, st);
    __syncwarp();
    leave_unwalked<true>(a, lane);
}

}  // namespace

cudaError_t launch_walk_replay(const ReplayArgs &a, int sm_count, cudaStream_t s, int *blocks) {
    *blocks = 0;
    if (a.total <= 0) return cudaSuccess;
    if (a.pol) {
        // three blocks an SM (140 registers), and as many lanes a photon as let all photons walk at
        // once: a lane more tests a candidate for nothing, but a photon more in a warp shares its rest
        const int64_t warps = 12 * (int64_t)std::max(1, sm_count);
        int glog = 5;
        while (glog > 0 && warps << (5 - glog) < a.total) --glog;
        const int64_t each = 4 << (5 - glog);                         // photons a block at a time
        const int64_t grid = std::min<int64_t>(3 * (int64_t)std::max(1, sm_count), (a.total + each - 1) / each);
        *blocks = (int)grid;
        walk_replay_pol_kernel<<<(unsigned)grid, 128, 0, s>>>(a, glog);
        return cudaGetLastError();
    }
    // four blocks an SM (126 registers), a warp of each part on each of its four FP64 pipes; few
    // photons are spread over all of them
    ReplayArgs b = a;
    const int64_t grid = std::min<int64_t>(4 * (int64_t)std::max(1, sm_count), a.total);
    const int64_t each = (a.total + grid - 1) / grid;
    b.slots = (int32_t)std::min<int64_t>(kSlots, each);
    b.claim = (int32_t)std::min<int64_t>(32, each);
    *blocks = (int)grid;
    walk_replay_kernel<<<(unsigned)grid, 128, 0, s>>>(b);
    return cudaGetLastError();
}

}  // namespace mcw
