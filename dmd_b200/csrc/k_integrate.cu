// k_integrate.cu -- Velocity Verlet with fused thermostat / barostat bookkeeping.
//
// Reference sequence (SimulationEngine::step, src/sim/simulation_engine.cpp:53-86):
//   compute; half_kick; advance; compute; half_kick; thermostat; barostat.
// Device form (per step, every replica of the batch in the same launches):
//   [eval #1]           only where the first evaluation would differ from the
//                       previous step's second one (REF barostat moved the atoms,
//                       no forces yet, or the REF list cadence rebuilds now)
//   k_kick_drift        pending thermostat scale, half kick, PHYS pending
//                       barostat scale, drift, clear forces, write the sorted
//                       FP32/FP64 mirror, skin check (replicas with step < target)
//   [eval #2]           (k_eval_begin, launched before the drift or, between the
//                       steps of one graph, done by k_replica_update, marks the
//                       replicas that advance and scales the PHYS box to match)
//   k_kick2             half kick (+ Andersen), per-tile KE / virial partials
//   k_replica_update    closes eval #2, KE, thermostat (Berendsen / Nose-Hoover
//                       scale, applied lazily in the next kick), Berendsen
//                       barostat factor (REF: applied now; PHYS: pending for the
//                       next drift)
//   k_apply_scale       REF barostat position scaling (only when a barostat exists)
// PHYS therefore evaluates forces once per step with or without a barostat:
// the first kick of a step uses the forces of the previous evaluation and the
// scaling is applied with the drift, so every evaluation sees the positions
// the next kick is for.
// Integration arithmetic is FP64 with the reference's operation order
// (src/integrate/integrator.cpp:4-20) and no FMA contraction.
#include "device.cuh"
#include "launch.h"

namespace dmd {

namespace {

// Work counters and the rebuild's grid barrier, before an evaluation.
__device__ __forceinline__ void reset_counters(const Dev& d) {
    *d.nb_work = 0;
    if (d.nb_work_mi) *d.nb_work_mi = 0;
    d.grid_bar[0] = 0;  // arrivals (the generation word keeps counting)
}

// A force evaluation of replica r (ev) is about to start.
__device__ __forceinline__ void begin_eval(RepState& s, const Rep& R, bool ev, bool want_e) {
    s.eval = ev;
    s.green_ok = (s.green_L == s.L) ? 1 : 0;
    s.want_e = want_e;
    if (ev) {
        for (int k = 0; k < N_EACC; ++k) s.e_acc[k] = 0;
        s.e_recip = 0.0;
        s.vir_recip = 0.0;
        if (!(R.flags & F_PHYS) && (R.flags & F_LJ) && s.lj_counter >= 10) s.rebuild = 1;
    }
}

// Start of a step, before its kick and drift: which replicas advance, the
// pending scales handed to k_kick_drift, the box that follows the positions it
// scales, and the step's (second) evaluation.  Runs in k_eval_begin ahead of
// the first step of a launch, and at the end of k_replica_update between the
// steps of one launch.
// skipped: the step's first evaluation was not issued (REF; no replica needed
// it), but LennardJones::compute advances its counter on every call
// (lennard_jones.cpp:91).
__device__ __forceinline__ void begin_step(RepState& s, const Rep& R, bool skipped) {
    s.active = (s.step < s.target_step) ? 1 : 0;
    if (skipped && s.active && !(R.flags & F_PHYS) && (R.flags & F_LJ)) s.lj_counter += 1;
    s.dr_move = s.active;
    s.dr_vscale = s.vscale;
    s.dr_pscale = s.pscale;
    s.dr_L = s.L;
    // a replica that has reached its target keeps its pending thermostat scale
    // for the next read of its velocities
    if (s.active) s.vscale = 1.0;
    if (s.active && (R.flags & F_PHYS) && s.pscale != 1.0) {
        s.L *= s.pscale;
        s.invL = 1.0 / s.L;
        s.pscale = 1.0;
    }
    // Pair energies and the pair virial are needed by single-point evaluations,
    // by the evaluation that ends a run (its energies are what the host reads; the
    // FP64 path forms them at the end of every call, read_step) and, with the PHYS
    // barostat, every step (its pressure uses the atomic virial).
    begin_eval(s, R, s.active, s.step + 1 >= s.target_step || s.step + 1 == s.read_step || ((R.flags & F_PHYS) && R.barostat));
}

__global__ void k_eval_begin(Dev d, int pass) {
    chain_wait();
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r == 0) reset_counters(d);
    if (r >= d.n_rep) return;
    RepState* s = d.st + r;
    const Rep& R = d.rep[r];
    if (pass == PASS_SECOND || pass == PASS_SECOND_ONLY) {
        begin_step(*s, R, pass == PASS_SECOND_ONLY);
        return;
    }
    bool ev = true;
    if (pass == PASS_FIRST) {
        const bool ref_lj = !(R.flags & F_PHYS) && (R.flags & F_LJ);
        // which replicas advance this step (the host may have moved the targets)
        s->active = (s->step < s->target_step) ? 1 : 0;
        // REF: the barostat scale of the previous step has been applied; PHYS keeps
        // its pending scale for the drift, so an evaluation before it sees the
        // unscaled pair.
        if (!(R.flags & F_PHYS)) s->pscale = 1.0;
        ev = s->active && ((R.barostat != 0 && !(R.flags & F_PHYS)) || !s->have_forces ||
                           (ref_lj && s->lj_counter >= 10));
        // LennardJones::compute advances its counter on every call (lennard_jones.cpp:91)
        if (s->active && !ev && ref_lj) s->lj_counter += 1;
    }
    // eval #1 never needs energies: eval #2 of the same step overwrites its sums
    begin_eval(*s, R, ev, pass == PASS_SINGLE);
}

// FP64: the replicas' energies are read after n more steps.
__global__ void k_mark_read(Dev d, int n) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < d.n_rep) d.st[r].read_step = d.st[r].step + n;
}

__global__ void k_eval_end(Dev d) {
    chain_wait();
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= d.n_rep) return;
    RepState* s = d.st + r;
    const Rep& R = d.rep[r];
    if (!s->eval) return;
    if (!(R.flags & F_PHYS) && (R.flags & F_LJ)) s->lj_counter += 1;
    s->have_forces = 1;
    if (R.flags & F_PME) s->green_L = s->L;  // the influence kernel has filled the cache
}

__global__ void k_clear_forces(Dev d) {
    chain_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < d.n_slots) {
        int r = d.tile_rep[i >> 5];
        if (d.st[r].eval) {
            d.fnx[i] = 0;
            d.fny[i] = 0;
            d.fnz[i] = 0;
        }
    }
    if (i < d.n_atoms) {
        int r = d.atom_rep[i];
        if (d.st[r].eval) {
            d.fbx[i] = 0;
            d.fby[i] = 0;
            d.fbz[i] = 0;
        }
    }
}

__device__ __forceinline__ void write_mirror(const Dev& d, int slot, int a, double x, double y, double z,
                                             double L) {
    if (d.xq32) {
        const int t = slot >> 5;
        d.xq32[slot] = make_float4(static_cast<float>((x - d.imgx[a] * L) - d.tcx[t]),
                                   static_cast<float>((y - d.imgy[a] * L) - d.tcy[t]),
                                   static_cast<float>((z - d.imgz[a] * L) - d.tcz[t]),
                                   static_cast<float>(d.q[a]));
    }
    if (d.xq64) d.xq64[slot] = make_double4(x, y, z, d.q[a]);
}

__device__ __forceinline__ void skin_check(const Dev& d, RepState* s, const Rep& R, int a, double x,
                                           double y, double z) {
    if (!(R.flags & F_PHYS)) return;
    const double dx = x - d.xr[a], dy = y - d.yr[a], dz = z - d.zr[a];
    if (dx * dx + dy * dy + dz * dz > R.half_skin2) s->rebuild = 1;
}

// Integrator::half_kick + advance (integrator.cpp:4-20), with the pending
// thermostat scale of the previous step applied first.  PHYS with a barostat:
// the pending position scale s (1 otherwise, an exact multiply) is applied
// before the drift, x <- s x + v dt, and the mirror is written for the box
// s L that begin_step has stored.
// One thread per atom in reference order: the FP64 state, masses and bonded
// forces are read and written coalesced; only the pair forces and the mirror
// are addressed through the atom's slot.
// The kernel before it (k_eval_begin or k_replica_update) writes replica state
// only, so a chained launch loads everything else before it waits for that
// kernel.  With k_kick2 and k_replica_update loading ahead the same way and the
// next step begun by k_replica_update, a step of 1,000 LJ atoms takes 13.5 us
// (18.8 with each kernel loading after its wait and k_eval_begin every step).
__global__ void k_kick_drift(Dev d) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = a < d.n_atoms;
    int r = 0, slot = 0;
    double inv_mass = 0, fx = 0, fy = 0, fz = 0, vx = 0, vy = 0, vz = 0, x = 0, y = 0, z = 0;
    if (in) {
        r = d.atom_rep[a];
        slot = d.slot_of_atom[a];
        inv_mass = 1.0 / d.mass[a];
        fx = from_fix(d.fnx[slot] + d.fbx[a], FSCALE);
        fy = from_fix(d.fny[slot] + d.fby[a], FSCALE);
        fz = from_fix(d.fnz[slot] + d.fbz[a], FSCALE);
        vx = d.vx[a];
        vy = d.vy[a];
        vz = d.vz[a];
        x = d.x[a];
        y = d.y[a];
        z = d.z[a];
    }
    chain_wait();
    if (!in) return;
    RepState* s = d.st + r;
    if (!s->dr_move) return;
    const Rep& R = d.rep[r];
    const double dt = R.dt, half_dt = 0.5 * dt;
    const double lam = s->dr_vscale;
    vx = __dadd_rn(__dmul_rn(vx, lam), __dmul_rn(__dmul_rn(fx, inv_mass), half_dt));
    vy = __dadd_rn(__dmul_rn(vy, lam), __dmul_rn(__dmul_rn(fy, inv_mass), half_dt));
    vz = __dadd_rn(__dmul_rn(vz, lam), __dmul_rn(__dmul_rn(fz, inv_mass), half_dt));
    const double sc = s->dr_pscale;
    x = __dadd_rn(__dmul_rn(x, sc), __dmul_rn(vx, dt));
    y = __dadd_rn(__dmul_rn(y, sc), __dmul_rn(vy, dt));
    z = __dadd_rn(__dmul_rn(z, sc), __dmul_rn(vz, dt));
    d.vx[a] = vx;
    d.vy[a] = vy;
    d.vz[a] = vz;
    d.x[a] = x;
    d.y[a] = y;
    d.z[a] = z;
    d.fnx[slot] = 0;
    d.fny[slot] = 0;
    d.fnz[slot] = 0;
    d.fbx[a] = 0;
    d.fby[a] = 0;
    d.fbz[a] = 0;
    write_mirror(d, slot, a, x, y, z, s->dr_L * sc);
    skin_check(d, s, R, a, x, y, z);
}

// Philox4x32-10 (Salmon et al., SC'11) for the PHYS Andersen thermostat.
__device__ __forceinline__ void philox(uint32_t c[4], uint32_t k0, uint32_t k1) {
#pragma unroll
    for (int i = 0; i < 10; ++i) {
        const uint32_t hi0 = __umulhi(0xD2511F53u, c[0]), lo0 = 0xD2511F53u * c[0];
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]), lo1 = 0xCD9E8D57u * c[2];
        const uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
        c[0] = n0;
        c[1] = lo1;
        c[2] = n2;
        c[3] = lo0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
}

// Second half kick, optional Andersen collisions, per-tile KE and r.F partials.
// Only the forces come from the kernel before it in a chained launch: the rest
// is loaded before the wait.
__global__ void k_kick2(Dev d, int andersen_ref, int andersen_phys) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int t = slot >> 5;
    const int r = (t < d.n_tiles) ? d.tile_rep[t] : 0;
    RepState* s = d.st + r;
    const Rep& R = d.rep[r];
    double ke = 0.0, w = 0.0;
    int a = -1;
    double m = 1, inv_mass = 1, vx = 0, vy = 0, vz = 0, x = 0, y = 0, z = 0;
    if (slot < d.n_slots && s->active) a = d.atom_of_slot[slot];
    if (a >= 0) {
        m = d.mass[a];
        inv_mass = 1.0 / m;
        vx = d.vx[a];
        vy = d.vy[a];
        vz = d.vz[a];
        x = d.x[a];
        y = d.y[a];
        z = d.z[a];
    }
    chain_wait();
    {
        if (a >= 0) {
            const double half_dt = 0.5 * R.dt;
            const double fx = from_fix(d.fnx[slot] + d.fbx[a], FSCALE);
            const double fy = from_fix(d.fny[slot] + d.fby[a], FSCALE);
            const double fz = from_fix(d.fnz[slot] + d.fbz[a], FSCALE);
            vx = __dadd_rn(vx, __dmul_rn(__dmul_rn(fx, inv_mass), half_dt));
            vy = __dadd_rn(vy, __dmul_rn(__dmul_rn(fy, inv_mass), half_dt));
            vz = __dadd_rn(vz, __dmul_rn(__dmul_rn(fz, inv_mass), half_dt));
            if (R.thermostat == 3 && R.t_freq * R.dt > 0.0) {
                if (andersen_ref && d.and_flag && d.and_flag[a]) {
                    vx = d.and_v[3 * a];
                    vy = d.and_v[3 * a + 1];
                    vz = d.and_v[3 * a + 2];
                } else if (andersen_phys && (R.flags & F_PHYS)) {
                    const uint32_t call = static_cast<uint32_t>(s->andersen_calls);
                    const uint32_t callh = static_cast<uint32_t>(s->andersen_calls >> 32);
                    const uint32_t li = static_cast<uint32_t>(a - R.atom_begin);
                    uint32_t c[4] = {li, call, callh, 0x414E4400u};
                    philox(c, R.key0, R.key1);
                    const double u = c[0] * 2.3283064365386963e-10;
                    if (u < R.t_freq * R.dt) {
                        const double sg = sqrt(KB * R.t_temp / m);
                        const double u1 = (c[1] + 1.0) * 2.3283064365386963e-10;
                        const double u2 = c[2] * 2.3283064365386963e-10;
                        const double rr = sqrt(-2.0 * log(u1));
                        uint32_t e[4] = {li, call, callh, 0x414E4401u};
                        philox(e, R.key0, R.key1);
                        const double u3 = (e[0] + 1.0) * 2.3283064365386963e-10;
                        const double u4 = e[1] * 2.3283064365386963e-10;
                        vx = rr * cos(2.0 * PI * u2) * sg;
                        vy = rr * sin(2.0 * PI * u2) * sg;
                        vz = sqrt(-2.0 * log(u3)) * cos(2.0 * PI * u4) * sg;
                    }
                }
            }
            d.vx[a] = vx;
            d.vy[a] = vy;
            d.vz[a] = vz;
            // kinetic_energy (thermostat.cpp:6-15) and virial (barostat.cpp:6-14) terms
            ke = __dmul_rn(__dmul_rn(0.5, m),
                           __dadd_rn(__dadd_rn(__dmul_rn(vx, vx), __dmul_rn(vy, vy)), __dmul_rn(vz, vz)));
            w = __dadd_rn(__dadd_rn(__dmul_rn(x, fx), __dmul_rn(y, fy)), __dmul_rn(z, fz));
        }
    }
    ke = warp_sum_d(ke);
    w = warp_sum_d(w);
    if (lane == 0 && t < d.n_tiles) {
        d.tile_ke[t] = ke;
        d.tile_vir[t] = w;
    }
}

// A rigid three-site molecule: constraints (p, q), (p, r), (q, r) in that
// sweep order.  Its three atoms then live in registers (index 0, 1, 2 = p, q,
// r) for all sweeps, and what a sweep does not change (1/m, d^2, the
// denominators) is formed once -- the same FP64 operations on the same
// operands, so the sweeps are bit for bit those of the general path, which
// re-reads every operand from global memory in each of its dependent steps.
// The sweeps are one dependent FP64 chain per thread, so their latency is the
// kernel's time: 522 molecules, 43.4 -> 14.3 us (SHAKE) and 60.6 -> 12.8 us
// (RATTLE) against the general path.
__device__ __forceinline__ bool is_triangle(const Dev& d, int c0, int c1, int3& at) {
    if (c1 - c0 != 3) return false;
    const int2 u = d.cons_ij[c0], v = d.cons_ij[c0 + 1], w = d.cons_ij[c0 + 2];
    at = make_int3(u.x, u.y, v.y);
    return v.x == u.x && w.x == u.y && w.y == v.y;
}

// d - round(d * inv) * L along each axis; a displacement inside half a box (the
// usual case) has round() = 0 and is returned as it is, which is the same value.
__device__ __forceinline__ void wrap_ref(double& dx, double& dy, double& dz, double L, double inv) {
    const double m = fmax(fmax(fabs(dx), fabs(dy)), fabs(dz));
    if (!(__dmul_rn(m, inv) >= 0.5)) return;
    dx = __dsub_rn(dx, __dmul_rn(round(__dmul_rn(dx, inv)), L));
    dy = __dsub_rn(dy, __dmul_rn(round(__dmul_rn(dy, inv)), L));
    dz = __dsub_rn(dz, __dmul_rn(round(__dmul_rn(dz, inv)), L));
}

// a / b with y = 1 / b (correctly rounded): Markstein's division (P. Markstein,
// IBM J. Res. Dev. 34, 1990), the quotient estimate a y and one correction by
// its exact remainder.  The correctly rounded quotient, in three dependent
// operations instead of a full division in every sweep (b does not change
// between sweeps).
__device__ __forceinline__ double div_known(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}

__device__ __forceinline__ double dot_ref(double ax, double ay, double az, double bx, double by, double bz) {
    return __dadd_rn(__dadd_rn(__dmul_rn(ax, bx), __dmul_rn(ay, by)), __dmul_rn(az, bz));
}

// SHAKE sweeps of one triangle (see k_shake).
__device__ __forceinline__ void shake_triangle(double (&x)[3], double (&y)[3], double (&z)[3], const double (&w)[3],
                                               const double (&dist)[3], double L, double inv, double tol) {
    double d2[3], den[3], rden[3];
    bool ok[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int a = c == 2 ? 1 : 0, b = c == 0 ? 1 : 2;
        d2[c] = __dmul_rn(dist[c], dist[c]);
        den[c] = __dmul_rn(__dmul_rn(2.0, d2[c]), __dadd_rn(w[a], w[b]));
        rden[c] = 1.0 / den[c];
    }
    for (int it = 0; it < 100; ++it) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int a = c == 2 ? 1 : 0, b = c == 0 ? 1 : 2;
            double dx = __dsub_rn(x[b], x[a]), dy = __dsub_rn(y[b], y[a]), dz = __dsub_rn(z[b], z[a]);
            wrap_ref(dx, dy, dz, L, inv);
            const double err = __dsub_rn(dot_ref(dx, dy, dz, dx, dy, dz), d2[c]);
            ok[c] = !(fabs(err) >= tol);
            if (fabs(err) > tol) {
                const double lam = div_known(err, den[c], rden[c]);
                const double lx = __dmul_rn(lam, dx), ly = __dmul_rn(lam, dy), lz = __dmul_rn(lam, dz);
                x[a] = __dadd_rn(x[a], __dmul_rn(lx, w[a]));
                y[a] = __dadd_rn(y[a], __dmul_rn(ly, w[a]));
                z[a] = __dadd_rn(z[a], __dmul_rn(lz, w[a]));
                x[b] = __dsub_rn(x[b], __dmul_rn(lx, w[b]));
                y[b] = __dsub_rn(y[b], __dmul_rn(ly, w[b]));
                z[b] = __dsub_rn(z[b], __dmul_rn(lz, w[b]));
            }
        }
        if (ok[0] & ok[1] & ok[2]) break;
    }
}

// RATTLE of one triangle (see k_rattle): its bond vectors and denominators do
// not change between sweeps.
struct TriangleBonds {
    double dx[3], dy[3], dz[3], den[3], rden[3];
    __device__ __forceinline__ void set(const double (&x)[3], const double (&y)[3], const double (&z)[3],
                                        const double (&w)[3], double L, double inv) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int a = c == 2 ? 1 : 0, b = c == 0 ? 1 : 2;
            dx[c] = __dsub_rn(x[b], x[a]);
            dy[c] = __dsub_rn(y[b], y[a]);
            dz[c] = __dsub_rn(z[b], z[a]);
            wrap_ref(dx[c], dy[c], dz[c], L, inv);
            den[c] = __dmul_rn(dot_ref(dx[c], dy[c], dz[c], dx[c], dy[c], dz[c]), __dadd_rn(w[a], w[b]));
            rden[c] = 1.0 / den[c];
        }
    }
};

__device__ __forceinline__ void rattle_triangle(const TriangleBonds& tb, double (&vx)[3], double (&vy)[3],
                                                double (&vz)[3], const double (&w)[3], double tol) {
    const double(&dx)[3] = tb.dx;
    const double(&dy)[3] = tb.dy;
    const double(&dz)[3] = tb.dz;
    bool ok[3];
    for (int it = 0; it < 100; ++it) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int a = c == 2 ? 1 : 0, b = c == 0 ? 1 : 2;
            const double rv = dot_ref(dx[c], dy[c], dz[c], __dsub_rn(vx[b], vx[a]), __dsub_rn(vy[b], vy[a]),
                                      __dsub_rn(vz[b], vz[a]));
            ok[c] = !(fabs(rv) >= tol);
            if (fabs(rv) > tol) {
                const double lam = div_known(rv, tb.den[c], tb.rden[c]);
                const double lx = __dmul_rn(lam, dx[c]), ly = __dmul_rn(lam, dy[c]), lz = __dmul_rn(lam, dz[c]);
                vx[a] = __dadd_rn(vx[a], __dmul_rn(lx, w[a]));
                vy[a] = __dadd_rn(vy[a], __dmul_rn(ly, w[a]));
                vz[a] = __dadd_rn(vz[a], __dmul_rn(lz, w[a]));
                vx[b] = __dsub_rn(vx[b], __dmul_rn(lx, w[b]));
                vy[b] = __dsub_rn(vy[b], __dmul_rn(ly, w[b]));
                vz[b] = __dsub_rn(vz[b], __dmul_rn(lz, w[b]));
            }
        }
        if (ok[0] & ok[1] & ok[2]) break;
    }
}

// Constraints::apply (src/integrate/constraints.cpp:9-47) after the drift: one
// thread per group of constraints that share atoms (a molecule), its
// constraints swept in their given order until the group's largest
// |r^2 - d^2| (measured before each correction) is below the tolerance, at
// most 100 sweeps.  Groups share no atoms, so this is the reference's
// Gauss-Seidel sweep over all constraints, group by group.  The FP64
// operations follow the reference's order; the moved atoms' mirror entries
// are written again.  PHYS: the box is the drifted frame's (L times the
// pending barostat scale), and SHAKE's displacement is also given to the
// half-step velocities (v += dx / dt).
__global__ void k_shake(Dev d) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = g < d.n_cgroups;
    // a triangle's data that the drift does not write are loaded before the wait
    // for it (and the mirror's and the skin check's before the sweeps)
    int r = 0, c0 = 0, c1 = 0;
    int3 at;
    bool tri = false;
    int id[3], slot[3], im[3][3];
    double w[3], dist[3], q[3], tc[3][3], xr[3][3];
    if (in) {
        r = d.cgroup_rep[g];
        c0 = d.cgroup_begin[g];
        c1 = d.cgroup_begin[g + 1];
        tri = is_triangle(d, c0, c1, at);
    }
    if (tri) {
        id[0] = at.x;
        id[1] = at.y;
        id[2] = at.z;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int a = id[k];
            w[k] = 1.0 / d.mass[a];
            dist[k] = d.cons_d[c0 + k];
            q[k] = d.q[a];
            slot[k] = d.slot_of_atom[a];
            im[k][0] = d.imgx[a];
            im[k][1] = d.imgy[a];
            im[k][2] = d.imgz[a];
            xr[k][0] = d.xr[a];
            xr[k][1] = d.yr[a];
            xr[k][2] = d.zr[a];
            tc[k][0] = d.tcx[slot[k] >> 5];
            tc[k][1] = d.tcy[slot[k] >> 5];
            tc[k][2] = d.tcz[slot[k] >> 5];
        }
    }
    chain_wait();
    if (!in) return;
    RepState* s = d.st + r;
    if (!s->dr_move) return;  // the replicas k_kick_drift moved
    const Rep& R = d.rep[r];
    const bool phys = (R.flags & F_PHYS) != 0;
    const double L = phys ? s->dr_L * s->dr_pscale : s->dr_L, inv = 1.0 / L, tol = R.cons_tol;
    const int na = d.n_atoms;
    if (tri) {
        double x[3], y[3], z[3], x0[3], y0[3], z0[3], vx[3], vy[3], vz[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int a = id[k];
            x0[k] = x[k] = d.x[a];
            y0[k] = y[k] = d.y[a];
            z0[k] = z[k] = d.z[a];
            vx[k] = d.vx[a];
            vy[k] = d.vy[a];
            vz[k] = d.vz[a];
        }
        shake_triangle(x, y, z, w, dist, L, inv, tol);
        const double dt = R.dt, rdt = 1.0 / dt;
        bool far = false;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int a = id[k];
            d.x[a] = x[k];
            d.y[a] = y[k];
            d.z[a] = z[k];
            if (phys) {
                d.vx[a] = __dadd_rn(vx[k], div_known(__dsub_rn(x[k], x0[k]), dt, rdt));
                d.vy[a] = __dadd_rn(vy[k], div_known(__dsub_rn(y[k], y0[k]), dt, rdt));
                d.vz[a] = __dadd_rn(vz[k], div_known(__dsub_rn(z[k], z0[k]), dt, rdt));
            }
            // write_mirror and skin_check on the loaded values
            if (d.xq32)
                d.xq32[slot[k]] = make_float4(static_cast<float>((x[k] - im[k][0] * L) - tc[k][0]),
                                              static_cast<float>((y[k] - im[k][1] * L) - tc[k][1]),
                                              static_cast<float>((z[k] - im[k][2] * L) - tc[k][2]),
                                              static_cast<float>(q[k]));
            if (d.xq64) d.xq64[slot[k]] = make_double4(x[k], y[k], z[k], q[k]);
            const double dx = x[k] - xr[k][0], dy = y[k] - xr[k][1], dz = z[k] - xr[k][2];
            far |= dx * dx + dy * dy + dz * dz > R.half_skin2;
        }
        if (phys && far) s->rebuild = 1;
        return;
    }
    const int q0 = d.cgroup_atom_begin[g], q1 = d.cgroup_atom_begin[g + 1];
    if (phys)
        for (int q = q0; q < q1; ++q) {
            const int a = d.cgroup_atoms[q];
            d.cons_x0[a] = d.x[a];
            d.cons_x0[na + a] = d.y[a];
            d.cons_x0[2 * na + a] = d.z[a];
        }
    for (int it = 0; it < 100; ++it) {
        double worst = 0.0;
        for (int c = c0; c < c1; ++c) {
            const int a = d.cons_ij[c].x, b = d.cons_ij[c].y;
            double dx = __dsub_rn(d.x[b], d.x[a]), dy = __dsub_rn(d.y[b], d.y[a]), dz = __dsub_rn(d.z[b], d.z[a]);
            dx = __dsub_rn(dx, __dmul_rn(round(__dmul_rn(dx, inv)), L));
            dy = __dsub_rn(dy, __dmul_rn(round(__dmul_rn(dy, inv)), L));
            dz = __dsub_rn(dz, __dmul_rn(round(__dmul_rn(dz, inv)), L));
            const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
            const double d2 = __dmul_rn(d.cons_d[c], d.cons_d[c]);
            const double err = __dsub_rn(r2, d2);
            if (fabs(err) > worst) worst = fabs(err);
            if (fabs(err) > tol) {
                const double wa = 1.0 / d.mass[a], wb = 1.0 / d.mass[b];
                const double lam = err / __dmul_rn(__dmul_rn(2.0, d2), __dadd_rn(wa, wb));
                d.x[a] = __dadd_rn(d.x[a], __dmul_rn(__dmul_rn(lam, dx), wa));
                d.y[a] = __dadd_rn(d.y[a], __dmul_rn(__dmul_rn(lam, dy), wa));
                d.z[a] = __dadd_rn(d.z[a], __dmul_rn(__dmul_rn(lam, dz), wa));
                d.x[b] = __dsub_rn(d.x[b], __dmul_rn(__dmul_rn(lam, dx), wb));
                d.y[b] = __dsub_rn(d.y[b], __dmul_rn(__dmul_rn(lam, dy), wb));
                d.z[b] = __dsub_rn(d.z[b], __dmul_rn(__dmul_rn(lam, dz), wb));
            }
        }
        if (worst < tol) break;
    }
    for (int q = q0; q < q1; ++q) {
        const int a = d.cgroup_atoms[q];
        const double x = d.x[a], y = d.y[a], z = d.z[a];
        if (phys) {
            d.vx[a] = __dadd_rn(d.vx[a], __dsub_rn(x, d.cons_x0[a]) / R.dt);
            d.vy[a] = __dadd_rn(d.vy[a], __dsub_rn(y, d.cons_x0[na + a]) / R.dt);
            d.vz[a] = __dadd_rn(d.vz[a], __dsub_rn(z, d.cons_x0[2 * na + a]) / R.dt);
        }
        write_mirror(d, d.slot_of_atom[a], a, x, y, z, L);
        skin_check(d, s, R, a, x, y, z);
    }
}

// Constraints::apply_rattle (constraints.cpp:49-91), after the second half
// kick: the same group sweeps on r.v, lambda = r.v / (r^2 (1/m_i + 1/m_j)).
__global__ void k_rattle(Dev d) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = g < d.n_cgroups;
    // only the velocities come from the kernel before it
    int r = 0, c0 = 0, c1 = 0;
    int3 at;
    bool tri = false, active = false;
    double L = 1.0, inv = 1.0, tol = 0.0;
    TriangleBonds tb;
    double w[3];
    if (in) {
        r = d.cgroup_rep[g];
        active = d.st[r].active != 0;
        L = d.st[r].L;
        inv = 1.0 / L;
        tol = d.rep[r].cons_tol;
        c0 = d.cgroup_begin[g];
        c1 = d.cgroup_begin[g + 1];
        tri = is_triangle(d, c0, c1, at);
    }
    const int id[3] = {at.x, at.y, at.z};
    if (tri) {
        double x[3], y[3], z[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            x[k] = d.x[id[k]];
            y[k] = d.y[id[k]];
            z[k] = d.z[id[k]];
            w[k] = 1.0 / d.mass[id[k]];
        }
        tb.set(x, y, z, w, L, inv);
    }
    chain_wait();
    if (!in || !active) return;
    if (tri) {
        double vx[3], vy[3], vz[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            vx[k] = d.vx[id[k]];
            vy[k] = d.vy[id[k]];
            vz[k] = d.vz[id[k]];
        }
        rattle_triangle(tb, vx, vy, vz, w, tol);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            d.vx[id[k]] = vx[k];
            d.vy[id[k]] = vy[k];
            d.vz[id[k]] = vz[k];
        }
        return;
    }
    for (int it = 0; it < 100; ++it) {
        double worst = 0.0;
        for (int c = c0; c < c1; ++c) {
            const int a = d.cons_ij[c].x, b = d.cons_ij[c].y;
            double dx = __dsub_rn(d.x[b], d.x[a]), dy = __dsub_rn(d.y[b], d.y[a]), dz = __dsub_rn(d.z[b], d.z[a]);
            dx = __dsub_rn(dx, __dmul_rn(round(__dmul_rn(dx, inv)), L));
            dy = __dsub_rn(dy, __dmul_rn(round(__dmul_rn(dy, inv)), L));
            dz = __dsub_rn(dz, __dmul_rn(round(__dmul_rn(dz, inv)), L));
            const double dvx = __dsub_rn(d.vx[b], d.vx[a]), dvy = __dsub_rn(d.vy[b], d.vy[a]),
                         dvz = __dsub_rn(d.vz[b], d.vz[a]);
            const double rv = __dadd_rn(__dadd_rn(__dmul_rn(dx, dvx), __dmul_rn(dy, dvy)), __dmul_rn(dz, dvz));
            const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
            const double e = fabs(rv);
            if (e > worst) worst = e;
            if (e > tol) {
                const double wa = 1.0 / d.mass[a], wb = 1.0 / d.mass[b];
                const double lam = rv / __dmul_rn(r2, __dadd_rn(wa, wb));
                d.vx[a] = __dadd_rn(d.vx[a], __dmul_rn(__dmul_rn(lam, dx), wa));
                d.vy[a] = __dadd_rn(d.vy[a], __dmul_rn(__dmul_rn(lam, dy), wa));
                d.vz[a] = __dadd_rn(d.vz[a], __dmul_rn(__dmul_rn(lam, dz), wa));
                d.vx[b] = __dsub_rn(d.vx[b], __dmul_rn(__dmul_rn(lam, dx), wb));
                d.vy[b] = __dsub_rn(d.vy[b], __dmul_rn(__dmul_rn(lam, dy), wb));
                d.vz[b] = __dsub_rn(d.vz[b], __dmul_rn(__dmul_rn(lam, dz), wb));
            }
        }
        if (worst < tol) break;
    }
}

// Per-tile kinetic-energy partials again after RATTLE (the thermostat reads the
// constrained velocities; same expression and order as k_kick2's).
__global__ void k_tile_ke(Dev d) {
    chain_wait();
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int t = slot >> 5;
    const int r = (t < d.n_tiles) ? d.tile_rep[t] : 0;
    double ke = 0.0;
    if (slot < d.n_slots && d.st[r].active) {
        const int a = d.atom_of_slot[slot];
        if (a >= 0) {
            const double m = d.mass[a], vx = d.vx[a], vy = d.vy[a], vz = d.vz[a];
            ke = __dmul_rn(__dmul_rn(0.5, m),
                           __dadd_rn(__dadd_rn(__dmul_rn(vx, vx), __dmul_rn(vy, vy)), __dmul_rn(vz, vz)));
        }
    }
    ke = warp_sum_d(ke);
    if (lane == 0 && t < d.n_tiles) d.tile_ke[t] = ke;
}

__device__ double block_sum(double v, double* sh) {
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    double r = sh[0];
    __syncthreads();
    return r;
}

// PME energy / virial partial sums of replica r (fixed order).
__device__ void reduce_pme(const Dev& d, int r, double* sh) {
    const Rep& R = d.rep[r];
    double e = 0.0, v = 0.0;
    if (R.flags & F_PME) {
        for (int b = threadIdx.x; b < R.pme_blocks; b += blockDim.x) {
            e += d.pme_part[2 * (R.pme_block_begin + b)];
            v += d.pme_part[2 * (R.pme_block_begin + b) + 1];
        }
    }
    e = block_sum(e, sh);
    v = block_sum(v, sh);
    if (threadIdx.x == 0) {
        d.st[r].e_recip = e;
        d.st[r].vir_recip = v;
    }
}

__global__ void k_energy_reduce(Dev d) {
    __shared__ double sh[256];
    const int r = blockIdx.x;
    if (!d.st[r].eval) return;
    reduce_pme(d, r, sh);
}

// Four block-wide sums at once in a fixed order: lane sums by shuffles, then
// the block's warps by warp 0 (256 or 512 threads; the warps beyond a
// replica's summing threads hold zeros, which leave its sums as they are).
__device__ void block_sum4(double v[4], double (*sh)[4]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = warp_sum_d(v[k]);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
        for (int k = 0; k < 4; ++k) sh[w][k] = v[k];
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        for (int k = 0; k < 4; ++k) {
            double x = (lane < nw) ? sh[lane][k] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(FULL, x, o);
            v[k] = x;
        }
    }
}

// Thermostat (berendsen.cpp:13-28, nose_hoover.cpp:6-32) and Berendsen barostat
// (berendsen_barostat.cpp:14-66); one block per replica.  Tile partials of KE
// and r.F and the PME blocks' energy / virial partials are summed together.
// With `next` the next step of the same launch begins here too (begin_step).
// In a chained launch only the tile partials come from the kernel before it:
// the replica's records and the PME partials are loaded before the wait.
__global__ void __launch_bounds__(512) k_replica_update(Dev d, int next) {
    __shared__ double sh[16][4];
    const int r = blockIdx.x;
    RepState* s = d.st + r;
    const Rep& R = d.rep[r];
    const bool active = s->active != 0;
    // Threads that sum: 256, or all 512 of a wide launch for a replica of many
    // tiles (by its own size, so its sums do not depend on what else is in the
    // table).  Water 750k, 23,438 tiles and 27,936 PME
    // partials (now 6,984): 59 -> 12 us.
    const int nt = R.n_tiles >= WIDE_TILES ? static_cast<int>(blockDim.x) : 256;
    const bool summing = static_cast<int>(threadIdx.x) < nt;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    RepState st;
    Rep Rr;
    if (active) {
        if ((R.flags & F_PME) && summing) {
            const double2* pp = reinterpret_cast<const double2*>(d.pme_part) + R.pme_block_begin;
            for (int b = threadIdx.x; b < R.pme_blocks; b += nt) {
                const double2 ev = pp[b];
                v[2] += ev.x;
                v[3] += ev.y;
            }
        }
        // one thread uses these: the replica's records copied to registers at
        // once (independent loads) and written back at the end
        if (threadIdx.x == 0) {
            st = *s;
            Rr = R;
        }
    }
    chain_wait();
    if (next && r == 0 && threadIdx.x == 0) reset_counters(d);
    if (!active) return;
    if (summing) {
#pragma unroll 4
        for (int t = R.tile_begin + threadIdx.x; t < R.tile_begin + R.n_tiles; t += nt) {
            v[0] += d.tile_ke[t];
            v[1] += d.tile_vir[t];
        }
    }
    block_sum4(v, sh);
    if (threadIdx.x != 0) return;
    const double ke = v[0], w = v[1];
    st.e_recip = v[2];
    st.vir_recip = v[3];
    // end of the step's second evaluation (k_eval_end's work, at the box it used)
    if (st.eval) {
        if (!(Rr.flags & F_PHYS) && (Rr.flags & F_LJ)) st.lj_counter += 1;
        st.have_forces = 1;
        if (Rr.flags & F_PME) st.green_L = st.L;
    }
    const double n = static_cast<double>(Rr.n_atoms);
    const double dt = Rr.dt;
    auto temp = [&](double ek) { return Rr.n_atoms < 2 ? 0.0 : 2.0 * ek / ((3.0 * n - 3.0) * KB); };
    double lam = 1.0;
    if (Rr.thermostat == 1) {
        if (Rr.t_tau > 0.0 && ke > 0.0) {
            const double T = temp(ke);
            const double l = sqrt(1.0 + dt / Rr.t_tau * (Rr.t_temp / T - 1.0));
            if (!(l <= 0.0)) lam = l;
        }
    } else if (Rr.thermostat == 2) {
        const double T = temp(ke);
        st.zeta += 0.5 * dt * KB * (T - Rr.t_temp) / Rr.nh_Q;
        lam = exp(-st.zeta * 0.5 * dt);
    } else if (Rr.thermostat == 3) {
        if (Rr.t_freq * dt > 0.0) st.andersen_calls += 1;
    }
    st.vscale = lam;
    const double ke_after = ke * lam * lam;
    st.ke = ke_after;
    const double L = st.L;
    const double V = L * (L * L);
    double W;
    if (Rr.flags & F_PHYS) W = from_fix(st.e_acc[E_VIR], ESCALE) + st.vir_recip;
    else W = w;
    st.virial = W;
    st.pressure = (V <= 0.0) ? 0.0 : (2.0 * ke_after + W) / (3.0 * V);
    if (Rr.barostat == 2 && V > 0.0) {
        // AndersenBarostat::apply (andersen_barostat.cpp:20-45), ref profile: half a
        // step of piston velocity from 3V (P - P0) / W (P0 in the reference's units),
        // positions and box scale by exp(eps_dot dt) (positions in k_apply_scale),
        // then the second half step with the same forcing
        const double forcing = 3.0 * V * (st.pressure - Rr.b_pressure) / Rr.piston_W;
        st.eps_dot = st.eps_dot + 0.5 * dt * forcing;
        const double sc = exp(st.eps_dot * dt);
        st.pscale = sc;
        st.L = L * sc;
        st.invL = 1.0 / st.L;
        st.eps_dot = st.eps_dot + 0.5 * dt * forcing;
    }
    if (Rr.barostat == 1 && Rr.b_tau > 0.0 && V > 0.0) {
        double mu;
        if (Rr.flags & F_PHYS) mu = 1.0 - (dt / Rr.b_tau) * Rr.b_compress * (Rr.b_pressure - st.pressure / BAR);
        else mu = 1.0 - (dt / Rr.b_tau) * (Rr.b_compress / BAR) * (Rr.b_pressure - st.pressure);
        if (mu <= 0.0) mu = 0.0;
        const double sc = cbrt(mu);
        st.pscale = sc;
        if (!(Rr.flags & F_PHYS)) {  // REF: positions and box scale now (k_apply_scale)
            st.L = L * sc;
            st.invL = 1.0 / st.L;
        }
    }
    st.step += 1;
    st.time += dt;
    if (next) begin_step(st, Rr, next == NEXT_SKIPS);
    *s = st;
}

// BerendsenBarostat position scaling (berendsen_barostat.cpp:60-65).
__global__ void k_apply_scale(Dev d) {
    chain_wait();
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= d.n_slots) return;
    const int r = d.tile_rep[slot >> 5];
    RepState* s = d.st + r;
    if (!s->active || s->pscale == 1.0) return;
    const int a = d.atom_of_slot[slot];
    if (a < 0) return;
    const double sc = s->pscale;
    const double x = d.x[a] * sc, y = d.y[a] * sc, z = d.z[a] * sc;
    d.x[a] = x;
    d.y[a] = y;
    d.z[a] = z;
    write_mirror(d, slot, a, x, y, z, s->L);
    skin_check(d, s, d.rep[r], a, x, y, z);
}

__global__ void k_finalize_v(Dev d) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= d.n_atoms) return;
    const double lam = d.st[d.atom_rep[a]].vscale;
    if (lam == 1.0) return;
    d.vx[a] = __dmul_rn(d.vx[a], lam);
    d.vy[a] = __dmul_rn(d.vy[a], lam);
    d.vz[a] = __dmul_rn(d.vz[a], lam);
}

// One replica's frame into a device staging buffer, without changing any
// state: [step, time, box, x[n], y[n], z[n], vx[n], vy[n], vz[n]], the
// velocities with the pending thermostat scale applied as k_finalize_v would.
__global__ void k_frame_snapshot(Dev d, int r, double* out) {
    const Rep& R = d.rep[r];
    const RepState& s = d.st[r];
    const int n = R.n_atoms;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        out[0] = static_cast<double>(s.step);
        out[1] = s.time;
        out[2] = s.L;
    }
    if (i >= n) return;
    const int a = R.atom_begin + i;
    const double lam = s.vscale;
    double* o = out + 3;
    o[i] = d.x[a];
    o[n + i] = d.y[a];
    o[2 * n + i] = d.z[a];
    o[3 * n + i] = lam == 1.0 ? d.vx[a] : __dmul_rn(d.vx[a], lam);
    o[4 * n + i] = lam == 1.0 ? d.vy[a] : __dmul_rn(d.vy[a], lam);
    o[5 * n + i] = lam == 1.0 ? d.vz[a] : __dmul_rn(d.vz[a], lam);
}

// n atoms from a0 on into host memory that the device can write (pinned): which
// 0 positions, 1 velocities with the pending thermostat scale applied as
// k_finalize_v would (no state is changed), 2 forces; rows: [n][3], otherwise
// three arrays `stride` apart.  256 threads per block; rows go through shared
// memory, so that the block writes its 6 KB contiguously (stores of 8 bytes
// every 24 left the link half empty: 30,000 atoms 33 -> 18 us).
__global__ void k_export_state(Dev d, int a0, int n, int which, int rows, long long stride, double* out) {
    __shared__ double s_row[768];
    const int i = blockIdx.x * 256 + threadIdx.x;
    double v[3] = {0.0, 0.0, 0.0};
    if (i < n) {
        const int a = a0 + i;
        if (which == 0) {
            v[0] = d.x[a];
            v[1] = d.y[a];
            v[2] = d.z[a];
        } else if (which == 1) {
            const double lam = d.st[d.atom_rep[a]].vscale;
            v[0] = lam == 1.0 ? d.vx[a] : __dmul_rn(d.vx[a], lam);
            v[1] = lam == 1.0 ? d.vy[a] : __dmul_rn(d.vy[a], lam);
            v[2] = lam == 1.0 ? d.vz[a] : __dmul_rn(d.vz[a], lam);
        } else {
            const int s = d.slot_of_atom[a];
            v[0] = from_fix(d.fbx[a] + d.fnx[s], FSCALE);
            v[1] = from_fix(d.fby[a] + d.fny[s], FSCALE);
            v[2] = from_fix(d.fbz[a] + d.fnz[s], FSCALE);
        }
    }
    if (!rows) {
        if (i < n)
            for (int c = 0; c < 3; ++c) out[c * stride + i] = v[c];
        return;
    }
    for (int c = 0; c < 3; ++c) s_row[3 * threadIdx.x + c] = v[c];
    __syncthreads();
    const long long o = 768LL * blockIdx.x, left = 3LL * n - o;
    for (int k = 0; k < 3; ++k) {
        const int e = 256 * k + threadIdx.x;
        if (e < left) out[o + e] = s_row[e];
    }
}

// The reverse for replica r's positions (0: its list and forces are then due)
// and velocities (1: any pending thermostat scale is dropped with the old ones).
__global__ void k_import_state(Dev d, int r, int a0, int n, int which, int rows, long long stride, const double* in) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i == 0) {
        if (which == 0) {
            d.st[r].rebuild = 1;
            d.st[r].have_forces = 0;
        } else {
            d.st[r].vscale = 1.0;
        }
    }
    if (i >= n) return;
    double v[3];
    for (int c = 0; c < 3; ++c) v[c] = in[rows ? 3LL * i + c : c * stride + i];
    const int a = a0 + i;
    double* x = which == 0 ? d.x : d.vx;
    double* y = which == 0 ? d.y : d.vy;
    double* z = which == 0 ? d.z : d.vz;
    x[a] = v[0];
    y[a] = v[1];
    z[a] = v[2];
}

__global__ void k_request_rebuild(Dev d, int r) { d.st[r].rebuild = 1; }

__global__ void k_finalize_reset(Dev d) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < d.n_rep) d.st[r].vscale = 1.0;
}

__global__ void k_write_mirror(Dev d) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= d.n_slots) return;
    const int a = d.atom_of_slot[slot];
    if (a < 0) return;
    const int r = d.tile_rep[slot >> 5];
    write_mirror(d, slot, a, d.x[a], d.y[a], d.z[a], d.st[r].L);
}

}  // namespace

void launch_eval_begin(const Dev& d, int pass, cudaStream_t st, long long* n) {
    launch_chained(k_eval_begin, (d.n_rep + 127) / 128, 128, st, d, pass);
    ++*n;
}
void launch_mark_read(const Dev& d, int n_steps, cudaStream_t st, long long* n) {
    k_mark_read<<<(d.n_rep + 127) / 128, 128, 0, st>>>(d, n_steps);
    ++*n;
}
void launch_clear_forces(const Dev& d, cudaStream_t st, long long* n) {
    const int m = d.n_slots > d.n_atoms ? d.n_slots : d.n_atoms;
    launch_chained(k_clear_forces, (m + 255) / 256, 256, st, d);
    ++*n;
}
void launch_eval_end(const Dev& d, cudaStream_t st, long long* n) {
    launch_chained(k_eval_end, (d.n_rep + 127) / 128, 128, st, d);
    ++*n;
}
void launch_kick_drift(const Dev& d, bool, cudaStream_t st, long long* n) {
    launch_chained(k_kick_drift, (d.n_atoms + 255) / 256, 256, st, d);
    ++*n;
}
void launch_kick2(const Dev& d, bool andersen_ref, bool andersen_phys, bool chained, cudaStream_t st, long long* n) {
    const int g = (d.n_slots + 255) / 256, ar = andersen_ref ? 1 : 0, ap = andersen_phys ? 1 : 0;
    if (chained) launch_chained(k_kick2, g, 256, st, d, ar, ap);
    else k_kick2<<<g, 256, 0, st>>>(d, ar, ap);
    ++*n;
}
void launch_shake(const Dev& d, cudaStream_t st, long long* n) {
    launch_chained(k_shake, (d.n_cgroups + 63) / 64, 64, st, d);
    ++*n;
}
void launch_rattle(const Dev& d, cudaStream_t st, long long* n) {
    launch_chained(k_rattle, (d.n_cgroups + 63) / 64, 64, st, d);
    launch_chained(k_tile_ke, (d.n_slots + 255) / 256, 256, st, d);
    *n += 2;
}
void launch_replica_update(const Dev& d, int next, cudaStream_t st, long long* n) {
    launch_chained(k_replica_update, d.n_rep, d.any_wide ? 512 : 256, st, d, next);
    ++*n;
}
void launch_apply_scale(const Dev& d, bool, cudaStream_t st, long long* n) {
    launch_chained(k_apply_scale, (d.n_slots + 255) / 256, 256, st, d);
    ++*n;
}
void launch_finalize_velocities(const Dev& d, cudaStream_t st, long long* n) {
    k_finalize_v<<<(d.n_atoms + 255) / 256, 256, 0, st>>>(d);
    k_finalize_reset<<<(d.n_rep + 127) / 128, 128, 0, st>>>(d);
    *n += 2;
}
void launch_frame_snapshot(const Dev& d, int r, int n_atoms, double* out, cudaStream_t st, long long* n) {
    k_frame_snapshot<<<(n_atoms + 255) / 256, 256, 0, st>>>(d, r, out);
    ++*n;
}
void launch_export_state(const Dev& d, int a0, int n, int which, bool rows, long long stride, double* out,
                         cudaStream_t st, long long* nl) {
    k_export_state<<<(n + 255) / 256, 256, 0, st>>>(d, a0, n, which, rows ? 1 : 0, stride, out);
    ++*nl;
}
void launch_import_state(const Dev& d, int r, int a0, int n, int which, bool rows, long long stride, const double* in,
                         cudaStream_t st, long long* nl) {
    k_import_state<<<(n + 255) / 256, 256, 0, st>>>(d, r, a0, n, which, rows ? 1 : 0, stride, in);
    ++*nl;
}
void launch_request_rebuild(const Dev& d, int r, cudaStream_t st, long long* n) {
    k_request_rebuild<<<1, 1, 0, st>>>(d, r);
    ++*n;
}
void launch_energy_reduce(const Dev& d, cudaStream_t st, long long* n) {
    k_energy_reduce<<<d.n_rep, 256, 0, st>>>(d);
    ++*n;
}
void launch_write_mirror(const Dev& d, bool, cudaStream_t st, long long* n) {
    k_write_mirror<<<(d.n_slots + 255) / 256, 256, 0, st>>>(d);
    ++*n;
}

}  // namespace dmd
