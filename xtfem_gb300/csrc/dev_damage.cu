// dev_damage.cu -- per-Gauss-point two-scale fatigue damage on the GPU.
//
// Implements the update of src/kokkos_kernel.h:45-344 (constants
// src/damage.h:9-17): for every spatial Gauss point and every temporal
// interpolation point of the slab, interpolate the strain, run the elastic
// predictor and, when the trial von Mises stress exceeds sig_f, the plastic
// corrector with stored energy ws and damage D, all state in FP64.  A thread
// screens the steps of one Gauss point; a point that yields goes to a team of 8
// or 32 lanes of its warp, in the reference's formulas with regrouped sums.
//
// The reference spends 144 FMAs per step re-interpolating the displacement
// of the 8 nodes (src/kokkos_kernel.h:55-71).  The strain is linear in the
// six temporal shape values Nt_k(t), so each point first forms its six
// strain "basis" vectors E_k = B u_k once per slab; the strain at any step is
// then sum_k Nt_k(t) E_k.  In the elastic predictor the deviatoric trial
// stress is affine in the strain as long as the internal variables (D,
// eps_pl, sig_back) do not change, i.e. between plastic steps:
//     tsig(t) = sum_k Nt_k(t) G_k + C0
// with G_k = c1 * m .* dev(E_k), C0 = (c3-1) * m .* dev(eps_pl) - sig_back
// (m = 2 mu on the normal terms, mu on the engineering shears).  A step is
// elastic iff 1.5 sum_n tsig_n^2 + 3 sum_s tsig_s^2 <= sig_f^2.
//
// GB300's FP64 rate is a small fraction of its FP32 rate, so every step is
// first screened in FP32 with a rigorous rounding bound: a whole chunk of the
// table at once, then runs of steps, then single steps.  Steps the screen
// proves elastic change nothing but the "last elastic" markers (sig_eff,
// eps_old, sig_d are overwritten by every elastic step, so only the last one
// before a plastic step, or before the slab ends, has to be evaluated).
// A point's first step the screen cannot decide, and all that follow, are the
// team's (Team).
#include <cstdlib>
#include <mutex>

#include "xt_device.h"

namespace xt {

namespace {

// src/damage.h:9-17
constexpr double CY = 1740.0, HH = 0.2, SD = 0.5, SIGF = 180.0, SIGU = 577.0, EPSD = 0.08;
constexpr double WD = (SIGU - SIGF) * EPSD;
constexpr int kNtChunk = 1024;  // temporal points per shared-memory chunk
constexpr int kRun = 32;        // steps proven elastic by one bound

struct Mat {
    double nu, E, ca, cb, coef;
};

__device__ __forceinline__ double vm_equiv(const double s[6])
{
    double e = 0.0;
    for (int i = 0; i < 3; ++i) e += 1.5 * s[i] * s[i];
    for (int i = 3; i < 6; ++i) e += 3.0 * s[i] * s[i];
    return sqrt(e);
}

__device__ __forceinline__ void deviator(const double s[6], double o[6])
{
    double tr = 0.0;
    for (int i = 0; i < 3; ++i) tr += s[i];
    tr = tr / 3.0;
    o[0] = s[0] - tr; o[1] = s[1] - tr; o[2] = s[2] - tr;
    o[3] = s[3]; o[4] = s[4]; o[5] = s[5];
}

// D times a Voigt vector with the reference's 6x6 dmat
// (src/kokkos_kernel.h:81-92), summed in the reference's order
__device__ __forceinline__ void dmat_mul(const Mat& m, const double v[6], double o[6])
{
    const double off = m.coef * m.nu, dia = m.coef * (1.0 - m.nu);
    const double sh = m.coef * (1.0 - 2.0 * m.nu) / 2.0;
    for (int i = 0; i < 3; ++i) {
        double acc = 0.0;
        for (int j = 0; j < 3; ++j) acc += (i == j ? dia : off) * v[j];
        for (int j = 3; j < 6; ++j) acc += 0.0 * v[j];
        o[i] = acc;
    }
    for (int i = 3; i < 6; ++i) {
        double acc = 0.0;
        for (int j = 0; j < 6; ++j) acc += (j == i ? sh : 0.0) * v[j];
        o[i] = acc;
    }
}

// Elastic predictor of src/kokkos_kernel.h:96-160 in FP64 and reference
// order.  Returns the equivalent trial stress; tse receives D * tee.
__device__ double predictor(const Mat& m, double d, const double eps[6], const double epl[6],
                            const double sbk[6], double tse[6])
{
    const double c1 = 1.0 / (1.0 - m.cb * d);
    const double c2 = (m.ca - m.cb) * d / ((1.0 - m.cb * d) * (1.0 - m.ca * d));
    const double c3 = m.cb * (1.0 - d) / (1.0 - m.cb * d);
    double tel[6], tee[6], tdev[6], tsig[6];
    for (int i = 0; i < 6; ++i) tel[i] = c1 * eps[i] + c3 * epl[i];
    double tr = 0.0;
    for (int i = 0; i < 3; ++i) tr += eps[i];
    tr = c2 * tr / 3.0;
    for (int i = 0; i < 3; ++i) tel[i] += tr;
    for (int i = 0; i < 6; ++i) tee[i] = tel[i] - epl[i];
    dmat_mul(m, tee, tse);
    deviator(tse, tdev);
    for (int i = 0; i < 6; ++i) tsig[i] = tdev[i] - sbk[i];
    return vm_equiv(tsig);
}

struct State {
    double epo[6], epl[6], sef[6], sbk[6];
    double p, d, ws, dpo, sigd;
};

// Affine screen coefficients for the current internal state: G (6x6, FP32,
// G[k][i]), C0 (6, FP32) and the absolute rounding bound of the screened
// teq^2.
__device__ void screen_setup(const Mat& m, const State& st, const double E[6][6],
                             const float* __restrict__ ntmax, float G[6][6], float C0[6],
                             float& err2, float ecomp[6])
{
    const double d = st.d;
    const double c1 = 1.0 / (1.0 - m.cb * d);
    const double c3 = m.cb * (1.0 - d) / (1.0 - m.cb * d);
    const double mn = m.coef * (1.0 - 2.0 * m.nu), ms = mn / 2.0;
    double dv[6];
    double S[6];
    // a third by multiplication: the bound covers its rounding
    auto dev3 = [](const double* v, double* o) {
        const double t = (v[0] + v[1] + v[2]) * (1.0 / 3.0);
        for (int i = 0; i < 6; ++i) o[i] = i < 3 ? v[i] - t : v[i];
    };
    dev3(st.epl, dv);
    for (int i = 0; i < 6; ++i) {
        const double c0 = (c3 - 1.0) * (i < 3 ? mn : ms) * dv[i] - st.sbk[i];
        C0[i] = (float)c0;
        S[i] = fabs(c0);
    }
    for (int k = 0; k < 6; ++k) {
        double ed[6];
        dev3(E[k], ed);
        for (int i = 0; i < 6; ++i) {
            const double gk = c1 * (i < 3 ? mn : ms) * ed[i];
            G[k][i] = (float)gk;
            S[i] += (double)ntmax[k] * fabs(gk);
        }
    }
    // Each screened component sums 7 rounded products of rounded inputs;
    // 32 units of 2^-24 of the absolute sum S_i bounds its error e_i, and
    // teq^2 = sum w_i tsig_i^2 then errs by at most sum w_i (2 S_i e_i +
    // e_i^2) plus the rounding of the final sum (another 16 units).
    const double u = 32.0 * 5.9604644775390625e-8;
    double e2 = 0.0, tot = 0.0;
    for (int i = 0; i < 6; ++i) {
        const double w = i < 3 ? 1.5 : 3.0;
        const double ei = u * S[i];
        ecomp[i] = (float)(ei * 1.0001);
        e2 += w * (2.0 * S[i] * ei + ei * ei);
        tot += w * S[i] * S[i];
    }
    err2 = (float)(e2 + 16.0 * 5.9604644775390625e-8 * tot) * 1.0001f + 1e-30f;
}

// Everything the rare exact FP64 path needs lives in one per-thread record
// that only no-inline functions touch, so the FP32 screening loop keeps just
// its 43 coefficients in registers (occupancy, no spills in the hot loop).
struct Slow {
    Mat m;
    State st;
    double E[6][6];
};
struct Screen {
    float G[6][6];
    float C0[6];
    float e[6];  // bound on each screened component's error
    float err2;
};

__device__ __noinline__ void slow_screen(const Slow* s, const float* __restrict__ ntmax, Screen* sc)
{
    screen_setup(s->m, s->st, s->E, ntmax, sc->G, sc->C0, sc->err2, sc->e);
}

__device__ __forceinline__ void strain_at(const Slow* s, const double* __restrict__ Nt, int jj,
                                          double eps[6])
{
    const double* ntr = Nt + (size_t)jj * 6;
    double w[6];
    for (int k = 0; k < 6; ++k) w[k] = ntr[k];
    for (int c = 0; c < 6; ++c) {
        double acc = 0.0;
        for (int k = 0; k < 6; ++k) acc = fma(w[k], s->E[k][c], acc);
        eps[c] = acc;
    }
}

// outputs of an elastic step (sig_eff, eps_old, sig_d), reference order
__device__ __noinline__ void slow_materialize(Slow* s, const double* __restrict__ Nt, int jj)
{
    double eps[6], tse[6];
    strain_at(s, Nt, jj, eps);
    const double teq = predictor(s->m, s->st.d, eps, s->st.epl, s->st.sbk, tse);
    for (int i = 0; i < 6; ++i) { s->st.sef[i] = tse[i]; s->st.epo[i] = eps[i]; }
    s->st.sigd = teq;
}

// ---------------------------------------------------------------------------
// Exact steps of one point by a team of L lanes of a warp.
//
// This part takes an FP64 instruction of one warp in 64 cycles whatever its
// live lanes, so a point's chain of plastic steps costs its FP64 instruction
// count: one thread doing the six components in turn took about 940 of them a
// step (29 us).  Here lane i < 6 of a team holds component i of every tensor,
// lane 6 the mean of every tensor as a component of its own (the predictor
// and the corrector act on the mean as on a component, so no trace is ever
// summed), and the scalars are held by all: about
// 87 instructions a plastic step without damage growth, 131 with it.  The
// factors of the damage (four quotients) are formed by four lanes in one
// division, and again only when the damage has changed.  A team's L lanes
// screen L steps at once between plastic phases.
//
// The formulas are those of src/kokkos_kernel.h:96-341 with the sums regrouped
// (c5 = 1 + gam dp / SIGF is qeq / SIGF; the deviator of D tee is
// a (tee - mean)); everything in FP64.
//
// Measured (GB300, against one thread a point): a slab of 25,600 steps on
// 192,000 points, displacement amplitudes of 115 MPa at other seeds, 122 to 159
// -> 21.2 to 26 ms; 1,536 points, 2,560 steps, host arrays, 31 to 33 -> 5.6 ms;
// no plastic point (192,000 points, 25,600 steps) 2.1 -> 0.45 ms, from the chunk
// bound and fused sums; every point of 24,000 yielding, 1,024 steps, 14.6 -> 11.4
// ms, with their damage growing 16.5 -> 16.0.
//
// L = 32 for a warp's only point that needs exact steps (32 steps a screening
// pass), else L = 8 (four points a warp, each FP64 instruction serving four; two
// points one after the other with L = 32 took 569 points of a 10 x 10 x 30 rod
// 8.3 ms in place of 4.9, 726 of a 14 x 14 x 40 one 11.9 in place of 6.7).  The
// teams of a warp run in step: every branch below is taken by the whole warp
// (a vote), and a team that does not take part keeps its values.
template <int L>
struct Team {
    // lane constants: elastic coefficients, weight in the equivalent stress,
    // share of the mean (shear 0, else 1)
    double a, off, w, nrm;
    double cb, ca, cacb, kb3, g3;     // factors of the moduli (load)
    double cden;                      // the coefficient of d in the lane's quotient of factors()
    double ky, kn;                    // (1 + nu) / 2E and 9 nu / 2E, divided by SD
    double E[6];                      // strain basis of the lane's component
    double epo, epl, sef, sbk;        // the lane's components
    double p, d, ws, dpo, sigd;       // the point's scalars
    double sold;                      // |sigd - SIGF|
    double c1, c3m1, c2i, Ai, Bi, rgam, cyd, hx2;  // factors of d
    float g[6][6], c0[6], err2;       // FP32 screen of the whole point
    double sumg;                      // sum_k ntmax_k |g_k| of the lane's component
    unsigned mask;
    int lane;

    __device__ __forceinline__ double get(double v, int src) const { return __shfl_sync(mask, v, src, L); }
    // a condition of any of the warp's teams (L = 32: of the one team)
    static __device__ __forceinline__ bool any(bool c) { return L == 32 ? c : __any_sync(0xffffffffu, c) != 0; }
    // sum over lanes 0..7 of the team
    __device__ __forceinline__ double sum8(double v) const
    {
        v += __shfl_xor_sync(mask, v, 4, L);
        v += __shfl_xor_sync(mask, v, 2, L);
        v += __shfl_xor_sync(mask, v, 1, L);
        return L == 8 ? v : get(v, 0);
    }

    __device__ void load(const DamageArgs& A, int gp)
    {
        const int i = lane;
        const double Ey = A.ym[gp], nu = A.nu[gp];
        ca = (1.0 + nu) / (3.0 * (1.0 - nu));
        cb = 2.0 * (4.0 - 5.0 * nu) / (15.0 * (1.0 - nu));
        cacb = ca - cb;
        g3 = 3.0 * (Ey / (2.0 * (1.0 + nu))) * (1.0 - cb);
        cden = i == 0 ? cb : (i == 1 ? ca : HH);
        ky = (1.0 + nu) / (2.0 * Ey) * (1.0 / SD);
        kn = 9.0 * (nu / (2.0 * Ey)) * (1.0 / SD);
        const double coef = Ey / ((1.0 + nu) * (1.0 - 2.0 * nu)), mn = coef * (1.0 - 2.0 * nu);
        const bool shear = i >= 3 && i < 6, norm = i < 3 || i == 6;  // normal component or mean
        a = shear ? 0.5 * mn : (norm ? mn : 0.0);
        off = norm ? 3.0 * coef * nu : 0.0;
        w = i < 3 ? 1.5 : (shear ? 3.0 : 0.0);
        nrm = norm ? 1.0 : 0.0;
        kb3 = norm ? Ey / (1.0 - 2.0 * nu) : 0.0;
        // component i of the strain rows: N_a u_x (+ N_b u_y for a shear)
        const double* Na = (i == 0 ? A.Nx : (i == 1 || i == 3 ? A.Ny : A.Nz)) + (size_t)gp * A.nnse;
        const double* Nb = (i == 4 ? A.Ny : A.Nx) + (size_t)gp * A.nnse;
        const int ux = i == 1 || i == 4 ? 1 : (i == 2 ? 2 : 0), uy = i == 3 ? 1 : 2;
        for (int k = 0; k < 6; ++k) E[k] = 0.0;
        if (i < 6)
            for (int n = 0; n < A.nnse; ++n) {
                const double* u = A.sol + (size_t)(A.nodes[(size_t)gp * A.nnse + n] - 1) * 3;
                const double na = Na[n], nb = shear ? Nb[n] : 0.0;
                for (int k = 0; k < 6; ++k) {
                    const double* uk = u + (size_t)k * A.nn * 3;
                    E[k] = fma(na, uk[ux], fma(nb, uk[uy], E[k]));
                }
            }
        const size_t b6 = (size_t)gp * A.ncmp + (i < 6 ? i : 0);
        epo = i < 6 ? A.eps_old[b6] : 0.0;
        epl = i < 6 ? A.eps_pl[b6] : 0.0;
        sef = i < 6 ? A.sig_eff[b6] : 0.0;
        sbk = i < 6 ? A.sig_back[b6] : 0.0;
        auto mean = [&](double& v) {
            const double t = (get(v, 0) + get(v, 1) + get(v, 2)) / 3.0;
            if (i == 6) v = t;
        };
        for (int k = 0; k < 6; ++k) mean(E[k]);
        mean(epo);
        mean(epl);
        mean(sef);
        mean(sbk);
        p = A.p[gp];
        d = A.D[gp];
        ws = A.ws[gp];
        dpo = A.del_po[gp];
        sigd = A.sig_d[gp];
        sold = fabs(sigd - SIGF);
    }

    // the factors of d: 1 / (1 - cb d), 1 / (1 - ca d), (1 - d) / (1 - H d) and
    // 1 / gam = (1 - cb d) / (CY (1 - d)(1 - cb d) + 3 G (1 - cb)), one division
    // in lanes 0..3
    __device__ __forceinline__ void factors()
    {
        const double omd = 1.0 - d, ncb = fma(-cb, d, 1.0), own = fma(-cden, d, 1.0);
        const double gd = fma(CY * omd, ncb, g3);
        const double quo = (lane == 2 ? omd : (lane == 3 ? ncb : 1.0)) / (lane == 3 ? gd : own);
        const double r1 = get(quo, 0), ra = get(quo, 1), x = get(quo, 2);
        rgam = get(quo, 3);
        c1 = r1;
        c3m1 = fma(cb * omd, r1, -1.0);
        const double c2 = cacb * d * r1 * ra;
        c2i = c2 * nrm;
        Ai = a * r1;
        Bi = fma(off, r1, kb3 * c2);
        cyd = (2.0 * CY / 3.0) * omd;
        hx2 = HH * x * x;
    }

    // screen coefficients of the strain basis (they change with d), then of
    // the internal variables; the bounds are those of screen_setup
    __device__ void screen_basis(const float* __restrict__ ntmax)
    {
        sumg = 0.0;
        for (int k = 0; k < 6; ++k) {
            const double gk = c1 * a * fma(-nrm, get(E[k], 6), E[k]);
            sumg = fma((double)__ldg(ntmax + k), fabs(gk), sumg);
            const float f = (float)gk;
#pragma unroll
            for (int i = 0; i < 6; ++i) g[k][i] = __shfl_sync(mask, f, i, L);
        }
    }
    __device__ __forceinline__ void screen_state()
    {
        const double c = fma(c3m1 * a, fma(-nrm, get(epl, 6), epl), -sbk);
        const float f = (float)c;
#pragma unroll
        for (int i = 0; i < 6; ++i) c0[i] = __shfl_sync(mask, f, i, L);
        const double S = fabs(c) + sumg;
        const double tot = sum8(w * S * S);
        const double u = 32.0 * 5.9604644775390625e-8;
        err2 = (float)(tot * (2.0 * u + u * u + 16.0 * 5.9604644775390625e-8)) * 1.0001f + 1e-30f;
    }
    // teq^2 of step j in FP32
    __device__ __forceinline__ float screen(const float2* __restrict__ nt2, int j) const
    {
        const float2 t0 = __ldg(nt2 + 3 * (size_t)j), t1 = __ldg(nt2 + 3 * (size_t)j + 1),
                     t2 = __ldg(nt2 + 3 * (size_t)j + 2);
        const float wv[6] = {t0.x, t0.y, t1.x, t1.y, t2.x, t2.y};
        float q = 0.0f;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            float acc = c0[i];
#pragma unroll
            for (int k = 0; k < 6; ++k) acc = fmaf(wv[k], g[k][i], acc);
            q = fmaf(i < 3 ? 1.5f : 3.0f, acc * acc, q);
        }
        return q;
    }

    __device__ __forceinline__ double strain(const double nt[6]) const
    {
        double e = nt[0] * E[0];
#pragma unroll
        for (int k = 1; k < 6; ++k) e = fma(nt[k], E[k], e);
        return e;
    }
    // elastic predictor: the trial elastic strain, its mean and teq^2
    __device__ __forceinline__ double predict(double eps, double& tee, double& tm) const
    {
        tee = fma(c2i, get(eps, 6), fma(c3m1, epl, c1 * eps));
        tm = get(tee, 6);
        const double ts = fma(a, fma(-nrm, tm, tee), -sbk);
        return sum8(w * ts * ts);
    }
    // outputs of an elastic step
    __device__ __forceinline__ void elastic(double eps, double tee, double tm, double q, bool take)
    {
        const double s = fma(off, tm, a * tee), t = sqrt(q);
        if (L == 32 || take) {
            sef = s;
            epo = eps;
            sigd = t;
            sold = fabs(t - SIGF);
        }
    }
    // plastic corrector; returns whether d changed
    __device__ __forceinline__ bool correct(double eps, bool part)
    {
        const bool take = L == 32 || part;
        const double de = eps - epo;
        const double qs = sbk - sef - fma(Ai, de, Bi * get(de, 6));
        // The mean of qs, the same number here and below: with a trace and a
        // third by multiplication, always too small, and a common factor for dsg
        // a chain of steps ended with 1.9 times the error of p and 1.4 times that
        // of the stresses that the reference's sequence has; this has 0.85 to 1.
        const double qm = get(qs, 6);
        const double dq = fma(-nrm, qm, qs);
        const double q2 = sum8(w * dq * dq);
        // qeq = sqrt(q2), and its reciprocal: one Newton step on q2 rsqrt(q2)
        const double rq = rsqrt(q2);
        double qeq = q2 * rq;
        qeq = fma(fma(-qeq, qeq, q2), 0.5 * rq, qeq);
        const double dp = (qeq - SIGF) * rgam;
        // dsg = -SIGF dq / qeq, each component's quotient corrected once
        const double q0 = dq * (SIGF * rq);
        const double dsg = -fma(fma(-qeq, q0, SIGF * dq), rq, q0);
        const double k1 = dp * (1.5 / SIGF);
        const double nepl = fma(dsg, k1, epl);
        const double nsbk = fma(dsg, k1 * cyd, sbk);
        const double nsef = fma(-nrm, qm, dsg) + nsbk;
        // the equivalent stress, and the damage rate's square where it may be
        // needed: both sums in one butterfly (lanes 0..3 the one, 4..7 the
        // other) and both roots in one
        const double m2 = get(nsef, 6);
        const double sd = fma(-nrm, m2, nsef);
        const double v = w * sd * sd;
        double seq, rate = 0.0;
        if (any(take && ws >= WD)) {
            const double y = lane < 3 ? (nsef < 0.0 ? hx2 : 1.0) * nsef * nsef : 0.0;
            const bool up = (lane & 4) != 0;
            double t = (up ? y : v) + __shfl_xor_sync(mask, up ? v : y, 4, L);
            t += __shfl_xor_sync(mask, t, 2, L);
            t += __shfl_xor_sync(mask, t, 1, L);
            const double yn = kn * (m2 >= 0.0 ? 1.0 : hx2) * m2 * m2;
            const double root = sqrt(up ? fma(ky, t, -yn) : t);
            seq = get(root, 0);
            rate = get(root, 4);
        } else {
            seq = sqrt(sum8(v));
        }
        const double snew = fabs(seq - SIGF);
        const double nws = fma(fma(snew, dp, sold * dpo), 0.5, ws);
        const bool grow = take && nws >= WD;
        if (any(grow && ws < WD)) {  // the step that crosses the threshold
            const double sp = sum8(lane < 3 ? (nsef < 0.0 ? hx2 : 1.0) * nsef * nsef : 0.0);
            const double yn = kn * (m2 >= 0.0 ? 1.0 : hx2) * m2 * m2;
            const double r = sqrt(fma(ky, sp, -yn));
            if (ws < WD) rate = r;
        }
        // (the exponent of the damage law, src/damage.h:15, is 1/2)
        const double nd = grow ? fma(rate, dp, d) : 0.0;
        const bool changed = take && nd != d;
        if (take) {
            p += dp;
            epl = nepl;
            sbk = nsbk;
            sef = nsef;
            ws = nws;
            d = nd;
            epo = eps;
            sigd = seq;
            sold = snew;
            dpo = dp;
        }
        return changed;
    }
};

// A step's six shape values, the same for the whole team.
__device__ __forceinline__ void shape_row(const double* __restrict__ Nt, int j, double nt[6])
{
    // a caller's table is aligned to 8 bytes only
#pragma unroll
    for (int k = 0; k < 6; ++k) nt[k] = __ldg(Nt + (size_t)j * 6 + k);
}

// The slab's remaining steps of the warp's points in `todo` (one bit a lane:
// the lane's point gp, from its step from, its last proven step last) by
// teams of L lanes, 32 / L points at a time.
template <int L>
__device__ __noinline__ void exact_points(const DamageArgs& A, const float* __restrict__ ntmax,
                                          unsigned todo, int gp_lane, int from_lane, int last_lane)
{
    constexpr int TEAMS = 32 / L;
    constexpr int kPasses = L == 32 ? 4 : 8;  // screening passes between two exact steps of other teams
    const unsigned full = 0xffffffffu;
    const float thr = (float)(SIGF * SIGF) * 0.99999976f;
    const int wl = threadIdx.x & 31, team = wl / L;
    const float2* nt2 = reinterpret_cast<const float2*>(A.Nt32);
    while (todo) {
        // the team's point: the team-th bit of todo (none: the team idles on
        // the first one's data and stores nothing)
        unsigned m = todo;
        int src = __ffs(todo) - 1;
        bool on = false;
        for (int t = 0; t < TEAMS; ++t) {
            const int b = m ? __ffs(m) - 1 : -1;
            if (t == team && b >= 0) {
                src = b;
                on = true;
            }
            if (b >= 0) m &= m - 1;
        }
        todo = m;
        const int gp = __shfl_sync(full, gp_lane, src);
        int jj = __shfl_sync(full, from_lane, src), last = __shfl_sync(full, last_lane, src);
        if (!on) jj = A.nip;
        Team<L> T;
        T.mask = L == 32 ? full : (0xffu << (wl & ~7));
        T.lane = wl % L;
        T.load(A, gp);
        T.factors();
        T.screen_basis(ntmax);
        T.screen_state();
        bool stale = false, fresh_basis = true;
        unsigned n_exact = 0, n_plastic = 0;
        // the first unproven step is exact; nt holds step jj's shape values
        // while the team is at an exact step
        bool exact = on;
        double nt[6];
        shape_row(A.Nt, on ? jj : 0, nt);
        while (Team<L>::any(jj < A.nip)) {
            // screening: L steps a pass, until a step is not proven
            for (int pass = 0; pass < kPasses; ++pass) {
                const bool scan = jj < A.nip && !exact && !stale;
                if (!Team<L>::any(scan)) break;
                bool fail = false;
                if (scan && jj + T.lane < A.nip) fail = !(T.screen(nt2, jj + T.lane) + T.err2 < thr);
                const unsigned b = (__ballot_sync(full, fail) & T.mask) >> (L == 32 ? 0 : (wl & ~7));
                if (scan) {
                    const int f = b ? __ffs(b) - 1 : min(L, A.nip - jj);
                    if (f > 0) last = jj + f - 1;
                    jj += f;
                    exact = b != 0;
                    if (exact) shape_row(A.Nt, jj, nt);
                }
            }
            const bool act = jj < A.nip && (exact || stale);
            if (!Team<L>::any(act)) continue;
            double nx[6];  // the next step's shape values, loaded meanwhile
            shape_row(A.Nt, min(jj + 1, A.nip - 1), nx);
            const double eps = T.strain(nt);
            double tee, tm;
            const double q = T.predict(eps, tee, tm);
            const bool plastic = act && !(q <= SIGF * SIGF);
            if (act) ++n_exact;
            // a plastic step after proven ones: their last one's outputs first
            const bool pend = plastic && last >= 0;
            if (Team<L>::any(pend)) {
                double lt[6], le_tee, le_tm;
                shape_row(A.Nt, last >= 0 ? last : 0, lt);
                const double le = T.strain(lt);
                const double lq = T.predict(le, le_tee, le_tm);
                T.elastic(le, le_tee, le_tm, lq, pend);
            }
            if (Team<L>::any(act && !plastic)) T.elastic(eps, tee, tm, q, act && !plastic);
            bool dch = false;
            if (Team<L>::any(plastic)) {
                dch = T.correct(eps, plastic);
                if (plastic) ++n_plastic;
                if (Team<L>::any(dch)) T.factors();
                if (dch) fresh_basis = false;
            }
            // the screen is rebuilt once a plastic phase has ended
            const bool rebuild = act && !plastic && stale;
            if (Team<L>::any(rebuild)) {
                if (Team<L>::any(rebuild && !fresh_basis)) {
                    T.screen_basis(ntmax);
                    if (rebuild) fresh_basis = true;
                }
                T.screen_state();
            }
            if (act) {
                stale = plastic;
                exact = false;
                last = -1;
                ++jj;
#pragma unroll
                for (int k = 0; k < 6; ++k) nt[k] = nx[k];
            }
        }
        // outputs of the last proven step
        if (Team<L>::any(last >= 0)) {
            double lt[6], tee, tm;
            shape_row(A.Nt, last >= 0 ? last : 0, lt);
            const double le = T.strain(lt);
            const double lq = T.predict(le, tee, tm);
            T.elastic(le, tee, tm, lq, last >= 0);
        }
        if (on) {
            const int i = T.lane;
            const size_t b6 = (size_t)gp * A.ncmp;
            if (i < 6) {
                A.eps_old[b6 + i] = T.epo;
                A.eps_pl[b6 + i] = T.epl;
                A.sig_eff[b6 + i] = T.sef;
                A.sig_back[b6 + i] = T.sbk;
            }
            if (i == 0) {
                const bool gone = A.gpsta && A.gpsta[gp] == 0;  // src/kokkos_damage.f90:102-107
                A.p[gp] = T.p;
                A.D[gp] = gone ? 0.0 : T.d;
                A.ws[gp] = gone ? 0.0 : T.ws;
                A.del_po[gp] = T.dpo;
                A.sig_d[gp] = T.sigd;
                if (A.counters) {
                    atomicAdd(&A.counters[0], (unsigned long long)n_plastic);
                    atomicAdd(&A.counters[1], (unsigned long long)A.nip - n_exact);
                    atomicAdd(&A.counters[2], (unsigned long long)n_exact);
                }
            }
        }
    }
}

// The larger of two numbers; NaN when one of them is.
__device__ __forceinline__ float nan_max(float m, float v) { return v > m || v != v ? v : m; }

// The slab's update of point gidx.  A thread without a point (gidx past the
// last one) loads and screens nothing: it is there for the barriers of the chunk
// loop and the warp's votes.
__device__ __forceinline__ void damage_point(const DamageArgs& a, const float* __restrict__ ntmax,
                                             int run_bound, long long gidx)
{
    const bool live = gidx < a.ngp;
    const int gp = live ? (int)gidx : 0;
    Slow s;
    State& st = s.st;
    const size_t b6 = (size_t)gp * a.ncmp;
    float G[6][6] = {}, C0[6] = {}, ecomp[6] = {}, err2 = 0.0f;
    if (live) {
        Mat& m = s.m;
        m.nu = a.nu[gp];
        m.E = a.ym[gp];
        m.ca = (1.0 + m.nu) / (3.0 * (1.0 - m.nu));
        m.cb = 2.0 * (4.0 - 5.0 * m.nu) / (15.0 * (1.0 - m.nu));
        m.coef = m.E / ((1.0 + m.nu) * (1.0 - 2.0 * m.nu));

        // strain basis E_k = B u_k (6 temporal blocks, checked on the host)
        for (int k = 0; k < 6; ++k)
            for (int c = 0; c < 6; ++c) s.E[k][c] = 0.0;
        for (int i = 0; i < a.nnse; ++i) {
            const int nd = a.nodes[(size_t)gp * a.nnse + i] - 1;
            const double nx = a.Nx[(size_t)gp * a.nnse + i];
            const double ny = a.Ny[(size_t)gp * a.nnse + i];
            const double nz = a.Nz[(size_t)gp * a.nnse + i];
            for (int k = 0; k < 6; ++k) {
                const double* u = a.sol + (size_t)k * a.nn * a.ndofn + (size_t)nd * a.ndofn;
                const double u0 = u[0], u1 = u[1], u2 = u[2];
                s.E[k][0] = fma(nx, u0, s.E[k][0]);
                s.E[k][1] = fma(ny, u1, s.E[k][1]);
                s.E[k][2] = fma(nz, u2, s.E[k][2]);
                s.E[k][3] = fma(ny, u0, fma(nx, u1, s.E[k][3]));
                s.E[k][4] = fma(nz, u1, fma(ny, u2, s.E[k][4]));
                s.E[k][5] = fma(nz, u0, fma(nx, u2, s.E[k][5]));
            }
        }
        for (int i = 0; i < 6; ++i) {
            st.epo[i] = a.eps_old[b6 + i];
            st.epl[i] = a.eps_pl[b6 + i];
            st.sef[i] = a.sig_eff[b6 + i];
            st.sbk[i] = a.sig_back[b6 + i];
        }
        st.p = a.p[gp];
        st.d = a.D[gp];
        st.ws = a.ws[gp];
        st.dpo = a.del_po[gp];
        st.sigd = a.sig_d[gp];

        Screen sc;
        slow_screen(&s, ntmax, &sc);
#pragma unroll
        for (int k = 0; k < 6; ++k)
#pragma unroll
            for (int i = 0; i < 6; ++i) G[k][i] = sc.G[k][i];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            C0[i] = sc.C0[i];
            ecomp[i] = sc.e[i];
        }
        err2 = sc.err2;
    }
    // proven elastic when q + err2 < sig_f^2 (margin covers the float add)
    const float thr = (float)(SIGF * SIGF) * 0.99999976f;
    int last_el = -1;  // last step known elastic whose outputs are pending
    int first = -1;    // first step the screen does not prove elastic
    // The FP32 shape table is shared by every point: the block streams it
    // through shared memory in chunks, so each step's six values are a
    // broadcast shared-memory read instead of an L2 round trip.
    __shared__ float2 sNt[3 * kNtChunk];
    __shared__ float sDel[kNtChunk / kRun][6];
    const float2* nt2 = reinterpret_cast<const float2*>(a.Nt32);
    for (int j0 = 0; j0 < a.nip; j0 += kNtChunk) {
    const int jn = min(kNtChunk, a.nip - j0);
    // One bound for the whole chunk first: |tsig_i| <= |C0_i| + e_i + sum_k
    // mx_k |g_ki| with mx_k the chunk's largest |Nt_k|, inflated as the run
    // bound below.  Most points (stress well under yield) need nothing else,
    // and a block of such points does not load the chunk's table.
    bool open = live && first < 0;
    if (run_bound && open && err2 < thr) {
        const float* mx = ntmax + 8 * (1 + j0 / kNtChunk);
        float qb = 0.0f;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            float dev = 0.0f;
#pragma unroll
            for (int k = 0; k < 6; ++k) dev = fmaf(__ldg(mx + k), fabsf(G[k][i]), dev);
            const float b = fabsf(C0[i]) + ecomp[i] + dev * 1.000001f;
            qb = fmaf(i < 3 ? 1.5f : 3.0f, b * b, qb);
        }
        if (qb * 1.0000039f < thr) {
            last_el = j0 + jn - 1;
            open = false;
        }
    }
    if (!__syncthreads_or(open)) continue;
    for (int i = threadIdx.x; i < 3 * jn; i += blockDim.x) sNt[i] = __ldg(nt2 + 3 * (size_t)j0 + i);
    __syncthreads();
    // Run bounds: delta_k >= |Nt_k(t) - Nt_k(t0)| of the FP64 table over each
    // run of kRun steps from its first step t0.  The FP32 table differs from
    // the FP64 one by at most u |Nt_k| <= u ntmax_k per entry (u = 2^-24),
    // and the FP32 difference by one more rounding: inflated accordingly.
    for (int t = threadIdx.x; t < (kNtChunk / kRun) * 8; t += blockDim.x) {
        const int run = t >> 3, k = t & 7;
        const int r0 = run * kRun;
        if (k < 6 && r0 < jn) {
            const float* f = reinterpret_cast<const float*>(sNt);
            const float base = f[r0 * 6 + k];
            float mx = 0.0f;
            for (int j = r0 + 1; j < min(r0 + kRun, jn); ++j) mx = nan_max(mx, fabsf(f[j * 6 + k] - base));
            sDel[run][k] = mx * 1.000001f + __ldg(ntmax + k) * 2.4e-7f;
        }
    }
    __syncthreads();
    for (int jr = 0; jr < jn && open && first < 0; jr += kRun) {
    const int jre = min(jn, jr + kRun);
    // One bound for the whole run: with acc_i(t0) the screened component at the run's
    // first step, every step of the run has |tsig_i| <= |acc_i(t0)| + e_i +
    // sum_k delta_k |g_ki| =: B_i (g the FP64 coefficient, |g| <= |G|(1 +
    // 1.01u); the FP32 sum of the six non-negative products is inflated by
    // 16u for that and its own rounding), so teq^2 <= sum w_i B_i^2; that
    // sum of non-negative FP32 terms is inflated by 2^-18 (64u) for its own
    // rounding.  Below the threshold, every step of the run is elastic.
    if (run_bound && err2 < thr) {
        const float2 t0 = sNt[3 * jr], t1 = sNt[3 * jr + 1], t2 = sNt[3 * jr + 2];
        const float w[6] = {t0.x, t0.y, t1.x, t1.y, t2.x, t2.y};
        float dl[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) dl[k] = sDel[jr / kRun][k];
        float qb = 0.0f;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            float acc = C0[i], dev = 0.0f;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                acc = fmaf(w[k], G[k][i], acc);
                dev = fmaf(dl[k], fabsf(G[k][i]), dev);
            }
            const float b = fabsf(acc) + ecomp[i] + dev * 1.000001f;
            qb = fmaf(i < 3 ? 1.5f : 3.0f, b * b, qb);
        }
        if (qb * 1.0000039f < thr) {
            last_el = j0 + jre - 1;
            continue;
        }
    }
    for (int jq = jr; jq < jre; ++jq) {
        const int jj = j0 + jq;
        const float2 t0 = sNt[3 * jq], t1 = sNt[3 * jq + 1], t2 = sNt[3 * jq + 2];
        const float w[6] = {t0.x, t0.y, t1.x, t1.y, t2.x, t2.y};
        float q = 0.0f;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            float acc = C0[i];
#pragma unroll
            for (int k = 0; k < 6; ++k) acc = fmaf(w[k], G[k][i], acc);
            q = fmaf(i < 3 ? 1.5f : 3.0f, acc * acc, q);
        }
        if (q + err2 < thr) {
            last_el = jj;
            continue;
        }
        first = jj;
        break;
    }
    }
    }
    // Points with an unproven step go to the whole warp, which takes the rest
    // of their slab; nothing of their state has changed yet.
    const unsigned todo = __ballot_sync(0xffffffffu, live && first >= 0);
    if (todo) {
        if (__popc(todo) == 1) exact_points<32>(a, ntmax, todo, gp, first, last_el);
        else exact_points<8>(a, ntmax, todo, gp, first, last_el);
    }
    if (!live || first >= 0) return;
    if (last_el >= 0) slow_materialize(&s, a.Nt, last_el);

    if (a.gpsta && a.gpsta[gp] == 0) {  // src/kokkos_damage.f90:102-107
        st.d = 0.0;
        st.ws = 0.0;
    }
    for (int i = 0; i < 6; ++i) {
        a.eps_old[b6 + i] = st.epo[i];
        a.eps_pl[b6 + i] = st.epl[i];
        a.sig_eff[b6 + i] = st.sef[i];
        a.sig_back[b6 + i] = st.sbk[i];
    }
    a.p[gp] = st.p;
    a.D[gp] = st.d;
    a.ws[gp] = st.ws;
    a.del_po[gp] = st.dpo;
    a.sig_d[gp] = st.sigd;
    if (a.counters) atomicAdd(&a.counters[1], (unsigned long long)a.nip);
}

// Points are dealt to blocks round-robin (pass it, slot s of block b takes
// point (it slots + s) gridDim + b): plastic points cluster in space, i.e. in
// consecutive point numbers, and their FP64 steps would otherwise pile up in
// a few blocks on a few SMs while the rest of the GPU idles.  One pass per
// slot is one slot per point; a small grid with several passes keeps the
// update on a few SMs.  A warp has ppw slots (its first ppw lanes; the others
// only keep its barriers and votes): fewer than 32 where the points
// do not fill the GPU, so that fewer plastic chains share a warp.
__global__ void __launch_bounds__(256)
k_damage(DamageArgs a, const float* __restrict__ ntmax, int run_bound, int passes, int ppw)
{
    const int lane = threadIdx.x & 31, slots = (int)(blockDim.x >> 5) * ppw;
    const int slot = (int)(threadIdx.x >> 5) * ppw + lane;
    for (int it = 0; it < passes; ++it)
        damage_point(a, ntmax, run_bound,
                     lane < ppw ? ((long long)it * slots + slot) * gridDim.x + blockIdx.x : (long long)a.ngp);
}

// max_t |Nt_k(t)| per k of each chunk of kNtChunk steps (one block a chunk)
// into out + 8 (1 + chunk), then of the whole slab into out.  A chunk that holds
// a NaN has a NaN maximum, so that no bound passes over it; the slab's leaves
// NaNs out.
__global__ void __launch_bounds__(256) k_ntmax(const float* __restrict__ nt32, int nip, float* __restrict__ out)
{
    __shared__ float sh[6][8];
    float m[6] = {0, 0, 0, 0, 0, 0};
    const int j1 = min(nip, ((int)blockIdx.x + 1) * kNtChunk);
    for (int j = blockIdx.x * kNtChunk + threadIdx.x; j < j1; j += blockDim.x)
        for (int k = 0; k < 6; ++k) m[k] = nan_max(m[k], fabsf(nt32[(size_t)j * 6 + k]));
    for (int k = 0; k < 6; ++k) {
        float v = m[k];
        for (int off = 16; off > 0; off >>= 1) v = nan_max(v, __shfl_xor_sync(0xffffffffu, v, off));
        if ((threadIdx.x & 31) == 0) sh[k][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        float v = 0.0f;
        for (int w = 0; w < 8; ++w) v = nan_max(v, sh[threadIdx.x][w]);
        out[8 * (1 + blockIdx.x) + threadIdx.x] = v * 1.000001f;
    }
}

__global__ void k_ntmax_all(int chunks, float* __restrict__ out)
{
    if (threadIdx.x >= 6) return;
    float v = 0.0f;
    for (int c = 0; c < chunks; ++c) v = fmaxf(v, out[8 * (1 + c) + threadIdx.x]);
    out[threadIdx.x] = v;
}

__global__ void k_nt_table(int nip, double t0, double t1, double t2, double w, double* nt64,
                           float* nt32)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nip) return;
    const double dt = t2 - t0;
    const double t = t0 + (double)i * dt / (double)nip;
    const double n1 = 2.0 * (t1 - t) * (t2 - t) / (dt * dt);
    const double n2 = -4.0 * (t0 - t) * (t2 - t) / (dt * dt);
    const double n3 = 2.0 * (t0 - t) * (t1 - t) / (dt * dt);
    const double swt = sin(w * t);
    const double r[6] = {n1, n2, n3, n1 * (swt - sin(w * t0)), n2 * (swt - sin(w * t1)),
                         n3 * (swt - sin(w * t2))};
    for (int k = 0; k < 6; ++k) {
        nt64[(size_t)i * 6 + k] = r[k];
        nt32[(size_t)i * 6 + k] = (float)r[k];
    }
}

// chkelesta: single block, elements in ascending order in chunks of
// blockDim.x, block-wide exclusive scan of the failure flags
__global__ void __launch_bounds__(1024)
k_chkelesta(int ne, int ngpe, double Dc, const double* __restrict__ D, int* elesta, int* gpsta,
            int* nefail, int* nef)
{
    __shared__ int warp_tot[32];
    __shared__ int base;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int e0 = 0; e0 < ne; e0 += blockDim.x) {
        const int e = e0 + threadIdx.x;
        int f = 0;
        if (e < ne)
            for (int g = 0; g < ngpe; ++g)
                if (D[(size_t)e * ngpe + g] >= Dc) f = 1;
        const unsigned bal = __ballot_sync(0xffffffffu, f);
        const int before = __popc(bal & ((1u << lane) - 1u));
        if (lane == 0) warp_tot[warp] = __popc(bal);
        __syncthreads();
        int off = base;
        for (int w = 0; w < warp; ++w) off += warp_tot[w];
        if (f) {
            nefail[off + before] = e + 1;
            elesta[e] = 0;
            for (int g = 0; g < ngpe; ++g) gpsta[(size_t)e * ngpe + g] = 0;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int t = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += warp_tot[w];
            base += t;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *nef = base;
}

__global__ void k_zero_int(int* a, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = 0;
}

__global__ void k_any_ge(const double* __restrict__ D, int n, double Dc, int* flag)
{
    int f = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (D[i] >= Dc) f = 1;
    if (__any_sync(0xffffffffu, f) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
}

// Scratch of the allocation-free damage entry point (xt_damage_device):
// the FP32 copy of the temporal shape table (6 values per step, up to
// kDamageStaticMaxNip steps), the shape-value bounds of the slab and of its
// chunks and the three step counters.  1.5 MB in all, part of the library image; one set per process
// and device, so concurrent calls share it.
constexpr size_t kStaticNt = (size_t)kDamageStaticMaxNip * 6;
constexpr size_t kStaticMax = 8 * (1 + (kDamageStaticMaxNip + kNtChunk - 1) / kNtChunk) * sizeof(float);
constexpr size_t kStaticBytes = kStaticNt * sizeof(float) + kStaticMax + 3 * sizeof(unsigned long long);
static_assert(kStaticMax % 8 == 0 && kNtChunk == kDamageChunk, "scratch layout");
static __device__ __align__(256) unsigned char g_damage_scratch[kStaticBytes];

}  // namespace

namespace {
// Per-device address of g_damage_scratch, looked up once per device and
// context.  A mutex guards it: two host threads making their first call at
// once must not race on the entry.  damage_static_forget() clears it when
// the library context is torn down (a new context may place the symbol at
// another address).
std::mutex g_scratch_mu;
constexpr int kMaxDevices = 64;
void* g_scratch_addr[kMaxDevices] = {nullptr};
}  // namespace

int damage_static_scratch(int device, float** nt32, float** ntmax, unsigned long long** counters)
{
    if (device < 0 || device >= kMaxDevices) {
        set_error("damage scratch: device index out of range");
        return XT_ERR_ARG;
    }
    void* base = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_scratch_mu);
        if (!g_scratch_addr[device]) {
            // the caller has made `device` current; cudaGetSymbolAddress can
            // load the module, so the first call must not sit inside a
            // stream capture
            int cur = -1;
            XT_CUDA(cudaGetDevice(&cur));
            if (cur != device) {
                set_error("damage scratch: the library's device is not current");
                return XT_ERR_CUDA;
            }
            void* p = nullptr;
            XT_CUDA(cudaGetSymbolAddress(&p, g_damage_scratch));
            g_scratch_addr[device] = p;
        }
        base = g_scratch_addr[device];
    }
    unsigned char* b = static_cast<unsigned char*>(base);
    *nt32 = reinterpret_cast<float*>(b);
    *ntmax = reinterpret_cast<float*>(b + kStaticNt * sizeof(float));
    *counters = reinterpret_cast<unsigned long long*>(b + kStaticNt * sizeof(float) + kStaticMax);
    return XT_OK;
}

void damage_static_forget()
{
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    for (int d = 0; d < kMaxDevices; ++d) g_scratch_addr[d] = nullptr;
}

int nt_table_device(int nip, double t0, double t1, double t2, double w, double* Nt64,
                    float* Nt32, cudaStream_t s)
{
    if (nip <= 0) return XT_OK;
    k_nt_table<<<(nip + 255) / 256, 256, 0, s>>>(nip, t0, t1, t2, w, Nt64, Nt32);
    note_launches(1);
    XT_CUDA(cudaGetLastError());
    return XT_OK;
}

int damage_update(const DamageArgs& a, cudaStream_t s)
{
    if (a.nnte != 3 || a.ndofn != 3 || a.ncmp != 6 || a.nnse < 1 || a.nnse > 8) {
        set_error("damage_update: the C3D8 kernel needs ndofn=3, nnte=3, ncmp=6, nnse<=8");
        return XT_ERR_ARG;
    }
    if (a.ngp <= 0 || a.nip <= 0) return XT_OK;
    // (the chunks' bounds lie behind the slab's: damage_bounds_floats)
    if (!a.ntmax) {
        set_error("damage_update: missing scratch for the shape-value bounds");
        return XT_ERR_ARG;
    }
    const int chunks = (a.nip + kNtChunk - 1) / kNtChunk;
    k_ntmax<<<chunks, 256, 0, s>>>(a.Nt32, a.nip, a.ntmax);
    k_ntmax_all<<<1, 32, 0, s>>>(chunks, a.ntmax);
    // XTFEM_DAMAGE_RUN=0: screen every step (no per-run bound)
    const char* e = std::getenv("XTFEM_DAMAGE_RUN");
    const int run_bound = (!e || std::atoi(e) != 0) ? 1 : 0;
    // 128 threads per block (XTFEM_DAMAGE_THREADS=256: 256).  A block that
    // holds a plastic point runs for the whole update; at 202 registers a
    // thread, a 128-thread block (26 K registers) leaves its SM room for the
    // solve's blocks beside it, a 256-thread block (52 K) for none of the dot
    // pass's.
    const char* et = std::getenv("XTFEM_DAMAGE_THREADS");
    const int nt = (et && std::atoi(et) == 256) ? 256 : 128;
    // XTFEM_DAMAGE_BLOCKS=B: a grid of B blocks, each thread taking several
    // points in turn (0: one thread per point)
    const char* eb = std::getenv("XTFEM_DAMAGE_BLOCKS");
    const long long want = eb ? std::atoll(eb) : 0;
    // slots per warp: as few as make no more than four warps an SM.  A plastic
    // chain that shares its warp with three others waits for each of theirs to
    // end, but every warp issues the strains and the screen's coefficients, some
    // 800 FP64 instructions.  1,536 points, 2,560 steps, without a plastic point,
    // with 97 and with 278 of them: at most twelve warps an SM 162 us, 5.02 and
    // 5.99 ms, six 122 us, 5.02 and 5.98, four 96 us, 5.02 and 6.19 (a thread a
    // point 146 us, 30.8 and 38.4).
    int ppw = 32;
    while (ppw > 1 && (long long)a.ngp <= (long long)(ppw / 2) * 152 * 4) ppw /= 2;
    const int slots = nt / 32 * ppw;
    const long long full = ((long long)a.ngp + slots - 1) / slots;
    const int grid = (int)((want > 0 && want < full) ? want : full);
    const int passes = (int)(((long long)a.ngp + (long long)grid * slots - 1) / ((long long)grid * slots));
    k_damage<<<grid, nt, 0, s>>>(a, a.ntmax, run_bound, passes, ppw);
    note_launches(3);
    XT_CUDA(cudaGetLastError());
    return XT_OK;
}

int chkelesta_device(int ne, int ngpe, double Dc, const double* D, int* elesta, int* gpsta,
                     int* nefail, int* nef, cudaStream_t s)
{
    if (ne <= 0) return XT_OK;
    k_zero_int<<<(ne + 255) / 256, 256, 0, s>>>(nefail, ne);
    k_chkelesta<<<1, 1024, 0, s>>>(ne, ngpe, Dc, D, elesta, gpsta, nefail, nef);
    note_launches(2);
    XT_CUDA(cudaGetLastError());
    return XT_OK;
}

int any_ge_device(const double* D, int ngp, double Dc, int* flag, cudaStream_t s)
{
    XT_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), s));
    if (ngp <= 0) return XT_OK;
    int blocks = (ngp + 255) / 256;
    if (blocks > 1024) blocks = 1024;
    k_any_ge<<<blocks, 256, 0, s>>>(D, ngp, Dc, flag);
    note_launches(1);
    XT_CUDA(cudaGetLastError());
    return XT_OK;
}

}  // namespace xt
