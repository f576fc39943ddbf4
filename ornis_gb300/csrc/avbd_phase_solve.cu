// avbd_phase_solve.cu — the AVBD iterations: per-colour primal block solves,
// the order-free dual update, then BDF1 velocities and sleep bookkeeping.
//
// Reference: crates/physics/src/avbd/assembly.rs:73-903 (solve_body),
// avbd/joints_ext.rs:464-919 (dual_update), avbd/mod.rs:1060-1142 (BDF1,
// sleep, driver baseline), avbd/sleep.rs:140-175.
#include "avbd_common.cuh"

// This file is compiled twice: the exact build (-fmad=false, IEEE divide and
// square root) reproduces the CPU oracle bit for bit with one thread per
// body; the fast build (-DAVBD_SOLVE_FAST: contracted multiply-adds,
// approximate divide and square root) stays within the 1e-5 pose tolerance
// and is what the benchmark runs.  Discovery is exact in both.
#ifdef AVBD_SOLVE_FAST
#define AVBD_SOLVE_NS fast
#else
#define AVBD_SOLVE_NS exact
#endif

namespace avbd {
namespace AVBD_SOLVE_NS {

static __device__ __forceinline__ void load_ctx(const DW& w, uint32_t p, uint2 ab, PairCtx& c) {
    float4 n4 = w.p_n[p];
    c.a = ab.x;
    c.b = ab.y;
    c.n = ld3(n4);
    c.gap = n4.w;
    c.mu = w.p_mu[p];
    c.np = w.p_np[p];
    const float4* ka = w.kin + (size_t)c.a * 4;
    const float4* kb = w.kin + (size_t)c.b * 4;
    float4 a0 = ka[0], a1 = ka[1], a2 = ka[2], a3 = ka[3];
    float4 b0 = kb[0], b1 = kb[1], b2 = kb[2], b3 = kb[3];
    c.pa = ld3(a0);
    c.pb = ld3(b0);
    c.qa = ldq(a1);
    c.qb = ldq(b1);
    c.dxa = ld3(a2);
    c.dxb = ld3(b2);
    c.dra = ld3(a3);
    c.drb = ld3(b3);
    c.sph_a = info_shape(__float_as_uint(a2.w)) == AVBD_SHAPE_SPHERE;
    c.sph_b = info_shape(__float_as_uint(b2.w)) == AVBD_SHAPE_SPHERE;
    c.rad_a = a0.w;
    c.rad_b = b0.w;
    c.t1 = ld3(w.p_t1[p]);
    c.t2 = cross(c.t1, c.n);
}
// the pair's rolling and torsion friction
static __device__ __forceinline__ void load_rolling(const DW& w, PairCtx& c) {
    const float4 ma = w.mat[c.a], mb = w.mat[c.b];
    c.mu_roll = fmaxf(ma.z, mb.z);
    c.mu_spin = fmaxf(ma.w, mb.w);
}
static __device__ __forceinline__ void load_ctx(const DW& w, uint32_t p, PairCtx& c) {
    load_ctx(w, p, w.p_ab[p], c);
    load_rolling(w, c);
}

// Where a body's rows go.  Sys adds each row to the body's 6x6 system in a
// thread's registers (stamp_row, stamp_angular in avbd_rows.cuh); RowSink
// stages three of them, [first, first + 3) in stamping order, in an item's
// shared-memory slot for the lanes that sum them.
//
// A slot holds three rows side by side: 8 float4, component k of which belongs
// to row k: direction x y z, penalty, lever torque x y z, force.
enum { ROW_NONE = 0, ROW_FULL = 1, ROW_ANG = 2, ROW_DIAG = 3 };  // 2 bits per row of a slot
struct RowSink {
    float* slot;
    int first, n;     // rows staged elsewhere before these; rows seen
    uint32_t types;
};
static __device__ __forceinline__ void put_row(RowSink& s, uint32_t type, V3 nn, float pen, V3 t, float f) {
    const int k = s.n++ - s.first;
    if (k < 0 || k >= 3) return;
    float* o = s.slot + k;
    o[0] = nn.x; o[4] = nn.y; o[8] = nn.z; o[12] = pen;
    o[16] = t.x; o[20] = t.y; o[24] = t.z; o[28] = f;
    s.types |= type << (2 * k);
}
static __device__ __forceinline__ void stamp_row(RowSink& s, V3 axis, float pen, float f, V3 r, float sign) {
    V3 nn = sign * axis;
    put_row(s, ROW_FULL, nn, pen, cross(r, nn), f);
}
static __device__ __forceinline__ void stamp_angular(RowSink& s, V3 g, float pen, float f) {
    put_row(s, ROW_ANG, V0(), pen, g, f);
}
// a joint's geometric stiffness on the angular diagonal
static __device__ __forceinline__ void stamp_diag(Sys& s, V3 d) {
    s.h[tri(3, 3)] += d.x;
    s.h[tri(4, 4)] += d.y;
    s.h[tri(5, 5)] += d.z;
}
static __device__ __forceinline__ void stamp_diag(RowSink& s, V3 d) { put_row(s, ROW_DIAG, V0(), 0.0f, d, 0.0f); }

// A point's levers and constraint values at the bodies' poses: the normal
// row's, and with `friction` the tangent rows'.
struct ContactGeo {
    V3 rup, rlo, raf, rbf;
    float cn, ct1, ct2;
};
static __device__ __forceinline__ ContactGeo contact_geo(const PairCtx& c, float4 ra, float4 rb, float c0, bool friction) {
    ContactGeo g;
    contact_levers(c, ra, rb, g.rup, g.rlo);
    g.cn = row_c_levers(c, c.n, c0, g.rup, g.rlo);
    g.raf = g.rup;
    g.rbf = g.rlo;
    g.ct1 = g.ct2 = 0.0f;
    if (friction) {
        friction_levers(c, g.rup, g.rlo, g.raf, g.rbf);
        g.ct1 = row_c_levers(c, c.t1, 0.0f, g.raf, g.rbf);
        g.ct2 = row_c_levers(c, c.t2, 0.0f, g.raf, g.rbf);
    }
    return g;
}
// Contact rows of a point for the body on side is_a (assembly.rs:99-252).
// live: bit k, row k is stamped (rows: normal, two tangents; a separated pair
// at most its damper as row 0).
struct ContactRows {
    uint32_t live;
    float pen[3], f[3];
    V3 lever, lever_f;  // of the normal row, of the tangent rows
};
static __device__ __forceinline__ ContactRows contact_rows(const DW& w, const PairCtx& c, const ContactGeo& g, bool is_a,
                                                           float4 lam, float4 pen) {
    ContactRows o;
    o.live = 0u;
    o.f[0] = o.f[1] = o.f[2] = 0.0f;
    o.pen[0] = pen.x;
    o.pen[1] = pen.y;
    o.pen[2] = pen.z;
    o.lever = is_a ? g.rup : g.rlo;
    o.lever_f = is_a ? g.raf : g.rbf;
    if (c.gap > 0.0f) {
        // separated damper, imminence-gated (assembly.rs:113-175)
        float approach = fmaxf(dot(ld3(w.vel[c.b]) - ld3(w.vel[c.a]), c.n), 0.0f);
        if (c.gap - approach * w.dt > 0.0f) return o;
        if (fabsf(g.cn) >= C_EPS) {
            float npts = (float)max(c.np, 1u);
            float ka = is_dynamic(w, c.a) ? w.inv_mass[c.a] : 0.0f;
            float kb = is_dynamic(w, c.b) ? w.inv_mass[c.b] : 0.0f;
            float m_red = ka + kb > NEAR_ZERO ? 1.0f / (ka + kb) : 0.0f;
            if (m_red > 0.0f) {
                float pen_d = fminf(2.0f * m_red / (w.dt * w.dt) / npts, PENALTY_MAX);
                o.pen[0] = pen_d;
                o.f[0] = fminf(pen_d * g.cn, 0.0f);
                o.live = 1u;
            }
        }
        return o;
    }
    if (!(c.gap <= 0.0f)) return o;
    contact_force(g.cn, pen, lam, g.ct1, g.ct2, c.mu, o.f);
    o.live = (row_live(g.cn, o.f[0]) ? 1u : 0u) | (row_live(g.ct1, o.f[1]) ? 2u : 0u) | (row_live(g.ct2, o.f[2]) ? 4u : 0u);
    return o;
}
// Rolling and torsion rows of a touching point of normal force fn.
template <class SINK>
static __device__ __forceinline__ void stamp_rolling(const DW& w, const PairCtx& c, uint32_t q, bool is_a, float fn,
                                                     SINK& s) {
    const float mu_roll = c.mu_roll, mu_spin = c.mu_spin;
    V3 wrel = c.dra - c.drb;
    float4 rl = w.q_roll[q];
    V3 rax[3] = {c.t1, c.t2, c.n};
    float murs[3] = {mu_roll, mu_roll, mu_spin};
    float rls[3] = {rl.x, rl.y, rl.z};
#pragma unroll
    for (int li = 0; li < 3; li++) {
        if (murs[li] <= 0.0f) continue;
        float cap = murs[li] * fabsf(fn);
        float fr = fclamp(ROLL_PEN * dot(wrel, rax[li]) + rls[li], -cap, cap);
        stamp_angular(s, is_a ? rax[li] : -rax[li], ROLL_PEN, fr);
    }
}
// Rows of point k of pair p for the body on side is_a.
static __device__ __forceinline__ void stamp_point(const DW& w, const PairCtx& c, uint32_t p, uint32_t k, bool is_a,
                                                   Sys& s) {
    const uint32_t q = p * MAX_PTS + k;
    const float4 lam = w.q_lam[q];
    const bool touching = c.gap <= 0.0f;
    const ContactGeo g = contact_geo(c, w.q_ra[q], w.q_rb[q], touching ? lam.w : 0.0f, touching);
    const ContactRows r = contact_rows(w, c, g, is_a, lam, w.q_pen[q]);
    const float sign = is_a ? 1.0f : -1.0f;
    if (r.live & 1u) stamp_row(s, c.n, r.pen[0], r.f[0], r.lever, sign);
    if (r.live & 2u) stamp_row(s, c.t1, r.pen[1], r.f[1], r.lever_f, sign);
    if (r.live & 4u) stamp_row(s, c.t2, r.pen[2], r.f[2], r.lever_f, sign);
    if (c.gap <= 0.0f && (c.mu_roll > 0.0f || c.mu_spin > 0.0f)) stamp_rolling(w, c, q, is_a, r.f[0], s);
}

// Joint rows for body h (assembly.rs:255-881): Ball, Revolute (and its
// limit), Prismatic (and its limit), Fixed, Distance, Rope, SixDof.
// ALL = false: the instantiation for worlds whose joints are all ball and
// revolute joints (the other kinds' rows would cost it registers).
// A gear's rows on body h, one of its coupled joints' bodies
// (assembly.rs:426-454 slides, :650-682 hinges): the shared force on the
// position-level row C = coord_a + ratio coord_b - constant, the slide
// sides first, then the hinge sides.
template <class SINK>
static __device__ __forceinline__ void stamp_gear(const DW& w, uint32_t j, uint32_t h, SINK& s) {
    const GearSide sd[2] = {gear_side(w, j, 0), gear_side(w, j, 1)};
    const float c = gear_error(w, j, sd[0], sd[1]);
    const float pen = w.j_pen_l[j].x;
    const float f = pen * c + w.j_lam_l[j].x;
    if (!row_live(c, f)) return;
    const float coef[2] = {1.0f, w.j_dref[j].x};
    for (int k = 0; k < 2; k++) {
        const GearSide& side = sd[k];
        if (side.angular || (h != side.a && h != side.b)) continue;
        stamp_row(s, side.axis, pen * coef[k] * coef[k], f * coef[k], h == side.a ? side.ra : side.rb,
                  h == side.a ? -1.0f : 1.0f);
    }
    for (int k = 0; k < 2; k++) {
        const GearSide& side = sd[k];
        if (!side.angular || (h != side.a && h != side.b)) continue;
        stamp_angular(s, h == side.a ? -side.axis : side.axis, pen * coef[k] * coef[k], f * coef[k]);
    }
}

template <bool ALL, class SINK>
static __device__ __forceinline__ void stamp_joint(const DW& w, uint32_t j, uint32_t h, SINK& s) {
    uint2 ab = w.j_ab[j];
    const uint32_t kind = w.j_kind[j];
    if (ALL && kind == AVBD_JOINT_GEAR) {
        stamp_gear(w, j, h, s);
        return;
    }
    const bool k_pri = ALL && kind == AVBD_JOINT_PRISMATIC, k_six = ALL && kind == AVBD_JOINT_SIXDOF;
    const bool k_dist = ALL && (kind == AVBD_JOINT_DISTANCE || kind == AVBD_JOINT_ROPE);
    const bool k_spr = ALL && kind == AVBD_JOINT_SPRING, k_whl = ALL && kind == AVBD_JOINT_WHEEL;
    bool is_a = ab.x == h;
    float sign = is_a ? 1.0f : -1.0f;
    float lsign = is_a ? -1.0f : 1.0f;  // rows measured B minus A flip the gradient
    Q qa = ldq(w.rot[ab.x]), qb = ldq(w.rot[ab.y]);
    Q qa0 = ldq(w.rot0[ab.x]), qb0 = ldq(w.rot0[ab.y]);
    V3 la = ld3(w.j_la[j]), lb = ld3(w.j_lb[j]);
    V3 pa = ld3(w.pos[ab.x]) + qrot(qa, la), pb = ld3(w.pos[ab.y]) + qrot(qb, lb);
    V3 pa0 = ld3(w.pos0[ab.x]) + qrot(qa0, la), pb0 = ld3(w.pos0[ab.y]) + qrot(qb0, lb);
    V3 live = pa - pb, c0v = pa0 - pb0;
    float4 axa4 = w.j_axa[j];
    V3 axa_l = ld3(axa4), axb_l = ld3(w.j_axb[j]);
    V3 wa = normalize_or(qrot(qa, axa_l), VZ());
    float4 pl = w.j_pen_l[j], ll = w.j_lam_l[j], pa4 = w.j_pen_a[j], la4 = w.j_lam_a[j];
    float penl[3] = {pl.x, pl.y, pl.z}, laml[3] = {ll.x, ll.y, ll.z};
    float pena[3] = {pa4.x, pa4.y, pa4.z}, lama[3] = {la4.x, la4.y, la4.z};
    const bool fixed = ALL && kind == AVBD_JOINT_FIXED;
    const V3 dref = fixed || k_six ? ld3(w.j_dref[j]) : V0();
    const float4 ref = w.j_ref[j];
    V3 r_plain = is_a ? qrot(qa, la) : qrot(qb, lb);
    V3 fl = V0();
    // linear rows
    if (kind == AVBD_JOINT_BALL || kind == AVBD_JOINT_REVOLUTE || fixed) {
        // Ball/Revolute levers carry a zero offset in the weld-offset slot
        V3 lever = is_a ? qrot(qa, la + (fixed ? dref : V0())) : qrot(qb, lb);
        V3 lv = fixed ? live + qrot(qa, dref) : live;
        V3 iv = fixed ? c0v + qrot(qa0, dref) : c0v;
        for (int k = 0; k < 3; k++) {
            V3 axis = V0();
            axis[k] = 1.0f;
            float cc = lv[k] - ALPHA * iv[k];
            float f = penl[k] * cc + laml[k];
            if (!row_live(cc, f)) continue;
            stamp_row(s, axis, penl[k], f, lever, sign);
            fl[k] = f;
        }
    } else if (k_pri) {
        V3 u = tangent_t1(wa);
        V3 v = cross(u, wa);
        V3 axs[2] = {u, v};
        for (int li = 0; li < 2; li++) {
            float cc = dot(live - ALPHA * c0v, axs[li]);
            float f = penl[li] * cc + laml[li];
            if (!row_live(cc, f)) continue;
            stamp_row(s, axs[li], penl[li], f, r_plain, sign);
            fl = fl + axs[li] * f;
        }
    } else if (k_dist) {
        float ln = len(live);
        if (kind == AVBD_JOINT_DISTANCE || ln > ref.x) {
            V3 dir = ln > NEAR_ZERO ? live / ln : VY();
            float cc = (ln - ref.x) - ALPHA * (len(c0v) - ref.x);
            float f = penl[0] * cc + laml[0];
            if (row_live(cc, f)) {
                stamp_row(s, dir, penl[0], f, r_plain, sign);
                fl = dir * f;
            }
        }
    } else if (k_whl) {
        // two rows across the suspension axis and the suspension spring
        // along it (assembly.rs:521-581); a zero frequency makes the spring a
        // rigid row on slot 2
        V3 u = tangent_t1(wa);
        V3 v = cross(u, wa);
        V3 axs[2] = {u, v};
        for (int li = 0; li < 2; li++) {
            float cc = dot(live - ALPHA * c0v, axs[li]);
            float f = penl[li] * cc + laml[li];
            if (!row_live(cc, f)) continue;
            stamp_row(s, axs[li], penl[li], f, r_plain, sign);
            fl = fl + axs[li] * f;
        }
        const float4 susp = w.j_lim[j];  // frequency, damping ratio
        const float sv = dot(pb - pa, wa) - ref.x;
        const V3 wa0 = normalize_or(qrot(qa0, axa_l), VZ());
        if (susp.x > 0.0f) {
            const float ka = eff_inv_mass(w, ab.x), kb = eff_inv_mass(w, ab.y);
            const float m = ka + kb > NEAR_ZERO ? 1.0f / (ka + kb) : 0.0f;
            if (m > 0.0f) {
                const float omega = TAU_F * susp.x;
                const float stiff = m * omega * omega, dampc = 2.0f * m * susp.y * omega;
                const float s0 = dot(pb0 - pa0, wa0) - ref.x;
                stamp_row(s, wa, stiff, stiff * sv + dampc * (sv - s0) / w.dt, r_plain, lsign);
            }
        } else {
            const float cc = sv - ALPHA * (dot(pb0 - pa0, wa0) - ref.x);
            const float f = penl[2] * cc + laml[2];
            if (row_live(cc, f)) stamp_row(s, wa, penl[2], f, r_plain, lsign);
        }
    } else if (k_spr) {
        // position-level spring about the rest length (assembly.rs:363-425):
        // penalty from the stiffness, damping from the step delta, no dual
        const float ln = len(live);
        const V3 dir = ln > NEAR_ZERO ? live / ln : VY();
        const float sv = ln - ref.x, s0 = len(c0v) - ref.x;
        const float ka = eff_inv_mass(w, ab.x), kb = eff_inv_mass(w, ab.y);
        const float m = ka + kb > NEAR_ZERO ? 1.0f / (ka + kb) : 0.0f;
        if (m > 0.0f) {
            const float4 mo = w.j_axb[j];  // stiffness, damping, max_force, target_velocity
            const bool force = (w.j_cfg[j] >> 4) == AVBD_MODEL_FORCE;
            const float stiff = force ? mo.x : mo.x * m, dampc = force ? mo.y : mo.y * m;
            if (stiff > 0.0f) {
                stamp_row(s, dir, stiff, stiff * sv + dampc * (sv - s0) / w.dt, r_plain, sign);
            } else if (dampc > 0.0f) {  // a pure damper: the viscous row only
                stamp_row(s, dir, dampc / w.dt, dampc * (sv - s0) / w.dt, r_plain, sign);
            }
        }
    } else if (k_six) {
        const uint32_t cfg = w.j_cfg[j];
        const float4 sa0 = w.j_sacc[2 * (size_t)j];
        const float sacc[3] = {sa0.x, sa0.y, sa0.z};
        for (int i = 0; i < 3; i++) {
            const uint32_t c = axis_cfg(cfg, i);
            if (c == AVBD_AXIS_FREE) continue;
            V3 e = V0();
            e[i] = 1.0f;
            V3 dir = normalize_or(qrot(qa, e), e);
            if (c == AVBD_AXIS_LOCKED) {
                float cc = dot((pb - pa) - qrot(qa, dref), dir);
                float f = penl[i] * cc + laml[i];
                if (!row_live(cc, f)) continue;
                stamp_row(s, dir, penl[i], f, r_plain, lsign);
            } else {
                float2 win = axis_window(w, j, i);
                float sep = dot((pb - pa) - qrot(qa, dref), dir);
                int stt = warm_limit_state(sep, win.x, win.y, LIMIT_SLOP_LIN, sacc[i]);
                if (stt < 0) continue;
                bool lower = stt == 1;
                V3 axis0 = normalize_or(qrot(qa0, e), e);
                float initial = dot((pb0 - pa0) - qrot(qa0, dref), axis0);
                float cc = regularized_limit(sep, initial, lower ? win.x : win.y, lower);
                float f_raw = penl[i] * cc + sacc[i];
                float f = lower ? fminf(f_raw, 0.0f) : fmaxf(f_raw, 0.0f);
                if (!row_live(cc, f)) continue;
                stamp_row(s, dir, penl[i], f, r_plain, lsign);
            }
        }
    }
    {
        // geometric stiffness (rows.rs:69-88, assembly.rs:589-618)
        V3 r = is_a ? qrot(qa, la + (fixed ? dref : V0())) : -qrot(qb, lb);
        float arr[3] = {r.x, r.y, r.z};
        float hm[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
        for (int k = 0; k < 3; k++) {
            float g[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
            g[0][0] = -arr[k];
            g[1][1] = -arr[k];
            g[2][2] = -arr[k];
            g[0][k] += arr[0];
            g[1][k] += arr[1];
            g[2][k] += arr[2];
            for (int x = 0; x < 3; x++)
                for (int y = 0; y < 3; y++) hm[x][y] += g[x][y] * fl[k];
        }
        stamp_diag(s, V3{len(V3{hm[0][0], hm[1][0], hm[2][0]}), len(V3{hm[0][1], hm[1][1], hm[2][1]}),
                         len(V3{hm[0][2], hm[1][2], hm[2][2]})});
    }
    // angular rows (a wheel's pair keys on its axle, in the weld-reference slots)
    if (kind == AVBD_JOINT_REVOLUTE || k_pri || k_whl) {
        const V3 hxa = k_whl ? ld3(w.j_dref[j]) : axa_l, hxb = k_whl ? ld3(w.j_qref[j]) : axb_l;
        V3 axa = qrot(qa, hxa), axb = qrot(qb, hxb);
        V3 axa0 = qrot(qa0, hxa), axb0 = qrot(qb0, hxb);
        V3 t1 = tangent_t1(axa0);
        V3 t2 = cross(t1, axa0);
        V3 ts[2] = {t1, t2};
        for (int li = 0; li < 2; li++) {
            float cc = dot(ts[li], axa - axb) - ALPHA * dot(ts[li], axa0 - axb0);
            float f = pena[li] * cc + lama[li];
            if (!row_live(cc, f)) continue;
            stamp_angular(s, is_a ? cross(axa, ts[li]) : -cross(axb, ts[li]), pena[li], f);
        }
    } else if (k_six) {
        const uint32_t cfg = w.j_cfg[j];
        const Q qref = ldq(w.j_qref[j]);
        const float4 sa0 = w.j_sacc[2 * (size_t)j], sa1 = w.j_sacc[2 * (size_t)j + 1];
        const float sacc[3] = {sa0.w, sa1.x, sa1.y};
        V3 diff = quat_diff_vec(qmul(conj(qa), qb), qref);
        for (int i = 0; i < 3; i++) {
            const uint32_t c = axis_cfg(cfg, 3 + i);
            if (c == AVBD_AXIS_FREE) continue;
            V3 e = V0();
            e[i] = 1.0f;
            V3 dir = normalize_or(qrot(qa, e), e);
            V3 g = is_a ? -dir : dir;
            if (c == AVBD_AXIS_LOCKED) {
                float cc = dot(diff, e);
                float f = pena[i] * cc + lama[i];
                if (!row_live(cc, f)) continue;
                stamp_angular(s, g, pena[i], f);
            } else {
                float2 win = axis_window(w, j, 3 + i);
                float travel = hinge_twist(qa, qb, e) - quat_twist(qref, e);
                int stt = warm_limit_state(travel, win.x, win.y, LIMIT_SLOP_ANG, sacc[i]);
                if (stt < 0) continue;
                bool lower = stt == 1;
                float initial = hinge_twist(qa0, qb0, e) - quat_twist(qref, e);
                float cc = regularized_limit(travel, initial, lower ? win.x : win.y, lower);
                float f_raw = pena[i] * cc + sacc[i];
                float f = lower ? fminf(f_raw, 0.0f) : fmaxf(f_raw, 0.0f);
                if (!row_live(cc, f)) continue;
                stamp_angular(s, g, pena[i], f);
            }
        }
    } else if (fixed) {
        const Q qref = ldq(w.j_qref[j]);
        V3 diff = quat_diff_vec(qmul(conj(qa), qb), qref);
        V3 diff0 = quat_diff_vec(qmul(conj(qa0), qb0), qref);
        for (int k = 0; k < 3; k++) {
            float cc = diff[k] - ALPHA * diff0[k];
            float f = pena[k] * cc + lama[k];
            if (!row_live(cc, f)) continue;
            V3 e = V0();
            e[k] = 1.0f;
            V3 dir = qrot(qa, e);
            stamp_angular(s, is_a ? -dir : dir, pena[k], f);
        }
    }
    // one-sided limit rows
    float4 lim = w.j_lim[j];
    if (lim.z != 0.0f && kind == AVBD_JOINT_REVOLUTE) {
        float refv = axa4.w;
        float angle = wrap_pi(hinge_twist(qa, qb, axa_l) - refv);
        int stt = warm_limit_state(angle, lim.x, lim.y, LIMIT_SLOP_ANG, lim.w);
        if (stt >= 0) {
            bool lower = stt == 1;
            float initial = wrap_pi(hinge_twist(qa0, qb0, axa_l) - refv);
            float cc = regularized_limit(angle, initial, lower ? lim.x : lim.y, lower);
            float f_raw = pa4.z * cc + lim.w;
            float f = lower ? fminf(f_raw, 0.0f) : fmaxf(f_raw, 0.0f);
            if (row_live(cc, f)) stamp_angular(s, is_a ? -wa : wa, pa4.z, f);
        }
    } else if (lim.z != 0.0f && k_pri) {
        float sv = dot(pb - pa, wa) - ref.x;
        int stt = warm_limit_state(sv, lim.x, lim.y, LIMIT_SLOP_LIN, ref.y);
        if (stt >= 0) {
            bool lower = stt == 1;
            V3 axis0 = normalize_or(qrot(qa0, axa_l), VZ());
            float initial = dot(pb0 - pa0, axis0) - ref.x;
            float cc = regularized_limit(sv, initial, lower ? lim.x : lim.y, lower);
            float f_raw = pl.z * cc + ref.y;
            float f = lower ? fminf(f_raw, 0.0f) : fmaxf(f_raw, 0.0f);
            if (row_live(cc, f)) stamp_row(s, wa, pl.z, f, r_plain, lsign);
        }
    }
}

// inertial block and rhs (assembly.rs:74-96); rdt2: the reciprocal of dt^2,
// shared by the block's ten divisions
static __device__ __forceinline__ Recip recip_dt2(const DW& w) {
    bool bad = false;
    return recip_of(w.dt * w.dt, bad);
}
static __device__ __forceinline__ float div_dt2(float a, const Recip& r) {
    bool bad = !(r.b >= 0x1p-40f && r.b <= 0x1p40f);
    const float q = div_by(a, r, bad);
    return bad ? a / r.b : q;
}
static __device__ __forceinline__ void inertial_block(const DW& w, uint32_t h, const Recip& rdt2, Sys& s) {
    const float4 rot4 = w.rot[h], in4 = w.inertia[h], pos4 = w.pos[h], y4 = w.inertial[h], qt4 = w.inertial_rot[h];
    float im = is_dynamic(w, h) ? w.inv_mass[h] : 0.0f;
    float m_dt2 = div_dt2(1.0f / im, rdt2);
    float iw[3][3];
    Q q = ldq(rot4);
    world_inertia(ld3(in4), q, iw);
    for (int i = 0; i < 21; i++) s.h[i] = 0.0f;
    s.h[tri(0, 0)] = m_dt2;
    s.h[tri(1, 1)] = m_dt2;
    s.h[tri(2, 2)] = m_dt2;
    for (int a = 0; a < 3; a++)
        for (int b = 0; b <= a; b++) s.h[tri(3 + a, 3 + b)] = div_dt2(iw[a][b], rdt2);
    V3 rl = m_dt2 * (ld3(pos4) - ld3(y4));
    s.r[0] = rl.x;
    s.r[1] = rl.y;
    s.r[2] = rl.z;
    V3 ra = mat3_vec(iw, quat_diff_vec(q, ldq(qt4)));
    s.r[3] = div_dt2(ra.x, rdt2);
    s.r[4] = div_dt2(ra.y, rdt2);
    s.r[5] = div_dt2(ra.z, rdt2);
}

// What a body's update reads besides its system, loaded ahead of the solve.
struct BodyPose {
    float4 pos, rot, pos0, rot0;
    float par;      // first shape parameter
    uint32_t info;
};
static __device__ __forceinline__ BodyPose load_pose(const DW& w, uint32_t h) {
    return BodyPose{w.pos[h], w.rot[h], w.pos0[h], w.rot0[h], w.shp[h].x, w.info[h]};
}
static __device__ __forceinline__ void apply_solve(const DW& w, uint32_t h, const BodyPose& b, const Sys& s) {
    float dx[6];
    if (solve_6x6_div(s, dx)) {
        V3 p = ld3(b.pos) + V3{dx[0], dx[1], dx[2]};
        Q q = quat_integrate(ldq(b.rot), V3{dx[3], dx[4], dx[5]});
        V3 d = p - ld3(b.pos0);
        V3 dr = quat_diff_vec(q, ldq(b.rot0));
        w.pos[h] = st3(p, 0.0f);
        w.rot[h] = stq(q);
        float4* k = w.kin + (size_t)h * 4;
        k[0] = st3(p, b.par);
        k[1] = stq(q);
        k[2] = st3(d, __uint_as_float(b.info));
        k[3] = st3(dr, 0.0f);
    } else {
        atomicAdd(&w.ctr[C_BREAKDOWN], 1u);  // breakdown: the body skips its update
    }
}

// JT: 0 for worlds without joints (the joint rows' code and registers stay
// out of the contact-only kernels), 1 with ball and revolute joints only,
// 2 with any joint kind.

// L lanes per body: the body's incident pairs are dealt round-robin over the
// lanes, the partial systems are summed with shuffles, lane 0 adds the
// inertial block and the joints and solves.
template <int L, int JT>
__global__ void k_primal_lanes(DW w, int colour) {
    if (aborted_solve(w)) return;
    uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t i = gid / L;
    int lane = threadIdx.x % L;
    uint32_t c0 = w.col_cnt[colour], c1 = w.col_cnt[colour + 1];
    bool active = c0 + i < c1;
    uint32_t h = active ? w.col_list[c0 + i] : 0u;
    Sys s;
#pragma unroll
    for (int k = 0; k < 21; k++) s.h[k] = 0.0f;
#pragma unroll
    for (int k = 0; k < 6; k++) s.r[k] = 0.0f;
    if (active) {
        uint32_t nb = w.offB[h + 1] - w.offB[h], na = w.offA[h + 1] - w.offA[h];
        for (uint32_t e = lane; e < nb + na; e += L) {
            uint32_t p = e < nb ? w.listB[w.offB[h] + e] : w.offA[h] + (e - nb);
            PairCtx c;
            load_ctx(w, p, c);
            for (uint32_t q = 0; q < c.np; q++) stamp_point(w, c, p, q, e >= nb, s);
        }
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < 21; k++) s.h[k] += __shfl_down_sync(0xffffffffu, s.h[k], o, L);
#pragma unroll
        for (int k = 0; k < 6; k++) s.r[k] += __shfl_down_sync(0xffffffffu, s.r[k], o, L);
    }
    if (!active || lane != 0) return;
    Sys t;
    inertial_block(w, h, recip_dt2(w), t);
#pragma unroll
    for (int k = 0; k < 21; k++) t.h[k] += s.h[k];
#pragma unroll
    for (int k = 0; k < 6; k++) t.r[k] += s.r[k];
    if (JT)
        for (uint32_t k = w.jofs[h]; k < w.jofs[h + 1]; k++) stamp_joint<JT == 2>(w, w.jlist[k], h, t);
    apply_solve(w, h, load_pose(w, h), t);
}

// ---- per-colour (pair, side) lists: what the reverse sweep's row kernel walks ------
// Slots: body h owns [offA[h] + offB[h], offA[h+1] + offB[h+1]), B sides first;
// the A side of pair p is slot p + offB[a+1], the B side slot offA[b] + posB[p].
constexpr int SIDE_BLOCK = 256;
__global__ void k_side_count(DW w) {
    if (aborted_solve(w)) return;
    __shared__ uint32_t hist[MAX_COLOURS];
    for (int c = threadIdx.x; c < MAX_COLOURS; c += blockDim.x) hist[c] = 0;
    __syncthreads();
    const uint32_t n = n_pairs(w);
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        uint2 ab = w.p_ab[p];
        int ca = w.colour[ab.x], cb = w.colour[ab.y];
        if (ca >= 0) atomicAdd(&hist[ca], 1u);
        if (cb >= 0) atomicAdd(&hist[cb], 1u);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < MAX_COLOURS; c += blockDim.x)
        if (hist[c]) atomicAdd(&w.side_cnt[MAX_COLOURS + 1 + c], hist[c]);
}
// one thread: list starts from the per-colour totals; cursors start there
__global__ void k_side_starts(DW w) {
    if (aborted_solve(w) || threadIdx.x != 0) return;
    uint32_t acc = 0;
    for (int c = 0; c < MAX_COLOURS; c++) {
        uint32_t t = w.side_cnt[MAX_COLOURS + 1 + c];
        w.side_cnt[c] = acc;
        w.side_cnt[MAX_COLOURS + 1 + c] = acc;
        acc += t;
    }
    w.side_cnt[MAX_COLOURS] = acc;
}
// Entries are placed with block-aggregated reservations, so a colour's list
// keeps roughly the pair order (neighbouring entries share bodies and point
// arrays: grouping entries by point count instead lost more in locality than
// it won in convergence); the exact order is irrelevant (each entry writes
// its own slot).
__global__ void k_side_place(DW w) {
    if (aborted_solve(w)) return;
    __shared__ uint32_t cnt[MAX_COLOURS], base[MAX_COLOURS];
    const uint32_t n = n_pairs(w);
    for (uint32_t p0 = blockIdx.x * blockDim.x; p0 < n; p0 += gridDim.x * blockDim.x) {
        for (int c = threadIdx.x; c < MAX_COLOURS; c += blockDim.x) cnt[c] = 0;
        __syncthreads();
        uint32_t p = p0 + threadIdx.x;
        int ca = -1, cb = -1;
        if (p < n) {
            uint2 ab = w.p_ab[p];
            ca = w.colour[ab.x];
            cb = w.colour[ab.y];
        }
        uint32_t ra = ca >= 0 ? atomicAdd(&cnt[ca], 1u) : 0u;
        uint32_t rb = cb >= 0 ? atomicAdd(&cnt[cb], 1u) : 0u;
        __syncthreads();
        for (int c = threadIdx.x; c < MAX_COLOURS; c += blockDim.x)
            base[c] = cnt[c] ? atomicAdd(&w.side_cnt[MAX_COLOURS + 1 + c], cnt[c]) : 0u;
        __syncthreads();
        if (ca >= 0) w.side_list[base[ca] + ra] = p * 2u + 1u;
        if (cb >= 0) w.side_list[base[cb] + rb] = p * 2u;
        __syncthreads();
    }
}

// Work lists are taken in chunks of one block (128 entries) whose entries are
// handed to the block's threads grouped by a small work class (the entry's
// loop length), so that the lanes of a warp run loops of the same length
// instead of idling behind the longest one.  The chunk keeps the list's
// locality; each entry writes only its own outputs, so which thread takes
// it changes no result.
constexpr int CHUNK = 128;
// Counting sort of the chunk's entries by class (0..MAX_PTS) into ent[].
// Every thread of the block calls it; returns the entries in the chunk.
static __device__ __forceinline__ uint32_t chunk_sort(uint32_t* cnt, uint32_t* ent, bool has, uint32_t e,
                                                      uint32_t cls, uint32_t n) {
    if (threadIdx.x <= MAX_PTS) cnt[threadIdx.x] = 0;
    __syncthreads();
    if (has) atomicAdd(&cnt[cls], 1u);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t acc = 0;
        for (int k = 0; k <= MAX_PTS; k++) {
            uint32_t c = cnt[k];
            cnt[k] = acc;
            acc += c;
        }
    }
    __syncthreads();
    if (has) ent[atomicAdd(&cnt[cls], 1u)] = e;
    __syncthreads();
    return n;
}
// ---- dual (joints_ext.rs:464-573 contacts, :574-896 joints) ----
// The dual update of a point from its constraint values: its new multipliers
// and penalties into lam and pen, stored with the grip flag (rbw: the flag as
// stored).
static __device__ __forceinline__ void dual_update(const DW& w, const PairCtx& c, const ContactGeo& g, uint32_t q, float rbw,
                                                   float4& lam, float4& pen) {
    const bool touching = c.gap <= 0.0f;
    float f[3];
    contact_force(g.cn, pen, lam, g.ct1, g.ct2, c.mu, f);
    float bnd = fabsf(f[0]) * fmaxf(c.mu.x, c.mu.y);
    float fu0 = pen.y * g.ct1 + lam.y, fu1 = pen.z * g.ct2 + lam.z;
    bool stuck = sqrt0(fu0 * fu0 + fu1 * fu1) <= bnd && sqrt0(g.ct1 * g.ct1 + g.ct2 * g.ct2) < STICK_THRESH;
    float4 nl = lam, np4 = pen;
    if (touching && fabsf(g.cn) >= C_EPS) {
        nl.x = f[0];
        if (f[0] < 0.0f) np4.x = fminf(pen.x + BETA * fabsf(g.cn), PENALTY_MAX);
    }
    float b1 = fabsf(f[0]) * c.mu.x, b2 = fabsf(f[0]) * c.mu.y;
    float s_ell = INFINITY;
    if (b1 > 0.0f && b2 > 0.0f) {
        const float g0 = div0(fu0, b1), g1 = div0(fu1, b2);
        s_ell = g0 * g0 + g1 * g1;
    }
    if (touching) {
        nl.y = f[1];
        nl.z = f[2];
        if (s_ell <= 1.0f) {
            if (fabsf(g.ct1) >= C_EPS) np4.y = fminf(pen.y + BETA * fabsf(g.ct1), PENALTY_MAX);
            if (fabsf(g.ct2) >= C_EPS) np4.z = fminf(pen.z + BETA * fabsf(g.ct2), PENALTY_MAX);
        }
    }
    w.q_lam[q] = nl;
    // penalties and the grip flag change in few iterations: store only changes
    if (np4.x != pen.x || np4.y != pen.y || np4.z != pen.z) w.q_pen[q] = np4;
    if (stuck != (rbw != 0.0f)) reinterpret_cast<float*>(&w.q_rb[q])[3] = stuck ? 1.0f : 0.0f;
    lam = nl;
    pen = np4;
}
static __device__ __forceinline__ void dual_point(const DW& w, const PairCtx& c, uint32_t q, float4& lam, float4& pen) {
    const bool touching = c.gap <= 0.0f;
    const float4 rb = w.q_rb[q];
    lam = w.q_lam[q];
    pen = w.q_pen[q];
    const ContactGeo g = contact_geo(c, w.q_ra[q], rb, touching ? lam.w : 0.0f, true);
    dual_update(w, c, g, q, rb.w, lam, pen);
    const float mu_roll = c.mu_roll, mu_spin = c.mu_spin;
    if (touching && (mu_roll > 0.0f || mu_spin > 0.0f)) {
        V3 wrel = c.dra - c.drb;
        float lam_n = fabsf(lam.x);
        float4 rl = w.q_roll[q];
        float rls[3] = {rl.x, rl.y, rl.z};
        V3 rax[3] = {c.t1, c.t2, c.n};
        float murs[3] = {mu_roll, mu_roll, mu_spin};
        for (int li = 0; li < 3; li++) {
            if (murs[li] <= 0.0f) continue;
            float cap = murs[li] * lam_n;
            rls[li] = fclamp(ROLL_PEN * dot(wrel, rax[li]) + rls[li], -cap, cap);
        }
        w.q_roll[q] = make_float4(rls[0], rls[1], rls[2], 0.0f);
    }
}
static __device__ __forceinline__ void dual_pair(const DW& w, uint32_t p) {
    uint32_t np = w.p_np[p];
    if (np == 0) return;
    PairCtx c;
    load_ctx(w, p, c);
    float4 lam, pen;
    for (uint32_t k = 0; k < np; k++) dual_point(w, c, p * MAX_PTS + k, lam, pen);
}
__global__ void __launch_bounds__(CHUNK) k_dual_pairs(DW w) {
    if (aborted_solve(w)) return;
    __shared__ uint32_t s_cnt[MAX_PTS + 1], s_ent[CHUNK];
    const uint32_t np = n_pairs(w);
    for (uint32_t base = blockIdx.x * CHUNK; base < np; base += gridDim.x * CHUNK) {
        const uint32_t p = base + threadIdx.x;
        const bool has = p < np;
        const uint32_t cls = has ? min(w.p_np[p], (uint32_t)MAX_PTS) : 0u;
        const uint32_t n = chunk_sort(s_cnt, s_ent, has, p, cls, min((uint32_t)CHUNK, np - base));
        if (threadIdx.x < n) dual_pair(w, s_ent[threadIdx.x]);
        __syncthreads();
    }
}
// joints_ext.rs:574-896: the joint rows' multipliers and penalties
static __device__ __forceinline__ float ramp(float pen, float c, float beta, float cap) {
    return fminf(pen + beta * fabsf(c), cap);
}
template <bool ALL>
static __device__ void dual_joint(const DW& w, uint32_t j) {
    uint2 ab = w.j_ab[j];
    const uint32_t kind = w.j_kind[j];
    if (ALL && kind == AVBD_JOINT_GEAR) {
        // reads only bodies and its own state: its place after every other
        // joint (joints_ext.rs:897-918) cannot change it; penalty capped
        // like a limit's
        const GearSide sa = gear_side(w, j, 0), sb = gear_side(w, j, 1);
        const float c = gear_error(w, j, sa, sb);
        if (fabsf(c) < C_EPS) return;
        float4 ll = w.j_lam_l[j], pl = w.j_pen_l[j];
        ll.x = ll.x + pl.x * c;
        pl.x = ramp(pl.x, c, BETA, LIM_PEN_MAX);
        w.j_lam_l[j] = ll;
        w.j_pen_l[j] = pl;
        return;
    }
    const bool k_pri = ALL && kind == AVBD_JOINT_PRISMATIC, k_six = ALL && kind == AVBD_JOINT_SIXDOF;
    Q qa = ldq(w.rot[ab.x]), qb = ldq(w.rot[ab.y]);
    Q qa0 = ldq(w.rot0[ab.x]), qb0 = ldq(w.rot0[ab.y]);
    V3 la = ld3(w.j_la[j]), lb = ld3(w.j_lb[j]);
    V3 pa = ld3(w.pos[ab.x]) + qrot(qa, la), pb = ld3(w.pos[ab.y]) + qrot(qb, lb);
    V3 pa0 = ld3(w.pos0[ab.x]) + qrot(qa0, la), pb0 = ld3(w.pos0[ab.y]) + qrot(qb0, lb);
    V3 live = pa - pb, c0v = pa0 - pb0;
    float4 ll = w.j_lam_l[j], pl = w.j_pen_l[j];
    float laml[3] = {ll.x, ll.y, ll.z}, penl[3] = {pl.x, pl.y, pl.z};
    float4 la4 = w.j_lam_a[j], pa4 = w.j_pen_a[j];
    float lama[3] = {la4.x, la4.y, la4.z}, pena[3] = {pa4.x, pa4.y, pa4.z};
    float4 ref = w.j_ref[j];
    // a soft joint (finite stiffness K) is a spring: penalty K, lambda zero,
    // for the anchor and hinge rows of ball and revolute joints; a hard one
    // is the reference's dual ascent
    const float K = w.joint_k;
    const bool soft = K > 0.0f && (kind == AVBD_JOINT_BALL || kind == AVBD_JOINT_REVOLUTE);
    const bool fixed = ALL && kind == AVBD_JOINT_FIXED;
    if (kind == AVBD_JOINT_BALL || kind == AVBD_JOINT_REVOLUTE || fixed) {
        const V3 dref = fixed ? ld3(w.j_dref[j]) : V0();
        V3 lv = fixed ? live + qrot(qa, dref) : live;
        V3 iv = fixed ? c0v + qrot(qa0, dref) : c0v;
        for (int k = 0; k < 3; k++) {
            float cc = lv[k] - ALPHA * iv[k];
            if (soft) {
                penl[k] = K;
            } else if (fabsf(cc) >= C_EPS) {
                laml[k] += penl[k] * cc;
                penl[k] = ramp(penl[k], cc, BETA, PENALTY_MAX);
            }
        }
    } else if (k_pri) {
        V3 wa = normalize_or(qrot(qa, ld3(w.j_axa[j])), VZ());
        V3 u = tangent_t1(wa);
        V3 v = cross(u, wa);
        V3 axs[2] = {u, v};
        for (int li = 0; li < 2; li++) {
            float cc = dot(live - ALPHA * c0v, axs[li]);
            if (fabsf(cc) >= C_EPS) {
                laml[li] += penl[li] * cc;
                penl[li] = ramp(penl[li], cc, BETA, PENALTY_MAX);
            }
        }
    } else if (ALL && kind == AVBD_JOINT_WHEEL) {
        // the rows across the suspension axis, and the rigid suspension row
        // when the frequency is zero (joints_ext.rs:738-764); a live spring
        // carries no dual state
        V3 wa = normalize_or(qrot(qa, ld3(w.j_axa[j])), VZ());
        V3 u = tangent_t1(wa);
        V3 v = cross(u, wa);
        V3 axs[2] = {u, v};
        for (int li = 0; li < 2; li++) {
            float cc = dot(live - ALPHA * c0v, axs[li]);
            if (fabsf(cc) >= C_EPS) {
                laml[li] += penl[li] * cc;
                penl[li] = ramp(penl[li], cc, BETA, PENALTY_MAX);
            }
        }
        if (w.j_lim[j].x <= 0.0f) {
            V3 wa0 = normalize_or(qrot(qa0, ld3(w.j_axa[j])), VZ());
            float cc = (-dot(live, wa) - ref.x) - ALPHA * (-dot(pa0 - pb0, wa0) - ref.x);
            if (fabsf(cc) >= C_EPS) {
                laml[2] += penl[2] * cc;
                penl[2] = ramp(penl[2], cc, BETA, LIM_PEN_MAX);
            }
        }
    } else if (ALL && kind == AVBD_JOINT_DISTANCE) {
        float cc = (len(live) - ref.x) - ALPHA * (len(c0v) - ref.x);
        if (fabsf(cc) >= C_EPS) {
            laml[0] += penl[0] * cc;
            penl[0] = ramp(penl[0], cc, BETA, PENALTY_MAX);
        }
    } else if (ALL && kind == AVBD_JOINT_ROPE) {
        float ln = len(live);
        if (ln > ref.x) {
            float cc = (ln - ref.x) - ALPHA * (len(c0v) - ref.x);
            if (fabsf(cc) >= C_EPS) {
                laml[0] = fmaxf(laml[0] + penl[0] * cc, 0.0f);
                penl[0] = ramp(penl[0], cc, BETA, LIM_PEN_MAX);
            }
        } else {
            laml[0] = 0.0f;
        }
    } else if (k_six) {
        const uint32_t cfg = w.j_cfg[j];
        const V3 dref = ld3(w.j_dref[j]);
        const Q qref = ldq(w.j_qref[j]);
        float4 sa0 = w.j_sacc[2 * (size_t)j], sa1 = w.j_sacc[2 * (size_t)j + 1];
        float sacc[6] = {sa0.x, sa0.y, sa0.z, sa0.w, sa1.x, sa1.y};
        for (int i = 0; i < 3; i++) {
            const uint32_t c = axis_cfg(cfg, i);
            if (c == AVBD_AXIS_FREE) continue;
            V3 e = V0();
            e[i] = 1.0f;
            V3 dir = normalize_or(qrot(qa, e), e);
            float sep = dot((pb - pa) - qrot(qa, dref), dir);
            if (c == AVBD_AXIS_LOCKED) {
                if (fabsf(sep) >= C_EPS) {
                    laml[i] += penl[i] * sep;
                    penl[i] = ramp(penl[i], sep, BETA, PENALTY_MAX);
                }
            } else {
                float2 win = axis_window(w, j, i);
                int stt = warm_limit_state(sep, win.x, win.y, LIMIT_SLOP_LIN, sacc[i]);
                if (stt >= 0) {
                    bool lower = stt == 1;
                    V3 axis0 = normalize_or(qrot(qa0, e), e);
                    float initial = dot((pb0 - pa0) - qrot(qa0, dref), axis0);
                    float cc = regularized_limit(sep, initial, lower ? win.x : win.y, lower);
                    if (fabsf(cc) >= C_EPS) {
                        float f = penl[i] * cc + sacc[i];
                        sacc[i] = lower ? fminf(f, 0.0f) : fmaxf(f, 0.0f);
                        penl[i] = ramp(penl[i], cc, BETA, LIM_PEN_MAX);
                    }
                } else {
                    sacc[i] = 0.0f;
                }
            }
        }
        V3 diff = quat_diff_vec(qmul(conj(qa), qb), qref);
        for (int i = 0; i < 3; i++) {
            const uint32_t c = axis_cfg(cfg, 3 + i);
            if (c == AVBD_AXIS_FREE) continue;
            V3 e = V0();
            e[i] = 1.0f;
            if (c == AVBD_AXIS_LOCKED) {
                float cc = dot(diff, e);
                if (fabsf(cc) >= C_EPS) {
                    lama[i] += pena[i] * cc;
                    pena[i] = ramp(pena[i], cc, BETA_ANG, PENALTY_MAX);
                }
            } else {
                float2 win = axis_window(w, j, 3 + i);
                float travel = hinge_twist(qa, qb, e) - quat_twist(qref, e);
                int stt = warm_limit_state(travel, win.x, win.y, LIMIT_SLOP_ANG, sacc[3 + i]);
                if (stt >= 0) {
                    bool lower = stt == 1;
                    float initial = hinge_twist(qa0, qb0, e) - quat_twist(qref, e);
                    float cc = regularized_limit(travel, initial, lower ? win.x : win.y, lower);
                    if (fabsf(cc) >= C_EPS) {
                        float f = pena[i] * cc + sacc[3 + i];
                        sacc[3 + i] = lower ? fminf(f, 0.0f) : fmaxf(f, 0.0f);
                        pena[i] = ramp(pena[i], cc, BETA_ANG, LIM_PEN_MAX);
                    }
                } else {
                    sacc[3 + i] = 0.0f;
                }
            }
        }
        w.j_sacc[2 * (size_t)j] = make_float4(sacc[0], sacc[1], sacc[2], sacc[3]);
        w.j_sacc[2 * (size_t)j + 1] = make_float4(sacc[4], sacc[5], 0.0f, 0.0f);
    }
    // angular equality rows (a wheel's keyed on its axle, joints_ext.rs:789-803)
    if (kind == AVBD_JOINT_REVOLUTE || k_pri || (ALL && kind == AVBD_JOINT_WHEEL)) {
        const bool whl = ALL && kind == AVBD_JOINT_WHEEL;
        V3 axa_l = whl ? ld3(w.j_dref[j]) : ld3(w.j_axa[j]), axb_l = whl ? ld3(w.j_qref[j]) : ld3(w.j_axb[j]);
        V3 axa = qrot(qa, axa_l), axb = qrot(qb, axb_l);
        V3 axa0 = qrot(qa0, axa_l), axb0 = qrot(qb0, axb_l);
        V3 t1 = tangent_t1(axa0);
        V3 t2 = cross(t1, axa0);
        V3 ts[2] = {t1, t2};
        for (int li = 0; li < 2; li++) {
            float cc = dot(ts[li], axa - axb) - ALPHA * dot(ts[li], axa0 - axb0);
            if (soft) {
                pena[li] = K;
                continue;
            }
            if (fabsf(cc) < C_EPS) continue;
            lama[li] = pena[li] * cc + lama[li];
            pena[li] = ramp(pena[li], cc, BETA_ANG, PENALTY_MAX);
        }
    } else if (fixed) {
        const Q qref = ldq(w.j_qref[j]);
        V3 diff = quat_diff_vec(qmul(conj(qa), qb), qref);
        V3 diff0 = quat_diff_vec(qmul(conj(qa0), qb0), qref);
        for (int k = 0; k < 3; k++) {
            float cc = diff[k] - ALPHA * diff0[k];
            if (fabsf(cc) < C_EPS) continue;
            lama[k] += pena[k] * cc;
            pena[k] = ramp(pena[k], cc, BETA_ANG, PENALTY_MAX);
        }
    }
    // one-sided limits
    float4 lim = w.j_lim[j];
    if (lim.z != 0.0f && kind == AVBD_JOINT_REVOLUTE) {
        V3 axa_l = ld3(w.j_axa[j]);
        float refv = w.j_axa[j].w;
        float angle = wrap_pi(hinge_twist(qa, qb, axa_l) - refv);
        int stt = warm_limit_state(angle, lim.x, lim.y, LIMIT_SLOP_ANG, lim.w);
        if (stt >= 0) {
            bool lower = stt == 1;
            float initial = wrap_pi(hinge_twist(qa0, qb0, axa_l) - refv);
            float cc = regularized_limit(angle, initial, lower ? lim.x : lim.y, lower);
            if (fabsf(cc) >= C_EPS) {
                float f = pena[2] * cc + lim.w;
                lim.w = lower ? fminf(f, 0.0f) : fmaxf(f, 0.0f);
                pena[2] = ramp(pena[2], cc, BETA_ANG, LIM_PEN_MAX);
            }
        } else {
            lim.w = 0.0f;
        }
        w.j_lim[j] = lim;
    } else if (lim.z != 0.0f && k_pri) {
        V3 axa_l = ld3(w.j_axa[j]);
        V3 wa = normalize_or(qrot(qa, axa_l), VZ());
        float sv = dot(pb - pa, wa) - ref.x;
        int stt = warm_limit_state(sv, lim.x, lim.y, LIMIT_SLOP_LIN, ref.y);
        if (stt >= 0) {
            bool lower = stt == 1;
            V3 axis0 = normalize_or(qrot(qa0, axa_l), VZ());
            float initial = dot(pb0 - pa0, axis0) - ref.x;
            float cc = regularized_limit(sv, initial, lower ? lim.x : lim.y, lower);
            if (fabsf(cc) >= C_EPS) {
                float f_raw = penl[2] * cc + ref.y;
                ref.y = lower ? fminf(f_raw, 0.0f) : fmaxf(f_raw, 0.0f);
                penl[2] = ramp(penl[2], cc, BETA, LIM_PEN_MAX);
            }
        } else {
            lim.w = 0.0f;
            ref.y = 0.0f;
        }
        w.j_lim[j] = lim;
        w.j_ref[j] = ref;
    }
    w.j_lam_l[j] = make_float4(laml[0], laml[1], laml[2], 0.0f);
    w.j_pen_l[j] = make_float4(penl[0], penl[1], penl[2], 0.0f);
    w.j_lam_a[j] = make_float4(lama[0], lama[1], lama[2], 0.0f);
    w.j_pen_a[j] = make_float4(pena[0], pena[1], pena[2], 0.0f);
}
template <bool ALL>
__global__ void k_dual_joints(DW w) {
    if (aborted_solve(w)) return;
    uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < (uint32_t)w.J) dual_joint<ALL>(w, j);
}

// ---- tile engine: every iteration of a substep in one launch --------------------
// A body's system is the inertial block plus its rows in incidence order
// (B-side pairs ascending, then A-side pairs ascending, their points in
// order, then its joints).  One thread per body pays a dependent chain of
// loads and about 600 instructions per point (46 us a colour for 35 cubes of
// 20 points each); one thread per (pair, side) writes and re-reads 112 bytes
// per incidence.  Here a warp takes up to 32 bodies of one colour and splits
// the work by what is independent:
//   rows   one lane per (point, side) or third of a joint computes its rows
//          into the warp's shared memory, 32 at a time;
//   sums   27 lanes, each owning one number of the 6x6 system, add the rows in
//          their order: the same additions in the same order as one thread
//          would make, so the sum is bit-identical;
//   solve  one lane per body factors and applies.
// Warps share nothing between barriers, so the latency of one (a chain of
// loads, then divisions and square roots) is covered by the others; bodies
// are dealt to as many warps as there are, 32 to a warp only once every warp
// has some.
// PS = false sums row by row (the thread-per-body order, the reference's);
// PS = true sums each pair's rows from zero first and adds the pair's sum
// (the split order).
//
// Bound by latency, not by bytes: a colour costs a lone warp about 2 us of
// item rows, 0.6 us of sums, 1.7 us of solves and 1 us of barrier; with every
// warp busy (100,000 bodies) the schedulers issue 40% of their slots.
// Iterations of a substep, before (a launch per colour) and after, in ms:
// 210-cube pyramid 3.25 -> 0.55, 1500-body heap 1.60 -> 0.27, 96 scenes of up
// to 400 bodies 1.44 -> 0.25, 1536 scenes of up to 1024 bodies 3.02 -> 2.42,
// 100,000 bodies on a plane 2.03 -> 1.07, 1200 ragdolls 2.37 -> 1.28.  A
// cluster per scene (its own barriers) was slower at every size but one
// (0.34, 0.33 and 3.1 ms for the heap and the two batches): warps idle at
// their own scene's barriers.
//
// k_entries lists, once per substep, every body's (point, side) items, so
// that an item's lane goes straight to its data.  The list lives in the
// previous generation's point anchors (q_ra, q_rb), which nothing reads once
// discovery has merged them.

constexpr uint32_t ENT_SIDE_A = 1u << 31;  // the body is the pair's A side
constexpr uint32_t ENT_LAST = 1u << 30;    // last item of its pair
constexpr uint32_t ENT_ROLL = 1u << 29;    // the point's rolling and torsion rows
constexpr uint32_t ENT_DUAL = 1u << 28;    // this side updates the point's dual (the pair's first swept colour)
constexpr uint32_t ENT_BODY = ENT_DUAL - 1u;  // the other body
constexpr uint32_t ENT_PER_SLOT = 2 * MAX_PTS;  // items of one incidence slot: 8 points, twice with rolling

// Eight lanes per body walk its incidence slots; einfo[h] = (first slot, items).
__global__ void __launch_bounds__(256) k_entries(DW w) {
    if (aborted_solve(w)) return;
    const uint32_t h = (blockIdx.x * blockDim.x + threadIdx.x) >> 3, l8 = threadIdx.x & 7u;
    if (h >= (uint32_t)w.N || w.colour[h] < 0) return;
    const uint32_t mask = 0xffu << (threadIdx.x & 24u);
    const uint32_t a0 = w.offA[h], b0 = w.offB[h], nB = w.offB[h + 1] - b0, n = nB + w.offA[h + 1] - a0;
    uint2* out = w.ent + (size_t)(a0 + b0) * ENT_PER_SLOT;
    uint32_t cnt = 0;
    for (uint32_t j0 = 0; j0 < n; j0 += 8) {
        const uint32_t j = j0 + l8;
        const bool side_a = j >= nB;
        uint32_t p = 0, np = 0, other = 0;
        bool roll = false, dual = false;
        if (j < n) {
            p = side_a ? a0 + (j - nB) : w.listB[b0 + j];
            np = min(w.p_np[p], (uint32_t)MAX_PTS);
            const uint2 ab = w.p_ab[p];
            other = side_a ? ab.y : ab.x;
            // neighbours have one colour only where the scene has more than the
            // solver's 64 (E_COLOUR_OVERFLOW): the lower handle's side then
            const int ch = w.colour[h], co = w.colour[other];
            dual = co < 0 || ch < co || (ch == co && h < other);
            if (w.p_n[p].w <= 0.0f) {
                const float4 ma = w.mat[ab.x], mb = w.mat[ab.y];
                roll = fmaxf(ma.z, mb.z) > 0.0f || fmaxf(ma.w, mb.w) > 0.0f;
            }
        }
        const uint32_t m = roll ? 2u * np : np;
        uint32_t inc = m;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const uint32_t v = __shfl_up_sync(mask, inc, o, 8);
            if (l8 >= (uint32_t)o) inc += v;
        }
        uint2* e = out + cnt + (inc - m);
        if (roll && np) w.ctr[C_ROLL] = 1u;
        const uint32_t tag = other | (side_a ? ENT_SIDE_A : 0u) | (dual ? ENT_DUAL : 0u);
        for (uint32_t k = 0; k < np; k++) {
            const uint32_t last = k + 1 == np ? ENT_LAST : 0u;
            *e++ = make_uint2(p * MAX_PTS + k, tag | (roll ? 0u : last));
            if (roll) *e++ = make_uint2(p * MAX_PTS + k, tag | ENT_ROLL | last);
        }
        cnt += __shfl_sync(mask, inc, 7, 8);
    }
    if (l8 == 0) w.einfo[h] = make_uint2(a0 + b0, cnt);
}

constexpr int SLOT = 36;        // floats of an item's slot: 8 float4, padded so that 32 slots spread over the banks
constexpr int SYS_STRIDE = 27;  // 21 Hessian + 6 right-hand-side numbers (odd: no bank conflicts)
constexpr uint32_t JOINT_PARTS = 3;  // items of a joint: up to 9 rows (revolute with a limit: 7)
// an item's control word: row types (6 bits), last item of its pair, a joint's
constexpr uint32_t CTL_LAST = 1u << 8, CTL_JOINT = 1u << 9;
constexpr uint32_t CTL_MIXED = 1u << 10;  // a row that is not ROW_FULL

struct WarpMem {
    float rows[35 * SLOT];  // the sums read up to three slots past the last
    float sys[32 * SYS_STRIDE];
    float ones[4];
};

// The number of the 6x6 system a lane owns, as float offsets into a slot:
// value += slot[c] * (slot[a] * slot[b]).
struct Elem {
    int a, b, c;
    int own;              // the number's index (a lane past 26 repeats 26)
    bool rhs, ang, diag;  // right-hand side; both factors angular; an angular diagonal
};
static __device__ __forceinline__ Elem elem_of(int lane) {
    Elem e;
    e.own = lane < SYS_STRIDE ? lane : SYS_STRIDE - 1;
    int i = 0, j = 0;
    e.rhs = lane >= 21;
    if (e.rhs) {
        i = lane < 27 ? lane - 21 : 0;
    } else {
        while (lane >= tri(i + 1, 0)) i++;
        j = lane - tri(i, 0);
    }
    e.a = 4 * (i < 3 ? i : i + 1);
    e.b = 4 * (j < 3 ? j : j + 1);
    e.c = e.rhs ? 28 : 12;
    e.ang = i >= 3 && (e.rhs || j >= 3);
    e.diag = !e.rhs && i >= 3 && i == j;
    return e;
}
// A lane's terms of a slot's three rows (dg: the value a diagonal row adds).
struct Terms {
    float x, y, z;
    float dx, dy, dz;
};
static __device__ __forceinline__ Terms slot_terms(const float* slot, const float* ones, const Elem& e) {
    const float4 A = *reinterpret_cast<const float4*>(slot + e.a);
    const float4 B = *reinterpret_cast<const float4*>(e.rhs ? ones : slot + e.b);
    const float4 C = *reinterpret_cast<const float4*>(slot + e.c);
    return Terms{C.x * (A.x * B.x), C.y * (A.y * B.y), C.z * (A.z * B.z), A.x, A.y, A.z};
}
static __device__ __forceinline__ void add_row(float& s, uint32_t type, float v, float diag, const Elem& e) {
    if (type == ROW_FULL || (type == ROW_ANG && e.ang)) s += v;
    else if (type == ROW_DIAG && e.diag) s += diag;
}
// Add a slot's rows, in order, to the lane's number.
static __device__ __forceinline__ void add_terms(const Terms& t, uint32_t ctl, const Elem& e, float& s) {
    add_row(s, ctl & 3u, t.x, t.dx, e);
    add_row(s, (ctl >> 2) & 3u, t.y, t.dy, e);
    add_row(s, (ctl >> 4) & 3u, t.z, t.dz, e);
}

// What a recording rollout keeps: a point's state after the dual of iteration
// slice - 1, a body's pose after the sweep of it (slice 0 is the start).
static __device__ __forceinline__ void record_point(const IterRec& rec, int slice, uint32_t q, float4 lam, float4 pen) {
    if (q >= rec.qcap) return;  // a frame too small: the host reports it
    rec.lam[(size_t)slice * rec.qstride + q] = lam;
    rec.pen[(size_t)slice * rec.qstride + q] = pen;
}
static __device__ __forceinline__ void record_pose(const DW& w, const IterRec& rec, int slice, uint32_t h) {
    const size_t i = (size_t)slice * (size_t)w.N + h;
    rec.pos[i] = w.pos[h];
    rec.rot[i] = w.rot[h];
}
// One iteration of the engine: whether this iteration's items first update
// their points' duals (of the iteration before), and what is recorded.
struct IterCtx {
    int it;
    bool dual;
    float* contrib;  // null, or recording: where the pairs' sums go, 28 floats per incidence slot
};
// the sum of the pair whose last item holds `slot`
static __device__ __forceinline__ void keep_pair(const IterRec& rec, const IterCtx& ic, const float* slot, float ps) {
    const uint32_t lane = threadIdx.x & 31u, q = __float_as_uint(slot[SLOT - 1]);
    if (lane < SYS_STRIDE && q < rec.slots) ic.contrib[(size_t)q * 28 + lane] = ps;  // else the host reports it
}
// An item of body h: a (point, side) of its list, or a third of joint e.x.
struct Item {
    uint32_t h;
    uint2 e;
    bool joint;
};
// The item's rows into the lane's slot; returns its control word.
template <int JT, bool PS, bool REC>
static __device__ __forceinline__ uint32_t item_rows(const DW& w, const IterRec& rec, const IterCtx& ic, float* slot,
                                                     const Item& im) {
    const uint32_t h = im.h;
    const uint2 e = im.e;
    if (JT && im.joint) {
        RowSink sink{slot, (int)(3u * e.y), 0, 0u};
        stamp_joint<JT == 2>(w, e.x, h, sink);
        return sink.types | CTL_JOINT | CTL_MIXED;
    }
    const bool side_a = (e.y & ENT_SIDE_A) != 0u, dual = ic.dual && (e.y & ENT_DUAL);
    const uint32_t other = e.y & ENT_BODY, p = e.x / MAX_PTS;
    const float4 ra = w.q_ra[e.x], rb = w.q_rb[e.x];
    float4 lam = w.q_lam[e.x], pen = w.q_pen[e.x];
    PairCtx c;
    load_ctx(w, p, side_a ? make_uint2(h, other) : make_uint2(other, h), c);
    const bool touching = c.gap <= 0.0f;
    const ContactGeo g = contact_geo(c, ra, rb, touching ? lam.w : 0.0f, touching || dual);
    if (dual) {
        dual_update(w, c, g, e.x, rb.w, lam, pen);
        if (REC && ic.contrib) record_point(rec, ic.it, e.x, lam, pen);
    }
    const ContactRows r = contact_rows(w, c, g, side_a, lam, pen);
    uint32_t ctl = (e.y & ENT_LAST) ? CTL_LAST : 0u;
    if (e.y & ENT_ROLL) {
        load_rolling(w, c);
        RowSink sink{slot, 0, 0, 0u};
        stamp_rolling(w, c, e.x, side_a, r.f[0], sink);
        ctl |= sink.types | CTL_MIXED;
    } else {
        const float sign = side_a ? 1.0f : -1.0f;
        const V3 n0 = sign * c.n, n1 = sign * c.t1, n2 = sign * c.t2;
        const V3 m0 = cross(r.lever, n0), m1 = cross(r.lever_f, n1), m2 = cross(r.lever_f, n2);
        float4* o = reinterpret_cast<float4*>(slot);
        o[0] = make_float4(n0.x, n1.x, n2.x, 0.0f);
        o[1] = make_float4(n0.y, n1.y, n2.y, 0.0f);
        o[2] = make_float4(n0.z, n1.z, n2.z, 0.0f);
        o[3] = make_float4(r.pen[0], r.pen[1], r.pen[2], 0.0f);
        o[4] = make_float4(m0.x, m1.x, m2.x, 0.0f);
        o[5] = make_float4(m0.y, m1.y, m2.y, 0.0f);
        o[6] = make_float4(m0.z, m1.z, m2.z, 0.0f);
        o[7] = make_float4(r.f[0], r.f[1], r.f[2], 0.0f);
        ctl |= (r.live & 1u) | (r.live & 2u) << 1 | (r.live & 4u) << 2;
    }
    if (REC && ic.contrib && (ctl & CTL_LAST))  // the pair's incidence slot, in the slot's padding
        slot[SLOT - 1] = __uint_as_float(side_a ? p + w.offB[h + 1] : w.offA[h] + w.posB[p]);
    return ctl;
}

// A warp's tile, bodies list[i0 .. i0 + nb) of one colour (nb <= 32): lane i
// holds body i's item count and its first item among the tile's `total`.
struct Tile {
    uint32_t nb, total;
    uint32_t h, first, ne, cnt, pre, j0;
    Item im;  // the lane's item of the first round
};
// The lane's item g of the tile (fetch: also its list entry), its body's lane.
template <int JT>
static __device__ __forceinline__ Item tile_item(const DW& w, const Tile& t, uint32_t g, uint32_t& b, bool fetch) {
    const uint32_t all = 0xffffffffu;
    // its body: the last lane whose first item is at or before it
    b = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
        const uint32_t v = __shfl_sync(all, t.pre, b + step);
        if (v <= g) b += step;
    }
    const uint32_t h = __shfl_sync(all, t.h, b), first = __shfl_sync(all, t.first, b), ne = __shfl_sync(all, t.ne, b);
    const uint32_t k = g - __shfl_sync(all, t.pre, b), j0 = JT ? __shfl_sync(all, t.j0, b) : 0u;
    Item im{h, make_uint2(0u, 0u), false};
    if (g < t.total) {
        if (JT && k >= ne) {
            im.joint = true;
            if (fetch) im.e = make_uint2(w.jlist[j0 + (k - ne) / JOINT_PARTS], (k - ne) % JOINT_PARTS);
        } else if (fetch) {
            im.e = w.ent[(size_t)first * ENT_PER_SLOT + k];
        }
    }
    return im;
}
// What a tile needs that no other body's move changes: its items and its
// bodies' inertial blocks (a body's own pose moves only in its own solve).
// Run while a barrier is being waited for.
template <int JT>
static __device__ __forceinline__ Tile open_tile(const DW& w, WarpMem& sm, const Recip& rdt2, const uint32_t* list,
                                                 uint32_t i0, uint32_t nb) {
    const uint32_t lane = threadIdx.x & 31u, all = 0xffffffffu;
    Tile t{nb, 0, 0, 0, 0, 0, 0, 0, Item{0, make_uint2(0u, 0u), false}};
    if (nb == 0) return t;
    uint32_t nj = 0;
    if (lane < nb) {
        t.h = list[i0 + lane];
        const uint2 ei = w.einfo[t.h];
        t.first = ei.x;
        t.ne = ei.y;
        if (JT) {
            t.j0 = w.jofs[t.h];
            nj = w.jofs[t.h + 1] - t.j0;
        }
    }
    t.cnt = t.ne + JOINT_PARTS * nj;
    uint32_t pre = t.cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(all, pre, o);
        if (lane >= (uint32_t)o) pre += v;
    }
    t.total = __shfl_sync(all, pre, 31);
    t.pre = pre - t.cnt;  // past the last body: total
    uint32_t b;
    t.im = tile_item<JT>(w, t, lane, b, true);
    if (lane < nb) {
        Sys s;
        inertial_block(w, t.h, rdt2, s);
        float* o = sm.sys + lane * SYS_STRIDE;
#pragma unroll
        for (int k = 0; k < 21; k++) o[k] = s.h[k];
#pragma unroll
        for (int k = 0; k < 6; k++) o[21 + k] = s.r[k];
    }
    return t;
}
// Solve a tile by its warp.  A caller whose next bodies read the moved poses
// synchronises first.
template <int JT, bool PS, bool REC>
static __device__ __forceinline__ void solve_tile(const DW& w, const IterRec& rec, const IterCtx& ic, WarpMem& sm,
                                                  const Elem& el, const Tile& tile) {
    const uint32_t lane = threadIdx.x & 31u, all = 0xffffffffu;
    const uint32_t h = tile.h, pre = tile.pre, cnt = tile.cnt, total = tile.total;
    __syncwarp();
    float ps = 0.0f;  // sum of the pair being added (a pair's items may span two rounds)
    for (uint32_t r0 = 0; r0 < total; r0 += 32) {
        const uint32_t g = r0 + lane;
        uint32_t b;
        Item im = tile_item<JT>(w, tile, g, b, r0 != 0);
        if (r0 == 0) im.e = tile.im.e;
        uint32_t ctl = 0;
        if (g < total) ctl = item_rows<JT, PS, REC>(w, rec, ic, sm.rows + lane * SLOT, im);
        __syncwarp();
        // which items have each row live, end a pair, hold other rows than ROW_FULL
        const uint32_t m0 = __ballot_sync(all, ctl & 1u), m1 = __ballot_sync(all, ctl & 4u), m2 = __ballot_sync(all, ctl & 16u);
        const uint32_t ml = PS ? __ballot_sync(all, ctl & CTL_LAST) : 0u;
        const bool plain = !__any_sync(all, ctl & CTL_MIXED);
        const uint32_t n = min(32u, total - r0);
        const uint32_t blast = __shfl_sync(all, b, n - 1);
        for (uint32_t bb = __shfl_sync(all, b, 0); bb <= blast; bb++) {
            const uint32_t f = __shfl_sync(all, pre, bb), e1 = min(f + __shfl_sync(all, cnt, bb), r0 + 32u) - r0;
            const uint32_t e0 = max(f, r0) - r0;
            if (f >= r0 + 32u || e0 >= e1) continue;
            float s = sm.sys[bb * SYS_STRIDE + el.own];
            if (plain) {
                // four items a round: their loads and products are independent, the sums follow in
                // order (bits past the body's last item are off)
                const uint32_t own = e1 < 32u ? (1u << e1) - 1u : all;
                const uint32_t x0 = m0 & own, x1 = m1 & own, x2 = m2 & own, xl = ml & own;
                for (uint32_t e = e0; e < e1; e += 4) {
                    Terms t[4];
#pragma unroll
                    for (uint32_t k = 0; k < 4; k++) t[k] = slot_terms(sm.rows + (e + k) * SLOT, sm.ones, el);
#pragma unroll
                    for (uint32_t k = 0; k < 4; k++) {
                        float& acc = PS ? ps : s;
                        if ((x0 >> e) & (1u << k)) acc += t[k].x;
                        if ((x1 >> e) & (1u << k)) acc += t[k].y;
                        if ((x2 >> e) & (1u << k)) acc += t[k].z;
                        if (PS && ((xl >> e) & (1u << k))) {
                            if (REC && ic.contrib) keep_pair(rec, ic, sm.rows + (e + k) * SLOT, ps);
                            s += ps;
                            ps = 0.0f;
                        }
                    }
                }
            } else {
                for (uint32_t e = e0; e < e1; e++) {
                    const uint32_t c = __shfl_sync(all, ctl, e);
                    const float* slot = sm.rows + e * SLOT;
                    const Terms t = slot_terms(slot, sm.ones, el);
                    if (PS && !(JT && (c & CTL_JOINT))) {
                        add_terms(t, c, el, ps);
                        if (c & CTL_LAST) {
                            if (REC && ic.contrib) keep_pair(rec, ic, slot, ps);
                            s += ps;
                            ps = 0.0f;
                        }
                    } else {
                        add_terms(t, c, el, s);
                    }
                }
            }
            if (lane < SYS_STRIDE) sm.sys[bb * SYS_STRIDE + lane] = s;
        }
        __syncwarp();
    }
    __syncwarp();
    if (lane < tile.nb) {
        const BodyPose pose = load_pose(w, h);
        Sys t;
        const float* o = sm.sys + lane * SYS_STRIDE;
#pragma unroll
        for (int k = 0; k < 21; k++) t.h[k] = o[k];
#pragma unroll
        for (int k = 0; k < 6; k++) t.r[k] = o[21 + k];
        apply_solve(w, h, pose, t);
        if (REC && ic.contrib) record_pose(w, rec, ic.it + 1, h);
    }
    __syncwarp();
}

// The duals of iterations [first, end) of every pair by threads t of n, four
// per pair; a pair without a swept body takes [unswept_first, end).
// A pair's dual reads its two bodies at the end of an iteration, and they hold
// still until the pair's first swept colour of the next one: there its item
// has the constraint values at hand, so it updates the dual before it stamps
// its rows (IterCtx::dual), and no pass over the points runs between
// iterations.  This pass then makes up the rest after the last iteration: its
// dual, and every iteration's for a pair that no item visits.
template <bool REC>
static __device__ __forceinline__ void dual_pass(const DW& w, const IterRec& rec, uint32_t t, uint32_t n, int first,
                                                 int unswept_first, int end) {
    const uint32_t np_all = n_pairs(w);
    for (uint32_t i = t; i < np_all * 4u; i += n) {
        const uint32_t p = i >> 2, np = w.p_np[p];
        if (REC && rec.contrib && np == 0u && (i & 3u) < 2u) {  // pairs without points: zero sums
            const uint2 ab = w.p_ab[p];
            const uint32_t slot = (i & 3u) ? p + w.offB[ab.x + 1] : w.offA[ab.y] + w.posB[p];
            for (int it = unswept_first; it < end && slot < rec.slots; it++)
                for (int k = 0; k < 7; k++)
                    rec.contrib[(size_t)it * rec.cstride + (size_t)slot * 7 + k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        if ((i & 3u) >= np) continue;
        PairCtx c;
        load_ctx(w, p, c);
        const int it0 = w.colour[c.a] < 0 && w.colour[c.b] < 0 ? unswept_first : first;
        for (uint32_t k = i & 3u; k < np; k += 4u) {
            const uint32_t q = p * MAX_PTS + k;
            for (int it = it0; it < end; it++) {
                float4 lam, pen;
                dual_point(w, c, q, lam, pen);
                if (REC && rec.contrib) record_point(rec, it + 1, q, lam, pen);
            }
        }
    }
}
static __device__ __forceinline__ void record_joint(const DW& w, const IterRec& rec, int it, uint32_t j) {
    const size_t J = (size_t)w.J;
    float4* o = rec.joint + (size_t)(it + 1) * 5 * J + j;
    o[0] = w.j_lam_l[j];
    o[J] = w.j_pen_l[j];
    o[2 * J] = w.j_lam_a[j];
    o[3 * J] = w.j_pen_a[j];
    o[4 * J] = w.j_lim[j];
}

// REC: the instantiation of differentiable worlds, recording or not: a
// rollout's plain and recorded passes run the same code, so they agree bit for
// bit in the fast build too, where contraction differs from one instantiation
// to the next.
// Every iteration: per colour its bodies dealt over all warps of the launch,
// a barrier, and with joints a pass over their duals.
template <int BS, int JT, bool PS, bool REC>
__global__ void __launch_bounds__(BS, 512 / BS) k_iterations(DW w, IterRec rec, int sync) {
    if (aborted_solve(w)) return;
    constexpr uint32_t NW = BS / 32;
    extern __shared__ float4 s_dyn[];
    WarpMem& sm = reinterpret_cast<WarpMem*>(s_dyn)[threadIdx.x >> 5];
    __shared__ uint32_t s_ok;
    const Elem el = elem_of(threadIdx.x & 31u);
    const Recip rdt2 = recip_dt2(w);
    if ((threadIdx.x & 31u) < 4u) sm.ones[threadIdx.x & 31u] = 1.0f;
    __syncwarp();
    const uint32_t warps = gridDim.x * NW, threads = gridDim.x * BS, tid = blockIdx.x * BS + threadIdx.x;
    // neighbouring blocks take neighbouring tiles: warp k of block b is number k * gridDim + b
    const uint32_t wid = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const int ncol = (int)min(w.ctr[C_NCOL], (uint32_t)MAX_COLOURS), iters = w.iterations;
    // rolling rows read what the dual writes: with any, the dual keeps its own pass
    const bool lazy = w.ctr[C_ROLL] == 0u;
    if (REC && rec.contrib)
        for (uint32_t h = tid; h < (uint32_t)w.N; h += threads)
            if (w.colour[h] < 0)
                for (int it = 0; it < iters; it++) record_pose(w, rec, it + 1, h);
    __shared__ uint32_t s_col[MAX_COLOURS + 1];
    for (uint32_t c = threadIdx.x; c <= MAX_COLOURS; c += BS) s_col[c] = w.col_cnt[c];
    __syncthreads();
    // bodies of colour c a warp takes at a time: every warp the same number of
    // equal tiles, as few of up to 32 bodies as hold the colour
    auto tile_size = [&](int c) {
        const uint32_t n = s_col[c + 1] - s_col[c], rounds = max(1u, (n + 32u * warps - 1u) / (32u * warps));
        return (n + rounds * warps - 1u) / (rounds * warps);
    };
    auto open = [&](int c, uint32_t i, uint32_t tb) {
        const uint32_t n = s_col[c + 1] - s_col[c];
        return open_tile<JT>(w, sm, rdt2, w.col_list, s_col[c] + i, i < n ? min(tb, n - i) : 0u);
    };
    if (iters <= 0) return;
    uint32_t* bar = &w.ctr[C_GBAR];
    uint32_t target = 0;
    uint32_t tb = ncol ? tile_size(0) : 0u;
    Tile tile = open(0, wid * tb, tb);
    for (int it = 0; it < iters; it++) {
        const IterCtx ic{it, lazy && it > 0,
                         REC && rec.contrib ? reinterpret_cast<float*>(rec.contrib + (size_t)it * rec.cstride) : nullptr};
        const bool last = it + 1 == iters;
        for (int c = 0; c < ncol; c++) {
            const uint32_t n = s_col[c + 1] - s_col[c];
            for (uint32_t i = wid * tb; i < n;) {
                solve_tile<JT, PS, REC>(w, rec, ic, sm, el, tile);
                i += warps * tb;
                if (i < n) tile = open(c, i, tb);
            }
            const int next = c + 1 < ncol ? c + 1 : 0;
            all_arrive(bar, sync);
            if (c + 1 < ncol || !last) {
                tb = tile_size(next);
                tile = open(next, wid * tb, tb);
            }
            if (!all_wait(w, bar, sync, target, &s_ok)) return;
        }
        if (!lazy || last) dual_pass<REC>(w, rec, tid, threads, it, lazy ? 0 : it, it + 1);
        if (JT)
            for (uint32_t j = tid; j < (uint32_t)w.J; j += threads) {
                dual_joint<JT == 2>(w, j);
                if (REC && ic.contrib) record_joint(w, rec, it, j);
            }
        if (!last && (JT || !lazy) && !all_sync(w, bar, sync, target, &s_ok)) return;
    }
}

template <int BS, int JT, bool PS, bool REC>
static void iterations_launch(const DW& w, const IterRec& rec, cudaStream_t st) {
    static Resident r;
    launch_synced(r, k_iterations<BS, JT, PS, REC>, BS, (BS / 32) * sizeof(WarpMem), w.N, st, w, rec);
}
// Every iteration of the substep in the thread-per-body order (lanes 1) or
// the split order (lanes 0, -1); r: what a rollout records of them.  A
// differentiable world (sort_static) runs the split order, without the joint
// kinds its reverse sweep refuses.
void launch_iterations(const DW& w, const Tune& tune, const IterRec& r, cudaStream_t st) {
    k_entries<<<nblk((size_t)w.N * 8, 256), 256, 0, st>>>(w);
    const bool ps = tune.primal_lanes <= 0;
    if (r.contrib || (w.sort_static && ps && !w.j_all)) {
        if (!w.J) iterations_launch<256, 0, true, true>(w, r, st);
        else iterations_launch<256, 1, true, true>(w, r, st);
        return;
    }
    const int jt = !w.J ? 0 : (w.j_all ? 2 : 1);
    if (jt == 0) ps ? iterations_launch<256, 0, true, false>(w, r, st) : iterations_launch<256, 0, false, false>(w, r, st);
    else if (jt == 1) ps ? iterations_launch<256, 1, true, false>(w, r, st) : iterations_launch<256, 1, false, false>(w, r, st);
    else ps ? iterations_launch<256, 2, true, false>(w, r, st) : iterations_launch<256, 2, false, false>(w, r, st);
}

void launch_side_lists(const DW& w, cudaStream_t st) {
    k_zero_u32<<<1, 256, 0, st>>>(w.side_cnt, 2 * MAX_COLOURS + 2);
    k_side_count<<<gsz(w.pair_cap, SIDE_BLOCK), SIDE_BLOCK, 0, st>>>(w);
    k_side_starts<<<1, 32, 0, st>>>(w);
    k_side_place<<<gsz(w.pair_cap, SIDE_BLOCK), SIDE_BLOCK, 0, st>>>(w);
}
// The lanes-per-body forms: one launch per colour.
template <int J>
static void primal_colour(const DW& w, const Tune& tune, int c, uint32_t max_bodies, cudaStream_t st) {
    int bs = tune.primal_block;
    switch (tune.primal_lanes) {
        case 4: k_primal_lanes<4, J><<<nblk((size_t)max_bodies * 4, bs), bs, 0, st>>>(w, c); break;
        case 8: k_primal_lanes<8, J><<<nblk((size_t)max_bodies * 8, bs), bs, 0, st>>>(w, c); break;
        case 16: k_primal_lanes<16, J><<<nblk((size_t)max_bodies * 16, bs), bs, 0, st>>>(w, c); break;
        default: k_primal_lanes<32, J><<<nblk((size_t)max_bodies * 32, bs), bs, 0, st>>>(w, c); break;
    }
}
void launch_primal_colour(const DW& w, const Tune& tune, int c, uint32_t max_bodies, cudaStream_t st) {
    if (!w.J) primal_colour<0>(w, tune, c, max_bodies, st);
    else if (!w.j_all) primal_colour<1>(w, tune, c, max_bodies, st);
    else primal_colour<2>(w, tune, c, max_bodies, st);
}
void launch_dual(const DW& w, const Tune& tune, cudaStream_t st) {
    k_dual_pairs<<<gsz(w.pair_cap, 128), 128, 0, st>>>(w);
    if (w.J) {
        if (w.j_all) k_dual_joints<true><<<nblk(w.J, 128), 128, 0, st>>>(w);
        else k_dual_joints<false><<<nblk(w.J, 128), 128, 0, st>>>(w);
    }
}
void launch_iteration(const DW& w, const Tune& tune, int ncolours, cudaStream_t st) {
    for (int c = 0; c < ncolours; c++) AVBD_SOLVE_NS::launch_primal_colour(w, tune, c, (uint32_t)w.N, st);
    AVBD_SOLVE_NS::launch_dual(w, tune, st);
}

// ---- BDF1 + sleep + driver baseline (mod.rs:1060-1142) -------------------------
// flag bits for the sleep pass: 1 joint-ready, 2 supported, 4 freeze.  Every
// writer of a flag byte within one kernel changes the same bit the same way.
__global__ void k_bdf1(DW w) {
    if (aborted_solve(w)) return;
    uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= (uint32_t)w.N) return;
    w.flag[h] = 1;
    w.comp_flag[h] = 0;
    if (!solved(w, h)) return;
    V3 p = ld3(w.pos[h]);
    w.vel[h] = st3((p - ld3(w.pos0[h])) / w.dt, 0.0f);
    Q q = ldq(w.rot[h]);
    V3 spin = quat_diff_vec(q, ldq(w.rot0[h]));
    w.angvel[h] = st3(len(spin) < SPIN_REST_EPS ? V0() : spin / w.dt, 0.0f);
    w.rot[h] = stq(qnormalize(q));
}
__global__ void k_ready_joint(DW w) {
    if (aborted_solve(w)) return;
    uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= (uint32_t)w.J) return;
    if (joint_driven(w, j) || joint_rest_error(w, j) > JOINT_REST_ERROR) {
        uint32_t m[4];
        const int nm = joint_members(w, j, m);
        for (int k = 0; k < nm; k++) w.flag[m[k]] &= (uint8_t)~1u;
    }
}
__global__ void k_ready_gather(DW w) {
    if (aborted_solve(w)) return;
    uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= (uint32_t)w.N) return;
    int c = w.comp[h];
    if (c >= 0 && is_dynamic(w, h) && !(w.flag[h] & 1)) w.comp_flag[c] = 1;
}
__global__ void k_ready_scatter(DW w) {
    if (aborted_solve(w)) return;
    uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= (uint32_t)w.N) return;
    int c = w.comp[h];
    if (c >= 0 && is_dynamic(w, h) && w.comp_flag[c]) w.flag[h] &= (uint8_t)~1u;
}
__global__ void k_support_joints(DW w) {
    if (aborted_solve(w)) return;
    uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= (uint32_t)w.J) return;
    uint2 ab = w.j_ab[j];
    w.flag[ab.x] |= 2;
    w.flag[ab.y] |= 2;
}
static __device__ __forceinline__ void k_support_one(const DW& w, uint32_t p) {
    if (w.p_n[p].w <= 0.0f && w.p_np[p] > 0) {
        uint2 ab = w.p_ab[p];
        w.flag[ab.x] |= 2;
        w.flag[ab.y] |= 2;
    }
}
__global__ void k_support(DW w) {
    if (aborted_solve(w)) return;
    const uint32_t n = n_pairs(w);
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x)
        k_support_one(w, p);
}

// Sleep timer of body h; returns whether it may freeze.
static __device__ __forceinline__ bool sleep_timer(const DW& w, uint32_t h) {
    uint8_t f = w.flag[h];
    bool freeze = w.asleep[h] != 0;
    if (solved(w, h)) {
        if (!(f & 2) || !(f & 1)) {
            w.sleep_timer[h] = 0.0f;
        } else if (len(ld3(w.vel[h])) < SLEEP_LIN && len(ld3(w.angvel[h])) < SLEEP_ANG) {
            float t = w.sleep_timer[h] + w.dt;
            w.sleep_timer[h] = t;
            freeze = t >= SLEEP_TIME;
        } else {
            w.sleep_timer[h] = 0.0f;
        }
    }
    return freeze;
}
static __device__ __forceinline__ void freeze_apply(const DW& w, uint32_t h, bool freeze, int sleep_on) {
    if (sleep_on) {
        if (freeze && !w.asleep[h] && is_dynamic(w, h)) {  // sleep_staticify (body.rs:403-408)
            w.vel[h] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            w.angvel[h] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            w.inv_mass[h] = 0.0f;
            w.inertia[h] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            w.asleep[h] = 1;
        }
        if (w.asleep[h]) agg_inc(&w.ctr[C_SLEEP]);
    }
    w.prev_pos[h] = w.pos[h];
    w.prev_rot[h] = w.rot[h];
}
// Without joints a body freezes by itself: timer and freeze in one launch.
__global__ void k_sleep(DW w, int sleep_on) {
    if (aborted_solve(w)) return;
    uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= (uint32_t)w.N) return;
    freeze_apply(w, h, sleep_on && sleep_timer(w, h), sleep_on);
}
__global__ void k_sleep_timer(DW w) {
    if (aborted_solve(w)) return;
    uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= (uint32_t)w.N) return;
    w.flag[h] = sleep_timer(w, h) ? 4 : 0;
    w.comp_flag[h] = 0;
}
__global__ void k_freeze_gather(DW w) {
    if (aborted_solve(w)) return;
    uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= (uint32_t)w.N) return;
    int c = w.comp[h];
    if (c >= 0 && is_dynamic(w, h) && !(w.flag[h] & 4)) w.comp_flag[c] = 1;
}
__global__ void k_freeze_apply(DW w) {
    if (aborted_solve(w)) return;
    uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= (uint32_t)w.N) return;
    bool freeze = (w.flag[h] & 4) != 0;
    int c = w.comp[h];
    if (c >= 0 && is_dynamic(w, h) && w.comp_flag[c]) freeze = false;
    freeze_apply(w, h, freeze, 1);
}

void launch_finish_substep(const DW& w, cudaStream_t st) {
    unsigned gb = nblk(w.N, 256);
    k_bdf1<<<gb, 256, 0, st>>>(w);
    if (w.enable_sleep) {
        if (w.J) {
            k_ready_joint<<<nblk(w.J, 128), 128, 0, st>>>(w);
            k_ready_gather<<<gb, 256, 0, st>>>(w);
            k_ready_scatter<<<gb, 256, 0, st>>>(w);
            k_support_joints<<<nblk(w.J, 128), 128, 0, st>>>(w);
        }
        k_support<<<gsz(w.pair_cap, 256), 256, 0, st>>>(w);
        if (w.J) {
            k_sleep_timer<<<gb, 256, 0, st>>>(w);
            k_freeze_gather<<<gb, 256, 0, st>>>(w);
            k_freeze_apply<<<gb, 256, 0, st>>>(w);
            return;
        }
    }
    k_sleep<<<gb, 256, 0, st>>>(w, w.enable_sleep);
}

}  // namespace AVBD_SOLVE_NS
}  // namespace avbd
