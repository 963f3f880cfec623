// pge_trace.cuh -- the exact pass's trace: one warp a droplet, records the change list only.
//
// Same steps, same operations and the same rounding as the record-only droplet_kernel (pge_droplets.cuh; the
// reference's trace loop, bake/globe/erosion/particle.py:421-815): the lists are identical bit for bit.  Included by
// pge_droplets_f64.cu behind that file, compiled without contraction.
//
// What bounds a wave is one droplet's serial chain of steps.  On a thread of its own a step is one long in-order run
// of ~1000 instructions, eleven divisions and roots of the path and seven of the mass transfer among them (305 us a
// wave of 2048 droplets on the N_c = 1024 sphere, some 6000 cycles a step).  But the path does not depend on the load:
// positions, directions and the volume are decided by the frozen surface alone, and the load only adds two ways to
// die, both at sea.  So a warp
//   1. walks the path up to TB steps ahead.  All lanes walk the same path; where a step needs several like things at
//      once (the four channels' bilinear samples, three roots, two rounds of quotients) each of four lane roles
//      computes one of them and a shuffle hands them round: the path's eleven divisions and roots become five, one
//      after another;
//   2. computes what the mass transfer needs that does not depend on the load (equilibrium, caps, their quotients by
//      the volume), a lane a step;
//   3. runs the load's own recurrence over the steps in order (a handful of operations and the quotient by the
//      evaporation, from its reciprocal), which also finds a death at sea that ends the path early;
//   4. writes the entries, a lane an entry.
// At sea the walk goes only TB_SEA steps ahead, since the load may end it.  Measured, a wave: 184 us (N_c = 1024 sphere),
// 297 with lakes (a thread a droplet: 493), 316 with banks (505), 82 where N_c = 32 (102).  A step's walk is ~2900
// cycles of it, ~800 of them the view's loads and ~1300 the five divisions and roots with their shuffles.
//
// The lanes agree on everything they walk, so one lane keeps the batch's record; a record stored by all 32 at once is
// a data race in the language's terms.
#pragma once

namespace pge {
namespace f64 {

namespace {

constexpr int TB = 32;
constexpr int TB_SEA = 8;
constexpr int RING = 64;  // active cells remembered: TB ahead, SPREAD behind, a power of two

// a step as the load sees it: from an active cell, at sea, at sea from its end on, crossing a lake, entering one, one
// with room
enum { TS_ACTIVE = 1, TS_SEA = 2, TS_SEA_NEXT = 4, TS_LAKE = 8, TS_TRAP = 16, TS_KEEPS = 32 };

// what the load's recurrence reads of a step (16-byte pieces)
struct __align__(16) LoadStep {
    double c_eq, k_up;     // towards c_eq: k_up from below it,
    double k_down, vol_rel;  // k_down from above
    double ecap, ecap_q;   // a pick-up's limit, and the concentration it allows
    double dcap, dcap_q;   // a deposit's
    double ev, inv_ev;     // inv_ev 0: divide
};
// the state a step starts from
struct __align__(16) PathStep {
    double x, y, vol, q, h0;
    float surf;
    int cell;
    float4 b;  // the cell's evaporation, hardness, sediment, base
    int face, nact;
};

// the bank beside a step (particle.py:699-738): what cutting it gives per unit of pick-up, and its limit
struct BankStep {
    double rate, lcap, lcap_q;
    double psa, psb;  // the direction the step started with
    double lat;       // cut, once the load is known
    int cell;
};

template <bool ROUTE, bool LATERAL>
struct TraceShared {
    LoadStep load[TB];
    PathStep path[TB + 1];  // n steps fill n + 1
    BankStep bank[LATERAL ? TB : 1];
    double2 dir[TB];  // the direction a step ends with
    double cdiff[TB];
    double rest[ROUTE ? TB : 1];
    int flags[TB];
    int ring[RING];
};

// what a step reads at a position, each lane its role's channel of the stencil
struct Spot {
    int cell, m;
    float surf;
    float4 b;  // evaporation, hardness, sediment, base
    double g0, g1, g2, q0, q1, q2;
    double h0, q, ma, mb;  // bilinear samples
    double hr, gi, gj;     // the surface steered on and its gradient
    float nflag;           // ROUTE: the cell's lake flag
};

template <bool ROUTE>
__device__ __forceinline__ void load_spot(const DropArgs &a, int role, int f, double x, double y, int ei, int ej, Spot &v)
{
    const int NE = a.NE;
    const double fi = x - 0.5 + double(a.H), fj = y - 0.5 + double(a.H);
    int i0 = (int)floor(fi), j0 = (int)floor(fj);
    if (i0 < 0) i0 = 0;
    if (i0 > NE - 2) i0 = NE - 2;
    if (j0 < 0) j0 = 0;
    if (j0 > NE - 2) j0 = NE - 2;
    const int c00 = (f * NE + i0) * NE + j0, cc = (f * NE + ei) * NE + ej;  // (cells fit 32 bits: check_shape)
    const float *A = reinterpret_cast<const float *>(a.A + c00);
    const float *A1 = reinterpret_cast<const float *>(a.A + c00 + NE);
    const float t00 = __ldg(A + role), t01 = __ldg(A + 4 + role), t10 = __ldg(A1 + role), t11 = __ldg(A1 + 4 + role);
    const float h00 = __ldg(A), h01 = __ldg(A + 4), h10 = __ldg(A1), h11 = __ldg(A1 + 4);
    v.b = __ldg(a.B + cc);
    const int mc = a.metric_shared ? ei * NE + ej : cc;
    const float4 g0 = __ldg(a.G + 2ll * mc), g1 = __ldg(a.G + 2ll * mc + 1);
    v.m = a.mask ? (int)__ldg(a.mask + cc) : PGE_MASK_ACTIVE;
    float2 r00, r01, r10, r11;
    if (ROUTE) {
        r00 = __ldg(a.R + c00);
        r01 = __ldg(a.R + c00 + 1);
        r10 = __ldg(a.R + c00 + NE);
        r11 = __ldg(a.R + c00 + NE + 1);
        v.nflag = a.lakes ? __ldg(&a.R[cc].y) : 0.0f;
    }
    const int di = ei - i0, dj = ej - j0;
    if ((unsigned)di <= 1u && (unsigned)dj <= 1u)
        v.surf = di ? (dj ? h11 : h10) : (dj ? h01 : h00);
    else
        v.surf = __ldg(&a.A[cc].x);
    double wi = fi - double(i0), wj = fj - double(j0);
    if (wi < 0.0) wi = 0.0;
    if (wi > 1.0) wi = 1.0;
    if (wj < 0.0) wj = 0.0;
    if (wj > 1.0) wj = 1.0;
    const double ui = 1.0 - wi, uj = 1.0 - wj;
    const double s = double(t00) * ui * uj + double(t10) * wi * uj + double(t01) * ui * wj + double(t11) * wi * wj;
    v.h0 = __shfl_sync(0xffffffffu, s, 0);
    v.q = __shfl_sync(0xffffffffu, s, 1);
    v.ma = __shfl_sync(0xffffffffu, s, 2);
    v.mb = __shfl_sync(0xffffffffu, s, 3);
    const float d10 = h10 - h00, d11 = h11 - h01, d01 = h01 - h00, d1110 = h11 - h10;
    v.gi = double(d10) * uj + double(d11) * wj;
    v.gj = double(d01) * ui + double(d1110) * wi;
    v.hr = v.h0;
    if (ROUTE) {
        // a lake or pit: steer on the routing surface where it is above the terrain (particle.py:453-460)
        float flag = r00.y + r10.y;
        flag = flag + r01.y;
        flag = flag + r11.y;
        if (flag != 0.0f) {
            const double r = double(r00.x) * ui * uj + double(r10.x) * wi * uj + double(r01.x) * ui * wj + double(r11.x) * wi * wj;
            if (r > v.h0) {
                const float e10 = r10.x - r00.x, e11 = r11.x - r01.x, e01 = r01.x - r00.x, e1110 = r11.x - r10.x;
                v.hr = r;
                v.gi = double(e10) * uj + double(e11) * wj;
                v.gj = double(e01) * ui + double(e1110) * wi;
            }
        }
    }
    v.cell = cc;
    v.g0 = double(g0.x);
    v.g1 = double(g0.y);
    v.g2 = double(g0.z);
    v.q0 = double(g0.w);
    v.q1 = double(g1.x);
    v.q2 = double(g1.y);
}

// whether |x| lies outside 2^-500 .. 2^500 (zero, infinity and NaN do)
__device__ __forceinline__ bool far_from_one(double x)
{
    return ((unsigned)__double2hiint(x) & 0x7fffffffu) - 0x20b00000u > 0x3e800000u;
}

__device__ __forceinline__ double norm2(const Spot &v, double a, double b)
{
    const double n2 = v.g0 * a * a + 2.0 * v.g1 * a * b + v.g2 * b * b;
    return n2 < 0.0 ? 0.0 : n2;
}

}  // namespace

template <bool ROUTE, bool LATERAL>
__global__ void __launch_bounds__(32, 14) trace_kernel(const DropArgs a)
{
    const PgeParams &p = a.p;
    __shared__ TraceShared<ROUTE, LATERAL> S;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x, role = lane & 3;
    const long long d = a.d_begin + blockIdx.x, row = d - a.rec_base;
    const int N = a.N, H = a.H, NE = a.NE;
    const double Nf = double(N), volume0 = a.volume0, inf = __longlong_as_double(0x7ff0000000000000ll);

    // the droplet, the same in every lane
    int f = a.sp_face[d];
    double x = a.sp_x[d], y = a.sp_y[d], sed = a.sp_sed[d], vol = volume0, sa = 0.0, sb = 0.0;
    if (sed > 0.0) {
        const Dir dd = a.cr_trig ? spawn_dir<true>(a.sp_dir[d]) : spawn_dir<false>(a.sp_dir[d]);
        sa = dd.c;
        sb = dd.s;
    }
    double accel = p.dt / (vol / volume0 * p.density);
    double fr = 1.0 - p.dt * p.friction;
    if (fr < 0.0) fr = 0.0;
    const double dt_evap = p.dt * p.evap_rate, sat2 = p.slope_sat > 0.0 ? p.slope_sat * p.slope_sat : 1.0;
    const double inv_sat = p.disc_saturation > 0.0 ? 1.0 / p.disc_saturation : 0.0;
    int step = 0, uphill = 0, sea_steps = 0, nact = 0, rec_n = 0;
    int nextra = 0, parked = 0;  // entries that are no steps: parks and banks; parks written
    [[maybe_unused]] int parks = 0;
    bool in_sea = false, in_lake = false;
    float h_prev = 0.0f;
    Spot v;
    load_spot<ROUTE>(a, role, f, x, y, cell_of(x, N) + H, cell_of(y, N) + H, v);
    if (v.surf < v.b.w && p.max_steps > 0 && v.m != PGE_MASK_OUTSIDE) in_sea = true;

    int cause = -1, at = 0, nring;  // death: its cause, the state it happened in, the ring's length there
    bool exited = false;
    do {
        // ---- 1. the path
        int n = 0;
        bool partial = false;  // the path ended inside step n, past its sea check
        bool sea_check = false;
        const int step0 = step;
        const float h_prev0 = h_prev;
        while (true) {
            if (lane == 0) {
                PathStep &t = S.path[n];
                *reinterpret_cast<double2 *>(&t.x) = make_double2(x, y);
                *reinterpret_cast<double2 *>(&t.vol) = make_double2(vol, v.q);
                t.h0 = v.h0;
                t.surf = v.surf;
                t.cell = v.cell;
                t.b = v.b;
                t.face = f;
                t.nact = nact;
            }
            if (cause >= 0 || n >= (in_sea ? TB_SEA : TB)) break;
            if (step >= p.max_steps) { cause = PGE_DEATH_AGE; break; }
            int fl = 0;
            if (v.m != PGE_MASK_ACTIVE || in_sea) {
                if (v.m == PGE_MASK_OUTSIDE) { exited = true; cause = PGE_DEATH_EXIT; break; }
                if (in_sea) {
                    if (v.surf >= v.b.w || sea_steps >= p.ocean_steps) { cause = PGE_DEATH_OCEAN; break; }
                    sea_steps++;
                    fl = TS_SEA;
                }
            }
            partial = true;
            sea_check = in_sea;
            if (v.m == PGE_MASK_ACTIVE) {
                fl |= TS_ACTIVE;
                if (lane == 0) S.ring[nact & (RING - 1)] = v.cell;
                nact++;
            }
            const double q = v.q < 0.0 ? 0.0 : v.q;
            double ev = 1.0 - dt_evap * double(v.b.x);
            if (ev < 0.01) ev = 0.01;
            const double vol1 = vol * ev;
            // forces
            const double di = v.q0 * v.gi + v.q1 * v.gj;
            const double dj = v.q1 * v.gi + v.q2 * v.gj;
            double s2 = v.gi * di + v.gj * dj;
            if (s2 < 0.0) s2 = 0.0;
            if (LATERAL && lane == 0) {
                S.bank[n].psa = sa;
                S.bank[n].psb = sb;
            }
            sa *= fr;
            sb *= fr;
            // roots: the slope's, the momentum's length, the direction's
            const double n2 = norm2(v, role == 1 ? v.ma : sa, role == 1 ? v.mb : sb);
            const double cosn = v.g0 * v.ma * sa + v.g1 * (v.ma * sb + v.mb * sa) + v.g2 * v.mb * sb;
            const double kden = vol + p.mom_scale * q;
            const double rt = sqrt(role == 0 ? s2 + sat2 : n2);
            const double mlen = __shfl_sync(full, rt, 1), slen0 = __shfl_sync(full, rt, 2);
            const bool mom = mlen > 1e-12 && slen0 > 1e-12;
            // quotients: the slope's gain, the momentum's cosine, the next step's relative volume
            double num = role == 0 ? p.slope_gain : vol1, den = role == 0 ? rt : volume0;
            num = role == 1 ? cosn : num;
            den = role == 1 ? (mom ? mlen * slen0 : 1.0) : den;
            const double qt = num / den;
            const double nrm = __shfl_sync(full, qt, 0), cosang = __shfl_sync(full, qt, 1), vol_rel1 = __shfl_sync(full, qt, 3);
            // ... the momentum's push, the next step's acceleration
            num = role == 3 ? p.dt : p.k_mom * cosang * p.mom_scale;
            den = role == 3 ? vol_rel1 * p.density : (mom ? kden : 1.0);
            const double qk = num / den;
            const double k = __shfl_sync(full, qk, 0), accel1 = __shfl_sync(full, qk, 3);
            const double na = -di * nrm, nb = -dj * nrm;
            if (mom) {
                sa += k * v.ma;
                sb += k * v.mb;
            }
            sa += accel * na;
            sb += accel * nb;
            const double slen = sqrt(norm2(v, sa, sb));
            if (slen < 1e-12) { cause = PGE_DEATH_STOP; break; }
            const double un = (role & 1 ? sb : sa) / slen;
            sa = __shfl_sync(full, un, 0);
            sb = __shfl_sync(full, un, 1);
            double nx = x + sa, ny = y + sb;
            int nf = f;
            if (nx < 0.0 || nx >= Nf || ny < 0.0 || ny >= Nf) {
                if (a.spherical) {
                    double cu = nx / Nf, cw = ny / Nf;
                    nf = cross_face(a.cr_trig != 0, f, cu, cw, sa, sb);
                    nx = cu * Nf;
                    ny = cw * Nf;
                    if (nx >= Nf) nx = Nf * 0.999999999;
                    if (ny >= Nf) ny = Nf * 0.999999999;
                    if (nx < 0.0) nx = 0.0;
                    if (ny < 0.0) ny = 0.0;
                } else if (nx < double(-H) || nx >= Nf + double(H) || ny < double(-H) || ny >= Nf + double(H)) {
                    exited = true; cause = PGE_DEATH_EXIT; break;
                }
            }
            const int nei = (int)floor(nx) + H, nej = (int)floor(ny) + H;
            if ((unsigned)nei >= (unsigned)NE || (unsigned)nej >= (unsigned)NE) { exited = true; cause = PGE_DEATH_EXIT; break; }
            const double hr0 = v.hr;
            h_prev = v.surf;
            load_spot<ROUTE>(a, role, nf, nx, ny, nei, nej, v);
            if (v.m == PGE_MASK_OUTSIDE) { exited = true; cause = PGE_DEATH_EXIT; break; }
            if (ROUTE) {
                if (in_lake) fl |= TS_LAKE;
                if (v.nflag >= 1.5f) fl |= TS_TRAP;
                if (v.nflag >= 2.5f) fl |= TS_KEEPS;
                in_lake = v.nflag >= 1.5f;
            }
            vol = vol1;
            accel = accel1;
            x = nx;
            y = ny;
            f = nf;
            step++;
            partial = false;
            // stop conditions
            if (v.surf < v.b.w && !in_sea) {
                in_sea = true;
                fl |= TS_SEA_NEXT;
            }
            const bool up = hr0 - v.hr < 0.0 && !in_lake;
            uphill = up ? uphill + 1 : 0;
            if (vol < p.min_volume) cause = in_sea ? PGE_DEATH_OCEAN : PGE_DEATH_EVAP;
            else if (up && uphill > p.pit_steps) cause = in_sea ? PGE_DEATH_OCEAN : PGE_DEATH_PIT;
            if (lane == 0) {
                S.dir[n] = make_double2(sa, sb);
                S.flags[n] = fl;
            }
            n++;
        }
        __syncwarp();

        // ---- 2. the mass transfer's terms that do not depend on the load, a lane a step (particle.py:562-671)
        if (lane < n) {
            const int fl = S.flags[lane];
            const PathStep &t = S.path[lane];
            const float h_here = t.surf;
            const double vr = t.vol / volume0, q0 = t.q;
            const bool has_hprev = step0 + lane > 0;
            const double rise = double(lane ? S.path[lane - 1].surf : h_prev0) - double(h_here);
            LoadStep &l = S.load[lane];
            double ev = 1.0 - dt_evap * double(t.b.x);
            if (ev < 0.01) ev = 0.01;
            l.ev = ev;
            l.inv_ev = far_from_one(ev) ? 0.0 : 1.0 / ev;
            l.vol_rel = vr;
            if (!(fl & TS_ACTIVE)) {  // no exchange: a change of zero
                l.c_eq = l.k_up = l.k_down = l.ecap_q = l.dcap_q = 0.0;
                l.ecap = l.dcap = inf;
            } else {
                if (fl & TS_SEA) {
                    double room = has_hprev ? rise : p.fan_room;
                    if (room < p.fan_room) room = p.fan_room;
                    const double lim = double(t.b.w) - p.dep_floor - double(h_here);
                    if (lim < room) room = lim;
                    if (room < 0.0) room = 0.0;
                    l.c_eq = -0.0;  // the load falls out: -ocean_rate * load
                    l.k_up = l.k_down = p.ocean_rate;
                    l.ecap = inf;
                    l.ecap_q = 0.0;
                    l.dcap = room;
                    l.dcap_q = -room / vr;
                } else {
                    const double q = q0 < 0.0 ? 0.0 : q0;
                    const double h1 = S.path[lane + 1].h0, b1 = double(S.path[lane + 1].b.w);
                    const double dh = t.h0 - (h1 > b1 ? h1 : b1);
                    double qe;
                    if (inv_sat <= 0.0) qe = 0.0;
                    else if (p.disc_exponent == 0.5) qe = sqrt(q * inv_sat);
                    else if (p.disc_exponent > 0.0) qe = pow(q * inv_sat, p.disc_exponent);
                    else qe = erf(q * inv_sat);
                    double c_eq = p.erodibility * dh * (1.0 + p.k_disc * qe);
                    if (c_eq < 0.0) c_eq = 0.0;
                    const float sthick = t.b.z;
                    double w_cover;
                    if (p.cover_depth > 0.0) {
                        w_cover = double(sthick) / p.cover_depth;
                        if (w_cover > 1.0) w_cover = 1.0;
                    } else {
                        w_cover = sthick > 0.0f ? 1.0 : 0.0;
                    }
                    double k_up = p.deposition_rate * (w_cover + (1.0 - w_cover) * (1.0 - double(t.b.y)));
                    double k_down = p.deposition_rate;
                    if (a.roots) {  // roots hold the ground (particle.py:615-618)
                        const double held = 1.0 - double(__ldg(a.roots + t.cell));
                        k_up *= held;
                        k_down *= held;
                    }
                    const double kexp = 1.0 + q * p.conc_scale;
                    double ecap = dh / kexp;
                    if (ecap > p.max_erode) ecap = p.max_erode;
                    if (ecap > double(h_here)) ecap = h_here > 0.0f ? double(h_here) : 0.0;
                    double room = has_hprev ? rise : p.dep_floor;
                    if (room < p.dep_floor) room = p.dep_floor;
                    const double dcap = room / kexp;
                    l.c_eq = c_eq;
                    l.k_up = k_up;
                    l.k_down = k_down;
                    l.ecap = ecap;
                    l.ecap_q = ecap / vr;
                    l.dcap = dcap;
                    l.dcap_q = -dcap / vr;
                    if (LATERAL) {
                        // the outside of the bend: a droplet cutting and turning also cuts the bank one cell across
                        // the flow, down towards the bed it just eroded
                        BankStep &b = S.bank[lane];
                        b.rate = 0.0;
                        const double na = S.dir[lane].x, nb = S.dir[lane].y;
                        const double cross = b.psa * nb - b.psb * na;
                        const double turn = cross > 0.0 ? cross : -cross;
                        if (turn > 1e-6) {
                            const double sgn = cross > 0.0 ? 1.0 : -1.0;
                            const double bx = t.x + sgn * nb, by = t.y - sgn * na;
                            const int bei = (int)floor(bx) + H, bej = (int)floor(by) + H;
                            if (bei >= 0 && bei < NE && bej >= 0 && bej < NE) {
                                const int bc = (t.face * NE + bei) * NE + bej;
                                const int bm = a.mask ? (int)__ldg(a.mask + bc) : PGE_MASK_ACTIVE;
                                const float bank = bm == PGE_MASK_ACTIVE ? __ldg(&a.A[bc].x) - h_here : 0.0f;
                                if (bank > 0.0f) {
                                    double lcap = double(bank) / kexp;
                                    if (lcap > p.max_erode) lcap = p.max_erode;
                                    b.rate = p.lateral_rate * turn;
                                    b.lcap = lcap;
                                    b.lcap_q = lcap / vr;
                                    b.cell = bc;
                                }
                            }
                        }
                    }
                }
            }
        }
        __syncwarp();

        // ---- 3. the load, step after step, the same in every lane
        int nv = n;  // steps the droplet lived through
        nring = nact;
        at = n;
        bool drowned = false;
        LoadStep l = S.load[0];
        int fl = S.flags[0];
        for (int i = 0; i < n; i++) {
            const int i1 = i + 1 < TB ? i + 1 : i;
            const LoadStep ln = S.load[i1];
            const int fln = S.flags[i1];
            if ((fl & TS_SEA) && sed * S.path[i].vol / volume0 < 1e-4) {
                drowned = true;
                nv = at = i;
                break;
            }
            const double vr = l.vol_rel;
            double cdiff = (l.c_eq > sed ? l.k_up : l.k_down) * (l.c_eq - sed);
            [[maybe_unused]] double trapped = 0.0;
            if (ROUTE && (fl & (TS_LAKE | TS_TRAP)) && (fl & (TS_ACTIVE | TS_SEA)) == TS_ACTIVE) {
                if (fl & TS_LAKE) {
                    cdiff = 0.0;  // crossing a lake: the bed sees nothing (particle.py:626-629)
                } else if (sed > 0.0) {
                    const double trap = -p.lake_trap * sed;  // entering a lake: the load drops at the shore (630-634)
                    if (trap < cdiff) cdiff = trap;
                    if (fl & TS_KEEPS) trapped = p.lake_trap * sed;  // ...and this lake has room for the rest (636)
                }
            }
            const double moved = cdiff * vr;
            const bool pick = cdiff > 0.0 && moved > l.ecap, drop = cdiff < 0.0 && -moved > l.dcap;
            cdiff = pick ? l.ecap_q : (drop ? l.dcap_q : cdiff);
            sed += cdiff;
            if (lane == 0) S.cdiff[i] = cdiff;
            if (ROUTE) {
                // a lake with room keeps what its shore did not take (particle.py:672-696)
                double rest = 0.0;
                if (trapped > 0.0 && a.parks && parks < LAKE_PARKS) {
                    rest = trapped + cdiff;  // cdiff <= 0: what the shore took
                    if (rest > 0.0) {
                        parks++;
                        sed -= rest;
                    } else {
                        rest = 0.0;
                    }
                }
                if (lane == 0) S.rest[i] = rest;
            }
            if (LATERAL) {
                double lat = 0.0;
                if (cdiff > 0.0 && (fl & (TS_ACTIVE | TS_SEA)) == TS_ACTIVE) {
                    lat = S.bank[i].rate * cdiff;
                    if (lat > 0.0) {
                        if (lat * vr > S.bank[i].lcap) lat = S.bank[i].lcap_q;
                        if (lat > 0.0) sed += lat;
                    }
                }
                if (lane == 0) S.bank[i].lat = lat;
            }
            // sed / ev, correctly rounded: 1/ev is, q1 is faithful, so the last step rounds as the quotient does
            // (P. Markstein, IBM J. Res. Dev. 34, 1990)
            double q1 = sed * l.inv_ev;
            q1 = __fma_rn(__fma_rn(-l.ev, q1, sed), l.inv_ev, q1);
            q1 = __fma_rn(__fma_rn(-l.ev, q1, sed), l.inv_ev, q1);
            if (l.inv_ev == 0.0 || (far_from_one(sed) && __double_as_longlong(sed) != 0)) q1 = sed / l.ev;
            sed = q1;
            if ((fl & TS_SEA_NEXT) && sed <= 0.0) {
                drowned = true;
                nv = at = i + 1;
                break;
            }
            l = ln;
            fl = fln;
        }
        if (!drowned && partial && sea_check && sed * S.path[n].vol / volume0 < 1e-4) drowned = true;  // (at == n)
        if (drowned) {
            cause = PGE_DEATH_OCEAN;
            exited = false;
            in_sea = true;
            nring = S.path[at].nact;
        }
        __syncwarp();

        // ---- 4. the entries, a lane a step; a park's entry, then a bank's, follows its step's own
        {
            const bool own = lane < nv && (S.flags[lane] & TS_ACTIVE);
            const bool park = ROUTE && own && S.rest[ROUTE ? lane : 0] > 0.0;
            const bool bank = LATERAL && own && S.bank[LATERAL ? lane : 0].lat > 0.0;
            const unsigned below = (1u << lane) - 1u, mown = __ballot_sync(full, own);
            const unsigned mpark = ROUTE ? __ballot_sync(full, park) : 0u, mbank = LATERAL ? __ballot_sync(full, bank) : 0u;
            int e = rec_n + __popc(mown & below) + __popc(mpark & below) + __popc(mbank & below);
            auto put = [&](int cell, double delta, float w, float2 m) {
                if (e < a.rec_cap) {
                    const long long o = row * a.rec_cap + e;
                    a.rec_cell[o] = cell;
                    a.rec_delta[o] = delta;
                    a.rec_vol[o] = w;
                    reinterpret_cast<float2 *>(a.rec_mom)[o] = m;
                }
            };
            const float2 none = make_float2(0.0f, 0.0f);
            if (own) {
                const bool land = !(S.flags[lane] & TS_SEA);
                const double w = S.path[lane].vol;
                put(S.path[lane].cell, -S.cdiff[lane] * S.load[lane].vol_rel, land ? (float)w : 0.0f,
                    land ? make_float2((float)(w * S.dir[lane].x), (float)(w * S.dir[lane].y)) : none);
                e++;
            }
            if (ROUTE && park) {
                put(S.path[lane + 1].cell, S.rest[ROUTE ? lane : 0] * S.load[lane].vol_rel, -3.0f, none);
                if (a.park_k) a.park_k[row * LAKE_PARKS + parked + __popc(mpark & below)] = e;
                e++;
            }
            if (LATERAL && bank) put(S.bank[LATERAL ? lane : 0].cell, -S.bank[LATERAL ? lane : 0].lat * S.load[lane].vol_rel, -2.0f, none);
            rec_n += __popc(mown) + __popc(mpark) + __popc(mbank);
            nextra += __popc(mpark) + __popc(mbank);
            parked += __popc(mpark);
        }
        __syncwarp();
    } while (cause < 0);

    // ---- death: final deposits (particle.py:770-815)
    if (in_sea && (cause == PGE_DEATH_AGE || cause == PGE_DEATH_STOP)) cause = PGE_DEATH_OCEAN;
    x = S.path[at].x;
    y = S.path[at].y;
    f = S.path[at].face;
    vol = S.path[at].vol;
    if (!exited) {
        const int c = (f * NE + cell_of(x, N) + H) * NE + cell_of(y, N) + H;
        const int mc = a.mask ? (int)__ldg(a.mask + c) : PGE_MASK_ACTIVE;
        const float sc = __ldg(&a.A[c].x), bc = __ldg(&a.B[c].w);
        if (mc == PGE_MASK_ACTIVE && !(in_sea && sc >= bc)) {
            if (nring == 0 || S.ring[(nring - 1) & (RING - 1)] != c) {
                if (lane == 0) S.ring[nring & (RING - 1)] = c;
                nring++;
            }
        }
    }
    __syncwarp();
    int nout = 0;
    double held = 0.0;
    if (sed > 0.0 && nring > 0 && (!exited || a.deposit_on_exit)) {
        held = sed * vol / volume0;
        nout = cause == PGE_DEATH_OCEAN ? 1 : (nring < SPREAD ? nring : SPREAD);
    }
    if (lane < nout && rec_n + lane < a.rec_cap) {
        const long long o = row * a.rec_cap + rec_n + lane;
        a.rec_cell[o] = S.ring[(nring - 1 - lane) & (RING - 1)];
        a.rec_delta[o] = lane == 0 ? held : 0.0;
        a.rec_vol[o] = -1.0f;
        reinterpret_cast<float2 *>(a.rec_mom)[o] = make_float2(0.0f, 0.0f);
    }
    if (lane == 0) {
        rec_n += nout;
        a.rec_count[row] = rec_n;
        a.rec_death[row] = (int8_t)cause;
        if (a.park_n) a.park_n[row] = parks;
        auto count = [](int64_t *c, long long v) { red_add(reinterpret_cast<long long *>(c), v); };
        count(&a.stats->droplets, 1);
        count(&a.stats->droplet_steps, step_entries(rec_n - nextra, nout));
        count(&a.stats->entries, rec_n);
        count(&a.stats->deaths[cause], 1);
    }
}

}  // namespace f64
}  // namespace pge
