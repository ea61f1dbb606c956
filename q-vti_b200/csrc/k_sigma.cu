// Stress kernel of the time step.
#include <algorithm>

#include "fft_pair.cuh"
#include "step_common.cuh"

namespace qvti {

namespace {

// Bulk prefetch of `bytes` (multiple of 16, 16-byte aligned) into L2.  The
// address operand is warp-uniform in hardware: issue it from one thread (a
// per-lane address makes the compiler serialise the lanes).
__device__ __forceinline__ void prefetch_l2(const void* p, unsigned bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
// ------------------------------------------------------------------ k_st --
// Compiled form of the stress update, one group of fields per block: NF = 9 the
// normal stresses (G 0..8), NF = 6 a shear stress (xz, xy, yz; G 9..26).  A block
// owns four or eight y rows and all z of one x; k_dz then takes the z
// derivatives.  (One block running the groups one after another and the z
// derivatives at the end measured 2.2 ms at 256^3, 0.57 of them the z pass on a
// third of its threads.)
//
// Rows 0 + i 1 and 2 + i 3 of a field are the two pencils of a packed pair
// (fft_pair.cuh): one thread transforms all four rows, and the slot its
// inverse leaves at height z holds rows 0, 2 in the first plane and 1, 3 in the
// second, so the update runs on pairs of rows in packed arithmetic.  C2R by the
// Hermitian extension: a butterfly's points below n/2 are loaded (two 16-byte
// loads of one sector: one 32-byte load per point measured 0.72 against 0.57 ms
// for the normal stresses), those above are the mirror of what the butterfly
// n/R - j loaded and come by shuffle where the threads of a pencil are 8, 16 or
// 32 neighbouring lanes (a second load otherwise: 2.65 against 2.2 ms).  With
// eight rows (Q = 2) the two row quads of a butterfly are neighbouring lanes and
// read 64 bytes of a line between them: a warp's load touches 16 lines instead
// of 32 (shear 0.68 against 0.78 ms at 256^3).
constexpr int st_threads(int n, int nf, int q) { return warps_up(nf * q * pair_tasks(n)); }
constexpr size_t st_smem(int n, int nf, int q) { return 16 * ((size_t)nf * q * pair_slots_q(n, q) + tw_rows_size(n)); }
// Blocks per SM the registers are sized for: 16 to 20 warps.
constexpr int st_blocks(int n, int nf, int q)
{
    const int warps = st_threads(n, nf, q) / 32, m = (int)(220 * 1024 / (st_smem(n, nf, q) + 2048));
    int b = (nf == 9 ? (q == 1 ? 16 : 18) : 20) / warps;
    if (b < 1) b = 1;
    return b < m ? b : m < 1 ? 1 : m;
}
// Whether stage 0 gets its mirror points by shuffle.
constexpr bool st_shuffles(int n, int q)
{
    const int lanes = pair_tasks(n) * q;
    return pair_rad(n, 0) % 2 == 0 && pair_k(n, 0) == 1 && (lanes == 8 || lanes == 16 || lanes == 32);
}
// Rows of a normal-stress block in quads where the shear blocks take q: one where
// four rows shuffle (nine fields of two quads leave 96 registers a thread at 256
// points, and spills: 1.48 against 1.40 ms for the whole update at 256^3, 0.220
// against 0.208 at 128^3), else the shear blocks' (98 points: 0.217 against 0.235).
constexpr int st_normal_q(int n, int q) { return st_shuffles(n, 1) ? 1 : q; }
// Whether a compiled z length takes sxy's two terms one after the other (see
// stress_pair): 64 and the 5-smooth lengths from 96, whose scalar kernel did (the
// other lengths had the runtime one).
constexpr bool st_halves(int n)
{
    if (n < 96) return n == 64;
    for (int r : {2, 3, 5})
        while (n % r == 0) n /= r;
    return n == 1;
}

__device__ __forceinline__ f2 bc(float a) { return pack2(a, a); }
__device__ __forceinline__ f2 sel2(bool a, bool b, f2 v)
{
    const float2 x = unpack2(v);
    return pack2(a ? x.x : 0.f, b ? x.y : 0.f);
}
__device__ __forceinline__ f2 rows2(const float* p, int n) { return pack2(p[0], p[n]); }
__device__ __forceinline__ f2 rows2_ro(const float* p, int n) { return pack2(__ldg(p), __ldg(p + n)); }
__device__ __forceinline__ void put2(float* p, int n, bool second, f2 v)
{
    const float2 x = unpack2(v);
    p[0] = x.x;
    if (second) p[n] = x.y;
}

// Constant-Q set of one modulus for two rows from its effective velocity
// c = v cos(pi g/2) (cuviscoelas_3D.cu:195-205): eta1 = -rho c g w0, eta2 =
// rho c^2, eta3 = rho c^3 g / w0, tau1 = rho c g pi, tau2 = rho c^2 g^2 pi / w0.
// c is built in FP64 at setup; the products are rebuilt here in FP32, one of the
// five at a time.  The last factor comes apart (o = m f), for sums that round the
// product only once.
struct Mod {
    f2 rc, c, g;
};
struct Coef {
    f2 m, f, o;
};
__device__ __forceinline__ Coef coef(const Mod& s, int j, float w0, float inv_w0)
{
    const float pi = 3.1415926f;
    Coef r;
    if (j == 0) { r.m = neg_(s.rc) * s.g; r.f = bc(w0); }
    else if (j == 1) { r.m = s.rc; r.f = s.c; }
    else if (j == 2) { r.m = s.rc * s.c * s.c * s.g; r.f = bc(inv_w0); }
    else if (j == 3) { r.m = s.rc * s.g; r.f = bc(pi); }
    else { r.m = s.rc * s.c * s.g * s.g * bc(pi); r.f = bc(inv_w0); }
    r.o = r.m * r.f;
    return r;
}
// a13 - 2 a55 of two sets, the product of a13 (but that of eta2, which eta3
// shares) not rounded by itself
__device__ __forceinline__ f2 less13(const Coef& a, const Coef& s5, int j)
{
    return j == 1 ? fma_(bc(-2.f), s5.o, a.o) : fma_(a.m, a.f, s5.o * bc(-2.f));
}
__device__ __forceinline__ f2 dot3(const f2* a, f2 x, f2 y, f2 z) { return fma_(a[2], z, fma_(a[0], x, a[1] * y)); }
__device__ __forceinline__ f2 dot2(const f2* a, f2 x, f2 y) { return fma_(a[3], x, a[4] * y); }

// One C-PML term of a row pair: the slab's memory variable and loss potential
// (second row n further on), loaded, then advanced by the term d and its new
// potential qn.  Rows outside the slab (on0, on1) keep zero.
struct Term {
    f2 po, qo;
};
__device__ __forceinline__ void term_load(Term& t, const float* ph, const float* q, int n, bool on0, bool on1)
{
    t.qo = pack2(on0 ? q[0] : 0.f, on1 ? q[n] : 0.f);
    t.po = pack2(on0 ? ph[0] : 0.f, on1 ? ph[n] : 0.f);
}
__device__ __forceinline__ f2 term_step(const Term& t, float* ph, float* q, int n, bool on0, bool on1, f2 a, f2 b, f2 d,
                                        f2 qn, f2 dt, f2 inv_dt)
{
    const f2 T = fma_(qn - t.qo, inv_dt, d);
    const f2 r = fma_(dt, fma_(neg_(a), t.po, neg_(b) * T), t.po);  // pml_step
    const float2 rv = unpack2(r), qv = unpack2(qn);
    if (on0) { q[0] = qv.x; ph[0] = rv.x; }
    if (on1) { q[n] = qv.y; ph[n] = rv.y; }
    return sel2(on0, on1, r);
}

// L2 prefetch of the rows y0 .. y0 + yv - 1 a group's update reads, issued
// ahead by one thread: fields and coefficients, and the C-PML variables
// of the slabs the rows are in.
__device__ __forceinline__ void prefetch_group(const KP& k, int n, int g, int x, int y0, int yv)
{
    const int c0 = cell(k, x, y0, 0);
    const unsigned run = 4u * yv * n;
    if (g == 0) {
        const float* arr[13] = {k.s[0], k.s[1], k.s[2], k.Q[0], k.Q[1], k.Q[2], k.mrho, k.mgp, k.mgs,
                                k.mcs, k.mc33, k.mc11, k.mc13};
#pragma unroll
        for (int a = 0; a < 13; ++a)
            if (a < 11 || k.mc11 != k.mc33) prefetch_l2(arr[a] + c0, run);
    } else {
        const int c = g == 1 ? 4 : g == 2 ? 3 : 5;
        prefetch_l2(k.s[c] + c0, run);
        prefetch_l2(k.Q[c] + c0, run);
#pragma unroll
        for (int j = 0; j < 5; ++j) prefetch_l2(k.MU[j] + c0, run);
    }
    auto pair = [&](float* const* a, float* const* b, int m, int at, unsigned bytes) {
        prefetch_l2(a[m] + at, bytes);
        prefetch_l2(b[m] + at, bytes);
    };
    const int zs = slab_z(k, x, y0, 0);
    const unsigned zrun = 8u * yv * k.pml;
    if (g == 0) {
        for (int m = 6; m < 8; ++m) pair(k.phn, k.qn, m, zs, zrun);
    } else if (g != 2) {
        pair(k.phs, k.qs, 2 * (g - 1), zs, zrun);
    }
    if (in_slab(x, k.nx, k.pml)) {
        const int xs = slab_x(k, x, y0, 0);
        if (g == 0) {
            for (int m = 0; m < 3; ++m) pair(k.phn, k.qn, m, xs, run);
        } else if (g != 3) {
            pair(k.phs, k.qs, 2 * g - 1, xs, run);
        }
    }
    if (in_slab(y0, k.ny, k.pml) && in_slab(y0 + yv - 1, k.ny, k.pml)) {  // whole tile (an edge tile's rows come on demand)
        const int ys = slab_y(k, x, y0, 0);
        if (g == 0) {
            for (int m = 3; m < 6; ++m) pair(k.phn, k.qn, m, ys, run);
        } else if (g != 1) {
            pair(k.phs, k.qs, g == 2 ? 2 : 5, ys, run);
        }
    }
}

// Source (cu:772-777), after the normal stresses' update of the block that
// holds it; one thread.
__device__ __forceinline__ void inject(const KP& k, int x, int y0, int yv)
{
    const int it = *k.d_it;
    if (x != k.s_ix || k.s_iy < y0 || k.s_iy >= y0 + yv || it >= k.nt_rec) return;
    const int ip = cell(k, x, k.s_iy, k.s_iz);
    const float w = k.rik[it];
    if (k.src_type == 1) {
        k.s[0][ip] += w;
        k.s[1][ip] += w;
        k.s[2][ip] += w;
    } else {
        k.v[0][ip] += w;
    }
}

// The z derivative d of a stress at (x, y, z) with its C-PML term (a, b) added.
__device__ __forceinline__ float z_term(const KP& k, float* ph, int x, int y, int z, float a, float b, float d)
{
    const int is = slab_z(k, x, y, z);
    const float nw = pml_step(ph[is], k.dt, a, b, d);
    ph[is] = nw;
    return d + nw;
}

// Stress update of one group at height z of rows y, y + D (constant-Q
// dispersion and loss, C-PML; cu:800-1015), in packed arithmetic; sv(f): the
// group's real field f at the two rows.  Not for the last x or z plane, nor y =
// ny - 1.  The C-PML terms sit behind branches that are uniform but for the z
// slab's edges; loads of a row pair that the compiler can all issue before the
// first store are what keeps the update fed.
// HALVES: sxy takes its y and its x term one after the other, each with its own
// part of the loss (dt L = ls (Qxy - Qxy_old), Qxy the sum of the two parts).
template <int D, bool HALVES, class SV>
__device__ __forceinline__ void stress_pair(const KP& k, int n, int grp, int x, int y, int z, SV sv)
{
    const int nx = k.nx, ny = k.ny, pml = k.pml;
    const float w0 = k.w0, inv_w0 = 1.0f / k.w0;
    // inv_dt enters only the loss terms (the spectral time derivative of the
    // constant-Q loss operator): their sign and presence follow the medium
    // (k.loss_scale: 1 viscoelastic, 0 dispersion only, -1 Q-compensated)
    const f2 dt = bc(k.dt), ls = bc(k.loss_scale), inv_dt = bc(k.loss_scale / k.dt);
    const bool sx = in_slab(x, nx, pml);
    const bool in1 = y + D < ny - 1;  // the last plane of an axis is never updated
    const int nd = in1 ? D * n : 0;   // to the second row; the first one again where there is none
    const int ip = cell(k, x, y, z);
    const bool sy0 = in_slab(y, ny, pml), sy1 = in1 && in_slab(y + D, ny, pml), sz = in_slab(z, n, pml);
    const int isx = sx ? slab_x(k, x, y, z) : 0, isz = sz ? slab_z(k, x, y, z) : 0;
    // row y + D of the y slab is D n further on; a pair whose first row is
    // outside starts at its second
    const int isy = sy0 ? slab_y(k, x, y, z) : sy1 ? slab_y(k, x, y + D, z) - D * n : 0;
    const bool sy = sy0 || sy1;
    const int nz2 = in1 ? 2 * D * pml : 0;
    // every load of the cell pair is issued before its first store: the arrays
    // cannot alias, but through the parameter struct the compiler cannot know
    Term tm[8];
    auto xload = [&](int i, float* ph, float* q) { term_load(tm[i], ph + isx, q + isx, nd, true, true); };
    auto yload = [&](int i, float* ph, float* q) { term_load(tm[i], ph + isy, q + isy, D * n, sy0, sy1); };
    auto zload = [&](int i, float* ph, float* q) { term_load(tm[i], ph + isz, q + isz, nz2, true, true); };
    auto xterm = [&](int i, float* ph, float* q, f2 a, f2 b, f2 d, f2 qn) {
        return term_step(tm[i], ph + isx, q + isx, nd, true, in1, a, b, d, qn, dt, inv_dt);
    };
    auto yterm = [&](int i, float* ph, float* q, f2 a, f2 b, f2 d, f2 qn) {
        return term_step(tm[i], ph + isy, q + isy, D * n, sy0, sy1, a, b, d, qn, dt, inv_dt);
    };
    auto zterm = [&](int i, float* ph, float* q, f2 a, f2 b, f2 d, f2 qn) {
        return term_step(tm[i], ph + isz, q + isz, nz2, true, in1, a, b, d, qn, dt, inv_dt);
    };
    auto yrow = [&](const float* p) { return pack2(p[y], p[in1 ? y + D : y]); };
    if (grp == 0) {
        f2 sxx = rows2(k.s[0] + ip, nd), syy = rows2(k.s[1] + ip, nd), szz = rows2(k.s[2] + ip, nd);
        const f2 qx = rows2(k.Q[0] + ip, nd), qy = rows2(k.Q[1] + ip, nd), qz = rows2(k.Q[2] + ip, nd);
        const f2 rho = rows2_ro(k.mrho + ip, nd), gp = rows2_ro(k.mgp + ip, nd), gs = rows2_ro(k.mgs + ip, nd);
        const f2 c33 = rows2_ro(k.mc33 + ip, nd), cs = rows2_ro(k.mcs + ip, nd);
        f2 c11 = c33, c13 = c33;
        const bool aniso = k.mc11 != k.mc33;
        if (aniso) {
            c11 = rows2_ro(k.mc11 + ip, nd);
            c13 = rows2_ro(k.mc13 + ip, nd);
        }
        if (sx) {
#pragma unroll
            for (int m = 0; m < 3; ++m) xload(m, k.phn[m], k.qn[m]);
        }
        if (sy) {
#pragma unroll
            for (int m = 3; m < 6; ++m) yload(m, k.phn[m], k.qn[m]);
        }
        if (sz) {
            zload(6, k.phn[6], k.qn[6]);
            zload(7, k.phn[7], k.qn[7]);
        }
        // the sets one coefficient at a time, each into the sums of all terms:
        // their products in the order 1, 0, 2 (d33z: 0, 1, 2) and 4, 3
        f2 d11x, d12x, d13x, d12y, d11y, d13y, d13z, d33z, q11x, q12x, q13x, q12y, q11y, q13y, q13z, q33z;
        {
            const Mod m33{rho * c33, c33, gp}, m11{rho * c11, c11, gp}, m13{rho * c13, c13, gp}, m5{rho * cs, cs, gs};
            auto sets = [&](int j, f2& a11, f2& a12, f2& a13, f2& a33) {
                const Coef s5 = coef(m5, j, w0, inv_w0), k33 = coef(m33, j, w0, inv_w0);
                const Coef k11 = aniso ? coef(m11, j, w0, inv_w0) : k33, k13 = aniso ? coef(m13, j, w0, inv_w0) : k33;
                a33 = k33.o;
                a11 = k11.o;
                a12 = fma_(bc(-2.f), s5.o, a11);
                a13 = less13(k13, s5, j);
            };
            f2 a11, a12, a13, a33;
            f2 X = sv(1), Y = sv(4), Z = sv(7);
            sets(1, a11, a12, a13, a33);
            d11x = a11 * X; d12x = a12 * X; d13x = a13 * X;
            d12y = a12 * Y; d11y = a11 * Y; d13y = a13 * Y;
            d13z = a13 * Z;
            const f2 a33_1 = a33;
            sets(4, a11, a12, a13, a33);
            q11x = a11 * X; q12x = a12 * X; q13x = a13 * X;
            q12y = a12 * Y; q11y = a11 * Y; q13y = a13 * Y;
            q13z = a13 * Z; q33z = a33 * Z;
            const f2 Z1 = Z;
            X = sv(0); Y = sv(3); Z = sv(6);
            sets(0, a11, a12, a13, a33);
            d11x = fma_(a11, X, d11x); d12x = fma_(a12, X, d12x); d13x = fma_(a13, X, d13x);
            d12y = fma_(a12, Y, d12y); d11y = fma_(a11, Y, d11y); d13y = fma_(a13, Y, d13y);
            d13z = fma_(a13, Z, d13z); d33z = fma_(a33_1, Z1, a33 * Z);
            sets(3, a11, a12, a13, a33);
            q11x = fma_(a11, X, q11x); q12x = fma_(a12, X, q12x); q13x = fma_(a13, X, q13x);
            q12y = fma_(a12, Y, q12y); q11y = fma_(a11, Y, q11y); q13y = fma_(a13, Y, q13y);
            q13z = fma_(a13, Z, q13z); q33z = fma_(a33, Z, q33z);
            X = sv(2); Y = sv(5); Z = sv(8);
            sets(2, a11, a12, a13, a33);
            d11x = fma_(a11, X, d11x); d12x = fma_(a12, X, d12x); d13x = fma_(a13, X, d13x);
            d12y = fma_(a12, Y, d12y); d11y = fma_(a11, Y, d11y); d13y = fma_(a13, Y, d13y);
            d13z = fma_(a13, Z, d13z); d33z = fma_(a33, Z, d33z);
        }
        // loss: sum_terms tau-coefficient x (S - S_prev)/dt = (Q - Q_prev)/dt
        const f2 Qxx = q11x + q12y + q13z, Qyy = q12x + q11y + q13z, Qzz = q13x + q13y + q33z;
        f2 txx = fma_(Qxx - qx, inv_dt, d11x + d12y + d13z);
        f2 tyy = fma_(Qyy - qy, inv_dt, d12x + d11y + d13z);
        f2 tzz = fma_(Qzz - qz, inv_dt, d13x + d13y + d33z);
        if (sx) {
            const f2 ax = bc(k.ax[x]), bx = bc(k.bx[x]);
            txx = txx + xterm(0, k.phn[0], k.qn[0], ax, bx, d11x, q11x);
            tyy = tyy + xterm(1, k.phn[1], k.qn[1], ax, bx, d12x, q12x);
            tzz = tzz + xterm(2, k.phn[2], k.qn[2], ax, bx, d13x, q13x);
        }
        if (sy) {
            const f2 a = yrow(k.ay), b = yrow(k.by);
            txx = txx + yterm(3, k.phn[3], k.qn[3], a, b, d12y, q12y);
            tyy = tyy + yterm(4, k.phn[4], k.qn[4], a, b, d11y, q11y);
            tzz = tzz + yterm(5, k.phn[5], k.qn[5], a, b, d13y, q13y);
        }
        if (sz) {
            const f2 a = bc(k.az[z]), b = bc(k.bz[z]);
            const f2 p = zterm(6, k.phn[6], k.qn[6], a, b, d13z, q13z);  // phi_vz_zx == phi_vz_zy
            txx = txx + p;
            tyy = tyy + p;
            tzz = tzz + zterm(7, k.phn[7], k.qn[7], a, b, d33z, q33z);
        }
        put2(k.s[0] + ip, nd, in1, fma_(dt, txx, sxx));
        put2(k.s[1] + ip, nd, in1, fma_(dt, tyy, syy));
        put2(k.s[2] + ip, nd, in1, fma_(dt, tzz, szz));
        put2(k.Q[0] + ip, nd, in1, Qxx);
        put2(k.Q[1] + ip, nd, in1, Qyy);
        put2(k.Q[2] + ip, nd, in1, Qzz);
    } else {
        // shear: xz, xy, yz (groups 1, 2, 3), each of two terms; A: dz vx, dy
        // vx, dz vy (z, y, z slab), B: dx vz, dx vy, dy vz (x, x, y slab)
        const int c = grp == 1 ? 4 : grp == 2 ? 3 : 5;
        float* __restrict__ sg = k.s[c] + ip;
        float* __restrict__ qg = k.Q[c] + ip;
        const f2 s_old = rows2(sg, nd), q_old = rows2(qg, nd);
        f2 mu[5];
#pragma unroll
        for (int j = 0; j < 5; ++j) mu[j] = rows2_ro(k.MU[j] + ip, nd);
        const int mA = 2 * (grp - 1), mB = mA + 1;
        const bool onA = grp == 2 ? sy : sz, onB = grp == 3 ? sy : sx;
        float *phA = k.phs[mA], *qsA = k.qs[mA], *phB = k.phs[mB], *qsB = k.qs[mB];
        if (onA) {
            if (grp == 2) yload(0, phA, qsA);
            else zload(0, phA, qsA);
        }
        if (onB) {
            if (grp == 3) yload(1, phB, qsB);
            else xload(1, phB, qsB);
        }
        f2 X = sv(0), Y = sv(1), Z = sv(2);
        const f2 dA = dot3(mu, X, Y, Z);
        const f2 qA = dot2(mu, X, Y);
        X = sv(3); Y = sv(4); Z = sv(5);
        const f2 dB = dot3(mu, X, Y, Z);
        const f2 qB = dot2(mu, X, Y);
        const f2 Qs = qA + qB;
        f2 pA = bc(0.f), pB = bc(0.f);
        if (onA) {
            if (grp == 2) pA = yterm(0, phA, qsA, yrow(k.ayh), yrow(k.byh), dA, qA);
            else pA = zterm(0, phA, qsA, bc(k.azh[z]), bc(k.bzh[z]), dA, qA);
        }
        if (onB) {
            if (grp == 3) pB = yterm(1, phB, qsB, yrow(k.ayh), yrow(k.byh), dB, qB);
            else pB = xterm(1, phB, qsB, bc(k.axh[x]), bc(k.bxh[x]), dB, qB);
        }
        f2 S;
        if (HALVES && grp == 2) {
            S = fma_(ls, qA - q_old, fma_(dt, dA + pA, s_old));
            S = fma_(ls, qB, fma_(dt, dB + pB, S));
        } else {
            S = fma_(dt, fma_(Qs - q_old, inv_dt, dA + pA + dB + pB), s_old);
        }
        put2(sg, nd, in1, S);
        put2(qg, nd, in1, Qs);
    }
}

template <int N, int NF, int Q>
__global__ void __launch_bounds__(st_threads(N, NF, Q), st_blocks(N, NF, Q)) k_st(KP k)
{
    using F = PairFFT<N, NF * Q, false, Q>;
    constexpr int NT = st_threads(N, NF, Q), R0 = F::R0, NR0 = N / R0, ROWS = 4 * Q, LANES = F::T * Q;
    constexpr bool SHFL = st_shuffles(N, Q);
    static_assert(NT <= 1024, "threads of a block");
    extern __shared__ float4 smem4[];
    f2* buf = reinterpret_cast<f2*>(smem4);
    float4* tw = smem4 + F::PLANE;
    const TwRows<N> W{tw};
    const int t = threadIdx.x, nx = k.nx, ny = k.ny, x = blockIdx.y;
    // the three shear blocks of a tile are neighbours: they share MU in L2
    const int y0 = ROWS * (NF == 9 ? blockIdx.x : blockIdx.x / 3);
    const int yv = min(ROWS, ny - y0);  // rows of the tile inside the grid (even)
    constexpr float inv_nz = 1.0f / N;
    const int grp = NF == 9 ? 0 : blockIdx.x % 3 + 1;
    if (x == nx - 1) {  // the last plane of an axis is never updated
        if (NF == 9 && t == 0) inject(k, x, y0, yv);
        return;
    }

    int p0, j0;
    const bool act = F::task(t, p0, j0);
    if (!act) { p0 = NF * Q - Q + t % Q; j0 = 0; }
    const int f0 = p0 / Q, q0 = 4 * (p0 % Q);  // field and first row of the pair

    c2 v[F::RM];
    // 1. C2R along z of the group's fields (whole warps: lanes without a
    //    butterfly follow along for the shuffles)
    if ((t & ~31) < NF * Q * F::T) {
        const int o = (NF == 9 ? 0 : 3 + 6 * grp) + f0;
        const bool gz = is_gz(o);
        const float2* src = gz ? k.H[o == 7 ? 2 : o == 10 ? 0 : 1]
                               : is_gy(o) ? k.Yv[o == 4 ? 1 : o == 16 ? 0 : 2] : k.G[o];
        const float2* M = o == 7 ? k.Fz : k.Bz;
        const bool r01 = q0 < yv, r23 = q0 + 2 < yv;
        src += (long long)x * ny + y0 + (r01 ? q0 : 0);
        const int ks = nx * ny;
        // the four rows at kz, the kz-only fields' multiplier applied
        // (imaginary parts dropped at kz = 0 and n/2 like a C2R)
        auto rows = [&](int kk, float2 a[4]) {
            const float2* at = src + (long long)kk * ks;
            const float4 u = *reinterpret_cast<const float4*>(at);
            const float4 w = r23 ? *reinterpret_cast<const float4*>(at + 2) : make_float4(0.f, 0.f, 0.f, 0.f);
            a[0] = make_float2(u.x, u.y); a[1] = make_float2(u.z, u.w);
            a[2] = make_float2(w.x, w.y); a[3] = make_float2(w.z, w.w);
            if (gz) {
                // (rounded as the scalar kernels of these lengths did)
                const float2 m = cscale(M[kk], inv_nz);
#pragma unroll
                for (int q = 0; q < 4; ++q) a[q] = st_halves(N) ? cmul_m(a[q], m) : cmul(a[q], m);
            }
            if (kk == 0 || 2 * kk == N) {
#pragma unroll
                for (int q = 0; q < 4; ++q) a[q].y = 0.f;
            }
        };
        auto direct = [](const float2 a[4]) {
            return c2{pack2(a[0].x - a[1].y, a[2].x - a[3].y), pack2(a[0].y + a[1].x, a[2].y + a[3].x)};
        };
        auto mirror = [](const float2 a[4]) {
            return c2{pack2(a[0].x + a[1].y, a[2].x + a[3].y), pack2(a[1].x - a[0].y, a[3].x - a[2].y)};
        };
        if constexpr (SHFL) {
            if (j0 >= NR0) j0 = 0;  // a pencil's lanes past its last butterfly
            c2 m[R0 / 2];
            float2 a[4];
#pragma unroll
            for (int r = 0; r < R0 / 2; ++r) {
                rows(j0 + r * NR0, a);
                v[r] = direct(a);
                m[r] = mirror(a);
            }
            const int from = (NR0 - j0) * Q + p0 % Q;  // the butterfly that holds the mirror points (j0 = 0: itself)
            auto swap1 = [&](f2 own, f2 send) {
                const float2 s = unpack2(send), w = unpack2(own);
                const float p = __shfl_sync(0xffffffffu, s.x, from, LANES), q = __shfl_sync(0xffffffffu, s.y, from, LANES);
                return j0 ? pack2(p, q) : pack2(w.x, w.y);
            };
            c2 ny2 = m[0];
            if (j0 == 0) {
                rows(N / 2, a);
                ny2 = direct(a);
            }
#pragma unroll
            for (int r = R0 / 2; r < R0; ++r) {
                const c2 own = r == R0 / 2 ? ny2 : m[R0 - r];
                v[r] = c2{swap1(own.x, m[R0 - 1 - r].x), swap1(own.y, m[R0 - 1 - r].y)};
            }
        } else {
            F::template each<0>(j0, [&](int m, int j) {
#pragma unroll
                for (int r = 0; r < R0; ++r) {
                    const int i = j + r * NR0;
                    float2 a[4];
                    rows(i <= N / 2 ? i : N - i, a);
                    const c2 d = direct(a), c = mirror(a);
                    v[m * R0 + r] = i <= N / 2 ? d : c;
                }
            });
        }
    }
    // behind the loads in flight (ahead of them its dozens of requests held up
    // the first warp: 1.40 against 1.38 ms at 256^3, 130 against 119 us at 96^3)
    if (t == 0) prefetch_group(k, N, grp, x, y0, yv);
    TwRows<N>::template fill<NT>(tw, k.tw_z);
    if (F::SYNC0) __syncthreads();
    F::template first<true>(W, buf, t, v);
    F::template finish<true>(W, buf, t, v);
    F::keep(buf, t, v);
    __syncthreads();

    // 2. stress update of the group: a thread takes rows 0, 2 or 1, 3 of a
    //    quad at z
    for (int w = t; w < ROWS / 2 * N; w += NT) {
        const int h = (unsigned)w / N, z = w - h * N, row = h / 2 * 4 + h % 2, y = y0 + row;
        if (row >= yv || y == ny - 1 || z == N - 1) continue;
        const f2* S = buf + (h & 1) * F::PLANE + F::slot(h / 2, z);
        stress_pair<2, st_halves(N)>(k, N, grp, x, y, z, [&](int f) { return S[f * Q * F::SL]; });
    }
    if constexpr (NF == 9) {
        __syncthreads();
        if (t == 0) inject(k, x, y0, yv);
    }
}

// ------------------------------------------------------------------ k_dz --
// z derivatives of the new szz (backward shift -> R_z), sxz (forward -> R_x),
// syz (forward -> R_y) with their C-PML z terms (blockIdx.z: the field); 16
// rows of one x per block, four rows per packed pair as in k_st, the
// multiplication and the epilogue in registers as in k_dv.
constexpr int kDzPairs = 4;
constexpr int dz_threads(int n) { return warps_up(kDzPairs * pair_tasks(n)); }
constexpr size_t dz_smem(int n) { return 16 * ((size_t)kDzPairs * pair_slots(n) + tw_rows_size(n)); }
constexpr int dz_blocks(int n)
{
    const int warps = dz_threads(n) / 32;
    int b = 65536 / (128 * dz_threads(n));
    while (b > 1 && b * warps % 4) --b;
    return b < 1 ? 1 : b;
}

template <int N>
__global__ void __launch_bounds__(dz_threads(N), dz_blocks(N)) k_dz(KP k)
{
    using D = PairFFT<N, kDzPairs, false>;
    constexpr int NT = dz_threads(N), R0 = D::R0, RL = D::RL;
    extern __shared__ float4 smem4[];
    f2* buf = reinterpret_cast<f2*>(smem4);
    float4* tw = smem4 + D::PLANE;
    const TwRows<N> W{tw};
    const int t = threadIdx.x, ny = k.ny, x = blockIdx.y, f = blockIdx.z;
    const float inv_n = 1.0f / N;
    c2 v[D::RM];
    int q, j;
    const bool act = D::task(t, q, j);
    const int y0 = (blockIdx.x * kDzPairs + q) * 4, yv = ny - y0;
    if (act) {
        const float* s = k.s[f == 0 ? 2 : f == 1 ? 4 : 5] + cell(k, x, y0, 0);
        D::template each<0>(j, [&](int m, int i) {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const float* p = s + i + r * (N / R0);
                const bool r01 = yv > 0, r23 = yv > 2;
                v[m * R0 + r] = c2{pack2(r01 ? p[0] : 0.f, r23 ? p[2 * N] : 0.f), pack2(r01 ? p[N] : 0.f, r23 ? p[3 * N] : 0.f)};
            }
        });
    }
    TwRows<N>::template fill<NT>(tw, k.tw_z);
    if (D::SYNC0) __syncthreads();
    D::template first<false>(W, buf, t, v);
    D::template finish<false>(W, buf, t, v);
    D::turn(buf, t, v);
    if (act) {
        const float2* T = f == 0 ? k.Bz : k.Fz;
        D::template each<0>(j, [&](int m, int i) {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const float2 c = cscale(__ldg(T + i + r * (N / R0)), inv_n);
                v[m * R0 + r] = cmul_m(v[m * R0 + r], bc(c.x), bc(c.y));
            }
        });
    }
    __syncthreads();
    D::template first<true>(W, buf, t, v);
    D::template finish<true>(W, buf, t, v);
    if (act) {
        float* __restrict__ R = k.R[f == 0 ? 2 : f == 1 ? 0 : 1] + cell(k, x, y0, 0);
        float* __restrict__ ph = k.php[f == 0 ? 8 : f == 1 ? 2 : 5];  // pzz_z, pxz_z, pyz_z
        const float* pa = f == 0 ? k.azh : k.az;
        const float* pb = f == 0 ? k.bzh : k.bz;
        D::template each<D::LAST>(j, [&](int m, int i0) {
#pragma unroll
            for (int r = 0; r < RL; ++r) {
                const int i = i0 + r * (N / RL);
                const float2 u = unpack2(v[m * RL + r].x), w = unpack2(v[m * RL + r].y);
                float d[4] = {u.x, w.x, u.y, w.y};
                if (x < k.nx - 1 && i < N - 1 && in_slab(i, N, k.pml)) {
                    const float a = pa[i], b = pb[i];
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (c < yv - 1) d[c] = z_term(k, ph, x, y0 + c, i, a, b, d[c]);
                }
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (c < yv) R[i + c * N] = d[c];
            }
        });
    }
}

#if QVTI_PART == 0
// The runtime-length forms: P rows of one x, scalar transforms of row pairs
// (2q, 2q + 1) packed as A + i B.  A block of k_sigma takes one group
// (blockIdx.z: normal, xz, xy, yz), k_dzr one stress: at the small grids that
// run here, blocks that took everything in turn left most of the chip idle.
__global__ void __launch_bounds__(kThreads, 2) k_sigma(KP k, int P)
{
    extern __shared__ float4 smem4[];
    float2* sm = reinterpret_cast<float2*>(smem4);
    const int n = k.nz, Qp = P / 2, np1 = n + 1, nx = k.nx, ny = k.ny;
    const int bufA = 9 * Qp * (n + n / 16);
    float2* tw = sm;
    float2* A = tw + n;
    float2* B = A + bufA;  // only with more than two stages
    float* S = reinterpret_cast<float*>(B + (k.pz.q.nst > 2 ? bufA : 0));  // [9][P][np1]: the group's real fields
    const int x = blockIdx.y, y0 = blockIdx.x * P, yv = min(P, ny - y0), grp = blockIdx.z;
    if (x == nx - 1) {  // the last plane of an axis is never updated
        if (grp == 0 && threadIdx.x == 0) inject(k, x, y0, yv);
        return;
    }
    const float inv_n = 1.0f / n;
    if (threadIdx.x == 0) prefetch_group(k, n, grp, x, y0, yv);
    load_table(tw, k.tw_z, n);
    __syncthreads();
    const int o0 = grp == 0 ? 0 : 3 + 6 * grp, npen = (grp == 0 ? 9 : 6) * Qp;
    auto load = [&](int pp, int i) -> float2 {
        const int f = pp / Qp, q = pp - f * Qp, o = o0 + f;
        if (2 * q >= yv) return make_float2(0.f, 0.f);
        const int kk = i <= n / 2 ? i : n - i;
        const float2* src = is_gz(o) ? k.H[o == 7 ? 2 : o == 10 ? 0 : 1]
                                     : is_gy(o) ? k.Yv[o == 4 ? 1 : o == 16 ? 0 : 2] : k.G[o];
        const float4 gg = *reinterpret_cast<const float4*>(src + spec(k, kk, x, y0 + 2 * q));
        float2 a = make_float2(gg.x, gg.y), b = make_float2(gg.z, gg.w);
        if (is_gz(o)) {  // kz-only field: M(kz) H(kz) / nz
            const float2 m = cscale((o == 7 ? k.Fz : k.Bz)[kk], inv_n);
            a = cmul(a, m);
            b = cmul(b, m);
        }
        if (kk == 0 || 2 * kk == n) { a.y = 0.f; b.y = 0.f; }
        if (i > n / 2) { a.y = -a.y; b.y = -b.y; }
        return make_float2(a.x - b.y, a.y + b.x);
    };
    auto store = [&](int pp, int i, float2 v) {
        const int f = pp / Qp, q = pp - f * Qp;
        S[(f * P + 2 * q) * np1 + i] = v.x;
        S[(f * P + 2 * q + 1) * np1 + i] = v.y;
    };
    fft_run<true, true>(k.pz, tw, A, B, npen, 1, npen, load, store, 4);
    for (int w = threadIdx.x; w < Qp * n; w += blockDim.x) {
        const int h = w / n, z = w - h * n;
        if (2 * h >= yv || z == n - 1) continue;
        stress_pair<1, false>(k, n, grp, x, y0 + 2 * h, z, [&](int f) {
            const float* p = S + (f * P + 2 * h) * np1 + z;
            return pack2(p[0], p[np1]);
        });
    }
    if (grp == 0) {
        __syncthreads();
        if (threadIdx.x == 0) inject(k, x, y0, yv);
    }
}

__global__ void __launch_bounds__(kThreads) k_dzr(KP k, int P)
{
    extern __shared__ float4 smem4[];
    float2* sm = reinterpret_cast<float2*>(smem4);
    const int n = k.nz, Qp = P / 2, ps = n + n / 16, ny = k.ny;
    float2* tw = sm;
    float2* A = tw + n;
    float2* B = A + Qp * ps;
    const int x = blockIdx.y, y0 = blockIdx.x * P, yv = min(P, ny - y0), f = blockIdx.z;
    const float inv_n = 1.0f / n;
    load_table(tw, k.tw_z, n);
    __syncthreads();
    const float* s = k.s[f == 0 ? 2 : f == 1 ? 4 : 5];
    auto load = [&](int q, int i) -> float2 {
        if (2 * q >= yv) return make_float2(0.f, 0.f);
        const float* p = s + cell(k, x, y0 + 2 * q, i);
        return make_float2(p[0], p[n]);
    };
    float2* Zf = fft_out_buf(k.pz, A, B);
    auto store_f = [&](int q, int i, float2 v) { Zf[q * ps + i] = v; };
    fft_run<false, false>(k.pz, tw, A, B, Qp, ps, 1, load, store_f, 4);
    float2* X1 = Zf == A ? B : A;
    const float2* T = f == 0 ? k.Bz : k.Fz;
    float* __restrict__ R = k.R[f == 0 ? 2 : f == 1 ? 0 : 1];
    float* __restrict__ ph = k.php[f == 0 ? 8 : f == 1 ? 2 : 5];  // pzz_z, pxz_z, pyz_z
    const float* pa = f == 0 ? k.azh : k.az;
    const float* pb = f == 0 ? k.bzh : k.bz;
    auto load_i = [&](int q, int i) -> float2 { return cmul_m(Zf[q * ps + i], cscale(T[i], inv_n)); };
    auto store_i = [&](int q, int i, float2 v) {
        if (2 * q >= yv) return;
        const int y = y0 + 2 * q;
        if (in_slab(i, n, k.pml) && i < n - 1 && x < k.nx - 1) {
            v.x = z_term(k, ph, x, y, i, pa[i], pb[i], v.x);
            if (y + 1 < ny - 1) v.y = z_term(k, ph, x, y + 1, i, pa[i], pb[i], v.y);
        }
        R[cell(k, x, y, i)] = v.x;
        R[cell(k, x, y + 1, i)] = v.y;
    };
    fft_run<false, true>(k.pz, tw, X1, Zf, Qp, ps, 1, load_i, store_i, 4);
}

#endif  // QVTI_PART == 0

}  // namespace

QVTI_DECLARE_PARTS(bool, st_launch, const KP& k, int P, cudaStream_t st);
QVTI_DECLARE_PARTS(bool, st_configure, SmemLimit& lim, int n);

template <>
bool st_launch<QVTI_PART>(const KP& k, int P, cudaStream_t st)
{
    return dispatch_len(k.nz, [&](auto NN) {
        constexpr int N = decltype(NN)::value;
        if constexpr (N >= kMinLong) {
            auto go = [&](auto QQ) {
                constexpr int q = decltype(QQ)::value, q9 = st_normal_q(N, q);
                k_st<N, 9, q9><<<dim3(cdiv(k.ny, 4 * q9), k.nx), st_threads(N, 9, q9), st_smem(N, 9, q9), st>>>(k);
                k_st<N, 6, q><<<dim3(3 * cdiv(k.ny, P), k.nx), st_threads(N, 6, q), st_smem(N, 6, q), st>>>(k);
            };
            if constexpr (st_eight_rows(N)) {
                if (P == 8) {
                    go(IntC<2>{});
                } else {
                    go(IntC<1>{});
                }
            } else {
                go(IntC<1>{});
            }
            k_dz<N><<<dim3(cdiv(k.ny, 4 * kDzPairs), k.nx, 3), dz_threads(N), dz_smem(N), st>>>(k);
        }
    });
}
template <>
bool st_configure<QVTI_PART>(SmemLimit& lim, int n)
{
    return dispatch_len(n, [&](auto NN) {
        constexpr int N = decltype(NN)::value;
        if constexpr (N >= kMinLong) {
            lim.set((const void*)k_st<N, 9, 1>);
            lim.set((const void*)k_st<N, 6, 1>);
            if constexpr (st_eight_rows(N)) {
                lim.set((const void*)k_st<N, 9, st_normal_q(N, 2)>);
                lim.set((const void*)k_st<N, 6, 2>);
            }
            lim.set((const void*)k_dz<N>);
        }
    });
}

#if QVTI_PART == 0
// Runtime layout of k_sigma: tw[nz] | A | B (with more than two stages) |
// S[9][P][nz+1]; k_dzr's tw | A | B is smaller.
size_t smem_sigma(const KP& k, int P, bool rt)
{
    if (!rt) return std::max(st_smem(k.nz, 9, P / 4), dz_smem(k.nz));
    const size_t bufA = (size_t)9 * (P / 2) * (k.nz + k.nz / 16);
    const int nb = k.pz.q.nst > 2 ? 2 : 1;
    return sizeof(float2) * (k.nz + nb * bufA) + sizeof(float) * (size_t)9 * P * (k.nz + 1);
}

void launch_sigma(const KP& k, int P, bool rt, cudaStream_t st)
{
    if (!rt) {
        (void)QVTI_CALL_PARTS(st_launch, k, P, st);
        return;
    }
    const int tiles = cdiv(k.ny, P);
    k_sigma<<<dim3(tiles, k.nx, 4), rt_threads(k.pz, 9 * P / 2), smem_sigma(k, P, true), st>>>(k, P);
    const size_t sm = sizeof(float2) * (k.nz + (size_t)P * (k.nz + k.nz / 16));
    k_dzr<<<dim3(tiles, k.nx, 3), rt_threads(k.pz, P / 2), sm, st>>>(k, P);
}

cudaError_t configure_sigma(int axis, int n)
{
    SmemLimit lim;
    if (axis < 0) {
        lim.set((const void*)k_sigma);
        lim.set((const void*)k_dzr);
    } else if (axis == 2) {
        (void)QVTI_CALL_PARTS(st_configure, lim, n);
    }
    return lim.e;
}
#endif  // QVTI_PART == 0

}  // namespace qvti
