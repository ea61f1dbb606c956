// Time-step kernels of the B200 viscoelastic pseudospectral engine.
//
// One time step of the reference (cuviscoelas_3D.cu:1255-1630: 29 launches,
// 63 cuFFT C2C transforms) becomes 10 launches here:
//
//   k_vy   y-pencils of the stresses: dy sxy, dy syy, dy syz (1D spectral
//          derivatives, C-PML memory terms in the y slab) added to R
//          (compiled lengths: k_dv)
//   k_vx   x-pencils: dx sxx, dx sxy, dx sxz, C-PML x terms, velocity update
//          (cuda_kernel_calculate_v, cu:1018-1101; compiled: k_dv)
//   k_fz   z-pencils: R2C of vx, vy, vz (two real pencils per complex FFT)
//   k_cy   y-lines: C2C forward of the 3 half spectra
//   k_mx   x-pencils in k-space: forward x, then the 21 constant-Q derivative
//          spectra Ap_j(|k|) * ik e^{+-ik d/2} * V (cu:475-744 fused) that
//          need it, each inverse-transformed along x on chip
//   k_cy   y-lines: C2C inverse of the 21 spectra
//   k_sigma  z-pencils: C2R of the 27 fields, stress update with constant-Q
//          dispersion + loss and C-PML (cuda_kernel_calculate_p,
//          cu:800-1015), source injection (cu:747-777); compiled: k_st, once
//          for the normal and once for the three shear stresses
//   k_dz   z derivatives of the new stresses for the next velocity update
//          (runtime lengths: k_dzr)
//   k_rec  receiver sampling (cu:782-791)
//
// The stress-divergence derivatives need no 3D transform at all: their
// multiplier depends on one wavenumber component, so IFFT3(M(kx) FFT3(f)) is
// the 1D spectral derivative along x of every x line (likewise y, z).
#include <algorithm>

#include "step_common.cuh"

namespace qvti {

namespace {

// ----------------------------------------------------------------- k_rec --
// Receivers (cu:782-791).  With traces to inject (back-propagation of
// recorded data, the adjoint of recording), sample nt - 1 - it of each
// component is first added to that component at the receiver, at the point
// of the step where the source is injected and the records are taken.
__global__ void k_rec(KP k)
{
    const int ir = blockIdx.x * blockDim.x + threadIdx.x;
    const int it = *k.d_it;
    if (ir >= k.rn || it < 0 || it >= k.nt_rec) return;
    const int ip = cell(k, k.r_ix[ir], k.r_iy[ir], k.r_iz);
    if (it < k.inj_nt) {
        const long long o = (long long)(k.inj_nt - 1 - it) * k.rn + ir;
        for (int c = 0; c < 3; ++c)
            if (k.inj[c]) k.v[c][ip] += k.inj[c][o];
    }
    const long long o = (long long)it * k.rn + ir;
    if (k.rec[0]) {
        k.rec[0][o] = k.v[0][ip];
        k.rec[1][o] = k.v[1][ip];
        k.rec[2][o] = k.v[2][ip];
    }
}

// ----------------------------------------------------- setup, FP64 kernels --
// Constant-Q sets (cuviscoelas_3D.cu:195-205) per modulus, FP64:
// c = v cos(pi g / 2); eta1 = -rho c g w0, eta2 = rho c^2, eta3 = rho c^3 g / w0,
// tau1 = rho c g pi, tau2 = rho c^2 g^2 pi / w0 (pi = 3.1415926, cu:15).
__device__ __forceinline__ void qset(double v, double g, double r, double w0, double o[5])
{
    const double pi = 3.1415926;
    const double c = v * cos(g * pi / 2.0);
    o[0] = -r * c * g * w0;
    o[1] = r * c * c;
    o[2] = r * c * c * c * g / w0;
    o[3] = r * c * g * pi;
    o[4] = r * c * c * g * g * pi / w0;
}

// Per-cell coefficient build, FP64.  out[0..7): rho, gamma_p, gamma_s and the
// effective velocities c = v cos(pi gamma / 2) of c11, c33, c13 (gamma_p) and
// c44 (gamma_s); out[7..12): the S set of c44, input of the 8-point average.
// VTI (project extension): c33 = rho vp^2, c44 = c66 = rho vs^2,
// c11 = c33 (1 + 2 eps), c13 = sqrt((c33 - c44)(c33 (1 + 2 delta) - c44)) - c44,
// each modulus taking the constant-Q set of its effective velocity
// (v11 = vp sqrt(1 + 2 eps), v13 = sqrt((c13 + 2 c44)/rho)); the off-diagonal
// sets are P(v) - 2 S(vs), which at eps = delta = 0 is the reference's
// eta_p - 2 eta_s (cu:851-898).
__global__ void k_coef(long long ntp, const float* velp, const float* vels, const float* rho, const float* gp,
                       const float* gs, const float* eps, const float* delta, int vti, double w0, int lossless,
                       float* const* out)
{
    const double pi = 3.1415926;
    for (long long ip = blockIdx.x * (long long)blockDim.x + threadIdx.x; ip < ntp;
         ip += (long long)gridDim.x * blockDim.x) {
        // lossless medium: gamma = 0 (Q infinite), the constant-Q sets reduce
        // to the elastic moduli
        const double r = rho[ip], vp = velp[ip], vs = vels[ip], g_p = lossless ? 0.0 : gp[ip],
                     g_s = lossless ? 0.0 : gs[ip];
        const double cp = cos(g_p * pi / 2.0), cq = cos(g_s * pi / 2.0);
        double v11 = vp, v13 = vp;
        if (vti) {
            const double e = eps[ip], dl = delta[ip];
            const double c33 = r * vp * vp, c44 = r * vs * vs;
            const double c13 = sqrt((c33 - c44) * (c33 * (1.0 + 2.0 * dl) - c44)) - c44;
            v11 = vp * sqrt(1.0 + 2.0 * e);
            v13 = sqrt((c13 + 2.0 * c44) / r);
        }
        out[0][ip] = (float)r;
        out[1][ip] = (float)g_p;
        out[2][ip] = (float)g_s;
        out[3][ip] = (float)(v11 * cp);
        out[4][ip] = (float)(vp * cp);
        out[5][ip] = (float)(v13 * cp);
        out[6][ip] = (float)(vs * cq);
        double s5[5];
        qset(vs, g_s, r, w0, s5);
        for (int j = 0; j < 5; ++j) out[7 + j][ip] = (float)s5[j];
    }
}

// 8-point averaged shear set (cu:956-971) and 1/rho-bar (cu:1077-1092).
struct MuArgs {
    const float* s[5];
    float* mu[5];
    const float* rho;
    float* rinv[3];
};
__global__ void k_mu_rinv(KP k, MuArgs a)
{
    const long long A = (long long)k.ny * k.nz;
    for (long long ip = blockIdx.x * (long long)blockDim.x + threadIdx.x; ip < k.ntp;
         ip += (long long)gridDim.x * blockDim.x) {
        const int z = ip % k.nz, y = (ip / k.nz) % k.ny, x = ip / A;
        const bool in = x < k.nx - 1 && y < k.ny - 1 && z < k.nz - 1;
        for (int j = 0; j < 5; ++j) {
            const float* s = a.s[j];
            double m = 0.0;
            if (in)
                m = 0.125 * ((double)s[ip] + s[ip + 1] + s[ip + k.nz] + s[ip + 1 + k.nz] + s[ip + A] + s[ip + A + 1] +
                             s[ip + A + k.nz] + s[ip + A + 1 + k.nz]);
            a.mu[j][ip] = (float)m;
        }
        const double r0 = a.rho[ip];
        a.rinv[0][ip] = in ? (float)(1.0 / (0.5 * (r0 + a.rho[ip + A]))) : 0.f;
        a.rinv[1][ip] = in ? (float)(1.0 / (0.5 * (r0 + a.rho[ip + k.nz]))) : 0.f;
        a.rinv[2][ip] = in ? (float)(1.0 / (0.5 * (r0 + a.rho[ip + 1]))) : 0.f;
    }
}

// 1D derivative along one axis of a real field (tests / diagnostics): out =
// Re IFFT(T(k)/n * FFT(in)) along `axis`, T the forward or backward shift.
__global__ void k_deriv1d(KP k, int axis, int fwd, const float* in, float* out, int P)
{
    extern __shared__ float4 smem4[];
    float2* sm = reinterpret_cast<float2*>(smem4);
    const FftPlan& pl = axis == 0 ? k.px : axis == 1 ? k.py : k.pz;
    const int n = pl.n;
    const float2* T = axis == 0 ? (fwd ? k.Fx : k.Bx) : axis == 1 ? (fwd ? k.Fy : k.By) : (fwd ? k.Fz : k.Bz);
    const float2* gtw = axis == 0 ? k.tw_x : axis == 1 ? k.tw_y : k.tw_z;
    float2* tw = sm;
    float2* A = tw + n;
    float2* B = A + n * P;
    load_table(tw, gtw, n);
    __syncthreads();
    // pencils: P/2 complex pairs; pencil index pp over the other two axes
    const int Qp = P / 2;
    const long long npen = k.ntp / n;
    const long long pen0 = (long long)blockIdx.x * P;
    auto addr = [&](long long pen, int i) -> long long {
        if (axis == 2) return pen * n + i;
        if (axis == 1) { const long long x = pen / k.nz, z = pen % k.nz; return (x * k.ny + i) * k.nz + z; }
        return (long long)i * k.ny * k.nz + pen;
    };
    float2* Zf = fft_out_buf(pl, A, B);
    auto load = [&](int q, int i) -> float2 {
        const long long p0 = pen0 + 2 * q, p1 = p0 + 1;
        return make_float2(p0 < npen ? in[addr(p0, i)] : 0.f, p1 < npen ? in[addr(p1, i)] : 0.f);
    };
    auto store = [&](int q, int i, float2 v) { Zf[i * Qp + q] = v; };
    fft_run<true, false>(pl, tw, A, B, Qp, 1, Qp, load, store);
    float2* X1 = Zf == A ? B : A;
    const float inv_n = 1.0f / n;
    auto load_i = [&](int q, int i) -> float2 { return cmul_m(Zf[i * Qp + q], cscale(T[i], inv_n)); };
    auto store_i = [&](int q, int i, float2 v) {
        const long long p0 = pen0 + 2 * q, p1 = p0 + 1;
        if (p0 < npen) out[addr(p0, i)] = v.x;
        if (p1 < npen) out[addr(p1, i)] = v.y;
    };
    fft_run<true, true>(pl, tw, X1, Zf, Qp, 1, Qp, load_i, store_i);
}

// ------------------------------------------- single-field constant-Q field --
// One of the 27 stress-side fields on its own: out = Re IFFT3(|k|^pw T(k_a)
// FFT3(in)) / ntp with T the forward or backward staggered shift along axis
// a (cu:475-744 with the transforms around them).  The half spectrum H[0]
// (kz-major, as in the step) is the scratch; k_fz and k_cy do the z and y
// passes, these two kernels the k-space x pass and the C2R along z.
__global__ void __launch_bounds__(kThreads) kq_mx(KP k, int P, int axis, int fwd, int pw)
{
    extern __shared__ float4 smem4[];
    float2* sm = reinterpret_cast<float2*>(smem4);
    const int n = k.nx;
    float2* tw = sm;
    float2* V = tw + n;   // [n][P]
    float2* A = V + n * P;
    float2* B = A + (n + n / 16) * P;
    load_table(tw, k.tw_x, n);
    __syncthreads();
    const int kz = blockIdx.y, y0 = blockIdx.x * P;
    float2* H = k.H[0];
    auto load = [&](int p, int i) -> float2 { return H[spec(k, kz, i, y0 + p)]; };
    auto store = [&](int p, int i, float2 v) { V[i * P + p] = v; };
    fft_run<true, false>(k.px, tw, A, B, P, 1, P, load, store, 4);
    const float kz2 = k.kz[kz] * k.kz[kz];
    auto load_i = [&](int p, int i) -> float2 {
        const float kyv = k.ky[y0 + p], kxv = k.kx[i];
        const float k2 = fmaxf(kxv * kxv + kyv * kyv + kz2, 1e-10f);
        const float ap = pw == 0 ? 1.0f : (pw < 0 ? 1.0f / sqrtf(k2) : sqrtf(k2));
        float2 T;
        if (axis == 0) T = fwd ? k.Fx[i] : k.Bx[i];
        else if (axis == 1) T = fwd ? k.Fy[y0 + p] : k.By[y0 + p];
        else T = fwd ? k.Fz[kz] : k.Bz[kz];
        return cmul(V[i * P + p], cscale(T, ap * k.inv_ntp));
    };
    auto store_i = [&](int p, int i, float2 v) { H[spec(k, kz, i, y0 + p)] = v; };
    fft_run<true, true>(k.px, tw, A, B, P, 1, P, load_i, store_i, 4);
}

__global__ void __launch_bounds__(kThreads) kq_iz(KP k, int P, float* out)
{
    extern __shared__ float4 smem4[];
    float2* sm = reinterpret_cast<float2*>(smem4);
    const int n = k.nz, Qp = P / 2;
    float2* tw = sm;
    float2* A = tw + n;
    float2* B = A + Qp * (n + n / 16);
    load_table(tw, k.tw_z, n);
    __syncthreads();
    const int x = blockIdx.y, y0 = blockIdx.x * P;
    const float2* g = k.H[0];
    auto load = [&](int q, int i) -> float2 {
        const int kk = i <= n / 2 ? i : n - i;
        const float4 gg = *reinterpret_cast<const float4*>(g + spec(k, kk, x, y0 + 2 * q));
        float2 a = make_float2(gg.x, gg.y), b = make_float2(gg.z, gg.w);
        if (kk == 0 || 2 * kk == n) { a.y = 0.f; b.y = 0.f; }
        if (i > n / 2) { a.y = -a.y; b.y = -b.y; }
        return make_float2(a.x - b.y, a.y + b.x);
    };
    auto store = [&](int q, int i, float2 v) {
        out[cell(k, x, y0 + 2 * q, i)] = v.x;
        out[cell(k, x, y0 + 2 * q + 1, i)] = v.y;
    };
    fft_run<true, true>(k.pz, tw, A, B, Qp, 1, Qp, load, store, 4);
}

// --------------------------------------------------------- tile selection --
int tile_of(int n, int want)
{
    int p = want;
    while (p > 2 && n % p) p >>= 1;
    return p;
}

}  // namespace

namespace {

bool ct_length(int n)
{
    for (int c : kCtLengths)
        if (c == n) return true;
    return false;
}
// Tiles of the step's launches.  A kernel whose transform length is compiled
// takes its full tile along the other axis, the last tile ragged (its rows
// or lines past the grid read as zeros and are not written); otherwise the
// runtime path takes the largest power-of-two divisor of the tiled axis up
// to the full tile.  A tile set in KP::tile_rt selects the runtime path with
// that tile.
//
// The compiled velocity kernels take 32 z (whole 128-byte rows: 16 z left
// half of every L1 line it fetched unused and measured 0.21 against 0.15 ms
// for k_vy, 0.34 against 0.22 for k_vx at 256^3, with the epilogue on registers)
// unless that leaves fewer than two blocks per SM.
int dv_tile(int nz, int lines) { return 3ll * cdiv(nz, 64) * lines >= 2 * 148 ? 32 : 16; }
// The compiled stress kernels take eight rows (half-line accesses, see k_st)
// unless that leaves fewer than four blocks per SM.
int st_rows(const KP& k)
{
    return st_eight_rows(k.nz) && (long long)cdiv(k.ny, 8) * k.nx >= 4 * 148 ? 8 : kSigmaRows;
}
struct StepTiles {
    int vy, vx, fz, cy, mx, sigma;
    bool rt[kNumTiled];  // runtime path, in the order above
};
StepTiles step_tiles(const KP& k)
{
    StepTiles t;
    auto tile = [&](int i, int len, int tiled, int want) {
        if (k.tile_rt[i] > 0) {
            t.rt[i] = true;
            return k.tile_rt[i];
        }
        t.rt[i] = !ct_length(len) || ((i == 1 || i == 4 || i == 5) && len < kMinLong);
        return t.rt[i] ? tile_of(tiled, std::min(want, 16)) : want;
    };
    t.vy = tile(0, k.ny, k.nz, dv_tile(k.nz, k.nx));
    t.vx = tile(1, k.nx, k.nz, dv_tile(k.nz, k.ny));
    t.fz = tile(2, k.nz, k.ny, 16);
    t.cy = tile(3, k.ny, k.nx, 8);
    t.mx = tile(4, k.nx, k.ny, 16);
    if (!t.rt[4]) t.mx = mp_rows(k.nx);
    t.sigma = tile(5, k.nz, k.ny, k.nz < kMinLong ? 16 : kSigmaRows);
    if (!t.rt[5]) t.sigma = st_rows(k);
    return t;
}

}  // namespace

int configure_kernels()
{
    SmemLimit lim;
    lim.set((const void*)k_deriv1d);
    lim.set((const void*)kq_mx);
    lim.set((const void*)kq_iz);
    for (cudaError_t r : {configure_velocity(-1, 0), configure_spectral(-1, 0), configure_sigma(-1, 0)})
        if (r != cudaSuccess) lim.e = r;
    const int et = configure_tc_kernels();
    if (et) lim.e = (cudaError_t)et;
    return (int)lim.e;
}

int configure_length(int axis, int n)
{
    cudaError_t e = cudaSuccess;
    for (cudaError_t r : {configure_velocity(axis, n), configure_spectral(axis, n), configure_sigma(axis, n)})
        if (r != cudaSuccess) e = r;
    return (int)e;
}

const char* const kStepKernelNames[kStepKernels] = {"k_vy",  "k_vx",     "k_fz",    "k_cy_fwd",
                                                     "k_mx",  "k_cy_inv", "k_sigma", "k_rec"};

// One time step.  With a profile sink, an event is recorded before the first
// kernel and after every launch, tagged with the launch's kernel index.
void launch_step(const KP& k, cudaStream_t st, StepProfile* prof)
{
    auto mark = [&](int kind) {
        if (prof && prof->n < StepProfile::kMax) {
            cudaEventRecord(prof->ev[prof->n], st);
            prof->kind[prof->n++] = kind;
        }
    };
    // the compile-time path of a kernel fixes its tile: 16 or 32 z (k_vy, k_vx;
    // dv_tile), 16 y rows (k_fz), 16 or 8 (k_mx; mp_rows), 8 lines (k_cy), 4 or
    // 8 y rows (k_sigma; st_rows)
    const StepTiles T = step_tiles(k);
    mark(-1);
    launch_vy(k, T.vy, T.rt[0], st);
    mark(0);
    launch_vx(k, T.vx, T.rt[1], st);
    mark(1);
    launch_fz(k, T.fz, T.rt[2], 3, st);
    mark(2);
    // k-space passes, optionally in batches of kz planes (KP::kz_batch).
    const int batch = k.kz_batch > 0 ? k.kz_batch : k.nkz;
    for (int kz0 = 0; kz0 < k.nkz; kz0 += batch) {
        const int nb = kz0 + batch <= k.nkz ? batch : k.nkz - kz0;
        const long long line0 = (long long)kz0 * k.nx, line_end = line0 + (long long)nb * k.nx;
        const bool tc = k.form == kFormTc && tc_cy_available(k);
        if (tc) launch_cy_tc(k, false, 3, line0, line_end, st);
        else launch_cy(k, T.cy, T.rt[3], false, 3, true, line0, line_end, st);
        mark(3);
        launch_mx(k, T.mx, T.rt[4], kz0, nb, st);
        mark(4);
        if (tc) launch_cy_tc(k, true, kNumGxy, line0, line_end, st);
        else launch_cy(k, T.cy, T.rt[3], true, kNumGxy, false, line0, line_end, st);
        mark(5);
    }
    launch_sigma(k, T.sigma, T.rt[5], st);
    mark(6);
    if (k.rn > 0) {
        k_rec<<<(k.rn + 255) / 256, 256, 0, st>>>(k);
        mark(7);
    }
}

// Largest dynamic shared memory of the step's launches for this grid.
size_t step_smem_bytes(const KP& k)
{
    const StepTiles T = step_tiles(k);
    size_t m = smem_vyx(k.ny, T.vy, T.rt[0]);
    m = std::max(m, smem_vyx(k.nx, T.vx, T.rt[1]));
    m = std::max(m, smem_fz(k, T.fz, T.rt[2]));
    m = std::max(m, smem_cy(k, T.cy, true, T.rt[3]));
    m = std::max(m, smem_mx(k, T.mx, T.rt[4]));
    m = std::max(m, smem_sigma(k, T.sigma, T.rt[5]));
    // the grids and tiles that are supported at runtime lengths are those of
    // layouts with a second transform buffer from three radices on, and on the z
    // axis with room for the z derivatives and their tables beside the fields
    if (T.rt[4] && k.px.q.radices > 2 && k.px.q.nst == 2)
        m = std::max(m, smem_mx(k, T.mx, true) + sizeof(float2) * (k.nx + k.nx / 16) * T.mx);
    if (T.rt[5]) {
        const size_t more = k.pz.q.radices > 2 && k.pz.q.nst == 2 ? sizeof(float2) * 9 * (T.sigma / 2) * (k.nz + k.nz / 16) : 0;
        m = std::max(m, smem_sigma(k, T.sigma, true) + more + sizeof(float2) * 2 * k.nz +
                            sizeof(float) * ((size_t)3 * T.sigma * (k.nz + 1) + 4 * k.nz + 4 * T.sigma));
    }
    return m;
}

void step_tile_set(const KP& k, int tiles[kNumTiled], int runtime[kNumTiled])
{
    const StepTiles T = step_tiles(k);
    const int t[kNumTiled] = {T.vy, T.vx, T.fz, T.cy, T.mx, T.sigma};
    for (int i = 0; i < kNumTiled; ++i) {
        if (tiles) tiles[i] = t[i];
        if (runtime) runtime[i] = T.rt[i] ? 1 : 0;
    }
}

bool tiles_valid(const KP& k)
{
    // the axis each kernel tiles: z rows (k_vy, k_vx), y rows (k_fz, k_mx,
    // k_sigma); k_cy's lines need not divide anything (a batch's last tile
    // is partial)
    const int axis[kNumTiled] = {k.nz, k.nz, k.ny, 0, k.ny, k.ny};
    for (int i = 0; i < kNumTiled; ++i) {
        const int t = k.tile_rt[i];
        if (t == 0) continue;
        if (t < 2 || t > 32 || (t & 1) || (axis[i] && axis[i] % t)) return false;
    }
    return step_smem_bytes(k) <= kMaxSmem;
}

void launch_coef_build(const KP& k, const float* velp, const float* vels, const float* rho, const float* gp,
                       const float* gs, const float* eps, const float* delta, int vti, float w0, int lossless,
                       float* const* coef_out, cudaStream_t st)
{
    k_coef<<<148 * 8, 256, 0, st>>>(k.ntp, velp, vels, rho, gp, gs, eps, delta, vti, (double)w0, lossless, coef_out);
}

void launch_mu_rinv(const KP& k, const float* rho, const float* const* sset, cudaStream_t st)
{
    MuArgs a;
    for (int j = 0; j < 5; ++j) { a.s[j] = sset[j]; a.mu[j] = const_cast<float*>(k.MU[j]); }
    a.rho = rho;
    for (int c = 0; c < 3; ++c) a.rinv[c] = const_cast<float*>(k.rinv[c]);
    k_mu_rinv<<<148 * 8, 256, 0, st>>>(k, a);
}

// k.v[0] = input field, k.H[0] = k.G[0] = half-spectrum scratch (nkz*nx*ny).
void launch_q_derivative(const KP& k_in, int axis, int fwd, int pw, float* out, cudaStream_t st)
{
    KP k = k_in;
    k.Hy[0] = k.H[0];  // the forward y pass works in place on the one scratch spectrum
    for (int c = 0; c < 3; ++c) k.Yv[c] = nullptr;  // and writes no y derivative
    const long long lines = (long long)k.nkz * k.nx;
    launch_fz(k, tile_of(k.ny, 16), true, 1, st);
    const int L = tile_of(k.nx, 8);
    launch_cy(k, L, true, false, 1, false, 0, lines, st);
    const int Pm = tile_of(k.ny, 8);
    kq_mx<<<dim3(k.ny / Pm, k.nkz), kThreads, sizeof(float2) * (k.nx + k.nx * Pm + 2 * (k.nx + k.nx / 16) * Pm), st>>>(
        k, Pm, axis, fwd, pw);
    launch_cy(k, L, true, true, 1, false, 0, lines, st);
    const int Pi = tile_of(k.ny, 8);
    kq_iz<<<dim3(k.ny / Pi, k.nx), kThreads, sizeof(float2) * (k.nz + 2 * (Pi / 2) * (k.nz + k.nz / 16)), st>>>(k, Pi,
                                                                                                               out);
}

void launch_derivative_1d(const KP& k, int axis, int fwd, const float* in, float* out, cudaStream_t st)
{
    const int n = axis == 0 ? k.nx : axis == 1 ? k.ny : k.nz;
    const int P = 16;
    const long long npen = k.ntp / n;
    const unsigned nb = (unsigned)((npen + P - 1) / P);
    k_deriv1d<<<nb, kThreads, sizeof(float2) * (n + 2 * n * P), st>>>(k, axis, fwd, in, out, P);
}

}  // namespace qvti
