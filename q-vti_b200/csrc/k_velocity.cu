// Velocity kernels of the time step: the y and x derivatives of the stresses
// and the velocity update.
#include "fft_pair.cuh"
#include "step_common.cuh"

namespace qvti {

namespace {

#if QVTI_PART == 0
// ------------------------------------------------------------------ k_vy --
// The runtime-length kernels (k_dv below is the compiled form); blockIdx.z: the
// pass (two fields, or one).
// y-derivatives of sxy (+, -> vx), syy (-, -> vy), syz (+, -> vz) for one x
// and P consecutive z; C-PML y terms; accumulate into R.  Each pass parks its
// derivatives in shared memory; the epilogue then loads everything a cell
// needs before storing anything (no store can delay a later load).
__global__ void __launch_bounds__(kThreads) k_vy(KP k, int P)
{
    extern __shared__ float4 smem4[];
    float2* sm = reinterpret_cast<float2*>(smem4);
    const int n = k.ny, ny = n, pml = k.pml;
    float2* tw = sm;
    float2* tF = tw + n;   // forward shift; the backward one is (-F.x, F.y)
    float2* A = tF + n;
    float2* B = A + (n + n / 16) * P;
    load_table(tw, k.tw_y, n);
    load_table(tF, k.Fy, n);
    if (blockIdx.x + blockIdx.y + blockIdx.z == 0 && threadIdx.x == 0) *k.d_it += 1;  // step counter
    __syncthreads();
    const int x = blockIdx.y, z0 = blockIdx.x * P;
    const int zv = min(P, k.nz - z0);  // rows of the tile inside the grid (even)
    const float dt = k.dt, inv_n = 1.0f / n;
    const bool xin = x < k.nx - 1;
    const float* __restrict__ sxy = k.s[3];
    const float* __restrict__ syy = k.s[1];
    const float* __restrict__ syz = k.s[5];
    float* __restrict__ R0 = k.R[0];
    float* __restrict__ R1 = k.R[1];
    float* __restrict__ R2 = k.R[2];
    float* __restrict__ f1 = k.php[1];  // phi_pxy_y, b_y
    float* __restrict__ f4 = k.php[4];  // phi_pyy_y, averaged b_y
    float* __restrict__ f7 = k.php[7];  // phi_pyz_y, b_y

    // pass 1: sxy + i syy -> dy+ sxy (vx), dy- syy (vy)
    if (blockIdx.z == 0) {
        float2* Zf = fft_out_buf(k.py, A, B);
        auto load = [&](int p, int i) -> float2 {
            if (p >= zv) return make_float2(0.f, 0.f);
            const int ip = cell(k, x, i, z0 + p);
            return make_float2(sxy[ip], syy[ip]);
        };
        auto store = [&](int p, int i, float2 v) { Zf[i * P + p] = v; };
        fft_rt<kPencil, false>(k.py, tw, A, B, P, 1, P, load, store);
        float2* X1 = Zf == A ? B : A;
        // [2][n][P] in the buffer the last stage does not read
        float* D = reinterpret_cast<float*>(fft_out_buf(k.py, X1, Zf));
        auto load_i = [&](int p, int i) -> float2 {
            const int im = i ? n - i : 0;
            return two_shift(Zf[i * P + p], cconj(Zf[im * P + p]), cscale(tF[i], inv_n), 1.0f);
        };
        auto store_i = [&](int p, int i, float2 v) {
            D[i * P + p] = v.x;
            D[(n + i) * P + p] = v.y;
        };
        fft_rt<kPencil, true>(k.py, tw, X1, Zf, P, 1, P, load_i, store_i);
        // kEpi cells per thread and trip: all their loads are in flight at once
        for (int t0 = threadIdx.x; t0 < n * P; t0 += kEpi * blockDim.x) {
            int ipu[kEpi], iu[kEpi], pu[kEpi], isu[kEpi];
            bool ok[kEpi], slab[kEpi];
            float r0[kEpi], r1[kEpi], p1[kEpi], p4[kEpi];
#pragma unroll
            for (int u = 0; u < kEpi; ++u) {
                const int t = t0 + u * blockDim.x;
                pu[u] = t % P;
                iu[u] = t / P;
                ok[u] = t < n * P && pu[u] < zv;
                const int z = z0 + pu[u];
                ipu[u] = cell(k, x, iu[u], z);
                slab[u] = ok[u] && in_slab(iu[u], ny, pml) && xin && iu[u] < ny - 1 && z < k.nz - 1;
                isu[u] = slab[u] ? slab_y(k, x, iu[u], z) : 0;
                r0[u] = ok[u] ? R0[ipu[u]] : 0.f;
                r1[u] = ok[u] ? R1[ipu[u]] : 0.f;
                p1[u] = slab[u] ? f1[isu[u]] : 0.f;
                p4[u] = slab[u] ? f4[isu[u]] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < kEpi; ++u) {
                if (!ok[u]) continue;
                const int i = iu[u], p = pu[u], ip = ipu[u];
                const float dx = D[i * P + p], dy = D[(n + i) * P + p];
                float rx = r0[u] + dx, ry = r1[u] + dy;
                if (slab[u]) {
                    const float q1 = p1[u] + dt * (-k.ay[i] * p1[u] - k.by[i] * dx);
                    const float q4 = p4[u] + dt * (-k.ayh[i] * p4[u] - k.byh[i] * dy);
                    rx += q1;
                    ry += q4;
                    f1[isu[u]] = q1;
                    f4[isu[u]] = q4;
                }
                R0[ip] = rx;
                R1[ip] = ry;
            }
        }
        return;
    }
    // pass 2: syz, pencils (2q, 2q+1) -> dy+ syz (vz)
    {
        const int Qp = P / 2;
        float2* Zf = fft_out_buf(k.py, A, B);
        auto load = [&](int q, int i) -> float2 {
            if (2 * q >= zv) return make_float2(0.f, 0.f);
            const int ip = cell(k, x, i, z0 + 2 * q);
            return *reinterpret_cast<const float2*>(syz + ip);
        };
        auto store = [&](int q, int i, float2 v) { Zf[i * Qp + q] = v; };
        fft_rt<kPencil, false>(k.py, tw, A, B, Qp, 1, Qp, load, store);
        float2* X1 = Zf == A ? B : A;
        float* D = reinterpret_cast<float*>(fft_out_buf(k.py, X1, Zf));  // [n][P]
        auto load_i = [&](int q, int i) -> float2 { return cmul_m(Zf[i * Qp + q], cscale(tF[i], inv_n)); };
        auto store_i = [&](int q, int i, float2 v) {
            D[i * P + 2 * q] = v.x;
            D[i * P + 2 * q + 1] = v.y;
        };
        fft_rt<kPencil, true>(k.py, tw, X1, Zf, Qp, 1, Qp, load_i, store_i);
        for (int t0 = threadIdx.x; t0 < n * P; t0 += kEpi * blockDim.x) {
            int ipu[kEpi], iu[kEpi], pu[kEpi], isu[kEpi];
            bool ok[kEpi], slab[kEpi];
            float r2[kEpi], p7[kEpi];
#pragma unroll
            for (int u = 0; u < kEpi; ++u) {
                const int t = t0 + u * blockDim.x;
                pu[u] = t % P;
                iu[u] = t / P;
                ok[u] = t < n * P && pu[u] < zv;
                const int z = z0 + pu[u];
                ipu[u] = cell(k, x, iu[u], z);
                slab[u] = ok[u] && in_slab(iu[u], ny, pml) && xin && iu[u] < ny - 1 && z < k.nz - 1;
                isu[u] = slab[u] ? slab_y(k, x, iu[u], z) : 0;
                r2[u] = ok[u] ? R2[ipu[u]] : 0.f;
                p7[u] = slab[u] ? f7[isu[u]] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < kEpi; ++u) {
                if (!ok[u]) continue;
                const int i = iu[u], ip = ipu[u];
                const float dz = D[i * P + pu[u]];
                float rz = r2[u] + dz;
                if (slab[u]) {
                    const float q7 = p7[u] + dt * (-k.ay[i] * p7[u] - k.by[i] * dz);
                    rz += q7;
                    f7[isu[u]] = q7;
                }
                R2[ip] = rz;
            }
        }
    }
}

// ------------------------------------------------------------------ k_vx --
// x-derivatives of sxx (-, vx), sxy (+, vy), sxz (+, vz); C-PML x terms and
// the velocity update (cuda_kernel_calculate_v, cu:1018-1101); same
// park-then-epilogue structure as k_vy.
__global__ void __launch_bounds__(kThreads) k_vx(KP k, int P)
{
    extern __shared__ float4 smem4[];
    float2* sm = reinterpret_cast<float2*>(smem4);
    const int n = k.nx, nx = n, pml = k.pml;
    float2* tw = sm;
    float2* tF = tw + n;   // forward shift; the backward one is (-F.x, F.y)
    float2* A = tF + n;
    float2* B = A + (n + n / 16) * P;
    load_table(tw, k.tw_x, n);
    load_table(tF, k.Fx, n);
    __syncthreads();
    const int y = blockIdx.y, z0 = blockIdx.x * P;
    const int zv = min(P, k.nz - z0);  // rows of the tile inside the grid (even)
    const float dt = k.dt, inv_n = 1.0f / n;
    const bool yin = y < k.ny - 1;
    const float* __restrict__ sxx = k.s[0];
    const float* __restrict__ sxy = k.s[3];
    const float* __restrict__ sxz = k.s[4];
    float* __restrict__ v0 = k.v[0];
    float* __restrict__ v1 = k.v[1];
    float* __restrict__ v2 = k.v[2];
    const float* __restrict__ R0 = k.R[0];
    const float* __restrict__ R1 = k.R[1];
    const float* __restrict__ R2 = k.R[2];
    const float* __restrict__ ri0 = k.rinv[0];
    const float* __restrict__ ri1 = k.rinv[1];
    const float* __restrict__ ri2 = k.rinv[2];
    float* __restrict__ f0 = k.php[0];  // phi_pxx_x, averaged b_x
    float* __restrict__ f3 = k.php[3];  // phi_pxy_x, b_x
    float* __restrict__ f6 = k.php[6];  // phi_pxz_x, b_x

    // pass 1: sxx + i sxy -> dx- sxx (vx), dx+ sxy (vy)
    if (blockIdx.z == 0) {
        float2* Zf = fft_out_buf(k.px, A, B);
        auto load = [&](int p, int i) -> float2 {
            if (p >= zv) return make_float2(0.f, 0.f);
            const int ip = cell(k, i, y, z0 + p);
            return make_float2(sxx[ip], sxy[ip]);
        };
        auto store = [&](int p, int i, float2 v) { Zf[i * P + p] = v; };
        fft_rt<kPencil, false>(k.px, tw, A, B, P, 1, P, load, store);
        float2* X1 = Zf == A ? B : A;
        float* D = reinterpret_cast<float*>(fft_out_buf(k.px, X1, Zf));  // [2][n][P]
        auto load_i = [&](int p, int i) -> float2 {
            const int im = i ? n - i : 0;
            return two_shift(Zf[i * P + p], cconj(Zf[im * P + p]), cscale(tF[i], inv_n), -1.0f);
        };
        auto store_i = [&](int p, int i, float2 v) {
            D[i * P + p] = v.x;
            D[(n + i) * P + p] = v.y;
        };
        fft_rt<kPencil, true>(k.px, tw, X1, Zf, P, 1, P, load_i, store_i);
        for (int t0 = threadIdx.x; t0 < n * P; t0 += kEpi * blockDim.x) {
            int ipu[kEpi], iu[kEpi], pu[kEpi], isu[kEpi];
            bool ok[kEpi], slab[kEpi];
            float a0[kEpi], a1[kEpi], r0[kEpi], r1[kEpi], w0[kEpi], w1[kEpi], p0[kEpi], p3[kEpi];
#pragma unroll
            for (int u = 0; u < kEpi; ++u) {
                const int t = t0 + u * blockDim.x;
                pu[u] = t % P;
                iu[u] = t / P;
                const int z = z0 + pu[u];
                ok[u] = t < n * P && iu[u] < nx - 1 && yin && z < k.nz - 1;
                ipu[u] = cell(k, iu[u], y, z);
                slab[u] = ok[u] && in_slab(iu[u], nx, pml);
                isu[u] = slab[u] ? slab_x(k, iu[u], y, z) : 0;
                const int ip = ipu[u];
                a0[u] = ok[u] ? v0[ip] : 0.f;
                a1[u] = ok[u] ? v1[ip] : 0.f;
                r0[u] = ok[u] ? R0[ip] : 0.f;
                r1[u] = ok[u] ? R1[ip] : 0.f;
                w0[u] = ok[u] ? ri0[ip] : 0.f;
                w1[u] = ok[u] ? ri1[ip] : 0.f;
                p0[u] = slab[u] ? f0[isu[u]] : 0.f;
                p3[u] = slab[u] ? f3[isu[u]] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < kEpi; ++u) {
                if (!ok[u]) continue;
                const int i = iu[u], p = pu[u], ip = ipu[u];
                float px = D[i * P + p], py = D[(n + i) * P + p];
                if (slab[u]) {
                    const float q0 = p0[u] + dt * (-k.axh[i] * p0[u] - k.bxh[i] * px);
                    const float q3 = p3[u] + dt * (-k.ax[i] * p3[u] - k.bx[i] * py);
                    px += q0;
                    py += q3;
                    f0[isu[u]] = q0;
                    f3[isu[u]] = q3;
                }
                v0[ip] = a0[u] + dt * w0[u] * (px + r0[u]);
                v1[ip] = a1[u] + dt * w1[u] * (py + r1[u]);
            }
        }
        return;
    }
    // pass 2: sxz pencils (2q, 2q+1) -> dx+ sxz (vz)
    {
        const int Qp = P / 2;
        float2* Zf = fft_out_buf(k.px, A, B);
        auto load = [&](int q, int i) -> float2 {
            if (2 * q >= zv) return make_float2(0.f, 0.f);
            const int ip = cell(k, i, y, z0 + 2 * q);
            return *reinterpret_cast<const float2*>(sxz + ip);
        };
        auto store = [&](int q, int i, float2 v) { Zf[i * Qp + q] = v; };
        fft_rt<kPencil, false>(k.px, tw, A, B, Qp, 1, Qp, load, store);
        float2* X1 = Zf == A ? B : A;
        float* D = reinterpret_cast<float*>(fft_out_buf(k.px, X1, Zf));  // [n][P]
        auto load_i = [&](int q, int i) -> float2 { return cmul_m(Zf[i * Qp + q], cscale(tF[i], inv_n)); };
        auto store_i = [&](int q, int i, float2 v) {
            D[i * P + 2 * q] = v.x;
            D[i * P + 2 * q + 1] = v.y;
        };
        fft_rt<kPencil, true>(k.px, tw, X1, Zf, Qp, 1, Qp, load_i, store_i);
        for (int t0 = threadIdx.x; t0 < n * P; t0 += kEpi * blockDim.x) {
            int ipu[kEpi], iu[kEpi], pu[kEpi], isu[kEpi];
            bool ok[kEpi], slab[kEpi];
            float a2[kEpi], r2[kEpi], w2[kEpi], p6[kEpi];
#pragma unroll
            for (int u = 0; u < kEpi; ++u) {
                const int t = t0 + u * blockDim.x;
                pu[u] = t % P;
                iu[u] = t / P;
                const int z = z0 + pu[u];
                ok[u] = t < n * P && iu[u] < nx - 1 && yin && z < k.nz - 1;
                ipu[u] = cell(k, iu[u], y, z);
                slab[u] = ok[u] && in_slab(iu[u], nx, pml);
                isu[u] = slab[u] ? slab_x(k, iu[u], y, z) : 0;
                a2[u] = ok[u] ? v2[ipu[u]] : 0.f;
                r2[u] = ok[u] ? R2[ipu[u]] : 0.f;
                w2[u] = ok[u] ? ri2[ipu[u]] : 0.f;
                p6[u] = slab[u] ? f6[isu[u]] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < kEpi; ++u) {
                if (!ok[u]) continue;
                const int i = iu[u], ip = ipu[u];
                float pz = D[i * P + pu[u]];
                if (slab[u]) {
                    const float q6 = p6[u] + dt * (-k.ax[i] * p6[u] - k.bx[i] * pz);
                    pz += q6;
                    f6[isu[u]] = q6;
                }
                v2[ip] = a2[u] + dt * w2[u] * (pz + r2[u]);
            }
        }
    }
}

#endif  // QVTI_PART == 0

// ------------------------------------------------------------------ k_dv --
// Compiled form of both velocity kernels.  AX = 1 (k_vy's job): the y
// derivatives of sxy (+), syy (-), syz (+) with their C-PML terms added to R.
// AX = 0 (k_vx's): the x derivatives of sxx (-), sxy (+), sxz (+), their C-PML
// terms and the velocity update (cu:1018-1101).  A block owns consecutive z of
// one line: the first blocks of a line 2 PP z of the first two fields, which
// share one complex transform (two_shift), z and z + 1 in a packed pair; the
// others 4 PP z of the third, z + 1 the imaginary part of z, two such pencils in
// a pair.
//
// The derivatives go back to the exchange for the epilogue, a loop in which
// consecutive lanes take consecutive z, two cells at a time with all their loads
// ahead of their stores.  (As straight code on the registers the inverse ends in
// the epilogue was four fifths of the kernel's instructions and 83 MB of the
// library.)  The kernels they replace ran scalar transforms at 55 % issue between
// barriers.
constexpr int dv_threads(int n, int pp) { return warps_up(pp * pair_tasks(n)); }
constexpr size_t dv_smem(int n, int pp) { return 16 * ((size_t)pp * pair_slots(n) + 2 * (size_t)n); }
// Blocks per SM the registers are sized for: a thread holds the pair's
// butterflies (4 registers a point) and the loads of the epilogue.
// Warps come in fours, one per scheduler, or a scheduler's registers are split
// more ways than the others'.
constexpr int dv_blocks(int n, int pp)
{
    const int warps = dv_threads(n, pp) / 32;
    int b = 65536 / (128 * dv_threads(n, pp));
    const int m = (int)(220 * 1024 / (dv_smem(n, pp) + 1024));
    if (m < b) b = m;
    while (b > 1 && b * warps % 4) --b;
    return b < 1 ? 1 : b;
}

// W = 2 or 4 consecutive z of a row of which `left` remain (even): 8-byte
// accesses, or one of 16 (v4: the rows are 16-byte aligned).
template <int W>
__device__ __forceinline__ void ldz(float* o, const float* p, int left, bool v4)
{
    if (W == 4 && v4) {
        const float4 a = left > 0 ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
        o[0] = a.x; o[1] = a.y; o[W - 2] = a.z; o[W - 1] = a.w;
    } else {
#pragma unroll
        for (int u = 0; u < W; u += 2) {
            const float2 a = left > u ? *reinterpret_cast<const float2*>(p + u) : make_float2(0.f, 0.f);
            o[u] = a.x; o[u + 1] = a.y;
        }
    }
}
template <int W>
__device__ __forceinline__ void stz(float* p, int left, bool v4, const float* v)
{
    if (W == 4 && v4) {
        if (left > 0) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[W - 2], v[W - 1]);
    } else {
#pragma unroll
        for (int u = 0; u < W; u += 2)
            if (left > u) *reinterpret_cast<float2*>(p + u) = make_float2(v[u], v[u + 1]);
    }
}

__device__ __forceinline__ void prefetch_line(const float* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// A velocity field's part of the epilogue: W z from z on at index i of the line;
// back: the shift is backward, the C-PML profile the half-point average.
template <int W>
struct DvCell {
    float r[W], o[W], w[W], q[W];
    int ip, is;
    bool on, slab;
};
template <int N, int AX, int W>
struct DvEpi {
    const KP& k;
    int line, base, stride;
    bool lin, v4;  // lin: cells of this line are updated (k_vx), or have C-PML terms (k_vy)
    float *R, *vel, *ph;
    const float *ri, *pa, *pb;
    __device__ __forceinline__ DvEpi(const KP& k_, int f, bool back, int line_)
        : k(k_), line(line_), v4(k_.nz % 4 == 0), R(k_.R[f]), vel(k_.v[f]), ph(k_.php[AX ? 3 * f + 1 : 3 * f]),
          ri(k_.rinv[f]), pa(AX ? (back ? k_.ayh : k_.ay) : (back ? k_.axh : k_.ax)),
          pb(AX ? (back ? k_.byh : k_.by) : (back ? k_.bxh : k_.bx))
    {
        stride = AX ? k.nz : k.ny * k.nz;
        base = AX ? line * k.ny * k.nz : line * k.nz;
        lin = AX ? line < k.nx - 1 : line < k.ny - 1;
    }
    __device__ __forceinline__ int slab_at(int i, int z) const { return AX ? slab_y(k, line, i, z) : slab_x(k, i, line, z); }
    __device__ __forceinline__ void prefetch(int i, int z) const
    {
        const int ip = base + i * stride + z;
        prefetch_line(R + ip);
        if (AX == 0) {
            prefetch_line(vel + ip);
            prefetch_line(ri + ip);
        }
        if (lin && in_slab(i, N, k.pml)) prefetch_line(ph + slab_at(i, z));
    }
    __device__ __forceinline__ void load(DvCell<W>& c, bool ok, int i, int z) const
    {
        const int left = k.nz - z;
        const bool in = lin && i < N - 1;
        c.on = ok && left > 0 && (AX || in);
        c.slab = c.on && in && in_slab(i, N, k.pml);
        c.ip = base + i * stride + z;
        c.is = c.slab ? slab_at(i, z) : 0;
        ldz<W>(c.r, R + c.ip, c.on ? left : 0, v4);
        if (AX == 0) {
            ldz<W>(c.o, vel + c.ip, c.on ? left : 0, v4);
            ldz<W>(c.w, ri + c.ip, c.on ? left : 0, v4);
        }
        ldz<W>(c.q, ph + c.is, c.slab ? left : 0, v4);
    }
    __device__ __forceinline__ void store(DvCell<W>& c, int i, int z, float* d) const
    {
        const int left = k.nz - z;
        const float dt = k.dt;
        if (!c.on) return;
        if (AX == 1) {
#pragma unroll
            for (int u = 0; u < W; ++u) c.r[u] += d[u];
        }
        if (c.slab) {
            const float a = pa[i], b = pb[i];
#pragma unroll
            for (int u = 0; u < W; ++u)
                if (u < left - 1) {  // all but the last plane
                    c.q[u] = pml_step(c.q[u], dt, a, b, d[u]);
                    (AX ? c.r : d)[u] += c.q[u];
                }
            stz<W>(ph + c.is, left, v4, c.q);
        }
        if (AX == 1) {
            stz<W>(R + c.ip, left, v4, c.r);
        } else {
#pragma unroll
            for (int u = 0; u < W; ++u)
                if (u < left - 1) c.o[u] = fmaf(dt * c.w[u], d[u] + c.r[u], c.o[u]);
            stz<W>(vel + c.ip, left, v4, c.o);
        }
    }
};

template <int N, int PP, int AX>
__global__ void __launch_bounds__(dv_threads(N, PP), dv_blocks(N, PP)) k_dv(KP k)
{
    using F = PairFFT<N, PP, true>;
    constexpr int NT = dv_threads(N, PP), R0 = F::R0;
    static_assert(NT <= 1024, "threads of a block");
    extern __shared__ float4 smem4[];
    f2* buf = reinterpret_cast<f2*>(smem4);
    float4* tw = smem4 + PP * pair_slots(N);
    float4* tf = tw + N;  // forward shift over n, doubled like the twiddles; the backward one is (-F.x, F.y)
    if (AX == 1 && blockIdx.x + blockIdx.y == 0 && threadIdx.x == 0) *k.d_it += 1;  // step counter
    const int t = threadIdx.x, nz = k.nz;
    const int line = blockIdx.y;  // x (AX = 1) or y
    const int stride = AX ? nz : k.ny * nz;
    const int base = AX ? line * k.ny * nz : line * nz;
    const int pairs = (nz + 2 * PP - 1) / (2 * PP);  // blocks of the first two fields
    int p, j;
    const bool act = F::task(t, p, j);
    c2 v[F::RM];
    auto tables = [&] {  // behind the loads in flight (read after the exchange's barrier)
        const float2* gtw = AX ? k.tw_y : k.tw_x;
        const float2* gf = AX ? k.Fy : k.Fx;
        constexpr float inv_n = 1.0f / N;
        for (int i = threadIdx.x; i < N; i += NT) {
            const float2 w = gtw[i], f = gf[i];
            tw[i] = make_float4(w.x, w.x, w.y, w.y);
            tf[i] = make_float4(f.x * inv_n, f.x * inv_n, f.y * inv_n, f.y * inv_n);
        }
        if (F::SYNC0) __syncthreads();
    };
    const TwAll<N> W{tw};
    if (blockIdx.x < pairs) {
        const int z0 = blockIdx.x * 2 * PP, z = z0 + 2 * p, left = nz - z;
        const float* sa = k.s[AX ? 3 : 0] + base + z;
        const float* sb = k.s[AX ? 1 : 3] + base + z;
        if (act)
            F::template each<0>(j, [&](int m, int i) {
#pragma unroll
                for (int r = 0; r < R0; ++r) {
                    const int at = (i + r * (N / R0)) * stride;
                    float a[2], b[2];
                    ldz<2>(a, sa + at, left, false);
                    ldz<2>(b, sb + at, left, false);
                    v[m * R0 + r] = c2{pack2(a[0], a[1]), pack2(b[0], b[1])};
                }
            });
        // k_vy: sxy forward, syy backward; k_vx: sxx backward, sxy forward
        const DvEpi<N, AX, 2> ea(k, 0, AX == 0, line), eb(k, 1, AX == 1, line);
        // the epilogue's operands start their way from HBM to L2 now
        for (int i = t; i < 2 * N; i += NT) {
            const int zp = min(z0 + (i & 1 ? 2 * PP - 1 : 0), nz - 1);
            ea.prefetch(i / 2, zp);
            eb.prefetch(i / 2, zp);
        }
        tables();
        F::template first<false>(W, buf, t, v);
        F::template finish<false>(W, buf, t, v);
        F::keep(buf, t, v);
        __syncthreads();
        if (act)
            F::template each<0>(j, [&](int m, int i0) {
#pragma unroll
                for (int r = 0; r < R0; ++r) {
                    const int i = i0 + r * (N / R0);
                    const c2 z = F::ld(buf + F::slot(p, i)), c = F::ld(buf + F::slot(p, i ? N - i : 0));
                    const float4 f = tf[i];
                    // two_shift, sgn = 1 (k_vy) or -1
                    const f2 fx = pack2(AX ? f.x : -f.x, AX ? f.x : -f.x), nx = pack2(AX ? -f.x : f.x, AX ? -f.x : f.x);
                    const f2 fy = pack2(f.z, f.z), ny = pack2(-f.z, -f.z);
                    v[m * R0 + r] = c2{fma_(fx, c.x, ny * z.y), fma_(nx, c.y, fy * z.x)};
                }
            });
        __syncthreads();
        F::template first<true>(W, buf, t, v);
        F::template finish<true>(W, buf, t, v);
        F::keep(buf, t, v);
        __syncthreads();
#pragma unroll 1
        for (int w = t; w < N * PP; w += 2 * NT) {
            DvCell<2> a[2], b[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = (unsigned)(w + u * NT) / PP, zc = z0 + 2 * ((w + u * NT) % PP);
                ea.load(a[u], i < N, i, zc);
                eb.load(b[u], i < N, i, zc);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = (unsigned)(w + u * NT) / PP, q = (w + u * NT) % PP;
                if (i >= N) break;
                const c2 d = F::ld(buf + F::slot(q, i));
                const float2 x = unpack2(d.x), y = unpack2(d.y);
                float da[2] = {x.x, x.y}, db[2] = {y.x, y.y};
                ea.store(a[u], i, z0 + 2 * q, da);
                eb.store(b[u], i, z0 + 2 * q, db);
            }
        }
    } else {
        const int z0 = (blockIdx.x - pairs) * 4 * PP, z = z0 + 4 * p, left = nz - z;
        const float* src = k.s[AX ? 5 : 4] + base + z;
        const DvEpi<N, AX, 4> e(k, 2, false, line);
        if (act)
            F::template each<0>(j, [&](int m, int i) {
#pragma unroll
                for (int r = 0; r < R0; ++r) {
                    float a[4];
                    ldz<4>(a, src + (i + r * (N / R0)) * stride, left, e.v4);
                    v[m * R0 + r] = c2{pack2(a[0], a[2]), pack2(a[1], a[3])};
                }
            });
        for (int i = t; i < 3 * N; i += NT) e.prefetch(i / 3, min(z0 + (i % 3 * (4 * PP - 1)) / 2, nz - 1));
        tables();
        F::template first<false>(W, buf, t, v);
        F::template finish<false>(W, buf, t, v);
        F::turn(buf, t, v);
        if (act)
            F::template each<0>(j, [&](int m, int i) {
#pragma unroll
                for (int r = 0; r < R0; ++r) {
                    const float4 f = tf[i + r * (N / R0)];
                    v[m * R0 + r] = cmul_m(v[m * R0 + r], pack2(f.x, f.y), pack2(f.z, f.w));
                }
            });
        __syncthreads();
        F::template first<true>(W, buf, t, v);
        F::template finish<true>(W, buf, t, v);
        F::keep(buf, t, v);
        __syncthreads();
#pragma unroll 1
        for (int w = t; w < N * PP; w += 2 * NT) {
            DvCell<4> a[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = (unsigned)(w + u * NT) / PP;
                e.load(a[u], i < N, i, z0 + 4 * ((w + u * NT) % PP));
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = (unsigned)(w + u * NT) / PP, q = (w + u * NT) % PP;
                if (i >= N) break;
                const c2 c = F::ld(buf + F::slot(q, i));
                const float2 x = unpack2(c.x), y = unpack2(c.y);
                float d[4] = {x.x, y.x, x.y, y.y};
                e.store(a[u], i, z0 + 4 * q, d);
            }
        }
    }
}

}  // namespace

QVTI_DECLARE_PARTS(bool, dv_launch, const KP& k, int ax, int P, cudaStream_t st);
QVTI_DECLARE_PARTS(bool, dv_configure, SmemLimit& lim, int ax, int n);

template <>
bool dv_launch<QVTI_PART>(const KP& k, int ax, int P, cudaStream_t st)
{
    return dispatch_len(ax ? k.ny : k.nx, [&](auto NN) {
        constexpr int N = decltype(NN)::value;
        const dim3 grid(cdiv(k.nz, P) + cdiv(k.nz, 2 * P), ax ? k.nx : k.ny);
        auto go = [&](auto AX) {
            constexpr int ax_ = decltype(AX)::value;
            const size_t sm = dv_smem(N, P / 2);
            if (P == 16) k_dv<N, 8, ax_><<<grid, dv_threads(N, 8), sm, st>>>(k);
            else k_dv<N, 16, ax_><<<grid, dv_threads(N, 16), sm, st>>>(k);
        };
        if (ax) {
            go(IntC<1>{});
        } else {
            if constexpr (N >= kMinLong) go(IntC<0>{});
        }
    });
}
template <>
bool dv_configure<QVTI_PART>(SmemLimit& lim, int ax, int n)
{
    return dispatch_len(n, [&](auto NN) {
        constexpr int N = decltype(NN)::value;
        auto set = [&](auto AX) {
            constexpr int ax_ = decltype(AX)::value;
            lim.set((const void*)k_dv<N, 8, ax_>);
            lim.set((const void*)k_dv<N, 16, ax_>);
        };
        if (ax) {
            set(IntC<1>{});
        } else {
            if constexpr (N >= kMinLong) set(IntC<0>{});
        }
    });
}

#if QVTI_PART == 0
// rt: the runtime kernels' layout.
size_t smem_vyx(int n, int P, bool rt) { return rt ? sizeof(float2) * (2 * n + 2 * (n + n / 16) * P) : dv_smem(n, P / 2); }

void launch_vy(const KP& k, int P, bool rt, cudaStream_t st)
{
    if (rt) k_vy<<<dim3(cdiv(k.nz, P), k.nx, 2), rt_threads(k.py, P), smem_vyx(k.ny, P, true), st>>>(k, P);
    else (void)QVTI_CALL_PARTS(dv_launch, k, 1, P, st);
}
void launch_vx(const KP& k, int P, bool rt, cudaStream_t st)
{
    if (rt) k_vx<<<dim3(cdiv(k.nz, P), k.ny, 2), rt_threads(k.px, P), smem_vyx(k.nx, P, true), st>>>(k, P);
    else (void)QVTI_CALL_PARTS(dv_launch, k, 0, P, st);
}

cudaError_t configure_velocity(int axis, int n)
{
    SmemLimit lim;
    if (axis < 0) {
        lim.set((const void*)k_vy);
        lim.set((const void*)k_vx);
    } else if (axis < 2) {
        (void)QVTI_CALL_PARTS(dv_configure, lim, axis, n);
    }
    return lim.e;
}
#endif  // QVTI_PART == 0

}  // namespace qvti
