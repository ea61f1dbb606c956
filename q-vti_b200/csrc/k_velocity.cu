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
        auto load_i = [&](int q, int i) -> float2 { return cmul(Zf[i * Qp + q], cscale(tF[i], inv_n)); };
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
        auto load_i = [&](int q, int i) -> float2 { return cmul(Zf[i * Qp + q], cscale(tF[i], inv_n)); };
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
// terms and the velocity update (cu:1018-1101).  A block owns 16 consecutive z
// of one line and takes the three fields one after another.
//
// Four consecutive z of a field are two complex pencils, (z + 2) i added to z
// and (z + 3) i to z + 1: one multiplier serves all, a 16-byte load IS the
// packed pair, and what the inverse's last stage leaves in a thread is four
// consecutive z of the derivative, so the epilogue reads and writes the other
// arrays 16 bytes at a time straight from registers.  Per field: two exchanges
// through shared memory (forward and inverse, reversed radices: nothing is
// exchanged at the multiplication).  The kernels they replace kept every
// derivative in shared memory for a scalar epilogue and ran at 55 % issue
// between barriers.
constexpr int dv_threads(int n, int pp) { return warps_up(pp * pair_tasks(n)); }
constexpr size_t dv_smem(int n, int pp) { return 16 * ((size_t)pp * pair_slots(n) + 2 * (size_t)n); }
// Blocks per SM the registers are sized for: a thread holds the pair's
// butterfly (4 registers a point) and the loads of the epilogue.
// Warps come in fours, one per scheduler, or a scheduler's registers are split
// more ways than the others'.
constexpr int dv_blocks(int n, int pp)
{
    const int warps = dv_threads(n, pp) / 32, regs = pair_rmax(n) >= 10 ? 128 : 96;
    int b = 65536 / (regs * dv_threads(n, pp));
    const int m = (int)(220 * 1024 / (dv_smem(n, pp) + 1024));
    if (m < b) b = m;
    while (b > 1 && b * warps % 4) --b;
    return b < 1 ? 1 : b;
}

template <bool V4>
__device__ __forceinline__ float4 ld4(const float* p, int left)  // `left` values of the row remain (even)
{
    if constexpr (V4) return left > 0 ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float2 a = left > 0 ? *reinterpret_cast<const float2*>(p) : make_float2(0.f, 0.f);
    const float2 b = left > 2 ? *reinterpret_cast<const float2*>(p + 2) : make_float2(0.f, 0.f);
    return make_float4(a.x, a.y, b.x, b.y);
}
template <bool V4>
__device__ __forceinline__ void st4(float* p, int left, float4 v)
{
    if constexpr (V4) {
        if (left > 0) *reinterpret_cast<float4*>(p) = v;
    } else {
        if (left > 0) *reinterpret_cast<float2*>(p) = make_float2(v.x, v.y);
        if (left > 2) *reinterpret_cast<float2*>(p + 2) = make_float2(v.z, v.w);
    }
}

__device__ __forceinline__ void prefetch_line(const float* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

template <int N, int PP, int AX, bool V4>
__global__ void __launch_bounds__(dv_threads(N, PP), dv_blocks(N, PP)) k_dv(KP k)
{
    using F = PairFFT<N, PP, true, false>;
    using I = PairFFT<N, PP, true, true>;
    constexpr int NT = dv_threads(N, PP), RM = pair_rmax(N), RL = F::RL, R0 = F::R0;
    extern __shared__ float4 smem4[];
    f2* buf = reinterpret_cast<f2*>(smem4);
    float4* tw = smem4 + PP * pair_slots(N);
    float4* tf = tw + N;  // forward shift over n, doubled like the twiddles; the backward one is (-F.x, F.y)
    if (AX == 1 && blockIdx.x + blockIdx.y + blockIdx.z == 0 && threadIdx.x == 0) *k.d_it += 1;  // step counter
    const int t = threadIdx.x, nz = k.nz, pml = k.pml;
    const int line = blockIdx.y;  // x (AX = 1) or y
    const int stride = AX ? nz : k.ny * nz;
    const float dt = k.dt;
    // cells of this line are updated (k_vx), or have C-PML terms (k_vy)
    const bool lin = AX ? line < k.nx - 1 : line < k.ny - 1;
    const float* pa = AX ? k.ay : k.ax;
    const float* pb = AX ? k.by : k.bx;
    const float* pah = AX ? k.ayh : k.axh;
    const float* pbh = AX ? k.byh : k.bxh;
    int p0, j0, pl, jl, pe, je;
    const bool act0 = F::template task<0>(t, p0, j0);
    const bool actl = F::template task<F::NST - 1>(t, pl, jl);
    const bool acte = I::template task<I::NST - 1>(t, pe, je);
    const int zl = blockIdx.x * (4 * PP) + 4 * p0, ze = blockIdx.x * (4 * PP) + 4 * pe;
    const int f = blockIdx.z;
    {
        // the field, its target, and the one with the backward shift (whose
        // C-PML profile is the half-point average)
        const float* src = k.s[AX ? (f == 0 ? 3 : f == 1 ? 1 : 5) : (f == 0 ? 0 : f == 1 ? 3 : 4)];
        const bool back = f == (AX ? 1 : 0);
        c2 v[RM];
        if (act0) {
            const int b0 = (AX ? line * k.ny * nz : line * nz) + j0 * stride + zl;
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const float4 a = ld4<V4>(src + b0 + r * (N / R0) * stride, nz - zl);
                v[r] = c2{pack2(a.x, a.y), pack2(a.z, a.w)};
            }
        }
        float* __restrict__ ph = k.php[AX ? 3 * f + 1 : 3 * f];
        float* __restrict__ R = k.R[f];
        float* __restrict__ vel = k.v[f];
        const float* __restrict__ ri = k.rinv[f];
        const int left = nz - ze;
        const int be = (AX ? line * k.ny * nz : line * nz) + ze;
        // the epilogue's operands start their way from HBM to L2 now
        if (acte && left > 0) {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const int i = je + r * (N / R0), ip = be + i * stride;
                prefetch_line(R + ip);
                if (AX == 0) {
                    prefetch_line(vel + ip);
                    prefetch_line(ri + ip);
                }
                if (lin && in_slab(i, N, pml)) prefetch_line(ph + (AX ? slab_y(k, line, i, ze) : slab_x(k, i, line, ze)));
            }
        }
        {  // tables, behind the loads in flight (read after the exchange's barrier)
            const float2* gtw = AX ? k.tw_y : k.tw_x;
            const float2* gf = AX ? k.Fy : k.Fx;
            constexpr float inv_n = 1.0f / N;
            for (int i = threadIdx.x; i < N; i += NT) {
                const float2 w = gtw[i], f = gf[i];
                tw[i] = make_float4(w.x, w.x, w.y, w.y);
                tf[i] = make_float4(f.x * inv_n, f.x * inv_n, f.y * inv_n, f.y * inv_n);
            }
        }
        F::template first<false>(buf, t, v);
        F::template finish<false>(TwAll<N>{tw}, buf, t, v);
        if (actl) {
#pragma unroll
            for (int r = 0; r < RL; ++r) {
                const float4 m = tf[jl + r * (N / RL)];
                f2 mx = pack2(m.x, m.y);
                const f2 my = pack2(m.z, m.w);
                if (back) mx = neg_(mx);
                v[r] = cmul_tw<false>(v[r], mx, my);
            }
        }
        __syncthreads();
        I::template first<true>(buf, t, v);
        I::template finish<true>(TwAll<N>{tw}, buf, t, v);
        if (!acte || left <= 0) return;
#pragma unroll
        for (int r = 0; r < R0; ++r) {
            const int i = je + r * (N / R0);
            const int ip = be + i * stride;
            const bool in = lin && i < N - 1;
            if (AX == 0 && !in) continue;
            const float2 dx = unpack2(v[r].x), dy = unpack2(v[r].y);
            float d[4] = {dx.x, dx.y, dy.x, dy.y};
            const float4 rr = ld4<V4>(R + ip, left);
            float4 vv, wi;
            if (AX == 0) {
                vv = ld4<V4>(vel + ip, left);
                wi = ld4<V4>(ri + ip, left);
            }
            if (in && in_slab(i, N, pml)) {
                const int is = (AX ? slab_y(k, line, i, ze) : slab_x(k, i, line, ze));
                const float a = back ? pah[i] : pa[i], b = back ? pbh[i] : pb[i];
                const float4 o = ld4<V4>(ph + is, left);
                float q[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (u < left - 1) {  // all but the last plane
                        q[u] = q[u] + dt * (-a * q[u] - b * d[u]);
                        d[u] += q[u];
                    }
                st4<V4>(ph + is, left, make_float4(q[0], q[1], q[2], q[3]));
            }
            if (AX == 1) {
                st4<V4>(R + ip, left, make_float4(rr.x + d[0], rr.y + d[1], rr.z + d[2], rr.w + d[3]));
            } else {
                const float o[4] = {vv.x, vv.y, vv.z, vv.w}, w[4] = {wi.x, wi.y, wi.z, wi.w}, q[4] = {rr.x, rr.y, rr.z, rr.w};
                float n[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) n[u] = u < left - 1 ? o[u] + dt * w[u] * (d[u] + q[u]) : o[u];
                st4<V4>(vel + ip, left, make_float4(n[0], n[1], n[2], n[3]));
            }
        }
    }
}

}  // namespace

QVTI_DECLARE_PARTS(bool, dv_launch, const KP& k, int ax, int P, cudaStream_t st);
QVTI_DECLARE_PARTS(bool, dv_configure, SmemLimit& lim);

template <>
bool dv_launch<QVTI_PART>(const KP& k, int ax, int P, cudaStream_t st)
{
    return dispatch_len(ax ? k.ny : k.nx, [&](auto NN) {
        constexpr int N = decltype(NN)::value;
        const dim3 grid(cdiv(k.nz, P), ax ? k.nx : k.ny, 3);
        auto go = [&](auto AX) {
            constexpr int ax_ = decltype(AX)::value;
            const size_t sm = dv_smem(N, P / 4);
            if (k.nz % 4) k_dv<N, 8, ax_, false><<<grid, dv_threads(N, 8), sm, st>>>(k);  // rows only 8-byte aligned
            else if (P == 16) k_dv<N, 4, ax_, true><<<grid, dv_threads(N, 4), sm, st>>>(k);
            else k_dv<N, 8, ax_, true><<<grid, dv_threads(N, 8), sm, st>>>(k);
        };
        if (ax) {
            go(IntC<1>{});
        } else {
            if constexpr (N >= kMinLong) go(IntC<0>{});
        }
    });
}
template <>
bool dv_configure<QVTI_PART>(SmemLimit& lim)
{
    for (int n : kMyLengths)
        dispatch_len(n, [&](auto NN) {
            constexpr int N = decltype(NN)::value;
            lim.set((const void*)k_dv<N, 8, 1, true>);
            lim.set((const void*)k_dv<N, 4, 1, true>);
            lim.set((const void*)k_dv<N, 8, 1, false>);
            if constexpr (N >= kMinLong) {
                lim.set((const void*)k_dv<N, 8, 0, true>);
                lim.set((const void*)k_dv<N, 4, 0, true>);
                lim.set((const void*)k_dv<N, 8, 0, false>);
            }
        });
    return false;
}

#if QVTI_PART == 0
// rt: the runtime kernels' layout.
size_t smem_vyx(int n, int P, bool rt) { return rt ? sizeof(float2) * (2 * n + 2 * (n + n / 16) * P) : dv_smem(n, P / 4); }

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

cudaError_t configure_velocity()
{
    SmemLimit lim;
    lim.set((const void*)k_vy);
    lim.set((const void*)k_vx);
    (void)QVTI_CALL_PARTS(dv_configure, lim);
    return lim.e;
}
#endif  // QVTI_PART == 0

}  // namespace qvti
