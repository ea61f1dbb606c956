// qvti_q_derivative_noalloc: one constant-Q derivative field for callers that
// cannot allocate device memory.
//
// Some callers own every byte of device memory through their own budget --
// a serving process whose footprint is fixed at start-up, a host framework
// that hands libraries pre-planned buffers from its own pool, or a latency-
// critical loop that cannot absorb the implicit device-wide synchronisation
// of cudaMalloc/cudaFree.  They cannot use qvti_q_derivative, which allocates
// device copies of its host arrays and a simulation's spectra as scratch.
// This variant takes device pointers for the input and output and keeps its
// scratch (the half spectrum) in a file-scope __device__ array of a fixed
// maximum size, so a call allocates nothing; its 1D tables are built in shared
// memory where they are used.
#include <algorithm>
#include <cstdio>
#include <mutex>

#include "engine.cuh"
#include "../../include/qvti.h"

namespace qvti {
namespace {

// Largest half spectrum (nz/2 + 1) * nx * ny the static scratch holds:
// 2^19 complex values = 4 MiB (e.g. 96^3, 64 x 64 x 128, 128 x 128 x 60).
constexpr long long kNoAllocSpectrum = 1ll << 19;
constexpr int kNoAllocAxis = 1024;  // longest axis

// Held by every GPU that loads the library, until the process exits.
static __device__ __align__(256) float2 g_na_scratch[kNoAllocSpectrum];
// Device address of the array above, looked up once per device with that
// device current (a host-side use of the array name would not be a device
// address), and the device's SM count.
struct NoAllocDev {
    bool ready = false;
    float2* scratch = nullptr;
    int sms = 0;
};
NoAllocDev g_na_dev[kMaxDevices];
std::mutex g_na_mu;

// ------------------------------------------------------------------ k_qd --
// The derivative in five launches, one per pass: z forward (R2C), y forward, x
// forward - multiplier - x inverse, y inverse, z inverse (C2R).  The fields are
// small (at most 4 MiB of spectrum, resident in L2), so as eight launches --
// three table builds and five passes -- a call was launch gaps and ramp-up: 49
// us at 32 x 48 x 40, 78 us at 96^3 (now 31 and 41).  A pass takes tiles of P
// pencils, block after block; the twiddles of its axis are built in FP64 in
// shared memory.  One kernel takes the pass as an argument: five kernels fetched
// their instructions anew at every launch (16^3 28.6 against 22.9 us, 96^3 49.2
// against 41.4).  The launches are programmatically dependent: the next pass is
// launched as the blocks before it end (with plain launches, 16^3 34.9 against
// 28.6 us); releasing it earlier takes shared memory from the running one (96^3
// 53.5 against 49.2).  Nothing needs its blocks on the GPU all at once, so the
// call runs in a context that owns a few SMs and beside kernels that hold the
// others; one cooperative launch with grid barriers between the passes needed
// them all, and took 22.6 and 43.0 us.
struct QdArgs {
    const float* in;
    float* out;
    float2* H;  // [kz][x][y]
    FftPlan pl[3];
    int n[3], nkz;
    float h[3];
    float inv_ntp;
    int axis, fwd, pw;
    int P;  // pencils per tile
};
constexpr int kQdThreads = 128;

template <bool INV>
__device__ __noinline__ void qd_lines(const FftPlan& pl, const float2* tw, float2* X, float2* A, float2* B, int P)
{
    const int ps = pl.n + pl.n / 16;
    auto load = [&](int p, int i) -> float2 { return X[p * ps + i + (i >> 4)]; };
    auto store = [&](int p, int i, float2 v) { X[p * ps + i + (i >> 4)] = v; };
    fft_run<false, INV>(pl, tw, A, B, P, ps, 1, load, store, 4);
}

// |k| of an index, the staggered shift multiplier (see k_axis_tables).
__device__ __forceinline__ float qd_kmag(int i, int n, float h)
{
    const int m = i <= n / 2 ? i : n - i;
    return (float)(2.0 * 3.1415926 / n / (double)h * m);
}
__device__ __forceinline__ float2 qd_shift(int i, int n, float h, int fwd)
{
    const double pi_ref = 3.1415926;
    const int m = i <= n / 2 ? i : n - i;
    const double t = 2.0 * pi_ref / n / (double)h * m, sn = sin(m * pi_ref / n), cs = cos(m * pi_ref / n);
    return make_float2((float)(fwd ? -t * sn : t * sn), 2 * i == n ? 0.f : (float)(i <= n / 2 ? t * cs : -t * cs));
}

__global__ void __launch_bounds__(kQdThreads) k_qd(const __grid_constant__ QdArgs a, int pass)
{
    extern __shared__ float4 smem4[];
    float2* sm = reinterpret_cast<float2*>(smem4);
    const int nx = a.n[0], ny = a.n[1], nz = a.n[2], P = a.P, t = threadIdx.x;
    float2 *tw = sm, *X, *A, *B;
    auto layout = [&](int ax) {
        const int n = a.n[ax], ps = n + n / 16;
        X = tw + n;
        A = X + P * ps;
        B = A + P * ps;  // used (and counted in the launch) only with more than two stages
        for (int i = t; i < n; i += kQdThreads) {
            double s, c;
            sincospi(-2.0 * i / n, &s, &c);
            tw[i] = make_float2((float)c, (float)s);
        }
        return ps;
    };
    auto ready = [] {  // the tables, and what the passes before this one wrote
        asm volatile("griddepcontrol.wait;" ::: "memory");
        __syncthreads();
    };
    // z forward: pencil q of a tile = rows (2q, 2q + 1) of the flattened (x, y)
    if (pass == 0) {
        const int ps = layout(2), npair = nx * ny / 2, tiles = (npair + P - 1) / P;
        ready();
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            const int q0 = tile * P, qn = min(P, npair - q0);
            for (int w = t; w < P * nz; w += kQdThreads) {
                const int q = w / nz, i = w - q * nz;
                const float* r = a.in + (long long)(q0 + q) * 2 * nz + i;
                X[q * ps + i + (i >> 4)] = q < qn ? make_float2(r[0], r[nz]) : make_float2(0.f, 0.f);
            }
            __syncthreads();
            qd_lines<false>(a.pl[2], tw, X, A, B, P);
            for (int w = t; w < P * a.nkz; w += kQdThreads) {
                const int q = w % P, kz = w / P, im = kz ? nz - kz : 0;
                if (q >= qn) continue;
                const float2 z = X[q * ps + kz + (kz >> 4)], zm = cconj(X[q * ps + im + (im >> 4)]);
                const float2 u = unpack_a(z, zm), v = unpack_b(z, zm);
                reinterpret_cast<float4*>(a.H + (long long)kz * nx * ny)[q0 + q] = make_float4(u.x, u.y, v.x, v.y);
            }
            __syncthreads();
        }
    }
    // a y pass over the contiguous lines (kz, x)
    if (pass == 1 || pass == 3) {
        const int ps = layout(1), lines = a.nkz * nx, tiles = (lines + P - 1) / P;
        ready();
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            const int l0 = tile * P, ln = min(P, lines - l0);
            float2* H = a.H + (long long)l0 * ny;
            for (int w = t; w < P * ny; w += kQdThreads) {
                const int p = w / ny, i = w - p * ny;
                X[p * ps + i + (i >> 4)] = p < ln ? H[w] : make_float2(0.f, 0.f);
            }
            __syncthreads();
            if (pass == 3) qd_lines<true>(a.pl[1], tw, X, A, B, P);
            else qd_lines<false>(a.pl[1], tw, X, A, B, P);
            for (int w = t; w < ln * ny; w += kQdThreads) {
                const int p = w / ny, i = w - p * ny;
                H[w] = X[p * ps + i + (i >> 4)];
            }
            __syncthreads();
        }
    }
    // x forward, |k|^pw T(k_axis) / ntp, x inverse: P consecutive y of one kz
    if (pass == 2) {
        const int ps = layout(0), chunks = (ny + P - 1) / P, tiles = chunks * a.nkz;
        float2* tT = B + (a.pl[0].q.nst > 2 ? P * ps : 0);  // the shift over the axis it varies on
        float* tk = reinterpret_cast<float*>(tT + max(nx, P));
        float* tky = tk + nx;
        for (int i = t; i < nx; i += kQdThreads) {
            const float kx = qd_kmag(i, nx, a.h[0]);
            tk[i] = kx * kx;
            if (a.axis == 0) tT[i] = cscale(qd_shift(i, nx, a.h[0], a.fwd), a.inv_ntp);
        }
        ready();
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            const int kz = tile / chunks, y0 = (tile - kz * chunks) * P, yn = min(P, ny - y0);
            float2* H = a.H + (long long)kz * nx * ny + y0;
            if (t < yn) {
                const float ky = qd_kmag(y0 + t, ny, a.h[1]), kk = qd_kmag(kz, nz, a.h[2]);
                tky[t] = ky * ky + kk * kk;
                if (a.axis == 1) tT[t] = cscale(qd_shift(y0 + t, ny, a.h[1], a.fwd), a.inv_ntp);
                else if (a.axis == 2) tT[t] = cscale(qd_shift(kz, nz, a.h[2], a.fwd), a.inv_ntp);
            }
            for (int w = t; w < P * nx; w += kQdThreads) {
                const int p = w % P, i = w / P;
                X[p * ps + i + (i >> 4)] = p < yn ? H[(long long)i * ny + p] : make_float2(0.f, 0.f);
            }
            __syncthreads();
            qd_lines<false>(a.pl[0], tw, X, A, B, P);
            for (int w = t; w < yn * nx; w += kQdThreads) {
                const int p = w / nx, i = w - p * nx;
                const float k2 = fmaxf(tk[i] + tky[p], 1e-10f);  // the reference sets |k|^2 = 1e-10 at DC (cu:74)
                const float ap = a.pw == 0 ? 1.0f : (a.pw < 0 ? 1.0f / sqrtf(k2) : sqrtf(k2));
                float2* x = X + p * ps + i + (i >> 4);
                *x = cmul(*x, cscale(tT[a.axis == 0 ? i : p], ap));
            }
            __syncthreads();
            qd_lines<true>(a.pl[0], tw, X, A, B, P);
            for (int w = t; w < P * nx; w += kQdThreads) {
                const int p = w % P, i = w / P;
                if (p < yn) H[(long long)i * ny + p] = X[p * ps + i + (i >> 4)];
            }
            __syncthreads();
        }
    }
    // z inverse (C2R)
    if (pass == 4) {
        const int ps = layout(2), npair = nx * ny / 2, tiles = (npair + P - 1) / P;
        ready();
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            const int q0 = tile * P, qn = min(P, npair - q0);
            for (int w = t; w < P * a.nkz; w += kQdThreads) {
                const int q = w % P, kz = w / P;
                if (q >= qn) continue;
                const float4 g = reinterpret_cast<const float4*>(a.H + (long long)kz * nx * ny)[q0 + q];
                float2 u = make_float2(g.x, g.y), v = make_float2(g.z, g.w);
                const bool edge = kz == 0 || 2 * kz == nz;  // imaginary parts dropped like a C2R
                if (edge) u.y = v.y = 0.f;
                X[q * ps + kz + (kz >> 4)] = make_float2(u.x - v.y, u.y + v.x);
                const int im = nz - kz;
                if (!edge) X[q * ps + im + (im >> 4)] = make_float2(u.x + v.y, v.x - u.y);
            }
            __syncthreads();
            qd_lines<true>(a.pl[2], tw, X, A, B, P);
            for (int w = t; w < qn * nz; w += kQdThreads) {
                const int q = w / nz, i = w - q * nz;
                const float2 z = X[q * ps + i + (i >> 4)];
                float* r = a.out + (long long)(q0 + q) * 2 * nz + i;
                r[0] = z.x;
                r[nz] = z.y;
            }
            __syncthreads();
        }
    }
}

size_t qd_smem(const QdArgs& a, int P)
{
    size_t m = 0;
    for (int ax = 0; ax < 3; ++ax) {
        const size_t n = a.n[ax], ps = n + n / 16, nb = a.pl[ax].q.nst > 2 ? 3 : 2;
        size_t b = sizeof(float2) * (n + nb * P * ps);
        if (ax == 0) b += sizeof(float2) * std::max<size_t>(n, P) + sizeof(float) * (n + P);
        m = std::max(m, b);
    }
    return m;
}

int setup_device(int dev, NoAllocDev** out)
{
    if (dev < 0 || dev >= kMaxDevices) return QVTI_ERR_ARG;
    std::lock_guard<std::mutex> lk(g_na_mu);
    NoAllocDev& d = g_na_dev[dev];
    if (!d.ready) {
        cudaError_t e = cudaGetSymbolAddress((void**)&d.scratch, g_na_scratch);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_qd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
        if (e != cudaSuccess) {
            fprintf(stderr, "qvti_q_derivative_noalloc: set-up: %s\n", cudaGetErrorString(e));
            return QVTI_ERR_CUDA;
        }
        d.ready = true;
    }
    *out = &d;
    return QVTI_OK;
}

bool smooth_even(int n)
{
    if (n < 16 || n > kNoAllocAxis || (n & 1)) return false;
    int m = n;
    for (int r : {2, 3, 5, 7})
        while (m % r == 0) m /= r;
    return m == 1;
}

}  // namespace
}  // namespace qvti

extern "C" int qvti_q_derivative_noalloc(const float* d_in, float* d_out, int ntx, int nty, int ntz, float dx,
                                         float dy, float dz, int axis, int fwd, int power, void* stream)
{
    using namespace qvti;
    if (!d_in || !d_out || axis < 0 || axis > 2 || power < -1 || power > 1 || !(dx > 0 && dy > 0 && dz > 0))
        return fail(QVTI_ERR_ARG);
    if (!smooth_even(ntx) || !smooth_even(nty) || !smooth_even(ntz)) return fail(QVTI_ERR_UNSUPPORTED);
    const long long nkz = ntz / 2 + 1;
    if (nkz * ntx * nty > kNoAllocSpectrum) {
        fprintf(stderr,
                "qvti_q_derivative_noalloc: grid %dx%dx%d needs %lld spectrum values, the static scratch holds %lld\n",
                ntx, nty, ntz, nkz * ntx * nty, kNoAllocSpectrum);
        return fail(QVTI_ERR_UNSUPPORTED);
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return fail(QVTI_ERR_CUDA);
    NoAllocDev* d = nullptr;
    int rc = setup_device(dev, &d);
    if (rc) return fail(rc);

    QdArgs a{};
    a.in = d_in;
    a.out = d_out;
    a.H = d->scratch;  // every pass overwrites what it reads: nothing needs clearing
    const int n[3] = {ntx, nty, ntz};
    const float h[3] = {dx, dy, dz};
    for (int i = 0; i < 3; ++i) {
        a.n[i] = n[i];
        a.h[i] = h[i];
        if (!make_fft_plan(n[i], &a.pl[i])) return fail(QVTI_ERR_UNSUPPORTED);
    }
    a.nkz = (int)nkz;
    a.inv_ntp = (float)(1.0 / ((double)ntx * nty * ntz));
    a.axis = axis;
    a.fwd = fwd;
    a.pw = power;
    // tiles of 8 pencils; of 4 where the passes have few, so more SMs get one
    // (20 x 28 x 150: 37 against 44 us; 64 x 64 x 128: 47 against 37), or where
    // the longest axis leaves no room for 8
    const long long pencils = (long long)ntx * nty / 2 + nkz * ntx + nkz * nty;
    a.P = pencils < 64ll * d->sms || qd_smem(a, 8) > kMaxSmem ? 4 : 8;
    const size_t sm = qd_smem(a, a.P);
    const long long pairs = (long long)ntx * nty / 2, chunks = nkz * ((nty + a.P - 1) / a.P);
    const long long tiles[5] = {(pairs + a.P - 1) / a.P, (nkz * ntx + a.P - 1) / a.P, chunks, (nkz * ntx + a.P - 1) / a.P,
                                (pairs + a.P - 1) / a.P};
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    for (int p = 0; p < 5; ++p) {
        cudaLaunchConfig_t c{};
        c.gridDim = dim3((unsigned)std::min<long long>(tiles[p], 4ll * d->sms));
        c.blockDim = dim3(kQdThreads);
        c.dynamicSmemBytes = sm;
        c.stream = static_cast<cudaStream_t>(stream);
        c.attrs = &at;
        c.numAttrs = p ? 1 : 0;  // the first pass waits for what the caller queued
        if (cudaLaunchKernelEx(&c, k_qd, a, p) != cudaSuccess) break;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        fprintf(stderr, "qvti_q_derivative_noalloc: launch: %s\n", cudaGetErrorString(e));
        return fail(QVTI_ERR_CUDA);
    }
    return QVTI_OK;
}
