// Spectral passes of the time step: z transforms of the velocities, y lines,
// and the k-space x pass with the constant-Q operators.
#include "fft_pair.cuh"
#include "step_common.cuh"

namespace qvti {

namespace {

#if QVTI_PART == 0
// Derivative bookkeeping for the 9 stress-side derivatives d (G index
// o = 3 d + j): component, axis, forward(1)/backward(0) staggered shift.
// d: 0 dx vx, 1 dy vy, 2 dz vz (forward shift, kvx_x kvy_y kvz_z),
//    3 dz vx, 4 dx vz, 5 dy vx, 6 dx vy, 7 dz vy, 8 dy vz (backward shift)
// -- the table assignment of cuviscoelas_3D.cu:1342-1562.
__constant__ int c_comp[9] = {0, 1, 2, 0, 2, 0, 1, 1, 2};
__constant__ int c_axis[9] = {0, 1, 2, 2, 0, 1, 0, 2, 1};
__constant__ int c_fwd[9] = {1, 1, 1, 0, 0, 0, 0, 0, 0};
#endif
// G indices that go through the x and y passes (all but kGz)
__constant__ int c_gxy[kNumGxy] = {0, 1, 2, 3, 5, 6, 8, 9, 11, 12, 13, 14, 15, 17, 18, 19, 20, 21, 23, 24, 26};

#if QVTI_PART == 0
// ------------------------------------------------------------------ k_fz --
// The runtime-length kernel (k_fp below is the compiled form).
// R2C along z of vx, vy, vz.  Tile: one x, P consecutive y rows (P even);
// rows (2q, 2q+1) share one complex transform.  Output H[f][kz][x][y].
__global__ void __launch_bounds__(kThreads) k_fz(KP k, int P)
{
    extern __shared__ float4 smem4[];
    float2* sm = reinterpret_cast<float2*>(smem4);
    const int n = k.nz, Qp = P / 2, ps = n + n / 16;
    float2* tw = sm;
    float2* A = tw + n;
    float2* B = A + Qp * ps;
    load_table(tw, k.tw_z, n);
    __syncthreads();
    const int f = blockIdx.z, x = blockIdx.y, y0 = blockIdx.x * P;
    const int yv = min(P, k.ny - y0);  // rows of the tile inside the grid (even)
    const float* src = k.v[f];
    float2* Z = fft_out_buf(k.pz, A, B);
    auto load = [&](int q, int i) -> float2 {
        if (2 * q >= yv) return make_float2(0.f, 0.f);
        const int b = cell(k, x, y0 + 2 * q, i);
        return make_float2(src[b], src[b + n]);
    };
    auto store = [&](int q, int i, float2 v) { Z[q * ps + i] = v; };
    fft_rt<kLinePad, false>(k.pz, tw, A, B, Qp, ps, 1, load, store);
    float2* H = k.H[f];
    for (int t = threadIdx.x; t < k.nkz * P; t += blockDim.x) {
        const int p = t % P, kz = t / P, q = p >> 1;
        if (p >= yv) continue;
        const float2 z = Z[q * ps + kz];
        const float2 zm = cconj(Z[q * ps + (kz ? n - kz : 0)]);
        H[spec(k, kz, x, y0 + p)] = (p & 1) ? unpack_b(z, zm) : unpack_a(z, zm);
    }
}
#endif  // QVTI_PART == 0

// ------------------------------------------------------------------ k_fp --
// Compiled form of k_fz: 16 rows as four packed pairs, rows 0 + i 1 and 2 + i 3
// of a quad in each (fft_pair.cuh), the four quads of a butterfly on
// neighbouring lanes; the unpacking reads the planes pair-fastest, so four
// lanes write one 128-byte line of the spectrum.
constexpr int kFpPairs = 4;
constexpr int fp_threads(int n) { return warps_up(kFpPairs * pair_tasks(n)); }
constexpr size_t fp_smem(int n) { return 16 * ((size_t)kFpPairs * pair_slots_q(n, kFpPairs) + tw_rows_size(n)); }
constexpr int fp_blocks(int n)
{
    const int warps = fp_threads(n) / 32;
    int b = 65536 / (128 * fp_threads(n));
    while (b > 1 && b * warps % 4) --b;
    return b < 1 ? 1 : b;
}

template <int N>
__global__ void __launch_bounds__(fp_threads(N), fp_blocks(N)) k_fp(KP k)
{
    using F = PairFFT<N, kFpPairs, false, kFpPairs>;
    constexpr int NT = fp_threads(N), R0 = F::R0;
    extern __shared__ float4 smem4[];
    f2* buf = reinterpret_cast<f2*>(smem4);
    float4* tw = smem4 + F::PLANE;
    const int t = threadIdx.x, x = blockIdx.y, y0 = blockIdx.x * 4 * kFpPairs;
    c2 v[F::RM];
    int p, j;
    if (F::task(t, p, j)) {
        const int left = k.ny - y0 - 4 * p;  // rows of the quad inside the grid: 4 or more, 2, none
        const float* s = k.v[blockIdx.z] + cell(k, x, y0 + 4 * p, 0);
        F::template each<0>(j, [&](int m, int i) {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const float* a = s + i + r * (N / R0);
                const bool r01 = left > 0, r23 = left > 2;
                v[m * R0 + r] = c2{pack2(r01 ? a[0] : 0.f, r23 ? a[2 * N] : 0.f), pack2(r01 ? a[N] : 0.f, r23 ? a[3 * N] : 0.f)};
            }
        });
    }
    TwRows<N>::template fill<NT>(tw, k.tw_z);
    if (F::SYNC0) __syncthreads();
    F::template first<false>(TwRows<N>{tw}, buf, t, v);
    F::template finish<false>(TwRows<N>{tw}, buf, t, v);
    F::keep(buf, t, v);
    __syncthreads();
    float2* H = k.H[blockIdx.z];
    const f2 half = pack2(0.5f, 0.5f);
    for (int w = t; w < kFpPairs * (N / 2 + 1); w += NT) {
        const int q = w % kFpPairs, kz = (unsigned)w / kFpPairs, y = y0 + 4 * q;
        if (y >= k.ny) continue;
        const c2 z = F::ld(buf + F::slot(q, kz)), m = F::ld(buf + F::slot(q, kz ? N - kz : 0));
        // rows 0, 2: (Z + conj Z(-k)) / 2; rows 1, 3: (Z - conj Z(-k)) / 2i
        const float2 ar = unpack2((z.x + m.x) * half), ai = unpack2((z.y - m.y) * half);
        const float2 br = unpack2((z.y + m.y) * half), bi = unpack2((m.x - z.x) * half);
        float4* to = reinterpret_cast<float4*>(H + spec(k, kz, x, y));
        to[0] = make_float4(ar.x, ai.x, br.x, bi.x);
        if (y + 2 < k.ny) to[1] = make_float4(ar.y, ai.y, br.y, bi.y);
    }
}

#if QVTI_PART == 0
// ------------------------------------------------------------------ k_cy --
// The runtime-length kernel (k_cp below is the compiled form).
// C2C along y, in place, on L contiguous y lines per block (lines (kz, x)
// starting at line0).  Line-major mapping on a padded tile: each half warp
// reads or writes 16 consecutive points (128 bytes) of one line, so a warp
// access touches two lines, and the radix-16 shared-memory stages are
// conflict-free.  The field is H[0..2] (forward) or G[0..26] (inverse), by
// blockIdx.y.
constexpr int kCyThreads = 128;

template <bool INV>
__global__ void __launch_bounds__(kCyThreads) k_cy(KP k, int L, long long line0, long long line_end)
{
    extern __shared__ float4 smem4[];
    float2* sm = reinterpret_cast<float2*>(smem4);
    const int n = k.ny;
    float2* tw = sm;
    float2* A = tw + n;
    float2* B = A + L * (n + n / 16);
    float2* C = B + L * (n + n / 16);  // forward with Yv: the lines' y spectra, [L][n]
    load_table(tw, k.tw_y, n);
    __syncthreads();
    // forward: H -> Hy (H stays for k_sigma's kz-only fields); inverse: G in
    // place, blockIdx.y over the fields that went through k_mx
    const int c = blockIdx.y;
    const long long first = line0 + (long long)blockIdx.x * L;
    const int lv = (int)min((long long)L, line_end - first);  // lines of the tile inside the batch
    const long long off = first * n;
    const float2* src = (INV ? k.G[c_gxy[c]] : k.H[c]) + off;
    float2* dst = (INV ? k.G[c_gxy[c]] : k.Hy[c]) + off;
    const bool ydv = !INV && k.Yv[c] != nullptr;
    auto load = [&](int p, int i) -> float2 { return p < lv ? src[(long long)p * n + i] : make_float2(0.f, 0.f); };
    auto store = [&](int p, int i, float2 v) {
        if (p < lv) dst[(long long)p * n + i] = v;
        if (ydv) C[p * n + i] = v;
    };
    fft_rt<kLinePad, INV>(k.py, tw, A, B, L, n + n / 16, 1, load, store);
    if constexpr (!INV) {
        if (ydv) {
            // the y derivative with the identity dispersion operator, scaled
            // by 1/(ny nz) like a field of the x and y passes (1/ntp times
            // the x round trip's nx): dy vy (c = 1, forward shift), dy vx and
            // dy vz (backward)
            const float2* T = c == 1 ? k.Fy : k.By;
            const float inv_n = 1.0f / ((float)n * (float)k.nz);
            float2* yd = k.Yv[c] + off;
            auto load_d = [&](int p, int i) -> float2 { return cmul_m(C[p * n + i], cscale(T[i], inv_n)); };
            auto store_d = [&](int p, int i, float2 v) {
                if (p < lv) yd[(long long)p * n + i] = v;
            };
            fft_rt<kLinePad, true>(k.py, tw, A, B, L, n + n / 16, 1, load_d, store_d);
        }
    }
}

#endif  // QVTI_PART == 0

// ------------------------------------------------------------------ k_cp --
// Compiled form of k_cy: eight lines as four packed pairs (fft_pair.cuh), the
// y derivative of the forward pass taken from the registers the transform
// ends in.
constexpr int kCpPairs = 4;
constexpr int cp_threads(int n) { return warps_up(kCpPairs * pair_tasks(n)); }
constexpr size_t cp_smem(int n) { return 16 * ((size_t)kCpPairs * pair_slots(n) + tw_rows_size(n)); }
constexpr int cp_blocks(int n)
{
    const int warps = cp_threads(n) / 32;
    int b = 65536 / (128 * cp_threads(n));
    while (b > 1 && b * warps % 4) --b;
    return b < 1 ? 1 : b;
}

template <int N, bool INV>
__global__ void __launch_bounds__(cp_threads(N), cp_blocks(N)) k_cp(KP k, long long line0, long long line_end)
{
    using F = PairFFT<N, kCpPairs, false>;
    constexpr int NT = cp_threads(N), R0 = F::R0, RL = F::RL;
    extern __shared__ float4 smem4[];
    f2* buf = reinterpret_cast<f2*>(smem4);
    float4* tw = smem4 + F::PLANE;
    const TwRows<N> W{tw};
    const int c = blockIdx.y, t = threadIdx.x;
    const long long first = line0 + (long long)blockIdx.x * 2 * kCpPairs, left = line_end - first;
    const float2* src = (INV ? k.G[c_gxy[c]] : k.H[c]) + first * N;
    float2* dst = (INV ? k.G[c_gxy[c]] : k.Hy[c]) + first * N;
    c2 v[F::RM];
    int p, j;
    const bool act = F::task(t, p, j);
    const bool in0 = 2 * p < left, in1 = 2 * p + 1 < left;
    if (act)
        F::template each<0>(j, [&](int m, int i) {
            const float2* a = src + 2 * p * N + i;
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const float2 x = in0 ? a[r * (N / R0)] : make_float2(0.f, 0.f);
                const float2 y = in1 ? a[r * (N / R0) + N] : make_float2(0.f, 0.f);
                v[m * R0 + r] = c2{pack2(x.x, y.x), pack2(x.y, y.y)};
            }
        });
    TwRows<N>::template fill<NT>(tw, k.tw_y);
    if (F::SYNC0) __syncthreads();
    F::template first<INV>(W, buf, t, v);
    F::template finish<INV>(W, buf, t, v);
    auto store = [&](float2* to) {
        if (act)
            F::template each<F::LAST>(j, [&](int m, int i) {
#pragma unroll
                for (int r = 0; r < RL; ++r) {
                    const float2 re = unpack2(v[m * RL + r].x), im = unpack2(v[m * RL + r].y);
                    const int at = 2 * p * N + i + r * (N / RL);
                    if (in0) to[at] = make_float2(re.x, im.x);
                    if (in1) to[at + N] = make_float2(re.y, im.y);
                }
            });
    };
    store(dst);
    if constexpr (!INV) {
        // the y derivative with the identity dispersion operator, scaled by
        // 1/(ny nz) like a field of the x and y passes (1/ntp times the x round
        // trip's nx): dy vy (c = 1, forward shift), dy vx and dy vz (backward)
        const float2* T = c == 1 ? k.Fy : k.By;
        const float inv_n = 1.0f / ((float)N * (float)k.nz);
        F::turn(buf, t, v);
        if (act)
            F::template each<0>(j, [&](int m, int i) {
#pragma unroll
                for (int r = 0; r < R0; ++r) {
                    const float2 f = cscale(__ldg(T + i + r * (N / R0)), inv_n);
                    v[m * R0 + r] = cmul_m(v[m * R0 + r], pack2(f.x, f.x), pack2(f.y, f.y));
                }
            });
        __syncthreads();
        F::template first<true>(W, buf, t, v);
        F::template finish<true>(W, buf, t, v);
        store(k.Yv[c] + first * N);
    }
}

#if QVTI_PART == 0
// ------------------------------------------------------------------ k_mx --
// The runtime-length kernel (k_mp below is the compiled form).
// x-pencils of a (kz, y-chunk) tile in k-space for one velocity component c
// (blockIdx.z): forward x-FFT of V_c, then the 9 fields that use V_c --
// 3 derivatives x 3 dispersion operators Ap_j D_d V_c -- each inverse
// x-transformed on chip.  blockIdx.y + kz0 is the kz plane.
__global__ void __launch_bounds__(kThreads) k_mx(KP k, int P, int kz0)
{
    extern __shared__ float4 smem4[];
    float2* sm = reinterpret_cast<float2*>(smem4);
    const int n = k.nx;
    // the second transform buffer exists only for transforms of more than
    // two stages (a two-stage transform reads its input through `load` and
    // writes its output through `store`)
    const int nbuf = k.px.q.nst > 2 ? 2 : 1;
    float2* tw = sm;
    float2* tFx = tw + n;
    float2* tBx = tFx + n;
    float2* V = tBx + n;            // [n][P]
    float2* A = V + n * P;
    float2* B = A + (n + n / 16) * P;
    float2* tFBy = A + nbuf * (n + n / 16) * P;  // [2][P]: Fy, By of the tile's rows
    float* tkx = reinterpret_cast<float*>(tFBy + 2 * P);
    float* tky = tkx + n;                         // [P]
    const int kz = kz0 + blockIdx.y, y0 = blockIdx.x * P, c = blockIdx.z % 3;
    const int part = blockIdx.z / 3, parts = gridDim.z / 3;  // of the three directions of c
    const int yv = min(P, k.ny - y0);  // rows of the tile inside the grid
    load_table(tw, k.tw_x, n);
    load_table(tFx, k.Fx, n);
    load_table(tBx, k.Bx, n);
    for (int i = threadIdx.x; i < n; i += blockDim.x) tkx[i] = k.kx[i];
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
        const bool in = i < yv;
        tky[i] = in ? k.ky[y0 + i] : 0.f;
        tFBy[i] = in ? k.Fy[y0 + i] : make_float2(0.f, 0.f);
        tFBy[P + i] = in ? k.By[y0 + i] : make_float2(0.f, 0.f);
    }
    __syncthreads();

    {
        const float2* H = k.Hy[c];
        auto load = [&](int p, int i) -> float2 { return p < yv ? H[spec(k, kz, i, y0 + p)] : make_float2(0.f, 0.f); };
        auto store = [&](int p, int i, float2 v) { V[i * P + p] = v; };
        fft_rt<kPencil, false>(k.px, tw, A, B, P, 1, P, load, store);
    }

    const float kzv = k.kz[kz];
    const float kz2 = kzv * kzv;
    const float2 tFz = k.Fz[kz], tBz = k.Bz[kz];
    for (int d = 0, nd = 0; d < 9; ++d) {
        if (c_comp[d] != c || nd++ % parts != part) continue;
        const int ax = c_axis[d], fw = c_fwd[d];
        for (int j = 0; j < 3; ++j) {
            if (is_gz(3 * d + j) || is_gy(3 * d + j)) continue;  // one-axis fields: formed elsewhere
            float2* G = k.G[3 * d + j];
            auto load = [&](int p, int i) -> float2 {
                const float kyv = tky[p];
                const float kxv = tkx[i];
                float k2 = kxv * kxv + kyv * kyv + kz2;
                k2 = fmaxf(k2, 1e-10f);  // the reference sets |k|^2 = 1e-10 at DC (cu:74)
                // |k|^-1 and |k| from the hardware reciprocal square root
                // (~2 ulp): far below the FP32 transforms' own rounding
                const float rk = rsqrtf(k2);
                const float ap = j == 1 ? 1.0f : (j == 0 ? rk : k2 * rk);
                float2 T;
                if (ax == 0) T = fw ? tFx[i] : tBx[i];
                else if (ax == 1) T = fw ? tFBy[p] : tFBy[P + p];
                else T = fw ? tFz : tBz;
                return cmul(V[i * P + p], cscale(T, ap * k.inv_ntp));
            };
            auto store = [&](int p, int i, float2 v) {
                if (p < yv) G[spec(k, kz, i, y0 + p)] = v;
            };
            fft_rt<kPencil, true>(k.px, tw, A, B, P, 1, P, load, store);
        }
    }
}

#endif  // QVTI_PART == 0

// ------------------------------------------------------------------ k_mp --
// Compiled form of k_mx: the same job on pairs of y rows in packed arithmetic
// (fft_pair.cuh).  V is turned once into the points each inverse's first stage
// takes, so it stays in registers for all seven fields and only the exchanges
// of the transforms go through shared memory.
// 16 y (128-byte rows); 8 at three stages.
constexpr int mp_pairs(int n) { return mp_rows(n) / 2; }
constexpr int mp_threads(int n) { return warps_up(mp_pairs(n) * pair_tasks(n)); }
constexpr size_t mp_smem(int n) { return 16 * ((size_t)mp_pairs(n) * pair_slots(n) + 2 * (size_t)n) + 4 * (size_t)n; }
// V and the working butterflies: 8 registers a point.
constexpr int mp_blocks(int n)
{
    const int regs = pair_rmax(n) >= 14 ? 168 : 128;
    const int b = 65536 / (regs * mp_threads(n)), m = (int)(220 * 1024 / (mp_smem(n) + 1024));
    return b < 1 ? 1 : b < m ? b : m;
}

template <int N>
__global__ void __launch_bounds__(mp_threads(N), mp_blocks(N)) k_mp(KP k, int kz0)
{
    constexpr int PP = mp_pairs(N), NT = mp_threads(N);
    using F = PairFFT<N, PP, true>;
    constexpr int R0 = F::R0, RL = F::RL;
    extern __shared__ float4 smem4[];
    f2* buf = reinterpret_cast<f2*>(smem4);
    float4* tw = smem4 + PP * pair_slots(N);
    float4* tx = tw + N;                                 // the component's x shift, doubled like the twiddles
    float* tk = reinterpret_cast<float*>(tx + N);        // |kx|
    const TwAll<N> W{tw};
    const int kz = kz0 + blockIdx.y, y0 = blockIdx.x * 2 * PP, c = blockIdx.z % 3, t = threadIdx.x;
    const int part = blockIdx.z / 3, parts = gridDim.z / 3;  // of the three directions of c
    const float sc = k.inv_ntp;
    c2 v[F::RM], V[F::RM];
    int p, j;
    const bool act = F::task(t, p, j);
    const int y = y0 + 2 * p;
    const bool in = y < k.ny;
    if (act)
        F::template each<0>(j, [&](int m, int i) {
            const float4* src = reinterpret_cast<const float4*>(k.Hy[c] + spec(k, kz, i, y));
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const float4 a = in ? src[(long long)r * (N / R0) * k.ny / 2] : make_float4(0.f, 0.f, 0.f, 0.f);
                V[m * R0 + r] = c2{pack2(a.x, a.z), pack2(a.y, a.w)};
            }
        });
    {
        const float2* gf = c == 0 ? k.Fx : k.Bx;
        for (int i = t; i < N; i += NT) {
            const float2 w = k.tw_x[i], f = gf[i];
            tw[i] = make_float4(w.x, w.x, w.y, w.y);
            tx[i] = make_float4(f.x, f.x, f.y, f.y);
            tk[i] = k.kx[i];
        }
    }
    __syncthreads();
    F::template first<false>(W, buf, t, V);
    F::template finish<false>(W, buf, t, V);
    F::turn(buf, t, V);

    const float kzv = k.kz[kz];
    const float kz2 = kzv * kzv;
    // rows of this thread's pair: wavenumbers and y shifts
    const int yr = min(y, k.ny - 2);
    const f2 ky = pack2(k.ky[yr], k.ky[yr + 1]);
    const float2* gy = c == 1 ? k.Fy : k.By;
    const float2 ya = gy[yr], yb = gy[yr + 1], zz = (c == 2 ? k.Fz : k.Bz)[kz];

    // seven fields: per axis |k|^-1 and |k|, on the x axis also the identity
    // operator (the other two have one-axis multipliers and are formed elsewhere)
#pragma unroll 1
    for (int f = 0; f < 7; ++f) {
        const int ax = f < 3 ? 0 : f < 5 ? 1 : 2, jj = f < 3 ? f : 2 * ((f - 3) & 1);
        if (parts == 3 && ax != part) continue;
        const int d = c == 0 ? (ax == 0 ? 0 : ax == 1 ? 5 : 3) : c == 1 ? (ax == 0 ? 6 : ax == 1 ? 1 : 7)
                                                                        : (ax == 0 ? 4 : ax == 1 ? 8 : 2);
        if (act) {
            const f2 cx = ax == 1 ? pack2(ya.x, yb.x) : pack2(zz.x, zz.x);
            const f2 cy = ax == 1 ? pack2(ya.y, yb.y) : pack2(zz.y, zz.y);
            F::template each<0>(j, [&](int m, int i0) {
#pragma unroll
                for (int r = 0; r < R0; ++r) {
                    const int i = i0 + r * (N / R0);
                    f2 mx = cx, my = cy;
                    if (ax == 0) {
                        const float4 T = tx[i];
                        mx = pack2(T.x, T.y);
                        my = pack2(T.z, T.w);
                    }
                    f2 s = pack2(sc, sc);
                    if (jj != 1) {
                        const f2 kx = pack2(tk[i], tk[i]);
                        const float2 s2 = unpack2(fma_(kx, kx, ky * ky) + pack2(kz2, kz2));
                        // the reference sets |k|^2 = 1e-10 at DC (cu:74)
                        const float a = fmaxf(s2.x, 1e-10f), b = fmaxf(s2.y, 1e-10f);
                        // |k|^-1 and |k| from the hardware reciprocal square root
                        // (~2 ulp): far below the FP32 transforms' own rounding
                        f2 ap = pack2(rsqrtf(a), rsqrtf(b));
                        if (jj == 2) ap = ap * pack2(a, b);
                        s = ap * s;
                    }
                    v[m * R0 + r] = cmul_tw<false>(V[m * R0 + r], mx * s, my * s);
                }
            });
        }
        __syncthreads();  // the previous transform's last reads of the exchange
        F::template first<true>(W, buf, t, v);
        F::template finish<true>(W, buf, t, v);
        if (act && in)
            F::template each<F::LAST>(j, [&](int m, int i) {
                float4* dst = reinterpret_cast<float4*>(k.G[3 * d + jj] + spec(k, kz, i, y));
#pragma unroll
                for (int r = 0; r < RL; ++r) {
                    const float2 x = unpack2(v[m * RL + r].x), q = unpack2(v[m * RL + r].y);
                    dst[(long long)r * (N / RL) * k.ny / 2] = make_float4(x.x, q.x, x.y, q.y);
                }
            });
    }
}

}  // namespace

// Parts k_mx splits each component's directions into: three (the forward
// transform repeated in each) where one block per component would leave SMs
// without a block.
static int mx_parts(const KP& k, int P, int nb) { return cdiv(k.ny, P) * nb * 3 < 2 * 148 ? 3 : 1; }

QVTI_DECLARE_PARTS(bool, fz_launch, const KP& k, int P, int ncomp, cudaStream_t st);
QVTI_DECLARE_PARTS(bool, cy_launch, const KP& k, bool inv, dim3 grid, long long line0, long long line_end,
                   cudaStream_t st);
QVTI_DECLARE_PARTS(bool, mx_launch, const KP& k, int P, int kz0, int nb, cudaStream_t st);
QVTI_DECLARE_PARTS(bool, sp_configure, SmemLimit& lim, int axis, int n);

template <>
bool fz_launch<QVTI_PART>(const KP& k, int P, int ncomp, cudaStream_t st)
{
    return dispatch_len(k.nz, [&](auto NN) {
        constexpr int N = decltype(NN)::value;
        k_fp<N><<<dim3(cdiv(k.ny, P), k.nx, ncomp), fp_threads(N), fp_smem(N), st>>>(k);
    });
}
template <>
bool cy_launch<QVTI_PART>(const KP& k, bool inv, dim3 grid, long long line0, long long line_end, cudaStream_t st)
{
    return dispatch_len(k.ny, [&](auto NN) {
        constexpr int N = decltype(NN)::value;
        if (inv) k_cp<N, true><<<grid, cp_threads(N), cp_smem(N), st>>>(k, line0, line_end);
        else k_cp<N, false><<<grid, cp_threads(N), cp_smem(N), st>>>(k, line0, line_end);
    });
}
template <>
bool mx_launch<QVTI_PART>(const KP& k, int P, int kz0, int nb, cudaStream_t st)
{
    return dispatch_len(k.nx, [&](auto NN) {
        constexpr int N = decltype(NN)::value;
        if constexpr (N >= kMinLong)
            k_mp<N><<<dim3(cdiv(k.ny, P), nb, 3 * mx_parts(k, P, nb)), mp_threads(N), mp_smem(N), st>>>(k, kz0);
    });
}
template <>
bool sp_configure<QVTI_PART>(SmemLimit& lim, int axis, int n)
{
    return dispatch_len(n, [&](auto NN) {
        constexpr int N = decltype(NN)::value;
        if (axis == 2) lim.set((const void*)k_fp<N>);
        if (axis == 1) {
            lim.set((const void*)k_cp<N, false>);
            lim.set((const void*)k_cp<N, true>);
        }
        if constexpr (N >= kMinLong)
            if (axis == 0) lim.set((const void*)k_mp<N>);
    });
}

#if QVTI_PART == 0
size_t smem_fz(const KP& k, int P, bool rt)
{
    if (!rt) return fp_smem(k.nz);
    return sizeof(float2) * (k.nz + 2 * (P / 2) * (k.nz + k.nz / 16));
}
size_t smem_cy(const KP& k, int L, bool ydv, bool rt)
{
    if (!rt) return cp_smem(k.ny);
    return sizeof(float2) * (k.ny + 2 * L * (k.ny + k.ny / 16) + (ydv ? (size_t)L * k.ny : 0));
}
size_t smem_mx(const KP& k, int P, bool rt)
{
    if (!rt) return mp_smem(k.nx);
    const int nbuf = k.px.q.nst > 2 ? 2 : 1;
    return sizeof(float2) * (3 * k.nx + k.nx * P + nbuf * (k.nx + k.nx / 16) * P + 2 * P) + sizeof(float) * (k.nx + P);
}

void launch_fz(const KP& k, int P, bool rt, int ncomp, cudaStream_t st)
{
    if (rt) k_fz<<<dim3(cdiv(k.ny, P), k.nx, ncomp), rt_threads(k.pz, P / 2), smem_fz(k, P, true), st>>>(k, P);
    else (void)QVTI_CALL_PARTS(fz_launch, k, P, ncomp, st);
}

void launch_cy(const KP& k, int L, bool rt, bool inv, int nfield, bool ydv, long long line0, long long line_end,
               cudaStream_t st)
{
    const dim3 grid((unsigned)((line_end - line0 + L - 1) / L), nfield);
    const size_t sm = smem_cy(k, L, ydv, true);
    if (!rt) (void)QVTI_CALL_PARTS(cy_launch, k, inv, grid, line0, line_end, st);
    else if (inv) k_cy<true><<<grid, kCyThreads, sm, st>>>(k, L, line0, line_end);
    else k_cy<false><<<grid, kCyThreads, sm, st>>>(k, L, line0, line_end);
}

void launch_mx(const KP& k, int P, bool rt, int kz0, int nb, cudaStream_t st)
{
    if (rt) k_mx<<<dim3(cdiv(k.ny, P), nb, 3 * mx_parts(k, P, nb)), rt_threads(k.px, P), smem_mx(k, P, true), st>>>(k, P, kz0);
    else (void)QVTI_CALL_PARTS(mx_launch, k, P, kz0, nb, st);
}

cudaError_t configure_spectral(int axis, int n)
{
    SmemLimit lim;
    if (axis < 0) {
        lim.set((const void*)k_fz);
        lim.set((const void*)k_cy<false>);
        lim.set((const void*)k_cy<true>);
        lim.set((const void*)k_mx);
    } else {
        (void)QVTI_CALL_PARTS(sp_configure, lim, axis, n);
    }
    return lim.e;
}
#endif  // QVTI_PART == 0

}  // namespace qvti
