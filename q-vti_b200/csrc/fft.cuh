// Shared-memory mixed-radix FFT building blocks for sm_100a.
//
// The spectral-derivative engine replaces the reference's 63 cuFFT C2C calls
// per step (cuviscoelas_3D.cu:1272-1562) with pencil kernels that transform a
// tile of P pencils of one axis on chip.  A transform of length n = prod(rad)
// runs as a Stockham autosort sequence of stages of up to 16 points:
//
//   * stage 0 reads its inputs through a caller-supplied `load(p, i)` functor
//     (straight from global memory, or from shared memory with a k-space
//     multiplier applied on the fly),
//   * middle stages ping-pong between two shared-memory buffers,
//   * the last stage hands its outputs to a `store(p, i, v)` functor (to global
//     memory, or into an update epilogue).
//
// so a pencil costs one trip through HBM no matter how many stages it has.
// Element (p, i) of a pencil tile lives at buf[p*ps + i*is]; the thread
// mapping is pencil-fastest (PF) when pencils are contiguous in global memory
// and index-fastest otherwise, so both the global and the shared-memory
// accesses of every stage are coalesced / bank-spread.
//
// Convention: forward e^{-2 pi i k m / n}, inverse e^{+...}, unnormalised,
// matching cuFFT's CUFFT_FORWARD / CUFFT_INVERSE used by the reference.
#pragma once
#include <cuda_runtime.h>

namespace qvti {

constexpr int kMaxStages = 4;

// Radix plan of a length, shared by the host, the runtime kernels and the
// compiled ones.  The arithmetic is that of the elementary radices 16, 8, 4, 2,
// 3, 5, 7 in this order (16 itself: 4 4); two neighbouring ones whose product is
// at most 16 run as ONE stage, the second on the first's outputs in the same
// registers (a then b; b = 1: a alone).  A stage is one exchange through shared
// memory and a barrier or two, whatever its radix, so 96 = 16 (2 3) is two
// stages; the values are those of the three separate ones.
struct RadixSeq {
    int nst;
    int a[kMaxStages], b[kMaxStages];
    int radices;  // elementary ones
    constexpr int rad(int s) const { return a[s] * b[s]; }
};
__host__ __device__ constexpr bool radix_pair(int a, int b)
{
    return (a == 2 && (b == 3 || b == 5 || b == 7)) || (a == 4 && b == 3) || (a == 3 && (b == 3 || b == 5));
}
__host__ __device__ constexpr RadixSeq radix_seq(int n)
{
    int el[12] = {}, ne = 0, m = n;
    const int order[7] = {16, 8, 4, 2, 3, 5, 7};
    if (n == 16) {
        el[0] = el[1] = 4;
        ne = 2;
        m = 1;
    }
    for (int i = 0; i < 7; ++i)
        while (m % order[i] == 0 && ne < 12) {
            el[ne++] = order[i];
            m /= order[i];
        }
    RadixSeq q{0, {1, 1, 1, 1}, {1, 1, 1, 1}, ne};
    if (m != 1 || ne < 2) return q;
    for (int i = 0; i < ne; ++q.nst) {
        if (q.nst == kMaxStages) return RadixSeq{0, {1, 1, 1, 1}, {1, 1, 1, 1}, ne};
        q.a[q.nst] = el[i++];
        if (i < ne && radix_pair(q.a[q.nst], el[i])) q.b[q.nst] = el[i++];
    }
    return q;
}

struct FftPlan {
    int n;      // transform length
    RadixSeq q;
};

// Two floats in one 64-bit register pair: sm_100a's packed FP32 instructions
// do the operation on both in one issue slot.
struct f2 {
    unsigned long long v;
};
__device__ __forceinline__ f2 pack2(float a, float b)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(f2 a)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
    return r;
}
__device__ __forceinline__ f2 operator+(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 operator-(f2 a, f2 b)
{
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 operator*(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 fma_(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ f2 neg_(f2 a) { return f2{a.v ^ 0x8000000080000000ull}; }
__device__ __forceinline__ f2 scale_(f2 a, float c) { return a * pack2(c, c); }
__device__ __forceinline__ f2 fmac_(f2 a, float c, f2 b) { return fma_(a, pack2(c, c), b); }
__device__ __forceinline__ float fma_(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ float neg_(float a) { return -a; }
__device__ __forceinline__ float scale_(float a, float c) { return a * c; }
__device__ __forceinline__ float fmac_(float a, float c, float b) { return fmaf(a, c, b); }

// A pair of complex numbers, real parts and imaginary parts packed: the
// complex type of transforms that run two pencils per thread.  The templates
// below take float2 (one complex number) or c2.
struct c2 {
    f2 x, y;
};

template <class C>
__device__ __forceinline__ C cmake(decltype(C::x) x, decltype(C::x) y)
{
    C r;
    r.x = x;
    r.y = y;
    return r;
}
template <class C>
__device__ __forceinline__ C cadd(C a, C b) { return cmake<C>(a.x + b.x, a.y + b.y); }
template <class C>
__device__ __forceinline__ C csub(C a, C b) { return cmake<C>(a.x - b.x, a.y - b.y); }
// a + rot(b) and a - rot(b), rot(b) = -i b (forward) or +i b (inverse)
template <bool INV, class C>
__device__ __forceinline__ C cadd_rot(C a, C b)
{
    return INV ? cmake<C>(a.x - b.y, a.y + b.x) : cmake<C>(a.x + b.y, a.y - b.x);
}
template <bool INV, class C>
__device__ __forceinline__ C csub_rot(C a, C b) { return cadd_rot<!INV>(a, b); }
// Complex products.  The rounding of each is fixed here, which product of a sum
// is rounded before the fused operation included: the scalar and the packed form
// agree bit for bit, whatever the compiler contracts elsewhere.
__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(fmaf(a.x, b.x, -(a.y * b.y)), fmaf(a.x, b.y, a.y * b.x));
}
// a times a multiplier m: the other product of the imaginary part first
__device__ __forceinline__ float2 cmul_m(float2 a, float2 m)
{
    return make_float2(fmaf(a.x, m.x, -(a.y * m.y)), fmaf(a.y, m.x, a.x * m.y));
}
__device__ __forceinline__ float2 cmulc(float2 a, float2 b)  // a * conj(b)
{
    return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -(a.x * b.y)));
}
// a times w (INV: conj(w)), w the same for both of a pair: (wx, wx), (wy, wy)
template <bool INV>
__device__ __forceinline__ c2 cmul_tw(c2 a, f2 wx, f2 wy)
{
    const f2 n = neg_(wy);
    c2 r;
    r.x = fma_(a.x, wx, a.y * (INV ? wy : n));
    r.y = INV ? fma_(a.y, wx, a.x * n) : fma_(a.x, wy, a.y * wx);
    return r;
}
__device__ __forceinline__ c2 cmul_m(c2 a, f2 mx, f2 my)
{
    c2 r;
    r.x = fma_(a.x, mx, a.y * neg_(my));
    r.y = fma_(a.y, mx, a.x * my);
    return r;
}
template <bool INV>
__device__ __forceinline__ float2 cmul_tw(float2 a, float2 w) { return INV ? cmulc(a, w) : cmul(a, w); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }

// ---------------------------------------------------------------- radix DFTs
template <int R>
struct Dft;

template <>
struct Dft<2> {
    template <bool INV, class C>
    static __device__ __forceinline__ void run(C* v)
    {
        const C a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    }
};

template <>
struct Dft<4> {
    template <bool INV, class C>
    static __device__ __forceinline__ void run(C* v, bool rot2 = false)  // rot2: v[2] stands for rot(v[2])
    {
        const C s0 = rot2 ? cadd_rot<INV>(v[0], v[2]) : cadd(v[0], v[2]);
        const C s1 = rot2 ? csub_rot<INV>(v[0], v[2]) : csub(v[0], v[2]);
        const C s2 = cadd(v[1], v[3]), s3 = csub(v[1], v[3]);
        v[0] = cadd(s0, s2);
        v[2] = csub(s0, s2);
        v[1] = cadd_rot<INV>(s1, s3);
        v[3] = csub_rot<INV>(s1, s3);
    }
};

template <>
struct Dft<8> {
    template <bool INV, class C>
    static __device__ __forceinline__ void run(C* v)
    {
        const float c = 0.70710678118654752f;
        C e[4] = {v[0], v[2], v[4], v[6]};
        C o[4] = {v[1], v[3], v[5], v[7]};
        Dft<4>::run<INV>(e);
        Dft<4>::run<INV>(o);
        // o[k] *= W8^k  (W8 = e^{-i pi/4} forward, conjugate inverse)
        const C r1 = cadd_rot<INV>(o[1], o[1]), r3 = csub_rot<INV>(o[3], o[3]);  // (1 -+ i) o1, (1 +- i) o3
        v[0] = cadd(e[0], o[0]);
        v[4] = csub(e[0], o[0]);
        v[1] = cmake<C>(fmac_(r1.x, c, e[1].x), fmac_(r1.y, c, e[1].y));
        v[5] = cmake<C>(fmac_(r1.x, -c, e[1].x), fmac_(r1.y, -c, e[1].y));
        v[2] = cadd_rot<INV>(e[2], o[2]);
        v[6] = csub_rot<INV>(e[2], o[2]);
        v[3] = cmake<C>(fmac_(r3.x, -c, e[3].x), fmac_(r3.y, -c, e[3].y));  // W8^3 o3 = -c r3
        v[7] = cmake<C>(fmac_(r3.x, c, e[3].x), fmac_(r3.y, c, e[3].y));
    }
};

// Odd radices 3, 5, 7: direct DFT.
template <int R>
__device__ constexpr float odd_cos(int k)
{
    k %= R;
    if (2 * k > R) k = R - k;
    if (k == 0) return 1.f;
    if (R == 3) return -0.5f;
    if (R == 5) return k == 1 ? 0.309016994f : -0.809016994f;
    return k == 1 ? 0.623489802f : k == 2 ? -0.222520934f : -0.900968868f;
}
template <int R>
__device__ constexpr float odd_sin(int k)
{
    k %= R;
    const float sg = 2 * k > R ? -1.f : 1.f;
    if (2 * k > R) k = R - k;
    if (k == 0) return 0.f;
    if (R == 3) return sg * 0.866025404f;
    if (R == 5) return sg * (k == 1 ? 0.951056516f : 0.587785252f);
    return sg * (k == 1 ? 0.781831482f : k == 2 ? 0.974927912f : 0.433883739f);
}

template <int R>
struct DftOdd {
    template <bool INV, class C>
    static __device__ __forceinline__ void run(C* v)
    {
        C o[R];
        o[0] = v[0];
#pragma unroll
        for (int r = 1; r < R; ++r) o[0] = cadd(o[0], v[r]);
#pragma unroll
        for (int q = 1; q < R; ++q) {
            o[q] = v[0];
#pragma unroll
            for (int r = 1; r < R; ++r) {
                const float c = odd_cos<R>(q * r), s = INV ? odd_sin<R>(q * r) : -odd_sin<R>(q * r);
                o[q] = cmake<C>(o[q].x + fmac_(v[r].x, c, scale_(v[r].y, -s)), o[q].y + fmac_(v[r].y, c, scale_(v[r].x, s)));
            }
        }
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = o[q];
    }
};
template <>
struct Dft<3> : DftOdd<3> {};
template <>
struct Dft<5> : DftOdd<5> {};
template <>
struct Dft<7> : DftOdd<7> {};

// Radix 16 in registers as 4 x 4: DFT-4 over n2 of v[n1 + 4 n2], twiddle
// W16^{n1 k2}, DFT-4 over n1; output X[k2 + 4 k1].
template <bool INV, class C>
__device__ __forceinline__ C w16(C a, int e)  // e = 1, 2, 3, 6, 9
{
    const float c1 = 0.923879533f, s1 = 0.382683432f, h = 0.707106781f;
    const float c = e == 1 ? c1 : e == 2 ? h : e == 3 ? s1 : e == 6 ? -h : -c1;
    float s = e == 1 ? s1 : e == 2 || e == 6 ? h : e == 3 ? c1 : -s1;
    if (!INV) s = -s;  // forward W16^e = cos - i sin, inverse its conjugate
    const auto x = !INV && e == 6 ? fmac_(a.y, -s, scale_(a.x, c)) : fmac_(a.x, c, scale_(a.y, -s));
    return cmake<C>(x, e == 2 ? fmac_(a.x, s, scale_(a.y, c)) : fmac_(a.y, c, scale_(a.x, s)));
}
template <>
struct Dft<16> {
    template <bool INV, class C>
    static __device__ __forceinline__ void run(C* v)
    {
        C y[16];
#pragma unroll
        for (int n1 = 0; n1 < 4; ++n1) {
            C t[4] = {v[n1], v[n1 + 4], v[n1 + 8], v[n1 + 12]};
            Dft<4>::run<INV>(t);
#pragma unroll
            for (int k2 = 0; k2 < 4; ++k2)  // W16^4 = -+ i is taken in the second pass
                y[n1 * 4 + k2] = n1 * k2 == 0 || n1 * k2 == 4 ? t[k2] : w16<INV>(t[k2], n1 * k2);
        }
#pragma unroll
        for (int k2 = 0; k2 < 4; ++k2) {
            C t[4] = {y[k2], y[4 + k2], y[8 + k2], y[12 + k2]};
            Dft<4>::run<INV>(t, k2 == 2);
#pragma unroll
            for (int k1 = 0; k1 < 4; ++k1) v[k2 + 4 * k1] = t[k1];
        }
    }
};

// A stage of radix A, then radix B on its outputs.  Point r of v is index
// j + r N / (A B); the second radix's butterflies take the same point o of B
// first-radix butterflies, each times the twiddle inner(o, r2) applies.
template <int A, int B, bool INV, class C, class In>
__device__ __forceinline__ void dft_stage(C* v, In inner)
{
    if constexpr (B == 1) {
        Dft<A>::template run<INV>(v);
    } else {
        C t[A * B];  // [o][r2]
#pragma unroll
        for (int r2 = 0; r2 < B; ++r2) {
            C u[A];
#pragma unroll
            for (int r1 = 0; r1 < A; ++r1) u[r1] = v[r2 + B * r1];
            Dft<A>::template run<INV>(u);
#pragma unroll
            for (int o = 0; o < A; ++o) t[o * B + r2] = r2 ? inner(u[o], o, r2) : u[o];
        }
#pragma unroll
        for (int o = 0; o < A; ++o) {
            Dft<B>::template run<INV>(t + o * B);
#pragma unroll
            for (int q = 0; q < B; ++q) v[o + A * q] = t[o * B + q];
        }
    }
}

// ------------------------------------------------------------------- stages
template <int V>
struct IntC {
    static constexpr int value = V;
};
// Shared-memory address of element (p, i): p*ps + i*is, plus one extra `is`
// row every 2^padsh indices when padsh > 0 (breaks the bank conflicts of the
// radix-16 stage-0 writes in pencil-fastest tiles).
__device__ __forceinline__ int smem_at(int p, int i, int ps, int is, int padsh)
{
    return p * ps + i * is + (padsh ? (i >> padsh) * is : 0);
}

template <int A, int B, bool PF, bool INV, class Load, class Store>
__device__ __forceinline__ void fft_stage(int n, int P, int ps, int is, int padsh, int Ns, bool first, bool last,
                                          const float2* __restrict__ tw, const float2* src, float2* dst,
                                          Load& load, Store& store)
{
    constexpr int R = A * B;
    const int nr = n / R;
    const int total = P * nr;
    const int tw1 = n / (Ns * A), tw2 = nr / Ns;  // twiddle strides of the two radices
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int p, j;
        if (PF) { p = t % P; j = t / P; }
        else    { j = t % nr; p = t / nr; }
        const int jm = j % Ns;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int idx = j + r * nr;
            v[r] = first ? load(p, idx) : src[smem_at(p, idx, ps, is, padsh)];
        }
        if (jm) {
#pragma unroll
            for (int r = B; r < R; ++r) v[r] = cmul_tw<INV>(v[r], tw[jm * (r / B) * tw1]);
        }
        dft_stage<A, B, INV>(v, [&](float2 u, int o, int r2) { return cmul_tw<INV>(u, tw[(jm + o * Ns) * r2 * tw2]); });
        const int base = (j - jm) * R + jm;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int idx = base + r * Ns;
            if (last) store(p, idx, v[r]);
            else dst[smem_at(p, idx, ps, is, padsh)] = v[r];
        }
    }
}

// Run a full transform of P pencils.  Stage 0 reads through `load`, writes
// bufA; stage s writes buf[s&1] (bufA, bufB alternating); the last stage
// writes through `store`.  Ends with __syncthreads().  Requires nst >= 2.
// Shared buffers must not alias anything `load` reads after stage 0.
template <bool PF, bool INV, class Load, class Store>
__device__ void fft_run(const FftPlan& pl, const float2* __restrict__ tw, float2* bufA, float2* bufB,
                        int P, int ps, int is, Load load, Store store, int padsh = 0)
{
    int Ns = 1;
    for (int s = 0; s < pl.q.nst; ++s) {
        const bool first = (s == 0), last = (s == pl.q.nst - 1);
        const float2* src = first ? nullptr : (((s - 1) & 1) ? bufB : bufA);
        float2* dst = (s & 1) ? bufB : bufA;
        auto stage = [&](auto AA, auto BB) {
            fft_stage<decltype(AA)::value, decltype(BB)::value, PF, INV>(pl.n, P, ps, is, padsh, Ns, first, last, tw,
                                                                         src, dst, load, store);
        };
        switch (pl.q.a[s] * 16 + pl.q.b[s]) {
            case 2 * 16 + 1: stage(IntC<2>{}, IntC<1>{}); break;
            case 2 * 16 + 3: stage(IntC<2>{}, IntC<3>{}); break;
            case 2 * 16 + 5: stage(IntC<2>{}, IntC<5>{}); break;
            case 2 * 16 + 7: stage(IntC<2>{}, IntC<7>{}); break;
            case 3 * 16 + 1: stage(IntC<3>{}, IntC<1>{}); break;
            case 3 * 16 + 3: stage(IntC<3>{}, IntC<3>{}); break;
            case 3 * 16 + 5: stage(IntC<3>{}, IntC<5>{}); break;
            case 4 * 16 + 1: stage(IntC<4>{}, IntC<1>{}); break;
            case 4 * 16 + 3: stage(IntC<4>{}, IntC<3>{}); break;
            case 5 * 16 + 1: stage(IntC<5>{}, IntC<1>{}); break;
            case 7 * 16 + 1: stage(IntC<7>{}, IntC<1>{}); break;
            case 8 * 16 + 1: stage(IntC<8>{}, IntC<1>{}); break;
            default: stage(IntC<16>{}, IntC<1>{}); break;
        }
        __syncthreads();
        Ns *= pl.q.rad(s);
    }
}

// Buffer that holds the output of fft_run when its store writes "the other"
// buffer of the pair (the one the last stage does not read).
__device__ __forceinline__ float2* fft_out_buf(const FftPlan& pl, float2* bufA, float2* bufB)
{
    return ((pl.q.nst - 1) & 1) ? bufB : bufA;
}

// Two real pencils a, b packed as z = a + i b and transformed together; this
// recovers A(k) and B(k) from Z(k) and Zc = conj(Z(n-k)).
__device__ __forceinline__ float2 unpack_a(float2 z, float2 zmc) { return make_float2(0.5f * (z.x + zmc.x), 0.5f * (z.y + zmc.y)); }
__device__ __forceinline__ float2 unpack_b(float2 z, float2 zmc)
{
    // (z - zmc) / (2i)
    return make_float2(0.5f * (z.y - zmc.y), -0.5f * (z.x - zmc.x));
}

// For z = a + i b transformed (a, b real), the spectrum of M1 a + i M2 b
// (M1, M2 Hermitian multipliers) is 1/2 [(M1+M2) Z(k) + (M1-M2) Zc] with
// Zc = conj(Z(n-k)).  For the staggered-shift pair of one axis, F = i k
// e^{+i k d/2} and B = i k e^{-i k d/2} satisfy B = (-F.x, F.y) exactly as
// tabulated (the Nyquist bin of both keeps only its real part), so
// (M1, M2) = (F, B) (sgn = 1) or (B, F) (sgn = -1) reduces it to
// i F.y Z + sgn F.x Zc.
__device__ __forceinline__ float2 two_shift(float2 z, float2 zmc, float2 f, float sgn)
{
    const float fx = sgn * f.x;
    return make_float2(fmaf(fx, zmc.x, -f.y * z.y), fmaf(fx, zmc.y, f.y * z.x));
}

}  // namespace qvti
