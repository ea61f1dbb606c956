// Shared-memory mixed-radix FFT building blocks for sm_100a.
//
// The spectral-derivative engine replaces the reference's 63 cuFFT C2C calls
// per step (cuviscoelas_3D.cu:1272-1562) with pencil kernels that transform a
// tile of P pencils of one axis on chip.  A transform of length n = prod(rad)
// runs as a Stockham autosort sequence of stages of radix up to 16:
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

struct FftPlan {
    int n;                   // transform length
    int nst;                 // number of stages (>= 2)
    int rad[kMaxStages];     // radix of each stage, first stage first
};

// Radix plan of a length, shared by the host, the runtime kernels and the
// compiled ones: the fewest stages of radices up to 16 (each stage is one
// exchange through shared memory and a barrier or two, whatever its radix:
// 96 = 12 8 instead of 16 2 3, 150 = 15 10 instead of 2 3 5 5), and among
// those the plan whose largest radix is smallest (512 = 8 8 8, not 16 16 2:
// a stage's task count is N / radix, so equal radices keep every thread busy
// in every stage), larger radices first.
__host__ __device__ constexpr bool radix_ok(int r)
{
    return (r >= 2 && r <= 10) || r == 12 || r == 14 || r == 15 || r == 16;
}
struct RadixSeq {
    int nst;
    int rad[4];
};
__host__ __device__ constexpr RadixSeq radix_seq(int n)
{
    RadixSeq best{0, {1, 1, 1, 1}};
    for (int a = 2; a <= 16 && !best.nst; ++a)  // two stages a >= b
        if (radix_ok(a) && n % a == 0 && n / a <= a && n / a >= 2 && radix_ok(n / a)) best = RadixSeq{2, {a, n / a, 1, 1}};
    for (int a = 2; a <= 16 && !best.nst; ++a)  // three, a >= b >= c, b smallest
        if (radix_ok(a) && n % a == 0)
            for (int b = 2; b <= a && !best.nst; ++b)
                if (radix_ok(b) && (n / a) % b == 0 && n / a / b <= b && n / a / b >= 2 && radix_ok(n / a / b))
                    best = RadixSeq{3, {a, b, n / a / b, 1}};
    return best;
}

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
__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmulc(float2 a, float2 b)  // a * conj(b)
{
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
// a times w (INV: conj(w)), w the same for both of a pair: (wx, wx), (wy, wy)
template <bool INV>
__device__ __forceinline__ c2 cmul_tw(c2 a, f2 wx, f2 wy)
{
    const f2 n = neg_(wy);
    c2 r;
    r.x = fma_(a.y, INV ? wy : n, a.x * wx);
    r.y = fma_(a.x, INV ? n : wy, a.y * wx);
    return r;
}
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
// a times cos - i sin (forward) or its conjugate (inverse), compile-time values
template <bool INV, class C>
__device__ __forceinline__ C cmul_cs(C a, float c, float s)
{
    if (INV) s = -s;
    return cmake<C>(fmac_(a.x, c, scale_(a.y, s)), fmac_(a.y, c, scale_(a.x, -s)));
}

// ---------------------------------------------------------------- radix DFTs
template <int R>
struct Dft;

template <>
struct Dft<1> {
    template <bool INV, class C>
    static __device__ __forceinline__ void run(C*) {}
};

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
        const C t1 = cmake<C>(scale_(r1.x, c), scale_(r1.y, c));
        const C t3 = cmake<C>(scale_(r3.x, c), scale_(r3.y, c));  // minus W8^3 o3
        v[0] = cadd(e[0], o[0]);
        v[4] = csub(e[0], o[0]);
        v[1] = cadd(e[1], t1);
        v[5] = csub(e[1], t1);
        v[2] = cadd_rot<INV>(e[2], o[2]);
        v[6] = csub_rot<INV>(e[2], o[2]);
        v[3] = csub(e[3], t3);
        v[7] = cadd(e[3], t3);
    }
};

// Odd radices 3, 5, 7: the sums t_h = v[h] + v[R-h] carry the cosines, the
// differences d_h the sines; outputs h and R-h share both products.
template <int R>
__device__ constexpr float odd_cos(int k)
{
    k %= R;
    if (2 * k > R) k = R - k;
    if (k == 0) return 1.f;
    if (R == 3) return -0.5f;
    if (R == 5) return k == 1 ? 0.30901699437494742f : -0.80901699437494742f;
    return k == 1 ? 0.62348980185873353f : k == 2 ? -0.22252093395631440f : -0.90096886790241913f;
}
template <int R>
__device__ constexpr float odd_sin(int k)
{
    k %= R;
    const float sg = 2 * k > R ? -1.f : 1.f;
    if (2 * k > R) k = R - k;
    if (k == 0) return 0.f;
    if (R == 3) return sg * 0.86602540378443865f;
    if (R == 5) return sg * (k == 1 ? 0.95105651629515357f : 0.58778525229247313f);
    return sg * (k == 1 ? 0.78183148246802981f : k == 2 ? 0.97492791218182361f : 0.43388373911755812f);
}

template <int R>
struct DftOdd {
    template <bool INV, class C>
    static __device__ __forceinline__ void run(C* v)
    {
        constexpr int H = (R - 1) / 2;
        C t[H], d[H];
#pragma unroll
        for (int h = 0; h < H; ++h) {
            t[h] = cadd(v[h + 1], v[R - 1 - h]);
            d[h] = csub(v[h + 1], v[R - 1 - h]);
        }
        const C v0 = v[0];
#pragma unroll
        for (int h = 0; h < H; ++h) v[0] = cadd(v[0], t[h]);
#pragma unroll
        for (int q = 1; q <= H; ++q) {
            C m = v0;
            C s = cmake<C>(scale_(d[0].x, odd_sin<R>(q)), scale_(d[0].y, odd_sin<R>(q)));
#pragma unroll
            for (int h = 1; h <= H; ++h)
                m = cmake<C>(fmac_(t[h - 1].x, odd_cos<R>(q * h), m.x), fmac_(t[h - 1].y, odd_cos<R>(q * h), m.y));
#pragma unroll
            for (int h = 2; h <= H; ++h)
                s = cmake<C>(fmac_(d[h - 1].x, odd_sin<R>(q * h), s.x), fmac_(d[h - 1].y, odd_sin<R>(q * h), s.y));
            v[q] = cadd_rot<INV>(m, s);
            v[R - q] = csub_rot<INV>(m, s);
        }
    }
};
template <>
struct Dft<3> : DftOdd<3> {};
template <>
struct Dft<5> : DftOdd<5> {};
template <>
struct Dft<7> : DftOdd<7> {};

// Radix A B with A and B coprime as A x B without twiddles (the prime-factor
// map: input B n1 + A n2, output the k with k = k1 mod A, k = k2 mod B).
// Inverse of a modulo m.
__host__ __device__ constexpr int inv_mod(int a, int m)
{
    for (int i = 1; i < m; ++i)
        if (a * i % m == 1) return i;
    return 1;
}
template <int A, int B>
struct DftCoprime {
    template <bool INV, class C>
    static __device__ __forceinline__ void run(C* v)
    {
        constexpr int E1 = B * inv_mod(B % A, A), E2 = A * inv_mod(A % B, B);
        C t[A * B];
#pragma unroll
        for (int n1 = 0; n1 < A; ++n1) {
            C u[B];
#pragma unroll
            for (int n2 = 0; n2 < B; ++n2) u[n2] = v[(B * n1 + A * n2) % (A * B)];
            Dft<B>::template run<INV>(u);
#pragma unroll
            for (int k2 = 0; k2 < B; ++k2) t[n1 * B + k2] = u[k2];
        }
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) {
            C u[A];
#pragma unroll
            for (int n1 = 0; n1 < A; ++n1) u[n1] = t[n1 * B + k2];
            Dft<A>::template run<INV>(u);
#pragma unroll
            for (int k1 = 0; k1 < A; ++k1) v[(E1 * k1 + E2 * k2) % (A * B)] = u[k1];
        }
    }
};
template <>
struct Dft<6> : DftCoprime<2, 3> {};
template <>
struct Dft<10> : DftCoprime<2, 5> {};
template <>
struct Dft<12> : DftCoprime<4, 3> {};
template <>
struct Dft<14> : DftCoprime<2, 7> {};
template <>
struct Dft<15> : DftCoprime<3, 5> {};

// Radix A^2 (9, 16) in registers as A x A: DFT-A over n2 of v[n1 + A n2],
// twiddle W^{n1 k2}, DFT-A over n1; output X[k2 + A k1].
__device__ constexpr float sq_cos(int n, int e)
{
    if (n == 16) {
        e %= 16;
        const float c[16] = {1.f, 0.92387953251128674f, 0.70710678118654752f, 0.38268343236508977f,
                             0.f, -0.38268343236508977f, -0.70710678118654752f, -0.92387953251128674f,
                             -1.f, -0.92387953251128674f, -0.70710678118654752f, -0.38268343236508977f,
                             0.f, 0.38268343236508977f, 0.70710678118654752f, 0.92387953251128674f};
        return c[e];
    }
    const float c[9] = {1.f, 0.76604444311897804f, 0.17364817766693035f, -0.5f, -0.93969262078590838f,
                        -0.93969262078590838f, -0.5f, 0.17364817766693035f, 0.76604444311897804f};
    return c[e % 9];
}
__device__ constexpr float sq_sin(int n, int e)
{
    if (n == 16) return sq_cos(16, e + 12);  // sin(x) = cos(x - pi/2)
    const float s[9] = {0.f, 0.64278760968653933f, 0.98480775301220806f, 0.86602540378443865f, 0.34202014332566873f,
                        -0.34202014332566873f, -0.86602540378443865f, -0.98480775301220806f, -0.64278760968653933f};
    return s[e % 9];
}
template <int A>
struct DftSquare {
    template <bool INV, class C>
    static __device__ __forceinline__ void run(C* v)
    {
        C y[A * A];
#pragma unroll
        for (int n1 = 0; n1 < A; ++n1) {
            C t[A];
#pragma unroll
            for (int n2 = 0; n2 < A; ++n2) t[n2] = v[n1 + A * n2];
            Dft<A>::template run<INV>(t);
#pragma unroll
            for (int k2 = 0; k2 < A; ++k2) {
                const int e = n1 * k2;
                if (e == 0) y[n1 * A + k2] = t[k2];
                else if (A == 4 && e == 4) y[n1 * A + k2] = t[k2];  // -+ i, taken in the second pass
                else y[n1 * A + k2] = cmul_cs<INV>(t[k2], sq_cos(A * A, e), sq_sin(A * A, e));
            }
        }
#pragma unroll
        for (int k2 = 0; k2 < A; ++k2) {
            C t[A];
#pragma unroll
            for (int n1 = 0; n1 < A; ++n1) t[n1] = y[n1 * A + k2];
            if constexpr (A == 4) Dft<4>::template run<INV>(t, k2 == 2);
            else Dft<A>::template run<INV>(t);
#pragma unroll
            for (int k1 = 0; k1 < A; ++k1) v[k2 + A * k1] = t[k1];
        }
    }
};
template <>
struct Dft<9> : DftSquare<3> {};
template <>
struct Dft<16> : DftSquare<4> {};

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

template <int R, bool PF, bool INV, class Load, class Store>
__device__ __forceinline__ void fft_stage(int n, int P, int ps, int is, int padsh, int Ns, bool first, bool last,
                                          const float2* __restrict__ tw, const float2* src, float2* dst,
                                          Load& load, Store& store)
{
    const int nr = n / R;
    const int total = P * nr;
    const int twstride = n / (Ns * R);
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
            for (int r = 1; r < R; ++r) {
                const float2 w = tw[jm * r * twstride];
                v[r] = INV ? cmulc(v[r], w) : cmul(v[r], w);
            }
        }
        Dft<R>::template run<INV>(v);
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
    for (int s = 0; s < pl.nst; ++s) {
        const bool first = (s == 0), last = (s == pl.nst - 1);
        const float2* src = first ? nullptr : (((s - 1) & 1) ? bufB : bufA);
        float2* dst = (s & 1) ? bufB : bufA;
        auto stage = [&](auto RR) {
            fft_stage<decltype(RR)::value, PF, INV>(pl.n, P, ps, is, padsh, Ns, first, last, tw, src, dst, load, store);
        };
        switch (pl.rad[s]) {
            case 2: stage(IntC<2>{}); break;
            case 3: stage(IntC<3>{}); break;
            case 4: stage(IntC<4>{}); break;
            case 5: stage(IntC<5>{}); break;
            case 6: stage(IntC<6>{}); break;
            case 7: stage(IntC<7>{}); break;
            case 8: stage(IntC<8>{}); break;
            case 9: stage(IntC<9>{}); break;
            case 10: stage(IntC<10>{}); break;
            case 12: stage(IntC<12>{}); break;
            case 14: stage(IntC<14>{}); break;
            case 15: stage(IntC<15>{}); break;
            default: stage(IntC<16>{}); break;
        }
        __syncthreads();
        Ns *= pl.rad[s];
    }
}

// Buffer that holds the output of fft_run when its store writes "the other"
// buffer of the pair (the one the last stage does not read).
__device__ __forceinline__ float2* fft_out_buf(const FftPlan& pl, float2* bufA, float2* bufB)
{
    return ((pl.nst - 1) & 1) ? bufB : bufA;
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
