// Transforms of two pencils per thread (sm_100a packed FP32).
//
// The same Stockham sequence as fft.cuh with the radix plan of radix_seq, but
// every thread carries the butterflies of TWO pencils in packed registers
// (c2: real parts and imaginary parts of the pair): one issue slot per two
// floating-point operations, one twiddle load and one address for both.  The kernels built on the scalar
// transforms were bound by issue slots and barriers (ncu at 128^3: 49..55 %
// issue, 4..9 cycles of barrier stall per instruction), not by the FP32 pipe,
// whose rate is the same for both forms.
//
// One exchange buffer: a stage's inputs are all in registers before any of
// its outputs is written (one butterfly pair per thread and stage), so a
// middle stage costs two barriers and no second buffer.  The stages are
// separate calls, so a kernel can keep what a last stage produced in
// registers: the inverse transform runs the radices in REVERSE order, its
// first stage takes exactly the points (j + r N/R) the forward transform's
// last stage left in the same thread, and a multiplication in between needs
// no exchange at all.
//
// The exchange is two planes of 8-byte words, the pairs' real and imaginary
// parts (16-byte slots tie the four registers of a point together, which cost
// register moves: see k_st).  Point (pair p, index i) lives in slot p-fastest
// (PF: pencils adjacent in memory) or line-major; one pad slot per first radix
// keeps the accesses of sixteen neighbouring lanes on distinct banks.
#pragma once
#include "fft.cuh"

namespace qvti {

// Radix of stage s of N's plan, forward or reversed order.
__host__ __device__ constexpr int pair_rad(int n, int s, bool rev)
{
    const RadixSeq q = radix_seq(n);
    return q.rad[rev ? q.nst - 1 - s : s];
}
__host__ __device__ constexpr int pair_ns(int n, int s, bool rev)
{
    int p = 1;
    for (int i = 0; i < s; ++i) p *= pair_rad(n, i, rev);
    return p;
}
// Butterflies per pencil of the stage with most of them, and the largest radix.
__host__ __device__ constexpr int pair_tasks(int n)
{
    const RadixSeq q = radix_seq(n);
    int m = 0;
    for (int s = 0; s < q.nst; ++s) m = n / q.rad[s] > m ? n / q.rad[s] : m;
    return m;
}
__host__ __device__ constexpr int pair_rmax(int n)
{
    const RadixSeq q = radix_seq(n);
    int m = 0;
    for (int s = 0; s < q.nst; ++s) m = q.rad[s] > m ? q.rad[s] : m;
    return m;
}
__host__ __device__ constexpr int warps_up(int t) { return (t + 31) / 32 * 32; }
// Slots of one pencil pair in the exchange: the pad is per first radix of the
// sequence that writes it, so size for both orders.
__host__ __device__ constexpr int pair_pad(int n, bool rev) { return pair_rad(n, 0, rev) % 2 == 0 ? n / pair_rad(n, 0, rev) : 0; }
__host__ __device__ constexpr int pair_slots(int n)
{
    return n + (pair_pad(n, false) > pair_pad(n, true) ? pair_pad(n, false) : pair_pad(n, true));
}

// Pairs on neighbouring lanes: 16 / Q butterflies of each of the Q pairs make up
// a 16-lane access, so the pairs' slots start 16 / Q banks apart.
__host__ __device__ constexpr int pair_slots_q(int n, int q)
{
    int s = pair_slots(n);
    if (q > 1)
        while (s % 16 != 16 / q) ++s;
    return s;
}

// Twiddles e^{-2 pi i e / N}, e = jm r N / (NS R) in stage S, as (c, c, s, s).
// TwAll: a shared-memory table of all N (pencil-fast tiles: the lanes of one
// butterfly read one entry).  TwRows: per stage rows r = 1 .. R-1 of NS
// entries, so neighbouring butterflies read neighbouring entries (line-major
// tiles).  TwGlobal: the plain table where it lies.
template <int N>
struct TwAll {
    const float4* tw;
    template <int S, bool REV>
    __device__ __forceinline__ float4 at(int r, int jm) const
    {
        constexpr int TWS = N / (pair_ns(N, S, REV) * pair_rad(N, S, REV));
        return tw[jm * r * TWS];
    }
};
constexpr int tw_rows_off(int n, int s) { return s <= 1 ? 0 : (pair_rad(n, 1, false) - 1) * pair_ns(n, 1, false); }
constexpr int tw_rows_size(int n)
{
    const int l = radix_seq(n).nst - 1;
    return tw_rows_off(n, l) + (pair_rad(n, l, false) - 1) * pair_ns(n, l, false);
}
template <int N>
struct TwRows {
    const float4* tw;
    static constexpr int off(int s) { return tw_rows_off(N, s); }
    // fill stages S.. from the plain table, by all threads of a block of NT
    template <int NT, int S = 1>
    static __device__ __forceinline__ void fill(float4* s, const float2* g)
    {
        constexpr int R = pair_rad(N, S, false), NS = pair_ns(N, S, false), O = off(S), TWS = N / (NS * R);
#pragma unroll
        for (int i0 = 0; i0 < (R - 1) * NS; i0 += NT) {
            const unsigned i = i0 + threadIdx.x;
            if (i < (R - 1) * NS) {
                const float2 w = __ldg(g + (i / NS + 1) * (i % NS) * TWS);
                s[O + i] = make_float4(w.x, w.x, w.y, w.y);
            }
        }
        if constexpr (S + 1 < radix_seq(N).nst) fill<NT, S + 1>(s, g);
    }
    template <int S, bool REV>
    __device__ __forceinline__ float4 at(int r, int jm) const
    {
        static_assert(!REV, "rows are laid out for the forward order");
        constexpr int O = off(S), NS = pair_ns(N, S, false);
        return tw[O + (r - 1) * NS + jm];
    }
};
template <int N>
struct TwGlobal {
    const float2* tw;
    template <int S, bool REV>
    __device__ __forceinline__ float4 at(int r, int jm) const
    {
        constexpr int TWS = N / (pair_ns(N, S, REV) * pair_rad(N, S, REV));
        const float2 w = __ldg(tw + jm * r * TWS);
        return make_float4(w.x, w.x, w.y, w.y);
    }
};

// N points, PP pencil pairs per block.  Q > 1 (line-major): Q neighbouring
// pairs on neighbouring lanes, for pencils that share memory lines.
template <int N, int PP, bool PF, bool REV, int Q = 1>
struct PairFFT {
    static constexpr int NST = radix_seq(N).nst;
    static constexpr int R0 = pair_rad(N, 0, REV), RL = pair_rad(N, NST - 1, REV);
    template <int S>
    static constexpr int rad() { return pair_rad(N, S, REV); }

    static constexpr int SL = pair_slots_q(N, Q);
    static constexpr int PLANE = PP * SL;  // words of one plane
    static __device__ __forceinline__ void st(f2* b, c2 v)
    {
        b[0] = v.x;
        b[PLANE] = v.y;
    }
    static __device__ __forceinline__ c2 ld(const f2* b) { return c2{b[0], b[PLANE]}; }

    template <int S>
    static __device__ __forceinline__ bool task(int t, int& p, int& j)
    {
        constexpr unsigned NR = N / pair_rad(N, S, REV);
        const unsigned u = t;
        if constexpr (PF) { p = u % PP; j = u / PP; }
        else if constexpr (Q == 1) { p = u / NR; j = u % NR; }
        else { p = u / (Q * NR) * Q + u % Q; j = u / Q % NR; }
        return u < PP * NR;
    }
    // Slots: one pad per R0 indices where R0 is even.  Every stage's accesses
    // are a base and a constant distance per point (its strides are multiples
    // of R0), which keeps the index arithmetic out of the unrolled loops.
    static constexpr bool PAD = R0 % 2 == 0;
    static constexpr int STEP = PF ? PP : 1;  // distance of neighbouring indices
    static constexpr int padded(int n) { return n + (PAD ? n / R0 : 0); }   // n a multiple of R0
    static __device__ __forceinline__ int slot(int p, int i)
    {
        const int q = PAD ? i + (int)((unsigned)i / R0) : i;
        return PF ? q * PP + p : p * SL + q;
    }
    // Slot of point r of stage S's butterfly j (S >= 1; its inputs, and the
    // last stage's outputs): slot(p, j) + r dist<S>().
    template <int S>
    static constexpr int dist() { return padded(N / pair_rad(N, S, REV)) * STEP; }  // (use as a constant expression)

    // Stage 0 on v (its R0 points j + r N/R0), written to the exchange.  The
    // caller has loaded v; the exchange must be free.
    template <bool INV>
    static __device__ __forceinline__ void first(f2* buf, int t, c2* v)
    {
        int p, j;
        if (task<0>(t, p, j)) {
            Dft<R0>::template run<INV>(v);
            f2* b = buf + slot(p, j * R0);
#pragma unroll
            for (int r = 0; r < R0; ++r) st(b + r * STEP, v[r]);
        }
    }
    // Inputs of stage S >= 1, twiddled and transformed, left in v.
    template <bool INV, int S, class Tw>
    static __device__ __forceinline__ void take(const Tw& tw, const f2* buf, int t, c2* v)
    {
        constexpr int R = pair_rad(N, S, REV), NS = pair_ns(N, S, REV), D = dist<S>();
        int p, j;
        if (task<S>(t, p, j)) {
            const int jm = (unsigned)j % NS;
            const f2* b = buf + slot(p, j);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                v[r] = ld(b + r * D);
                if (r) {
                    const float4 w = tw.template at<S, REV>(r, jm);
                    v[r] = cmul_tw<INV>(v[r], pack2(w.x, w.y), pack2(w.z, w.w));
                }
            }
            Dft<R>::template run<INV>(v);
        }
    }
    template <int S>
    static __device__ __forceinline__ void put(f2* buf, int t, const c2* v)
    {
        constexpr int R = pair_rad(N, S, REV), NS = pair_ns(N, S, REV), D = padded(NS) * STEP;
        int p, j;
        if (task<S>(t, p, j)) {
            const int jm = (unsigned)j % NS;
            f2* b = buf + slot(p, (j - jm) * R + jm);
#pragma unroll
            for (int r = 0; r < R; ++r) st(b + r * D, v[r]);
        }
    }
    // From stage 0's outputs in the exchange (written, not yet synchronised)
    // to the last stage's outputs in v: point r of v is index j + r N/RL of
    // the task<NST-1> pair and j.
    template <bool INV, class Tw>
    static __device__ __forceinline__ void finish(const Tw& tw, f2* buf, int t, c2* v)
    {
        __syncthreads();
        if constexpr (NST == 3) {
            take<INV, 1>(tw, buf, t, v);
            __syncthreads();
            put<1>(buf, t, v);
            __syncthreads();
        }
        take<INV, NST - 1>(tw, buf, t, v);
    }
};

}  // namespace qvti
