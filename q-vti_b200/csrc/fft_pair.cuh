// Transforms of two pencils per thread (sm_100a packed FP32).
//
// The same Stockham sequence and arithmetic as fft.cuh, but every thread
// carries the butterflies of TWO pencils in packed registers (c2: real parts
// and imaginary parts of the pair): one issue slot per two floating-point
// operations, one twiddle load and one address for both.  The kernels built on
// the scalar transforms were bound by issue slots and barriers (ncu at 128^3:
// 49..55 % issue, 4..9 cycles of barrier stall per instruction), not by the FP32
// pipe, whose rate is the same for both forms.
//
// One exchange buffer: a stage's inputs are all in registers before any of its
// outputs is written, so a middle stage costs two barriers and no second
// buffer.  A thread takes as many butterflies of a stage as 16 points hold (K:
// 128 = 16 8 has one of 16 or two of 8), so a short radix does not need a block
// several times as large.
// The stages are separate calls, so a kernel can keep what a last stage produced
// in registers; turn() hands it to the inverse transform's first stage, without
// an exchange where both stages leave a thread the same points (256, 128, 512).
//
// The exchange is two planes of 8-byte words, the pairs' real and imaginary
// parts (16-byte slots tie the four registers of a point together, which cost
// register moves: see k_st).  Point (pair p, index i) lives in slot p-fastest
// (PF: pencils adjacent in memory) or line-major; one pad slot per first radix
// keeps the accesses of sixteen neighbouring lanes on distinct banks.
#pragma once
#include "fft.cuh"

namespace qvti {

// Points of stage s of N's plan, and of all stages before it.
__host__ __device__ constexpr int pair_rad(int n, int s) { return radix_seq(n).rad(s); }
__host__ __device__ constexpr int pair_ns(int n, int s)
{
    int p = 1;
    for (int i = 0; i < s; ++i) p *= pair_rad(n, i);
    return p;
}
// Butterflies of stage s per thread (16 points), points per thread, and threads
// per pencil pair.
__host__ __device__ constexpr int pair_k(int n, int s) { return 16 / pair_rad(n, s); }
__host__ __device__ constexpr int pair_rmax(int n)
{
    const RadixSeq q = radix_seq(n);
    int m = 0;
    for (int s = 0; s < q.nst; ++s) m = q.rad(s) * pair_k(n, s) > m ? q.rad(s) * pair_k(n, s) : m;
    return m;
}
__host__ __device__ constexpr int pair_tasks(int n)
{
    const RadixSeq q = radix_seq(n);
    int m = 0;
    for (int s = 0; s < q.nst; ++s) {
        const int t = (n / q.rad(s) + pair_k(n, s) - 1) / pair_k(n, s);
        m = t > m ? t : m;
    }
    return m;
}
__host__ __device__ constexpr int warps_up(int t) { return (t + 31) / 32 * 32; }
// Slots of one pencil pair in the exchange.
__host__ __device__ constexpr int pair_slots(int n) { return pair_rad(n, 0) % 2 == 0 ? n + n / pair_rad(n, 0) : n; }

// Pairs on neighbouring lanes: 16 / Q butterflies of each of the Q pairs make up
// a 16-lane access, so the pairs' slots start 16 / Q banks apart.
__host__ __device__ constexpr int pair_slots_q(int n, int q)
{
    int s = pair_slots(n);
    if (q > 1)
        while (s % 16 != 16 / q) ++s;
    return s;
}

// Twiddles e^{-2 pi i e / N} as (c, c, s, s).  Those of a radix R after NS points
// are e = jm r N / (NS R); radix 2 s is stage s's first, 2 s + 1 its second.
__host__ __device__ constexpr int tw_radix(int n, int l) { return l % 2 ? radix_seq(n).b[l / 2] : radix_seq(n).a[l / 2]; }
__host__ __device__ constexpr int tw_ns(int n, int l) { return pair_ns(n, l / 2) * (l % 2 ? radix_seq(n).a[l / 2] : 1); }
// TwAll: a shared-memory table of all N (pencil-fast tiles: the lanes of one
// butterfly read one entry).  TwRows: per radix rows r = 1 .. R-1 of NS
// entries, so neighbouring butterflies read neighbouring entries (line-major
// tiles).  TwGlobal: the plain table where it lies.
template <int N>
struct TwAll {
    const float4* tw;
    template <int L>
    __device__ __forceinline__ float4 at(int r, int jm) const
    {
        constexpr int TWS = N / (tw_ns(N, L) * tw_radix(N, L));
        return tw[jm * r * TWS];
    }
};
__host__ __device__ constexpr int tw_rows_off(int n, int l)
{
    int o = 0;
    for (int i = 1; i < l; ++i) o += (tw_radix(n, i) - 1) * tw_ns(n, i);
    return o;
}
__host__ __device__ constexpr int tw_rows_size(int n) { return tw_rows_off(n, 2 * radix_seq(n).nst); }
template <int N>
struct TwRows {
    const float4* tw;
    // fill the rows of radices L.. from the plain table, by all threads of a block of NT
    template <int NT, int L = 1>
    static __device__ __forceinline__ void fill(float4* s, const float2* g)
    {
        constexpr int R = tw_radix(N, L), NS = tw_ns(N, L), O = tw_rows_off(N, L), TWS = N / (NS * R);
        if constexpr (R > 1) {
#pragma unroll
            for (int i0 = 0; i0 < (R - 1) * NS; i0 += NT) {
                const unsigned i = i0 + threadIdx.x;
                if (i < (R - 1) * NS) {
                    const float2 w = __ldg(g + (i / NS + 1) * (i % NS) * TWS);
                    s[O + i] = make_float4(w.x, w.x, w.y, w.y);
                }
            }
        }
        if constexpr (L + 1 < 2 * radix_seq(N).nst) fill<NT, L + 1>(s, g);
    }
    template <int L>
    __device__ __forceinline__ float4 at(int r, int jm) const
    {
        constexpr int O = tw_rows_off(N, L), NS = tw_ns(N, L);
        return tw[O + (r - 1) * NS + jm];
    }
};
template <int N>
struct TwGlobal {
    const float2* tw;
    template <int L>
    __device__ __forceinline__ float4 at(int r, int jm) const
    {
        constexpr int TWS = N / (tw_ns(N, L) * tw_radix(N, L));
        const float2 w = __ldg(tw + jm * r * TWS);
        return make_float4(w.x, w.x, w.y, w.y);
    }
};

// N points, PP pencil pairs per block.  Q > 1 (line-major): Q neighbouring
// pairs on neighbouring lanes, for pencils that share memory lines.
template <int N, int PP, bool PF, int Q = 1>
struct PairFFT {
    static constexpr int NST = radix_seq(N).nst, LAST = NST - 1;
    static constexpr int R0 = pair_rad(N, 0), RL = pair_rad(N, LAST);
    static constexpr int K0 = pair_k(N, 0), KL = pair_k(N, LAST);
    static constexpr int T = pair_tasks(N);  // threads per pair
    static constexpr int RM = pair_rmax(N);  // points per thread

    static constexpr int SL = pair_slots_q(N, Q);
    static constexpr int PLANE = PP * SL;  // words of one plane
    static __device__ __forceinline__ void st(f2* b, c2 v)
    {
        b[0] = v.x;
        b[PLANE] = v.y;
    }
    static __device__ __forceinline__ c2 ld(const f2* b) { return c2{b[0], b[PLANE]}; }

    // Pair and first butterfly of a thread (the same in every stage: its
    // butterflies are j, j + T, ..); false for the threads past the last pair.
    static __device__ __forceinline__ bool task(int t, int& p, int& j)
    {
        const unsigned u = t;
        if constexpr (PF) { p = u % PP; j = u / PP; }
        else if constexpr (Q == 1) { p = u / T; j = u % T; }
        else { p = u / (Q * T) * Q + u % Q; j = u / Q % T; }
        return u < PP * T;
    }
    // f(m, j) for the thread's butterflies m = 0 .. K-1 of stage S
    template <int S, class F>
    static __device__ __forceinline__ void each(int j, F&& f)
    {
        constexpr int NR = N / pair_rad(N, S), K = pair_k(N, S);
#pragma unroll
        for (int m = 0; m < K; ++m)
            if ((m + 1) * T <= NR || j + m * T < NR) f(m, j + m * T);
    }
    // Points of a thread in registers: v[m R + r], butterfly m, index
    // j + m T + r N / R.  Whether stage 0 and the last one have the same ones,
    // in the order i = m + K r of their distance T.
    static constexpr bool SAME = T * K0 * R0 == N && T * KL * RL == N;

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
    static constexpr int dist() { return padded(N / pair_rad(N, S)) * STEP; }  // (use as a constant expression)

    // The butterfly of stage S, twiddled inputs in v.
    template <bool INV, int S, class Tw>
    static __device__ __forceinline__ void fly(const Tw& tw, int jm, c2* v)
    {
        constexpr RadixSeq q = radix_seq(N);
        dft_stage<q.a[S], q.b[S], INV>(v, [&](c2 u, int o, int r2) {
            if (S == 0 && o == 0) return u;
            const float4 w = tw.template at<2 * S + 1>(r2, jm + o * pair_ns(N, S));
            return cmul_tw<INV>(u, pack2(w.x, w.y), pack2(w.z, w.w));
        });
    }
    // Stage 0 on v (its points), written to the exchange.  The caller has loaded
    // v; the exchange must be free, and the twiddles there where SYNC0.
    static constexpr bool SYNC0 = radix_seq(N).b[0] > 1;  // stage 0 reads twiddles
    template <bool INV, class Tw>
    static __device__ __forceinline__ void first(const Tw& tw, f2* buf, int t, c2* v)
    {
        int p, j;
        if (!task(t, p, j)) return;
        each<0>(j, [&](int m, int i) {
            c2* u = v + m * R0;
            fly<INV, 0>(tw, 0, u);
            f2* b = buf + slot(p, i * R0);
#pragma unroll
            for (int r = 0; r < R0; ++r) st(b + r * STEP, u[r]);
        });
    }
    // Inputs of stage S >= 1, twiddled and transformed, left in v.
    template <bool INV, int S, class Tw>
    static __device__ __forceinline__ void take(const Tw& tw, const f2* buf, int t, c2* v)
    {
        constexpr int R = pair_rad(N, S), NS = pair_ns(N, S), D = dist<S>(), B = radix_seq(N).b[S];
        int p, j;
        if (!task(t, p, j)) return;
        each<S>(j, [&](int m, int i) {
            const int jm = (unsigned)i % NS;
            const f2* b = buf + slot(p, i);
            c2* u = v + m * R;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                u[r] = ld(b + r * D);
                if (r >= B) {
                    const float4 w = tw.template at<2 * S>(r / B, jm);
                    u[r] = cmul_tw<INV>(u[r], pack2(w.x, w.y), pack2(w.z, w.w));
                }
            }
            fly<INV, S>(tw, jm, u);
        });
    }
    template <int S>
    static __device__ __forceinline__ void put(f2* buf, int t, const c2* v)
    {
        constexpr int R = pair_rad(N, S), NS = pair_ns(N, S), D = padded(NS) * STEP;
        int p, j;
        if (!task(t, p, j)) return;
        each<S>(j, [&](int m, int i) {
            const int jm = (unsigned)i % NS;
            f2* b = buf + slot(p, (i - jm) * R + jm);
#pragma unroll
            for (int r = 0; r < R; ++r) st(b + r * D, v[m * R + r]);
        });
    }
    // From stage 0's outputs in the exchange (written, not yet synchronised)
    // to the last stage's outputs in v.
    template <bool INV, int S = 1, class Tw>
    static __device__ __forceinline__ void finish(const Tw& tw, f2* buf, int t, c2* v)
    {
        __syncthreads();
        take<INV, S>(tw, buf, t, v);
        if constexpr (S < LAST) {
            __syncthreads();
            put<S>(buf, t, v);
            finish<INV, S + 1>(tw, buf, t, v);
        }
    }
    // The last stage's outputs back to the slots of its inputs (index order;
    // every thread overwrites only its own).
    static __device__ __forceinline__ void keep(f2* buf, int t, const c2* v) { put<LAST>(buf, t, v); }
    // Stage 0's points of another transform from what keep() left.
    static __device__ __forceinline__ void pick(const f2* buf, int t, c2* v)
    {
        constexpr int NR = N / R0;
        int p, j;
        if (!task(t, p, j)) return;
        each<0>(j, [&](int m, int i) {
#pragma unroll
            for (int r = 0; r < R0; ++r) v[m * R0 + r] = ld(buf + slot(p, i + r * NR));
        });
    }
    // The last stage's outputs as stage 0's points.  Leaves the exchange in use:
    // synchronise before it is written.
    static __device__ __forceinline__ void turn(f2* buf, int t, c2* v)
    {
        if constexpr (SAME) {
            if constexpr (K0 != KL) {
                constexpr int E = K0 * R0;
                c2 w[E];
#pragma unroll
                for (int i = 0; i < E; ++i) w[i % K0 * R0 + i / K0] = v[i % KL * RL + i / KL];
#pragma unroll
                for (int i = 0; i < E; ++i) v[i] = w[i];
            }
        } else {
            keep(buf, t, v);
            __syncthreads();
            pick(buf, t, v);
        }
    }
};

}  // namespace qvti
