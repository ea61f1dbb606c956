// Shared by the translation units of the time-step kernels (k_velocity.cu,
// k_spectral.cu, k_sigma.cu, step_kernels.cu): small helpers, the compiled
// transform lengths and the launchers of the single kernels.  One unit per
// kernel family lets the compiled lengths build in parallel.
#pragma once
#include <cstdio>
#include <type_traits>

#include "engine.cuh"

namespace qvti {

constexpr int kThreads = 256;
constexpr int kEpi = 4;  // cells per thread and trip in the velocity-kernel epilogues

constexpr int kSigmaRows = 4;  // y rows per k_sigma tile (compile-time path)

// Element offsets fit in 32 bits: the engine accepts at most 1024^3 cells
// (qvti_create), and 32-bit offsets take one multiply-add per address.
__device__ __forceinline__ int cell(const KP& k, int x, int y, int z) { return (x * k.ny + y) * k.nz + z; }
__device__ __forceinline__ int spec(const KP& k, int kz, int x, int y) { return (kz * k.nx + x) * k.ny + y; }
__device__ __forceinline__ bool in_slab(int i, int n, int pml) { return i < pml || i >= n - pml; }

// One step of a C-PML memory variable q with the term d of its axis.
__device__ __forceinline__ float pml_step(float q, float dt, float a, float b, float d)
{
    return fmaf(dt, fmaf(-a, q, -(b * d)), q);
}

__device__ __forceinline__ void load_table(float2* s, const float2* g, int n)
{
    for (int i = threadIdx.x; i < n; i += blockDim.x) s[i] = g[i];
}

// Tile layouts of the runtime kernels in shared memory: pencil-fastest (for
// pencils that are adjacent in memory) or line-major, both with one padding row
// every 16 indices.
constexpr int kPencil = 1, kLinePad = 2;
template <int LY, bool INV, class Load, class Store>
__device__ __forceinline__ void fft_rt(const FftPlan& pl, const float2* tw, float2* A, float2* B, int pencils, int ps,
                                       int is, Load load, Store store)
{
    fft_run<LY == kPencil, INV>(pl, tw, A, B, pencils, ps, is, load, store, 4);
}

// Transform lengths with a compile-time path: the 5-smooth lengths the
// batching and serving workloads draw between 96 and 384, 512, and most other
// even 7-smooth lengths from 24 to 252 (of those above, 280, 294, 336, 350 and
// 378 are not listed); a kernel takes it when its transform length is listed,
// otherwise the runtime path.  The
// shortest lengths, below 36, come for k_vy, k_fz and k_cy only: the tile tests
// run the x kernels' runtime form at 32, and the stress update of so short a z
// axis was faster in its runtime form with 16 rows per block (32^3: 26 us) than
// as the compiled kernels' three launches (28) when both ran 32 as 8 4; as 16 2 the
// runtime form takes 31.
constexpr int kMinLong = 36;
//
// The lengths are split into QVTI_PARTS lists: each unit of compiled kernels is
// built once per list (QVTI_PART), in parallel.
#define QVTI_PARTS 4
#define QVTI_LENGTHS0(X) X(36) X(48) X(56) X(72) X(90) X(100) X(120) X(140) X(160) X(180) X(200) X(224) X(252) X(288) X(324)
#define QVTI_LENGTHS1(X) X(40) X(50) X(60) X(80) X(96) X(108) X(126) X(144) X(162) X(192) X(210) X(240) X(256) X(300) X(360)
#define QVTI_LENGTHS2(X) X(42) X(54) X(64) X(84) X(98) X(112) X(128) X(150) X(168) X(196) X(216) X(250) X(270) X(320) X(384)
#define QVTI_LENGTHS3(X) X(24) X(28) X(30) X(32) X(70) X(512)
#define QVTI_LENGTHS(X) QVTI_LENGTHS0(X) QVTI_LENGTHS1(X) QVTI_LENGTHS2(X) QVTI_LENGTHS3(X)
#define QVTI_ITEM(N) N,
inline constexpr int kCtLengths[] = {QVTI_LENGTHS(QVTI_ITEM)};

#ifdef QVTI_PART
#if QVTI_PART == 0
#define QVTI_MY_LENGTHS QVTI_LENGTHS0
#elif QVTI_PART == 1
#define QVTI_MY_LENGTHS QVTI_LENGTHS1
#elif QVTI_PART == 2
#define QVTI_MY_LENGTHS QVTI_LENGTHS2
#else
#define QVTI_MY_LENGTHS QVTI_LENGTHS3
#endif
static constexpr int kMyLengths[] = {QVTI_MY_LENGTHS(QVTI_ITEM)};
// f(integral_constant n) if n is one of this part's lengths (internal linkage,
// like the list: every part has its own).
template <class F>
static bool dispatch_len(int n, F&& f)
{
    switch (n) {
#define QVTI_CASE(N) \
    case N: f(std::integral_constant<int, N>{}); return true;
        QVTI_MY_LENGTHS(QVTI_CASE)
#undef QVTI_CASE
        default: return false;
    }
}
#endif

// A function of one part (explicitly specialised in that part's object), and
// its call on the part that has the length.
#define QVTI_DECLARE_PARTS(RET, NAME, ...) \
    template <int PART>                    \
    RET NAME(__VA_ARGS__);                 \
    template <>                            \
    RET NAME<0>(__VA_ARGS__);              \
    template <>                            \
    RET NAME<1>(__VA_ARGS__);              \
    template <>                            \
    RET NAME<2>(__VA_ARGS__);              \
    template <>                            \
    RET NAME<3>(__VA_ARGS__)
#define QVTI_CALL_PARTS(NAME, ...) \
    (NAME<0>(__VA_ARGS__) || NAME<1>(__VA_ARGS__) || NAME<2>(__VA_ARGS__) || NAME<3>(__VA_ARGS__))

// Threads of a runtime-length block: its butterflies, at most kThreads (short
// transforms would otherwise hold registers for threads without work).
inline int rt_threads(const FftPlan& p, int pencils)
{
    int m = 0;
    for (int s = 0; s < p.q.nst; ++s) m = p.n / p.q.rad(s) > m ? p.n / p.q.rad(s) : m;
    const int t = (m * pencils + 31) / 32 * 32;
    return t < kThreads ? t : kThreads;
}

inline int cdiv(int a, int b) { return (a + b - 1) / b; }

// y rows of a compiled k_mx block.
__host__ __device__ constexpr int mp_rows(int n) { return radix_seq(n).nst > 2 ? 8 : 16; }

// Lengths whose compiled stress kernels also come with eight rows: those of two
// stages (at three, 18 .. 40 threads a pencil pair, eighteen pairs are a block of
// up to 720 threads, and its exchange most of an SM's shared memory).
__host__ __device__ constexpr bool st_eight_rows(int n) { return radix_seq(n).nst == 2; }

// One kernel of the step: tile `P`, rt = the runtime-length kernel.
void launch_vy(const KP& k, int P, bool rt, cudaStream_t st);
void launch_vx(const KP& k, int P, bool rt, cudaStream_t st);
void launch_fz(const KP& k, int P, bool rt, int ncomp, cudaStream_t st);
void launch_cy(const KP& k, int L, bool rt, bool inv, int nfield, bool ydv, long long line0, long long line_end,
               cudaStream_t st);
void launch_mx(const KP& k, int P, bool rt, int kz0, int nb, cudaStream_t st);
void launch_sigma(const KP& k, int P, bool rt, cudaStream_t st);
// Their dynamic shared memory (bytes).
size_t smem_vyx(int n, int P, bool rt);
size_t smem_fz(const KP& k, int P, bool rt);
size_t smem_cy(const KP& k, int L, bool ydv, bool rt);
size_t smem_mx(const KP& k, int P, bool rt);
size_t smem_sigma(const KP& k, int P, bool rt);
// Load kernels and raise their dynamic shared-memory limit: the runtime forms
// (axis < 0), or the compiled ones that transform axis 0 (x), 1 (y) or 2 (z) at
// length n; cudaError_t.
cudaError_t configure_velocity(int axis, int n);
cudaError_t configure_spectral(int axis, int n);
cudaError_t configure_sigma(int axis, int n);

// cudaFuncSetAttribute over kernels, keeping the last error.
struct SmemLimit {
    cudaError_t e = cudaSuccess;
    void set(const void* f)
    {
        const cudaError_t r = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
        if (r != cudaSuccess) e = r;
    }
};

}  // namespace qvti
