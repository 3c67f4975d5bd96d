// FP32 CUDA-core kernels: the plain path, the reference's arithmetic
// (crates/engine/src/cpu.rs) on the GPU. Token-level buffers are row-major
// [rows, features] over the rows of all instances of a launch; cell-level
// buffers are channel-last [cells, channels].
#pragma once

#include "common.cuh"

namespace jc {
namespace f32k {

// ---------------------------------------------------------------------------
// A-operand loaders of the tiled GEMM. `prologue` fills the CTA's shared
// memory with the rows' places in their grids (kCtx);
// `src(r, k, i, ctx)` is the address of A[r][k..k+3] (null: zeros), where i is
// the row's index in the tile; K and the loaders' channel counts are
// multiples of 4. kAligned = false: `src` may be on a 4-byte boundary only
// (copied by words).

struct NoCtx {};
struct GridCtx {
    int base;  // first row (token loader) or cell (cell loader) of the instance
    int y, x;  // coordinates inside the instance's grid
    int w, h;  // grid width and height
};

struct APlain {
    using Ctx = NoCtx;
    static constexpr bool kAligned = true, kCtx = false;
    const float* A;
    int lda, R, K;
    __device__ void prologue(int, int, Ctx*) const {}
    __device__ const float* src(int r, int k, int, const Ctx*) const {
        return r < R && k < K ? A + (size_t)r * lda + k : nullptr;
    }
};

// Patches of the state (cpu.rs:253-269), P a multiple of 4: feature
// k = c P P + py P + px of a token is a run of P cells of row py.
struct PatchCtx {
    const float* cell0;  // channel 0 of the patch's first cell; null past the last row
    int nx, inst;
    long long plane;
};
struct APatch {
    using Ctx = PatchCtx;
    static constexpr bool kAligned = false, kCtx = true;
    const InstDev* inst;
    int n_inst, R, K, P;
    __device__ void prologue(int row0, int bm, Ctx* ctx) const {
        for (int i = threadIdx.x; i < bm; i += blockDim.x) {
            const int r = row0 + i;
            PatchCtx c{nullptr, 0, 0, 0};
            if (r < R) {
                c.inst = inst_of_row(inst, n_inst, r);
                const InstDev& I = inst[c.inst];
                const int t = r - I.row0;
                c.nx = I.nx;
                c.plane = (long long)I.nx * I.ny;
                c.cell0 = I.state + (size_t)(t / I.tx) * P * I.nx + (size_t)(t % I.tx) * P;
            }
            ctx[i] = c;
        }
    }
    __device__ const float* src(int, int k, int i, const Ctx* ctx) const {
        const PatchCtx& c = ctx[i];
        if (!c.cell0 || k >= K) return nullptr;
        const int ch = k / (P * P), py = (k / P) % P, px = k % P;
        return c.cell0 + ch * c.plane + (size_t)py * c.nx + px;
    }
};

// 3x3 zero-padded cross-correlation (cpu.rs:171-205) as an implicit GEMM:
// A[r][tap*C + c] = X[neighbour(r, tap)][c], or 0 outside the grid; K = 9 C.
// CELL: rows are cells of each instance's cell grid, else tokens of its token
// grid; X is [rows, C].
template <bool CELL>
struct AConv3 {
    using Ctx = GridCtx;
    static constexpr bool kAligned = true, kCtx = true;
    const float* X;
    const InstDev* inst;
    int n_inst, R, C;
    __device__ void prologue(int row0, int bm, Ctx* ctx) const {
        for (int i = threadIdx.x; i < bm; i += blockDim.x) {
            const int r = row0 + i;
            GridCtx c{0, -100, -100, 0, 0};
            if (r < R) {
                const InstDev& I = inst[CELL ? inst_of_cell(inst, n_inst, r) : inst_of_row(inst, n_inst, r)];
                const int base = CELL ? (int)I.cell0 : I.row0, w = CELL ? I.nx : I.tx, h = CELL ? I.ny : I.ty;
                c = GridCtx{base, (r - base) / w, (r - base) % w, w, h};
            }
            ctx[i] = c;
        }
    }
    __device__ const float* src(int, int k, int i, const Ctx* ctx) const {
        const GridCtx& c = ctx[i];
        const int tap = k / C, ch = k - tap * C;
        const int y = c.y + tap / 3 - 1, x = c.x + tap % 3 - 1;
        if (tap >= 9 || y < 0 || x < 0 || y >= c.h || x >= c.w) return nullptr;
        return X + ((size_t)c.base + (size_t)y * c.w + x) * C + ch;
    }
};

// Epilogues: four consecutive outputs n..n+3 of row r, bias included; i is
// the row's index in the tile and ctx the loader's row contexts.
struct EStore {
    float* out;
    int ld;
    template <class Ctx>
    __device__ void operator()(int r, int n, float4 v, int, const Ctx*) const {
        *reinterpret_cast<float4*>(out + (size_t)r * ld + n) = v;
    }
};
__device__ __forceinline__ float4 gelu4(float4 v) {
    return make_float4(gelu_erf(v.x), gelu_erf(v.y), gelu_erf(v.z), gelu_erf(v.w));
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
struct EGelu {
    float* out;
    int ld;
    template <class Ctx>
    __device__ void operator()(int r, int n, float4 v, int, const Ctx*) const {
        *reinterpret_cast<float4*>(out + (size_t)r * ld + n) = gelu4(v);
    }
};
struct EResid {  // x += v (cpu.rs:306,312 add_inplace)
    float* x;
    int ld;
    template <class Ctx>
    __device__ void operator()(int r, int n, float4 v, int, const Ctx*) const {
        float4* p = reinterpret_cast<float4*>(x + (size_t)r * ld + n);
        *p = add4(*p, v);
    }
};
struct EGeluResidFrom {  // out = src + gelu(v) (cpu.rs:327-328)
    const float* src;
    float* out;
    int ld;
    template <class Ctx>
    __device__ void operator()(int r, int n, float4 v, int, const Ctx*) const {
        const size_t o = (size_t)r * ld + n;
        *reinterpret_cast<float4*>(out + o) = add4(*reinterpret_cast<const float4*>(src + o), gelu4(v));
    }
};
struct EEmbed {  // x = (v + pos) + meta linear (cpu.rs:270-280)
    const InstDev* inst;
    const float* Wm;
    const float* bm;
    int meta_dim, D;
    float* x;
    __device__ void operator()(int r, int n, float4 v, int i, const PatchCtx* ctx) const {
        const InstDev& I = inst[ctx[i].inst];
        float4 m = *reinterpret_cast<const float4*>(bm + n);
        for (int f = 0; f < meta_dim; f++) {
            const float4 w = *reinterpret_cast<const float4*>(Wm + (size_t)f * D + n);
            const float t = I.meta[f];
            m = make_float4(fmaf(t, w.x, m.x), fmaf(t, w.y, m.y), fmaf(t, w.z, m.z), fmaf(t, w.w, m.w));
        }
        const float4 p = *reinterpret_cast<const float4*>(I.pos + (size_t)(r - I.row0) * D + n);
        *reinterpret_cast<float4*>(x + (size_t)r * D + n) = add4(add4(v, p), m);
    }
};

// out[r][n] = epi(bias[n] + sum_k A[r][k] W[k][n]); W is [K, N] row-major
// (the checkpoint's Linear layout), N a multiple of 4.
//
// Arithmetic, the same for every tile shape, so that a row's result does not
// depend on how many rows the launch has: chain w (w < 4) is the fmaf chain
// from 0 over the k of the 16-wide groups w, w + 4, ... in order, and the
// result is (((bias + T0) + T1) + T2) + T3. The four chains run on separate
// warps and meet in shared memory: a quarter of the serial chain each.
//
// A warp owns 8 TM x 16 TN outputs of one chain: lane (lm = lane / 4, ln =
// lane % 4) the rows lm + 8 i and the columns 16 c + 4 ln... A rows lie
// K-contiguous with a pitch of KS + 4 floats, so the eight rows that a warp
// reads as float4s (4 k at once) fall on different banks; W rows lie as they
// come. Stages of KS = 64 columns arrive by asynchronous copies, NST - 1 of
// them in flight.
//
// What bounds it is shared-memory reads against FMAs: a thread reads
// TM / 4 + TN float4s per k for 4 TM TN FMAs (two to three wavefronts a
// read). ncu at 40 K rows, K = 512, N = 128: 4 x 4 a thread keeps the shared
// pipe at 77% and the FMA pipe at 56% (38 TFLOP/s).
//   4 x 4 (4 x 8) a thread, 32 x 16 (32 x 32) tiles: launches of few rows,
//     which cost the length of a CTA's K loop; more CTAs, a shorter loop body;
//   8 x 8 a thread, 64 x 32 tiles: large launches, half of the shared and of
//     the L2 reads per FMA (43-45 TFLOP/s; 8 x 4 a thread: 36-40).
template <int TM_, int TN_, int WM_, int WN_, int NST_>
struct Tile {
    static constexpr int TM = TM_, TN = TN_, WM = WM_, WN = WN_, NST = NST_, WK = 4;
    static constexpr int BM = 8 * TM * WM, BN = 16 * TN * WN, KG = 16, KS = KG * WK, NT = 32 * WM * WN * WK;
    static constexpr int PITCH = KS + 4;
    static constexpr int kStage = BM * PITCH + KS * BN;  // floats
    static size_t smem(int K) {  // as many stages as the K loop has, and room for the partial tiles
        const int stages = (K + KS - 1) / KS;
        const size_t a = (size_t)(stages < NST ? stages : NST) * kStage, b = (size_t)WK * BM * BN;
        return (a > b ? a : b) * 4;
    }
};

template <class T, class AL, class EP>
__global__ void __launch_bounds__(T::NT) gemm_kernel(AL aload, const float* __restrict__ W,
                                                     const float* __restrict__ bias, int R, int N, int K, EP epi) {
    constexpr int TM = T::TM, TN = T::TN, WN = T::WN, WK = T::WK, NST = T::NST;
    constexpr int BM = T::BM, BN = T::BN, KS = T::KS, NT = T::NT, PITCH = T::PITCH;
    extern __shared__ __align__(16) float gsm[];
    __shared__ typename AL::Ctx ctx[AL::kCtx ? BM : 1];
    const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nst = (K + KS - 1) / KS;
    constexpr int A4 = BM * KS / 4, B4 = KS * BN / 4;
    static_assert(A4 % NT == 0 && B4 % NT == 0, "stage copies");
    auto load_b = [&](int s) {
        float* dst = gsm + (size_t)(s % NST) * T::kStage + BM * PITCH;
#pragma unroll
        for (int q = 0; q < B4 / NT; q++) {
            const int e = tid + q * NT, kk = e / (BN / 4), j = (e % (BN / 4)) * 4;
            const bool in = s * KS + kk < K && col0 + j < N;
            cp_async16(dst + kk * BN + j, in ? W + (size_t)(s * KS + kk) * N + col0 + j : W, in);
        }
    };
    auto load_a = [&](int s) {
        float* dst = gsm + (size_t)(s % NST) * T::kStage;
#pragma unroll
        for (int u = 0; u < A4 / NT; u++) {
            const int e = tid + u * NT, i = e / (KS / 4), kk = (e % (KS / 4)) * 4;
            const float* p = aload.src(row0 + i, s * KS + kk, i, ctx);
            float* q = dst + i * PITCH + kk;
            if (AL::kAligned || (reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
                cp_async16(q, p ? p : W, p != nullptr);
            } else {
#pragma unroll
                for (int c = 0; c < 4; c++) cp_async4(q + c, p + c, true);
            }
        }
    };
    // the weights never change: their first stages start before the previous
    // kernel has finished
#pragma unroll
    for (int s = 0; s < NST - 1; s++)
        if (s < nst) load_b(s);
    JC_PDL_ENTRY;
    if (AL::kCtx) {
        aload.prologue(row0, BM, ctx);
        __syncthreads();
    }
#pragma unroll
    for (int s = 0; s < NST - 1; s++) {
        if (s < nst) load_a(s);
        cp_async_commit();
    }
    const int wk = warp % WK, wt = warp / WK, wn = wt % WN, wm = wt / WN;
    const int lm = lane >> 2, ln = lane & 3;
    float acc[TM][4 * TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int c = 0; c < 4 * TN; c++) acc[i][c] = 0.f;
    for (int s = 0; s < nst; s++) {
        cp_async_wait_group<NST - 2>();
        const float* As = gsm + (size_t)(s % NST) * T::kStage;
        __syncthreads();
        if (s + NST - 1 < nst) {
            load_b(s + NST - 1);
            load_a(s + NST - 1);
        }
        cp_async_commit();
        const float* a = As + (wm * 8 * TM + lm) * PITCH + wk * T::KG;
        const float* b = As + BM * PITCH + wk * T::KG * BN + wn * 16 * TN + 4 * ln;
        if (s * KS + wk * T::KG < K) {
            // unrolled twice only: most launches run the loop a few times, and
            // its instructions come from memory then (a 128 x 128 rollout's
            // ticks: 262 us unrolled four times, 245 us twice)
#pragma unroll 2
            for (int kk = 0; kk < T::KG; kk += 4) {
                float4 av[TM];
#pragma unroll
                for (int i = 0; i < TM; i++) av[i] = *reinterpret_cast<const float4*>(a + i * 8 * PITCH + kk);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    float4 bv[TN];
#pragma unroll
                    for (int c = 0; c < TN; c++) bv[c] = *reinterpret_cast<const float4*>(b + (kk + q) * BN + 16 * c);
#pragma unroll
                    for (int i = 0; i < TM; i++) {
                        const float x = q == 0 ? av[i].x : q == 1 ? av[i].y : q == 2 ? av[i].z : av[i].w;
#pragma unroll
                        for (int c = 0; c < TN; c++) {
                            fma2_f32(acc[i][4 * c], acc[i][4 * c + 1], x, x, bv[c].x, bv[c].y);
                            fma2_f32(acc[i][4 * c + 2], acc[i][4 * c + 3], x, x, bv[c].z, bv[c].w);
                        }
                    }
                }
            }
        }
    }
    cp_async_wait_all();
    __syncthreads();  // every warp is done with the stages: they take the four partial tiles
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int c = 0; c < TN; c++)
            *reinterpret_cast<float4*>(gsm + ((size_t)wk * BM + wm * 8 * TM + lm + 8 * i) * BN + wn * 16 * TN + 16 * c +
                                       4 * ln) =
                make_float4(acc[i][4 * c], acc[i][4 * c + 1], acc[i][4 * c + 2], acc[i][4 * c + 3]);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < BM * BN / 4 / NT; u++) {
        const int e = tid + u * NT, i = e / (BN / 4), j = (e % (BN / 4)) * 4, r = row0 + i;
        if (r >= R || col0 + j >= N) continue;
        float4 v = *reinterpret_cast<const float4*>(bias + col0 + j);
#pragma unroll
        for (int w = 0; w < WK; w++)
            v = add4(v, *reinterpret_cast<const float4*>(gsm + ((size_t)w * BM + i) * BN + j));
        epi(r, col0 + j, v, i, ctx);
    }
}

}  // namespace f32k
}  // namespace jc
