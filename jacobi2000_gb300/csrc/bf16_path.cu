// BF16 tensor-core forward path (sm_103a).
//
// Per tick and model group (crates/engine/src/cpu.rs:249-352 restated):
//   embed (CUDA cores)      patchify + embed + pos + meta -> x (f32), LN1(x) (bf16)
//   per layer:
//     qkv   (tcgen05 GEMM)  LN1(x) @ Wqkv + b                      -> qkv (bf16)
//     attention (CUDA cores) stencil-masked softmax over <= (2r+1)^2 keys -> attn (bf16)
//     proj  (tcgen05 GEMM)  x += attn @ Wp + b; LN2(x)             -> x (f32), LN2(x) (bf16)
//     mlp   (tcgen05, fused) x += gelu(LN2(x) @ W1 + b1) @ W2 + b2; LN(x) for the next step
//                           (at dim 128 one kernel with proj)
//   token_mix (tcgen05 conv) t1 = xn + gelu(conv3x3(xn) + b)        (bf16)
//   to_cells (tcgen05 GEMM) z0 = t1 @ Wtc + b                      (f32; one kernel
//                           with token_mix at dims up to 128)
//   upsample (CUDA cores)   zc = [upsample(z0), state]             (f16, 48 channels)
//   conv1 (tcgen05 conv)    c1 = gelu(conv3x3(zc) + b)             (f16)
//   conv2 + step (tcgen05 conv) next = state + conv3x3(c1) + b     (f32)
// The 3x3 convolutions are implicit GEMMs without an im2col copy: a halo tile
// (10 x 18 positions, all channels) is loaded once in the no-swizzle core-matrix
// layout and each of the 9 taps is the same tile addressed through a shifted
// shared-memory descriptor (conv2, with 3 outputs, is one GEMM over the halo whose
// 27 columns are then added up).
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <stdexcept>
#include <string>

#include "bf16_path.hpp"
#include "launch.hpp"
#include "tc.cuh"

namespace jc {

typedef __nv_bfloat16 bf16;

static void check_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

// ---------------------------------------------------------------------------
// host: bf16 conversion and tensor maps

static uint16_t f2bf(float f) {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    if ((u & 0x7fffffffu) > 0x7f800000u) return (uint16_t)((u >> 16) | 0x40);  // NaN stays NaN
    u += 0x7fffu + ((u >> 16) & 1u);  // round to nearest even
    return (uint16_t)(u >> 16);
}

// f32 -> IEEE binary16 bits, round to nearest even (host)
static uint16_t f2h(float f) {
    const __half h = __float2half_rn(f);
    uint16_t u;
    std::memcpy(&u, &h, 2);
    return u;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        cuda_check(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q),
                   "cuTensorMapEncodeTiled entry point");
        if (q != cudaDriverEntryPointSuccess || !p) throw Error(JC_CUDA_ERROR, "cuTensorMapEncodeTiled unavailable");
        fn = (EncodeTiledFn)p;
    }
    return fn;
}

// Tensor of `rank` dims (innermost first), strides in bytes of dims
// 1..rank-1, box dims; bf16 and no swizzle unless given; zero fill out of
// bounds.
static CUtensorMap make_map(const void* base, int rank, const uint64_t* dims, const uint64_t* strides,
                            const uint32_t* box, CUtensorMapDataType type = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                            CUtensorMapSwizzle swz = CU_TENSOR_MAP_SWIZZLE_NONE) {
    CUtensorMap m;
    cuuint64_t gd[5], gs[4];
    cuuint32_t bx[5], es[5];
    for (int i = 0; i < rank; i++) {
        gd[i] = dims[i];
        bx[i] = box[i];
        es[i] = 1;
    }
    for (int i = 0; i < rank - 1; i++) gs[i] = strides[i];
    CUresult r = encode_fn()(&m, type, rank, const_cast<void*>(base), gd, gs, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             swz,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw Error(JC_CUDA_ERROR, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
    return m;
}

// Rows of a [rows, cols] bf16 matrix, loaded as 8-column x 128-row boxes.
static CUtensorMap rows_map(const void* base, int cols, int rows) {
    uint64_t dims[2] = {(uint64_t)cols, (uint64_t)(rows > 0 ? rows : 1)};
    uint64_t strides[1] = {(uint64_t)cols * 2};
    uint32_t box[2] = {8, 128};
    return make_map(base, 2, dims, strides, box);
}

// Output tiles of a [rows, cols] matrix with row pitch `ld` elements (bf16,
// or f32 when f32): boxes of 128 bytes x 128 rows, stored from shared memory
// in the 128-byte swizzled layout (16-byte chunk j of tile row r at chunk
// j ^ (r % 8)).
static CUtensorMap store_map(const void* base, int cols, int rows, int ld, bool f32) {
    const int es = f32 ? 4 : 2;
    uint64_t dims[2] = {(uint64_t)cols, (uint64_t)(rows > 0 ? rows : 1)};
    uint64_t strides[1] = {(uint64_t)ld * es};
    uint32_t box[2] = {(uint32_t)(128 / es), 128};
    return make_map(base, 2, dims, strides, box, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                    CU_TENSOR_MAP_SWIZZLE_128B);
}

// Rows of a [rows, cols] f32 matrix, moved as 16-column x 128-row boxes.
static CUtensorMap resid_map(const void* base, int cols, int rows) {
    uint64_t dims[2] = {(uint64_t)cols, (uint64_t)(rows > 0 ? rows : 1)};
    uint64_t strides[1] = {(uint64_t)cols * 4};
    uint32_t box[2] = {16, 128};
    return make_map(base, 2, dims, strides, box, CU_TENSOR_MAP_DATA_TYPE_FLOAT32);
}

// One instance's [ny, nx, C] channel-last grid (bf16, or f32 when f32),
// stored as 128-byte x 8 x 16 boxes (one 8 x 16 conv tile, 128 bytes of
// channels) from 128-byte swizzled shared memory; positions outside the grid
// are not written.
static CUtensorMap tile_store_map(const void* base, int C, int nx, int ny, bool f32) {
    const int es = f32 ? 4 : 2;
    uint64_t dims[3] = {(uint64_t)C, (uint64_t)nx, (uint64_t)ny};
    uint64_t strides[2] = {(uint64_t)C * es, (uint64_t)nx * C * es};
    uint32_t box[3] = {(uint32_t)(128 / es), kConvTX, kConvTY};
    return make_map(base, 3, dims, strides, box, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                    CU_TENSOR_MAP_SWIZZLE_128B);
}

// One instance's plane-major f16 cell-head grid: `planes` planes of
// [ny][nx][8 channels], `plane` bytes apart, seen as a [planes][ny][nx * 8]
// tensor, so each box row is a run of whole positions (one 16-byte chunk
// each) and a box of a conv tile moves in a few long rows instead of one
// 16-byte row per position. Halo loads: 10 x 18 positions of every plane
// from element (x0 - 1) * 8 (a 16-byte boundary; the fill covers the grid's
// edges), landing as [planes][18][10][8].
static CUtensorMap cell_plane_map(const void* base, int planes, long long plane, int nx, int ny) {
    uint64_t dims[3] = {(uint64_t)nx * 8, (uint64_t)ny, (uint64_t)planes};
    uint64_t strides[2] = {(uint64_t)nx * 16, (uint64_t)plane};
    uint32_t box[3] = {(uint32_t)(kConvTX + 2) * 8, (uint32_t)kConvTY + 2, (uint32_t)planes};
    return make_map(base, 3, dims, strides, box, CU_TENSOR_MAP_DATA_TYPE_FLOAT16);
}

// One instance's qkv rows as a [ty, tx, 3D] grid, loaded as 64-channel boxes
// of side x side tokens in the 128-byte swizzled layout (attention tiles).
static CUtensorMap att_map(const void* base, int D, int tx, int ty, int side) {
    uint64_t dims[3] = {(uint64_t)(3 * D), (uint64_t)tx, (uint64_t)ty};
    uint64_t strides[2] = {(uint64_t)3 * D * 2, (uint64_t)tx * 3 * D * 2};
    uint32_t box[3] = {64, (uint32_t)side, (uint32_t)side};
    return make_map(base, 3, dims, strides, box, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, CU_TENSOR_MAP_SWIZZLE_128B);
}

// One instance's [ny, nx, C] channel-last grid, loaded as 8-channel x 10 x 18 halo boxes.
static CUtensorMap halo_map(const void* base, int C, int nx, int ny) {
    uint64_t dims[3] = {(uint64_t)C, (uint64_t)nx, (uint64_t)ny};
    uint64_t strides[2] = {(uint64_t)C * 2, (uint64_t)nx * C * 2};
    uint32_t box[3] = {8, kConvTX + 2, kConvTY + 2};
    return make_map(base, 3, dims, strides, box);
}

// ---------------------------------------------------------------------------
// device

// Cell-head input channels (f16, conv1's operand type; f16 keeps 3 more
// mantissa bits than bf16 and the values are far inside its range): 32 z,
// then the state split exactly into f16 parts, s = hi + lo: [hi (3), lo (3),
// hi (3)] multiplied by the conv1 weights [W_hi, W_hi, W_lo], so the state
// enters conv1 with ~22-bit precision; the remaining 7 channels are zero.
constexpr int kZcCh = 48;
constexpr int kZcState = 32;
constexpr int kHaloW = kConvTX + 2, kHaloH = kConvTY + 2;
// bytes of one 8-channel plane of a halo tile (2880 used), padded so every
// plane starts on a 128-byte boundary for TMA (token-level halos, one load
// per plane)
constexpr int kHaloPlane = (kHaloW * kHaloH * 16 + 127) / 128 * 128;
// one 8-channel plane of a cell-level halo tile, loaded with every other
// plane by one TMA box (planes packed)
constexpr int kCellPlane = kHaloW * kHaloH * 16;

__device__ __forceinline__ float bf2f(bf16 v) { return __bfloat162float(v); }

// Token embedding and the first LayerNorm (cpu.rs:253-280, 289). Persistent
// CTAs walk tiles of 8 RW token rows: the embed weights [pd][D] are staged in
// shared memory once per CTA, and each tile's patches arrive as 16-byte
// asynchronous copies (one per (row, channel, patch row): 4 cells), double-
// buffered so the next tile's patches are in flight while this one is
// summed. Patches sit as [channel, patch row][row][4] floats. Warp w owns
// RW rows from RW w and lane l owns the CPL = D/32 consecutive outputs
// [CPL l, CPL l + CPL): per group of 4 patch elements it reads RW patch
// float4s and 4 x CPL weights and does 4 x RW x CPL FMAs. Each output is summed in
// the reference's order (bias, then the patch elements in order, then + pos,
// + the meta linear); x is written f32 and LayerNorm(x) bf16, with vector
// stores. The pos rows of a warp's rows are loaded together before the
// LayerNorms, and the meta linear is kept while the instance stays the same
// (across tiles too).
constexpr int kEmbedGroups = 12;  // 3 channels x 4 patch rows, 4 patch columns each

__host__ __device__ constexpr size_t embed_smem(int D, int rows) {
    return ((size_t)48 * D + 2 * (size_t)kEmbedGroups * rows * 4) * sizeof(float);
}

template <int CPL, int RW>
__global__ void __launch_bounds__(256, (CPL <= 4 ? 3 : 1)) bf_embed_kernel(Dims d, const float* __restrict__ We,
                                                       const float* __restrict__ be, const float* __restrict__ Wm,
                                                       const float* __restrict__ bm, const float* __restrict__ g,
                                                       const float* __restrict__ b, const InstDev* inst, int n_inst,
                                                       int R, float* __restrict__ x, bf16* __restrict__ ln) {
    extern __shared__ __align__(16) float esm[];
    constexpr int D = 32 * CPL, kRows = 8 * RW;
    constexpr int P = 4, pd = 3 * P * P;  // 3 channels, patch 4 (checked when the path is built)
    float* sW = esm;                      // [pd][D]
    float4* sP = reinterpret_cast<float4*>(esm + (size_t)pd * D);  // 2 x [groups][kRows] float4
    __shared__ int rinst[2][kRows];
    const int n_tiles = (R + kRows - 1) / kRows;
    for (int i = threadIdx.x; i < pd * D / 4; i += blockDim.x)
        cp_async16(reinterpret_cast<float4*>(sW) + i, reinterpret_cast<const float4*>(We) + i, true);
    JC_PDL_ENTRY;  // the weights do not wait for the previous kernel
    // the patches of tile t into buffer `buf` (and each row's instance); with
    // 256 threads, a multiple of the tile's rows, a thread copies the patches
    // of one row (threadIdx.x % kRows), so it finds that row's instance once
    static_assert(256 % kRows == 0, "embed copy layout");
    auto issue = [&](int t, int buf) {
        const int i = threadIdx.x % kRows, r = t * kRows + i;
        // a warp's rows are consecutive: the instance of its first row by a
        // warp-wide search, then at most a step or two per lane
        int ii = warp_find_last_le(n_inst, __shfl_sync(0xffffffffu, r, 0), [&](int k) { return (long long)inst[k].row0; });
        while (ii + 1 < n_inst && inst[ii + 1].row0 <= r) ii++;
        if (r >= R) ii = -1;
        for (int e = threadIdx.x; e < kRows * kEmbedGroups; e += blockDim.x) {
            const int gq = e / kRows;  // (channel, patch row)
            if (gq == 0) rinst[buf][i] = ii;
            const float* src = We;
            if (ii >= 0) {
                const InstDev& I = inst[ii];
                const int tk = r - I.row0, c = gq / P, py = gq % P;
                src = I.state + (size_t)c * I.nx * I.ny + ((size_t)(tk / I.tx) * P + py) * I.nx +
                      (size_t)(tk % I.tx) * P;
            }
            cp_async16(sP + ((size_t)buf * kEmbedGroups + gq) * kRows + i, src, ii >= 0);
        }
        cp_async_commit();
    };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i0 = warp * RW;  // this warp's RW rows
    const int o0 = CPL * lane;
    int k = 0;
    int m_inst = -1;  // the instance whose meta linear m holds
    float m[CPL];
    if ((int)blockIdx.x < n_tiles) issue(blockIdx.x, 0);
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x, k++) {
        const int buf = k & 1;
        if (t + (int)gridDim.x < n_tiles) {
            issue(t + gridDim.x, buf ^ 1);
            cp_async_wait_group<1>();
        } else {
            cp_async_wait_group<0>();
        }
        __syncthreads();
        const int r0 = t * kRows;
        if (r0 + i0 < R) {
            float v[RW][CPL];
#pragma unroll
            for (int q = 0; q < RW; q++)
#pragma unroll
                for (int c = 0; c < CPL; c++) v[q][c] = be[o0 + c];
            const float4* pb = sP + (size_t)buf * kEmbedGroups * kRows + i0;
#pragma unroll 2
            for (int gq = 0; gq < kEmbedGroups; gq++) {
                float4 p4[RW];
#pragma unroll
                for (int q = 0; q < RW; q++) p4[q] = pb[gq * kRows + q];
#pragma unroll
                for (int px = 0; px < 4; px++) {
                    const int f = gq * 4 + px;
                    float wv[CPL];
                    if (CPL % 4 == 0) {
#pragma unroll
                        for (int c = 0; c < CPL; c += 4) {
                            const float4 w4 = *reinterpret_cast<const float4*>(sW + f * D + o0 + c);
                            wv[c] = w4.x; wv[c + 1] = w4.y; wv[c + 2] = w4.z; wv[c + 3] = w4.w;
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < CPL; c++) wv[c] = sW[f * D + o0 + c];
                    }
#pragma unroll
                    for (int q = 0; q < RW; q++) {
                        const float pv = px == 0 ? p4[q].x : px == 1 ? p4[q].y : px == 2 ? p4[q].z : p4[q].w;
                        if (CPL % 2 == 0) {
#pragma unroll
                            for (int c = 0; c < CPL; c += 2) fma2_f32(v[q][c], v[q][c + 1], pv, pv, wv[c], wv[c + 1]);
                        } else {
#pragma unroll
                            for (int c = 0; c < CPL; c++) v[q][c] = fmaf(pv, wv[c], v[q][c]);
                        }
                    }
                }
            }
            // + pos for the warp's rows, the loads of all rows in flight together
            int rii[RW];
#pragma unroll
            for (int q = 0; q < RW; q++) {
                const int r = r0 + i0 + q;
                rii[q] = r < R ? rinst[buf][i0 + q] : -1;
                if (rii[q] >= 0) {
                    const InstDev& I = inst[rii[q]];
                    const float* pos = I.pos + (size_t)(r - I.row0) * D + o0;
                    if (CPL % 4 == 0) {
#pragma unroll
                        for (int c = 0; c < CPL; c += 4) {
                            const float4 p4 = *reinterpret_cast<const float4*>(pos + c);
                            v[q][c] += p4.x; v[q][c + 1] += p4.y; v[q][c + 2] += p4.z; v[q][c + 3] += p4.w;
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < CPL; c++) v[q][c] += pos[c];
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < RW; q++) {
                const int r = r0 + i0 + q;
                if (r >= R) continue;  // warp-uniform
                const int ii = rii[q];
                if (ii != m_inst) {
                    // the meta linear depends only on the instance: computed
                    // again only where the instance changes (kept across tiles)
                    const InstDev& I = inst[ii];
                    m_inst = ii;
#pragma unroll
                    for (int c = 0; c < CPL; c++) {
                        m[c] = bm[o0 + c];
                        for (int f = 0; f < d.meta_dim; f++) m[c] = fmaf(I.meta[f], Wm[(size_t)f * D + o0 + c], m[c]);
                    }
                }
                float sum = 0.f;
#pragma unroll
                for (int c = 0; c < CPL; c++) {
                    v[q][c] = v[q][c] + m[c];
                    sum += v[q][c];
                }
                const float mean = warp_sum(sum) / (float)D;
                float sq = 0.f;
#pragma unroll
                for (int c = 0; c < CPL; c++) sq += (v[q][c] - mean) * (v[q][c] - mean);
                const float rstd = rsqrtf(warp_sum(sq) / (float)D + 1e-5f);  // 2 ulp
                float o[CPL];
#pragma unroll
                for (int c = 0; c < CPL; c++) o[c] = (v[q][c] - mean) * rstd * g[o0 + c] + b[o0 + c];
                float* xr = x + (size_t)r * D + o0;
                bf16* lr = ln + (size_t)r * D + o0;
                if (CPL % 4 == 0) {
#pragma unroll
                    for (int c = 0; c < CPL; c += 4) {
                        *reinterpret_cast<float4*>(xr + c) = make_float4(v[q][c], v[q][c + 1], v[q][c + 2], v[q][c + 3]);
                        __nv_bfloat162 lo = __floats2bfloat162_rn(o[c], o[c + 1]);
                        __nv_bfloat162 hi = __floats2bfloat162_rn(o[c + 2], o[c + 3]);
                        uint2 u;
                        u.x = *reinterpret_cast<uint32_t*>(&lo);
                        u.y = *reinterpret_cast<uint32_t*>(&hi);
                        *reinterpret_cast<uint2*>(lr + c) = u;
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < CPL; c++) {
                        xr[c] = v[q][c];
                        lr[c] = __float2bfloat16(o[c]);
                    }
                }
            }
        }
        __syncthreads();  // every warp is done with `buf` before it is refilled
    }
    cp_async_wait_group<0>();
}

// Packed bf16 vectors of 1, 4 or 8 elements <-> f32.
template <int FPL>
struct BfVec;
template <>
struct BfVec<1> {
    __device__ static void load(const bf16* p, float* o) { o[0] = bf2f(p[0]); }
    __device__ static void store(bf16* p, const float* o) { p[0] = __float2bfloat16(o[0]); }
};
template <>
struct BfVec<4> {
    __device__ static void load(const bf16* p, float* o) {
        uint2 u = *reinterpret_cast<const uint2*>(p);
        __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&u.x), b = *reinterpret_cast<__nv_bfloat162*>(&u.y);
        float2 fa = __bfloat1622float2(a), fb = __bfloat1622float2(b);
        o[0] = fa.x; o[1] = fa.y; o[2] = fb.x; o[3] = fb.y;
    }
    __device__ static void store(bf16* p, const float* o) {
        __nv_bfloat162 a = __floats2bfloat162_rn(o[0], o[1]), b = __floats2bfloat162_rn(o[2], o[3]);
        uint2 u;
        u.x = *reinterpret_cast<uint32_t*>(&a);
        u.y = *reinterpret_cast<uint32_t*>(&b);
        *reinterpret_cast<uint2*>(p) = u;
    }
};
template <>
struct BfVec<8> {
    __device__ static void load(const bf16* p, float* o) {
        uint4 u = *reinterpret_cast<const uint4*>(p);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&w[i]);
            float2 f = __bfloat1622float2(h);
            o[2 * i] = f.x;
            o[2 * i + 1] = f.y;
        }
    }
    __device__ static void store(bf16* p, const float* o) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            __nv_bfloat162 h = __floats2bfloat162_rn(o[2 * i], o[2 * i + 1]);
            w[i] = *reinterpret_cast<uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    }
};

// One thread per (token row, head): the head's query stays in registers and
// every dot product and weighted sum runs serially in the thread, so no
// shuffles are needed; the threads of one row read the key and value rows of
// a candidate as consecutive 16-byte pieces. Radius-1 stencil (any dilation):
// scores, max, exp, denominator and the (e / denom)-weighted sum in the
// reference's order (cpu.rs:121-158); a general stencil or the full mask uses
// the online (running max) form.
template <int HD>
__device__ __forceinline__ void load_head(const bf16* p, float* f) {
#pragma unroll
    for (int w = 0; w < HD / 8; w++) {
        const uint4 u = reinterpret_cast<const uint4*>(p)[w];
        const uint32_t a[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            f[8 * w + 2 * i] = __uint_as_float(a[i] << 16);
            f[8 * w + 2 * i + 1] = __uint_as_float(a[i] & 0xffff0000u);
        }
    }
}

template <int HD>
__device__ __forceinline__ float dot_head(const float* q, const bf16* kp) {
    float p0 = 0.f, p1 = 0.f;
#pragma unroll
    for (int w = 0; w < HD / 8; w++) {
        const uint4 u = reinterpret_cast<const uint4*>(kp)[w];
        const uint32_t a[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            p0 = fmaf(q[8 * w + 2 * i], __uint_as_float(a[i] << 16), p0);
            p1 = fmaf(q[8 * w + 2 * i + 1], __uint_as_float(a[i] & 0xffff0000u), p1);
        }
    }
    return p0 + p1;
}

template <int HD>
__device__ __forceinline__ void axpy_head(float wgt, const bf16* vp, float* acc) {
#pragma unroll
    for (int w = 0; w < HD / 8; w++) {
        const uint4 u = reinterpret_cast<const uint4*>(vp)[w];
        const uint32_t a[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            acc[8 * w + 2 * i] = fmaf(wgt, __uint_as_float(a[i] << 16), acc[8 * w + 2 * i]);
            acc[8 * w + 2 * i + 1] = fmaf(wgt, __uint_as_float(a[i] & 0xffff0000u), acc[8 * w + 2 * i + 1]);
        }
    }
}

template <int HD>
__device__ __forceinline__ void store_head(bf16* p, const float* acc) {
#pragma unroll
    for (int w = 0; w < HD / 8; w++) BfVec<8>::store(p + 8 * w, acc + 8 * w);
}

template <int HD>
__global__ void __launch_bounds__(256) bf_attn_head_r1_kernel(Dims d, const bf16* __restrict__ qkv,
                                                              const InstDev* inst, int n_inst, int R,
                                                              bf16* __restrict__ out) {
    JC_PDL_ENTRY;
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = gid / d.heads, h = gid - r * d.heads;
    if (r >= R) return;
    const int D = d.D;
    const size_t D3 = 3 * (size_t)D;
    const InstDev& I = inst[inst_of_row(inst, n_inst, r)];
    const int t = r - I.row0, qy = t / I.tx, qx = t - qy * I.tx, dil = d.dilation;
    const float scale = 1.0f / sqrtf((float)HD);
    float q[HD];
    load_head<HD>(qkv + (size_t)r * D3 + h * HD, q);
    float sc[9];
    int kr[9];
    float smax = -INFINITY;
#pragma unroll
    for (int j = 0; j < 9; j++) {
        const int ky = qy + (j / 3 - 1) * dil, kx = qx + (j % 3 - 1) * dil;
        const bool in = ky >= 0 && kx >= 0 && ky < I.ty && kx < I.tx;
        kr[j] = in ? I.row0 + ky * I.tx + kx : -1;
        sc[j] = in ? dot_head<HD>(q, qkv + (size_t)kr[j] * D3 + D + h * HD) * scale : -INFINITY;
        smax = fmaxf(smax, sc[j]);
    }
    float denom = 0.f;
#pragma unroll
    for (int j = 0; j < 9; j++) {
        sc[j] = kr[j] >= 0 ? __expf(sc[j] - smax) : 0.f;
        denom += sc[j];
    }
    const float inv = 1.0f / denom;
    float acc[HD];
#pragma unroll
    for (int i = 0; i < HD; i++) acc[i] = 0.f;
#pragma unroll
    for (int j = 0; j < 9; j++)
        if (kr[j] >= 0) axpy_head<HD>(sc[j] * inv, qkv + (size_t)kr[j] * D3 + 2 * D + h * HD, acc);
    store_head<HD>(out + (size_t)r * D + h * HD, acc);
}

template <int HD>
__global__ void __launch_bounds__(256) bf_attn_head_kernel(Dims d, const bf16* __restrict__ qkv, const InstDev* inst,
                                                           int n_inst, int R, bf16* __restrict__ out) {
    JC_PDL_ENTRY;
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = gid / d.heads, h = gid - r * d.heads;
    if (r >= R) return;
    const int D = d.D;
    const size_t D3 = 3 * (size_t)D;
    const InstDev& I = inst[inst_of_row(inst, n_inst, r)];
    const int t = r - I.row0, qy = t / I.tx, qx = t - qy * I.tx;
    const float scale = 1.0f / sqrtf((float)HD);
    float q[HD], acc[HD];
    load_head<HD>(qkv + (size_t)r * D3 + h * HD, q);
#pragma unroll
    for (int i = 0; i < HD; i++) acc[i] = 0.f;
    const int side = 2 * d.radius + 1;
    const int nc = d.mask_kind == 0 ? I.tx * I.ty : side * side;
    float m = -INFINITY, l = 0.f;
    for (int j = 0; j < nc; j++) {
        int kr;
        if (d.mask_kind == 0) {
            kr = I.row0 + j;
        } else {
            const int ky = qy + (j / side - d.radius) * d.dilation, kx = qx + (j % side - d.radius) * d.dilation;
            if (ky < 0 || kx < 0 || ky >= I.ty || kx >= I.tx) continue;
            kr = I.row0 + ky * I.tx + kx;
        }
        const float s = dot_head<HD>(q, qkv + (size_t)kr * D3 + D + h * HD) * scale;
        const float mn = fmaxf(m, s);
        const float c = __expf(m - mn), e = __expf(s - mn);
        l = l * c + e;
#pragma unroll
        for (int i = 0; i < HD; i++) acc[i] *= c;
        axpy_head<HD>(e, qkv + (size_t)kr * D3 + 2 * D + h * HD, acc);
        m = mn;
    }
    const float inv = 1.0f / l;
#pragma unroll
    for (int i = 0; i < HD; i++) acc[i] *= inv;
    store_head<HD>(out + (size_t)r * D + h * HD, acc);
}

// Radius-1, dilation-1 stencil attention over shared-memory tiles (cpu.rs:
// 97-164, mask.rs:18-30). A CTA takes one 8 x 8 block of an instance's token
// grid (half of an 8 x 16 conv tile) for the heads of one 64-channel box:
// TMA brings the block's queries and the keys and values of its 10 x 10 halo
// for those channels into shared memory as 128-byte swizzled boxes (zero fill
// outside the grid, where the mask excludes the candidates anyway); 34 KB per
// CTA keeps six CTAs on an SM. Thread (token, head) then does the
// arithmetic of bf_attn_head_r1_kernel, in the same order, on shared-memory
// operands: the eight lanes of a quarter warp are eight neighbouring tokens
// of one head, so the swizzle spreads their 16-byte reads over all banks.
constexpr int kAttTile = 8;                        // tokens per side of a CTA's block
constexpr int kAttHalo = kAttTile + 2;             // halo side
constexpr int kAttBoxKV = kAttHalo * kAttHalo * 128;   // one 64-channel halo box: 12800 bytes
constexpr int kAttBoxKVPad = 13 * 1024;                // 1024-aligned slot of one halo box
constexpr int kAttBoxQ = kAttTile * kAttTile * 128;    // one 64-channel query box: 8192 bytes

// 16-byte chunk c (0..7) of row rho of a 128-byte swizzled box
__device__ __forceinline__ const uint4* swz_chunk(const uint8_t* box, int rho, int c) {
    return reinterpret_cast<const uint4*>(box + (size_t)rho * 128 + ((c ^ (rho & 7)) << 4));
}

template <int HD>
__device__ __forceinline__ void axpy_head_s(float wgt, const uint8_t* boxes, int box_stride, int rho, int ch0,
                                            float* acc) {
#pragma unroll
    for (int w = 0; w < HD / 8; w++) {
        const int ch = ch0 + 8 * w;
        const uint4 u = *swz_chunk(boxes + (size_t)(ch >> 6) * box_stride, rho, (ch & 63) >> 3);
        const uint32_t a[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            acc[8 * w + 2 * i] = fmaf(wgt, __uint_as_float(a[i] << 16), acc[8 * w + 2 * i]);
            acc[8 * w + 2 * i + 1] = fmaf(wgt, __uint_as_float(a[i] & 0xffff0000u), acc[8 * w + 2 * i + 1]);
        }
    }
}

// lo += a.lo * b.lo, hi += a.hi * b.hi for bf16 pairs a, b with f32
// accumulators, one rounding each (mixed-precision fma.rn.f32.bf16).
__device__ __forceinline__ void fma2_bf16_f32(uint32_t a, uint32_t b, float& lo, float& hi) {
    asm("{\n\t.reg .b16 al, ah, bl, bh;\n\t"
        "mov.b32 {al, ah}, %2;\n\t"
        "mov.b32 {bl, bh}, %3;\n\t"
        "fma.rn.f32.bf16 %0, al, bl, %0;\n\t"
        "fma.rn.f32.bf16 %1, ah, bh, %1;\n\t}"
        : "+f"(lo), "+f"(hi)
        : "r"(a), "r"(b));
}

// One (token, head) of the radius-1 stencil attention from the staged boxes:
// query box sQ (8 x 8 tokens), key and value halo boxes sK, sV (10 x 10; the
// positions outside the grid hold the tensor map's zero fill), token (lx, ly)
// of the block, grid position (qx, qy) in a tx x ty token grid. The nine
// scores are accumulated together, channel chunk outer and key inner, so a
// thread has 18 independent FMA chains in flight; each chain adds its
// channels in the same order as dot_head (even channels in one, odd in the
// other, then the two added), so every attention form gives the same bits.
// Keys outside the grid get score
// -inf and weight 0 (their zero-filled values then add exact zeros).
template <int HD>
__device__ __forceinline__ void attn_stencil_token(const uint8_t* sQ, const uint8_t* sK, const uint8_t* sV, int lx,
                                                   int ly, int qx, int qy, int tx, int ty, int hl, float scale,
                                                   float* acc) {
    // the query stays packed (bf16 pairs); scores use the mixed-precision FMA
    // bf16 x bf16 + f32, whose product is exact in f32, so each step rounds
    // exactly like fmaf on the unpacked values
    uint32_t q[HD / 2];
#pragma unroll
    for (int w = 0; w < HD / 8; w++) {
        const int ch = hl * HD + 8 * w;
        const uint4 u = *swz_chunk(sQ + (size_t)(ch >> 6) * kAttBoxQ, ly * kAttTile + lx, (ch & 63) >> 3);
        q[4 * w] = u.x;
        q[4 * w + 1] = u.y;
        q[4 * w + 2] = u.z;
        q[4 * w + 3] = u.w;
    }
    float p0[9], p1[9];
#pragma unroll
    for (int j = 0; j < 9; j++) p0[j] = p1[j] = 0.f;
#pragma unroll
    for (int w = 0; w < HD / 8; w++) {
        const int ch = hl * HD + 8 * w;
#pragma unroll
        for (int j = 0; j < 9; j++) {
            const int rho = (ly + j / 3) * kAttHalo + (lx + j % 3);
            const uint4 u = *swz_chunk(sK + (size_t)(ch >> 6) * kAttBoxKVPad, rho, (ch & 63) >> 3);
            const uint32_t a[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int i = 0; i < 4; i++) fma2_bf16_f32(q[4 * w + i], a[i], p0[j], p1[j]);
        }
    }
    float sc[9];
    bool in[9];
    float smax = -INFINITY;
#pragma unroll
    for (int j = 0; j < 9; j++) {
        const int ky = qy + j / 3 - 1, kx = qx + j % 3 - 1;
        in[j] = ky >= 0 && kx >= 0 && ky < ty && kx < tx;
        sc[j] = in[j] ? (p0[j] + p1[j]) * scale : -INFINITY;
        smax = fmaxf(smax, sc[j]);
    }
    float denom = 0.f;
#pragma unroll
    for (int j = 0; j < 9; j++) {
        sc[j] = in[j] ? __expf(sc[j] - smax) : 0.f;
        denom += sc[j];
    }
    const float inv = 1.0f / denom;
#pragma unroll
    for (int i = 0; i < HD; i++) acc[i] = 0.f;
#pragma unroll
    for (int j = 0; j < 9; j++) {
        const int rho = (ly + j / 3) * kAttHalo + (lx + j % 3);
        axpy_head_s<HD>(sc[j] * inv, sV, kAttBoxKVPad, rho, hl * HD, acc);
    }
}

// Maps of an instance used here: slot kv_slot = halo boxes (64 ch x 10 x 10)
// over its qkv rows, slot q_slot = query boxes (64 ch x 8 x 8) over the same
// rows. D = 64 * (boxes per vector); threads = 64 tokens x heads.
template <int HD>
__global__ void __launch_bounds__(64 * (64 / HD), 5) bf_attn_tile_kernel(Dims d, const CUtensorMap* __restrict__ maps, int kv_slot,
                                                           int q_slot, const InstDev* inst, int n_inst,
                                                           bf16* __restrict__ out, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int D = d.D;
    constexpr int HPB = 64 / HD;                  // heads per 64-channel box
    const int bx = blockIdx.z;                    // this CTA's box: heads bx HPB ..
    uint8_t* sK = smem;                           // the halo box of the keys
    uint8_t* sV = sK + (size_t)kAttBoxKVPad;      // the halo box of the values
    uint8_t* sQ = sV + (size_t)kAttBoxKVPad;      // the query box
    __shared__ uint64_t bar;
    __shared__ volatile int failed;
    const int tile = blockIdx.x, half = blockIdx.y;
    const int lo = warp_find_last_le(n_inst, tile, [&](int i) { return (long long)inst[i].tt0; });
    // the instance's fields in registers (no reloads after the barriers)
    const int Itx = inst[lo].tx, Ity = inst[lo].ty, Itt0 = inst[lo].tt0, Irow0 = inst[lo].row0;
    const int tiles_x = (Itx + kConvTX - 1) / kConvTX;
    const int tl = tile - Itt0;
    const int x0 = (tl % tiles_x) * kConvTX, y0 = (tl / tiles_x) * kConvTY + half * kAttTile;
    const CUtensorMap* mkv = maps + kMapsPerInst * lo + kv_slot;
    const CUtensorMap* mq = maps + kMapsPerInst * lo + q_slot;
    if (threadIdx.x == 0) {
        tc::mbar_init(&bar, 1);
        tc::fence_barrier_init();
        failed = 0;
        if (tc::smem_u32(smem) & 1023u) {
            failed = 1;
            atomicExch(err, 2);
        }
    }
    __syncthreads();
    JC_PDL_ENTRY;
    if (y0 >= Ity) return;  // the lower half of a tile that overhangs the grid (uniform per CTA)
    if (threadIdx.x < 32 && tc::elect_one() && !failed) {
        tc::tensormap_acquire(mkv);
        tc::tensormap_acquire(mq);
        tc::mbar_expect_tx(&bar, (uint32_t)(2 * kAttBoxKV + kAttBoxQ));
        tc::tma_load_3d(sK, mkv, D + 64 * bx, x0 - 1, y0 - 1, &bar);
        tc::tma_load_3d(sV, mkv, 2 * D + 64 * bx, x0 - 1, y0 - 1, &bar);
        tc::tma_load_3d(sQ, mq, 64 * bx, x0, y0, &bar);
    }
    const bool ok = __syncthreads_and(tc::mbar_wait(&bar, 0, err, &failed) ? 1 : 0) != 0;
    if (!ok) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int hl = warp % HPB;                   // head within the box
    const int h = bx * HPB + hl;
    const int tok = (warp / HPB) * 32 + lane;    // 0..63 within the block
    if (tok >= kAttTile * kAttTile) return;
    const int lx = tok & 7, ly = tok >> 3;
    const int qx = x0 + lx, qy = y0 + ly;
    if (qx >= Itx || qy >= Ity) return;
    const float scale = 1.0f / sqrtf((float)HD);
    float acc[HD];
    attn_stencil_token<HD>(sQ, sK, sV, lx, ly, qx, qy, Itx, Ity, hl, scale, acc);
    store_head<HD>(out + ((size_t)Irow0 + (size_t)qy * Itx + qx) * D + h * HD, acc);
}

// to_cells' output (f32 [rows, HD]) -> the cell-head input zc (f16, 48
// channels, conv1's operand type, plane-major: [6][cells][8], `zc_plane`
// elements between planes): upsample along y then x (cpu.rs:211-245;
// weights (i + 1/2) / P, the far neighbour clamped to the grid), the state
// appended split exactly into f16 parts (cpu.rs:339-342), zero padding. One CTA per 8 x 16 cell tile
// (the conv tiles): the 5 x 3 tokens it reads are staged in shared memory
// (row pitch HD + 4 floats against bank conflicts), thread r makes cell
// (y0 + r / 8, x0 + r % 8).
constexpr int kUpTokY = kConvTY / 4 + 1, kUpTokX = kConvTX / 4 + 1, kUpPitch = 36;

template <int HD, int C>
__global__ void __launch_bounds__(128) bf_upsample_kernel(Dims d, const float* __restrict__ z0, const InstDev* inst,
                                                          int n_inst, __half* __restrict__ zc, long long zc_plane) {
    static_assert(kZcState == HD && kZcState + 3 * C <= kZcCh && HD + 4 <= kUpPitch, "zc layout");
    constexpr int P = 4;  // patch (the BF16 path is built for 4); (i + 1/2) / 4 is exact as a product
    __shared__ __align__(16) float win[kUpTokY * kUpTokX * kUpPitch];
    const int tile = blockIdx.x;
    // the instance descriptors are written before the forward's first kernel
    const int lo = warp_find_last_le(n_inst, tile, [&](int i) { return (long long)inst[i].ct0; });
    const InstDev I = inst[lo];
    JC_PDL_ENTRY;
    const int tiles_x = (I.nx + kConvTX - 1) / kConvTX;
    const int tl = tile - I.ct0;
    const int x0 = (tl % tiles_x) * kConvTX, y0 = (tl / tiles_x) * kConvTY;
    const int ty0 = y0 / P, tx0 = x0 / P;
    for (int e = threadIdx.x; e < kUpTokY * kUpTokX * (HD / 4); e += blockDim.x) {
        const int q = e % (HD / 4), t = e / (HD / 4), ty = ty0 + t / kUpTokX, tx = tx0 + t % kUpTokX;
        const bool in = ty < I.ty && tx < I.tx;
        cp_async16(win + t * kUpPitch + 4 * q, in ? z0 + (size_t)(I.row0 + ty * I.tx + tx) * HD + 4 * q : z0, in);
    }
    cp_async_wait_all();
    __syncthreads();
    const int r = threadIdx.x;
    const int y = y0 + r / kConvTX, x = x0 + r % kConvTX;
    if (y >= I.ny || x >= I.nx) return;
    const int yt = y / P, iy = y % P, xt = x / P, ix = x % P;
    const int yt2 = min(yt + 1, I.ty - 1), xt2 = min(xt + 1, I.tx - 1);
    const float wy = ((float)iy + 0.5f) * (1.0f / P), wx = ((float)ix + 0.5f) * (1.0f / P);
    auto tok = [&](int ty, int tx) {
        return reinterpret_cast<const float4*>(win + ((ty - ty0) * kUpTokX + (tx - tx0)) * kUpPitch);
    };
    const float4 *a = tok(yt, xt), *b = tok(yt, xt2), *c = tok(yt2, xt), *e = tok(yt2, xt2);
    const float uy = 1.0f - wy, ux = 1.0f - wx;
    float vals[kZcCh];
#pragma unroll
    for (int i = 0; i < kZcCh; i++) vals[i] = 0.f;
#pragma unroll
    for (int q = 0; q < HD / 4; q++) {
        float4 A = a[q], B = b[q], Cc = c[q], E = e[q];
        vals[4 * q + 0] = (A.x * uy + Cc.x * wy) * ux + (B.x * uy + E.x * wy) * wx;
        vals[4 * q + 1] = (A.y * uy + Cc.y * wy) * ux + (B.y * uy + E.y * wy) * wx;
        vals[4 * q + 2] = (A.z * uy + Cc.z * wy) * ux + (B.z * uy + E.z * wy) * wx;
        vals[4 * q + 3] = (A.w * uy + Cc.w * wy) * ux + (B.w * uy + E.w * wy) * wx;
    }
    const size_t plane = (size_t)I.nx * I.ny, cl = (size_t)y * I.nx + x;
#pragma unroll
    for (int ch = 0; ch < C; ch++) {
        const float sv = I.state[ch * plane + cl];
        const float hi = __half2float(__float2half_rn(sv));
        vals[kZcState + ch] = hi;
        vals[kZcState + 3 + ch] = sv - hi;  // exact in f32; rounded to f16 below
        vals[kZcState + 6 + ch] = hi;
    }
    __half* o = zc + ((size_t)I.cell0 + cl) * 8;
#pragma unroll
    for (int q = 0; q < kZcCh / 8; q++) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            __half2 h = __floats2half2_rn(vals[8 * q + 2 * i], vals[8 * q + 2 * i + 1]);
            w[i] = *reinterpret_cast<uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(o + q * zc_plane) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// ---------------------------------------------------------------------------
// tensor-core kernels

// Epilogue helpers: thread (warp w, lane) owns TMEM lane 32 w + lane = tile row.
__device__ __forceinline__ uint32_t lane_addr(uint32_t tmem) {
    return tmem + (((threadIdx.x >> 5) & 3u) * 32u << 16);
}

// GELU of v + b for two values, x Phi(x) (cpu.rs:67-74), as x * sigmoid(2 u) with
// the odd polynomial u = x (c1 + c3 x^2 + c5 x^4): the tanh form of Hendrycks &
// Gimpel (2016) with its coefficients refitted (minimax of the absolute GELU
// error on |x| <= 9; |x| is clamped to 9, where Phi is 0 or 1 to f32
// precision). Maximum absolute error 2.6e-5 against the exact erf form, far
// below the bf16 rounding of the values it feeds. Two MUFU operations a value
// (ex2, rcp); the adds, multiplies and multiply-adds are paired (add/mul/fma.rn.f32x2:
// each lane is the scalar operation with the same rounding).
__device__ __forceinline__ void gelu_fast_pair(float& v0, float& v1, float b0, float b1) {
    // coefficients of u, times -2 log2(e), so sigmoid(2u) = 1 / (1 + 2^t)
    constexpr float k1 = -2.0f * 1.4426950408889634f * 7.97506042e-01f;
    constexpr float k3 = -2.0f * 1.4426950408889634f * 3.70071725e-02f;
    constexpr float k5 = -2.0f * 1.4426950408889634f * -3.51557324e-04f;
    float x0, x1, e0, e1, r0, r1;
    asm("{\n\t.reg .b64 v, b;\n\tmov.b64 v, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
        "add.rn.f32x2 v, v, b;\n\tmov.b64 {%0, %1}, v;\n\t}"
        : "=f"(x0), "=f"(x1)
        : "f"(v0), "f"(v1), "f"(b0), "f"(b1));
    const float c0 = fminf(fmaxf(x0, -9.0f), 9.0f), c1 = fminf(fmaxf(x1, -9.0f), 9.0f);
    float t0, t1;
    asm("{\n\t.reg .b64 c, q, p, kk1, kk3, kk5;\n\tmov.b64 c, {%2, %3};\n\t"
        "mov.b64 kk1, {%4, %4};\n\tmov.b64 kk3, {%5, %5};\n\tmov.b64 kk5, {%6, %6};\n\t"
        "mul.rn.f32x2 q, c, c;\n\tfma.rn.f32x2 p, q, kk5, kk3;\n\tfma.rn.f32x2 p, q, p, kk1;\n\t"
        "mul.rn.f32x2 p, c, p;\n\tmov.b64 {%0, %1}, p;\n\t}"
        : "=f"(t0), "=f"(t1)
        : "f"(c0), "f"(c1), "f"(k1), "f"(k3), "f"(k5));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(t0));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(t1));
    float d0, d1;
    asm("{\n\t.reg .b64 e, one;\n\tmov.b64 e, {%2, %3};\n\tmov.b64 one, {%4, %4};\n\t"
        "add.rn.f32x2 e, one, e;\n\tmov.b64 {%0, %1}, e;\n\t}"
        : "=f"(d0), "=f"(d1)
        : "f"(e0), "f"(e1), "f"(1.0f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(d0));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(d1));
    asm("{\n\t.reg .b64 x, r;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 r, {%4, %5};\n\t"
        "mul.rn.f32x2 x, x, r;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(v0), "=f"(v1)
        : "f"(x0), "f"(x1), "f"(r0), "f"(r1));
}

__device__ __forceinline__ int slot_swz(int r, int D) { return D >= 128 ? (r & 31) : (r & (D / 4 - 1)); }

// Stage columns [c0, c1) of this thread's TMEM lane (tile row `r`) into the
// shared f32 tile [128][D]; float4 slot q of row r is stored at slot
// q ^ slot_swz(r, D), which keeps both the row-per-thread writes here and the
// row-per-warp reads below free of bank conflicts.
__device__ __forceinline__ void stage_rows(uint32_t ta, int r, int D, int c0, int c1, float* tile) {
    for (int c = c0; c < c1; c += 16) {
        float a[16];
        tc::tmem_ld16(ta + c, a);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int q = c / 4 + i;
            reinterpret_cast<float4*>(tile + (size_t)r * D)[q ^ slot_swz(r, D)] =
                make_float4(a[4 * i], a[4 * i + 1], a[4 * i + 2], a[4 * i + 3]);
        }
    }
}

// Residual + LayerNorm rows (two-pass mean and biased variance, eps 1e-5),
// in one fixed arithmetic shared by every kernel that produces them, so the
// MLP forms give the same bits: every operation is an explicitly rounded
// one (no compiler contraction), element v = x + (acc + bias); each
// 4-element slot contributes ((v0 + v1) + (v2 + v3)) and, for the variance,
// fma(e0, e0, e1 e1) + fma(e2, e2, e3 e3); slot q belongs to lane q % 32, a
// lane sums its slots in order starting from 0, and the 32 lane partials are
// added in the xor-butterfly order of warp_sum; rstd = ln_rstd(sum of
// squared deviations); out = fma((v - mean) rstd, g, b).
__device__ __forceinline__ float4 resid4(float4 x, float4 a, float4 bias) {
    return make_float4(__fadd_rn(x.x, __fadd_rn(a.x, bias.x)), __fadd_rn(x.y, __fadd_rn(a.y, bias.y)),
                       __fadd_rn(x.z, __fadd_rn(a.z, bias.z)), __fadd_rn(x.w, __fadd_rn(a.w, bias.w)));
}
__device__ __forceinline__ float sum4(float4 v) { return __fadd_rn(__fadd_rn(v.x, v.y), __fadd_rn(v.z, v.w)); }
__device__ __forceinline__ float sqdev4(float4 v, float m) {
    const float e0 = __fsub_rn(v.x, m), e1 = __fsub_rn(v.y, m), e2 = __fsub_rn(v.z, m), e3 = __fsub_rn(v.w, m);
    return __fadd_rn(__fmaf_rn(e0, e0, __fmul_rn(e1, e1)), __fmaf_rn(e2, e2, __fmul_rn(e3, e3)));
}
// 1 / sqrt(variance + eps) of the residual + LayerNorm rows: the hardware
// reciprocal square root (rsqrtf, 2 ulp), not a rounded square root and a
// rounded division (which cost the MLP kernel 7% of its time). Every kernel
// that forms these rows calls this, so they keep giving the same bits.
__device__ __forceinline__ float ln_rstd(float sq_sum, int D) { return rsqrtf(sq_sum / (float)D + 1e-5f); }

__device__ __forceinline__ float ln1(float v, float m, float rstd, float g, float b) {
    return __fmaf_rn(__fmul_rn(__fsub_rn(v, m), rstd), g, b);
}
// warp_sum of N independent values at once: the butterfly steps of all N are
// interleaved, so their shuffle latencies overlap; each value is added in
// warp_sum's order and gets warp_sum's bits.
template <int N>
__device__ __forceinline__ void warp_sum_n(float (&v)[N]) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < N; k++) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
}

// The 32 lane partials in the order warp_sum adds them.
__device__ __forceinline__ float tree32(float* a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < o; i++) a[i] = __fadd_rn(a[i], a[i + o]);
    return a[0];
}

// One warp per tile row over the staged accumulator tile (float4 slot q of
// row r at q ^ slot_swz(r, D)); x and ln are read and written coalesced, G
// rows in flight per warp. Rows [0, nrows) of the tile (a multiple of G),
// tile row r -> global row m0 + r. SPL = slots per lane (1: D <= 128, 2: 256).
// PRE: load every row group's residual rows up front (four groups at most).
// A warp's residual rows for rows_resid_ln_t at D = 128 (lane l's slot of
// each of its up to 16 rows), loaded ahead of the epilogue by load_xrows so
// the loads overlap an MMA wait.
struct XRows {
    float4 v[4][4];
};
__device__ __forceinline__ void load_xrows(const float* __restrict__ x, int m0, int R, int warp, int nwarps,
                                           int nrows, XRows& xr) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r0 = warp * 4 + i * nwarps * 4;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int row = m0 + r0 + k;
            xr.v[i][k] = r0 < nrows && row < R ? reinterpret_cast<const float4*>(x + (size_t)row * 128)[lane]
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
}

template <int SPL, bool FULL, bool PRE = false>  // FULL: every lane owns SPL slots (D = 128 SPL)
__device__ __forceinline__ void rows_resid_ln_t(const float* tile, int D, int m0, int R, const float* __restrict__ bias,
                                float* __restrict__ x, const float* __restrict__ g, const float* __restrict__ b,
                                bf16* __restrict__ ln, int warp, int nwarps, int nrows, const XRows* xin = nullptr) {
    const int lane = threadIdx.x & 31;
    const int nq = D / 4;
    const int swz = D >= 128 ? 31 : nq - 1;  // slot_swz mask
    constexpr int G = 4;
    auto on = [&](int j) { return FULL || lane + 32 * j < nq; };
    float4 bb[SPL], gg[SPL], be[SPL];
#pragma unroll
    for (int j = 0; j < SPL; j++) {
        const int q = on(j) ? lane + 32 * j : 0;
        bb[j] = reinterpret_cast<const float4*>(bias)[q];
        gg[j] = reinterpret_cast<const float4*>(g)[q];
        be[j] = reinterpret_cast<const float4*>(b)[q];
    }
    // at most four row groups per warp (D <= 128): every group's residual
    // rows are loaded up front, so their latencies overlap instead of
    // adding up group after group
    constexpr int PF = 4;
    float4 xpre[SPL == 1 && PRE ? PF : 1][G];
    const bool prefetched = PRE && SPL == 1 && nrows <= PF * nwarps * G;
    if (SPL == 1 && prefetched && xin) {
#pragma unroll
        for (int i = 0; i < PF; i++)
#pragma unroll
            for (int k = 0; k < G; k++) xpre[SPL == 1 && PRE ? i : 0][k] = xin->v[i][k];
    } else if (SPL == 1 && prefetched) {
#pragma unroll
        for (int i = 0; i < PF; i++) {
            const int r0 = warp * G + i * nwarps * G;
#pragma unroll
            for (int k = 0; k < G; k++) {
                const int row = m0 + r0 + k;
                const int q = on(0) ? lane : 0;
                xpre[SPL == 1 && PRE ? i : 0][k] = r0 < nrows && row < R
                                                ? reinterpret_cast<const float4*>(x + (size_t)row * D)[q]
                                                : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    }
    int grp = 0;
    for (int r0 = warp * G; r0 < nrows; r0 += nwarps * G, grp++) {
        float4 a[G][SPL], xv[G][SPL];
#pragma unroll
        for (int k = 0; k < G; k++) {
            const int r = r0 + k, row = m0 + r;
#pragma unroll
            for (int j = 0; j < SPL; j++) {
                const int q = on(j) ? lane + 32 * j : 0;
                a[k][j] = reinterpret_cast<const float4*>(tile + (size_t)r * D)[q ^ (r & swz)];
                if (SPL == 1 && prefetched) {
                    float4 t = xpre[0][k];
#pragma unroll
                    for (int i = 1; i < PF; i++)
                        if (grp == i) t = xpre[SPL == 1 && PRE ? i : 0][k];
                    xv[k][j] = t;
                } else {
                    xv[k][j] = row < R ? reinterpret_cast<const float4*>(x + (size_t)row * D)[q]
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
        }
        // the G rows' reductions run interleaved (warp_sum_n): the same
        // order and bits per row as one warp_sum after another
        float4 v[G][SPL];
        float mean[G], q2[G];
#pragma unroll
        for (int k = 0; k < G; k++) {
            float s = 0.f;
#pragma unroll
            for (int j = 0; j < SPL; j++) {
                v[k][j] = resid4(xv[k][j], a[k][j], bb[j]);
                if (on(j)) s = __fadd_rn(s, sum4(v[k][j]));
            }
            mean[k] = s;
        }
        warp_sum_n(mean);
#pragma unroll
        for (int k = 0; k < G; k++) {
            mean[k] = mean[k] / (float)D;
            float t = 0.f;
#pragma unroll
            for (int j = 0; j < SPL; j++)
                if (on(j)) t = __fadd_rn(t, sqdev4(v[k][j], mean[k]));
            q2[k] = t;
        }
        warp_sum_n(q2);
#pragma unroll
        for (int k = 0; k < G; k++) {
            const int row = m0 + r0 + k;
            if (row >= R) break;  // warp-uniform
            const float rstd = ln_rstd(q2[k], D);
#pragma unroll
            for (int j = 0; j < SPL; j++) {
                if (!on(j)) continue;
                const int q = lane + 32 * j;
                reinterpret_cast<float4*>(x + (size_t)row * D)[q] = v[k][j];
                float o[4] = {ln1(v[k][j].x, mean[k], rstd, gg[j].x, be[j].x),
                              ln1(v[k][j].y, mean[k], rstd, gg[j].y, be[j].y),
                              ln1(v[k][j].z, mean[k], rstd, gg[j].z, be[j].z),
                              ln1(v[k][j].w, mean[k], rstd, gg[j].w, be[j].w)};
                BfVec<4>::store(ln + (size_t)row * D + 4 * q, o);
            }
        }
    }
}

template <bool PRE = false>
__device__ __forceinline__ void rows_resid_ln_any(const float* tile, int D, int m0, int R, const float* bias, float* x,
                                  const float* g, const float* b, bf16* ln, int warp, int nwarps, int nrows = 128,
                                  const XRows* xin = nullptr) {
    if (D == 256) rows_resid_ln_t<2, true>(tile, D, m0, R, bias, x, g, b, ln, warp, nwarps, nrows);
    else if (D == 128) rows_resid_ln_t<1, true, PRE>(tile, D, m0, R, bias, x, g, b, ln, warp, nwarps, nrows, xin);
    else rows_resid_ln_t<1, false, PRE>(tile, D, m0, R, bias, x, g, b, ln, warp, nwarps, nrows);
}

enum { EPI_BF16 = 0, EPI_F32 = 1, EPI_RESID_LN = 2 };

struct GemmEpi {
    const float* bias;
    bf16* out_bf;    // EPI_BF16 / EPI_RESID_LN (LayerNorm output)
    float* out_f;    // EPI_F32
    float* x;        // EPI_RESID_LN residual stream
    const float* g;  // EPI_RESID_LN LayerNorm
    const float* b;
    int ldo;         // output row stride (elements)
};

// C[128-row tile, BN-column block] = A[rows, K] @ B^T for dims above 128 (256 is
// the one that the head widths leave). A via TMA (64-column swizzled boxes), B (one
// pre-arranged [K/8][BN][8] block) via a bulk copy ahead of the previous kernel's
// end; all of K is staged at once (K <= 512, a multiple of 64), one thread issues
// the MMAs, four warps run the epilogue from TMEM, sixteen the residual +
// LayerNorm (with four, and A in 32 boxes of 8 columns, 32 tiles of dim 256 took
// 15.5 us for the projection and 13.5 for q/k/v, now 11.3 and 10.8).
constexpr int gemm_threads(int epi) { return epi == EPI_RESID_LN ? 512 : 128; }

template <int EPI>
__global__ void __launch_bounds__(gemm_threads(EPI)) tc_gemm_kernel(const __grid_constant__ CUtensorMap tmA,
                                                      const __grid_constant__ CUtensorMap tmO,
                                                      const bf16* __restrict__ Bblk, int K, int BN, int R,
                                                      GemmEpi ep, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sA = smem;                       // swizzled boxes of 64 columns x 128 rows
    uint8_t* sB = smem + (size_t)K * 256;     // [K/8][BN][8]
    __shared__ __align__(16) float sbias[256];
    __shared__ uint64_t bar_load, bar_mma;
    __shared__ uint32_t tmem_base;
    __shared__ volatile int failed;
    const int warp = threadIdx.x >> 5;
    const int m0 = blockIdx.x * 128, nb = blockIdx.y;
    const uint32_t ncols = BN <= 32 ? 32 : (BN <= 64 ? 64 : (BN <= 128 ? 128 : 256));
    if (threadIdx.x == 0) {
        tc::mbar_init(&bar_load, 1);
        tc::mbar_init(&bar_mma, 1);
        tc::fence_barrier_init();
        failed = 0;
        if (tc::smem_u32(smem) & 1023u) {  // operand tiles need aligned shared memory
            failed = 1;
            atomicExch(err, 2);
        }
    }
    if (warp == 0) tc::tmem_alloc(&tmem_base, ncols);
    if (EPI != EPI_RESID_LN)
        for (int i = threadIdx.x; i < BN; i += blockDim.x) sbias[i] = ep.bias[nb * BN + i];
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0 && tc::elect_one() && !failed) {  // the weights do not wait for the previous kernel
        const uint32_t bytes_b = (uint32_t)K * BN * 2;
        tc::mbar_expect_tx(&bar_load, (uint32_t)K * 256 + bytes_b);
        tc::bulk_load(sB, Bblk + (size_t)nb * K * BN, bytes_b, &bar_load);
    }
    __syncwarp();
    JC_PDL_ENTRY;
    tc::tc_fence_after();
    const uint32_t tmem = tmem_base;
    if (warp == 0 && tc::elect_one() && !failed) {
        for (int c = 0; c < K / 64; c++) tc::tma_load_2d(sA + c * 16384, &tmA, 64 * c, m0, &bar_load);
        if (tc::mbar_wait(&bar_load, 0, err, &failed)) {
            tc::tc_fence_after();
            const uint32_t idesc = tc::idesc_bf16(128, BN);
            const uint64_t ad = tc::sdesc_sw128(tc::smem_u32(sA)), bd = tc::sdesc(tc::smem_u32(sB), BN * 16, 128);
            for (int k = 0; k < K / 16; k++)
                tc::mma_bf16(tmem, tc::sdesc_at(ad, (k >> 2) * 16384 + (k & 3) * 32), tc::sdesc_at(bd, k * 2 * BN * 16), idesc, k > 0 ? 1u : 0u);
            tc::mma_commit(&bar_mma);
        }
    }
    __syncwarp();
    const bool ok = __syncthreads_and(tc::mbar_wait(&bar_mma, 0, err, &failed) ? 1 : 0) != 0;
    tc::tc_fence_after();
    if (ok) {
        const uint32_t ta = lane_addr(tmem);
        const int n0 = nb * BN;
        if (EPI == EPI_RESID_LN) {
            // every MMA and TMA write is complete: the operand tiles' shared
            // memory now holds the f32 accumulator tile
            float* tile = reinterpret_cast<float*>(smem);
            constexpr int NW = gemm_threads(EPI) / 32, parts = NW / 4;
            stage_rows(ta, (warp & 3) * 32 + (threadIdx.x & 31), BN, warp / 4 * (BN / parts), (warp / 4 + 1) * (BN / parts), tile);
            __syncthreads();
            rows_resid_ln_any(tile, BN, m0, R, ep.bias, ep.x, ep.g, ep.b, ep.out_bf, warp, NW);
        } else {
            // stage the tile (bias added) in 128-byte swizzled boxes of 128
            // rows in the operand shared memory, then store it with TMA
            constexpr int EB = EPI == EPI_BF16 ? 2 : 4;  // bytes per element
            constexpr int PB = 128 / EB;                 // elements per box row
            const int r = threadIdx.x;
            for (int c = 0; c < BN; c += 16) {
                float a[16];
                tc::tmem_ld16(ta + c, a);  // collective: every lane of the warp loads
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const float4 bv = *reinterpret_cast<const float4*>(sbias + c + i);
                    a[i] += bv.x;
                    a[i + 1] += bv.y;
                    a[i + 2] += bv.z;
                    a[i + 3] += bv.w;
                }
                uint8_t* box = smem + (size_t)(c / PB) * 16384 + (size_t)r * 128;
                const int j0 = (c % PB) * EB / 16;  // first 16-byte chunk of these 16 columns
                if (EPI == EPI_BF16) {
                    BfVec<8>::store(reinterpret_cast<bf16*>(box + ((j0 ^ (r & 7)) << 4)), a);
                    BfVec<8>::store(reinterpret_cast<bf16*>(box + (((j0 + 1) ^ (r & 7)) << 4)), a + 8);
                } else {
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        *reinterpret_cast<float4*>(box + (((j0 + q) ^ (r & 7)) << 4)) =
                            make_float4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
                }
            }
            tc::fence_async_shared();
            __syncthreads();
            if (warp == 0 && tc::elect_one()) {
                for (int c = 0; c < BN; c += PB) tc::tma_store_2d(&tmO, smem + (size_t)(c / PB) * 16384, n0 + c, m0);
                tc::bulk_commit();
                tc::bulk_wait_read();
            }
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, ncols);
}

// Residual + LayerNorm of tile row r by the thread that owns it (TMEM lane
// r): v = x + (acc + bias) in place in the f32 row of sX (128-byte swizzled
// boxes of 32 columns x 128 rows: 16-byte chunk q of row r at box q / 8,
// chunk (q % 8) ^ (r % 8)), then mean and biased variance over the row (two
// passes) and LayerNorm(v) as bf16: into swizzled staging boxes of 64
// columns (sLn) or straight to the global row (lnrow).
__device__ __forceinline__ float4* xrow_chunk(uint8_t* sX, int r, int q) {
    return reinterpret_cast<float4*>(sX + (size_t)(q >> 3) * 16384 + (size_t)r * 128 + (((q & 7) ^ (r & 7)) << 4));
}

// DT > 0: the width as a compile-time constant (every loop unrolled, so the
// shared-memory reads of a pass are all in flight at once); DT = 0: D.
template <int DT>
__device__ void row_resid_ln_t(uint32_t ta, int r, int D_, uint8_t* sX, const float* sbias, const float* sg,
                               const float* sb, bf16* lnrow) {
    const int D = DT > 0 ? DT : D_;
    // D <= 128: slot q is lane q's only slot, so lane partial q = 0 + sum4
    const int nq = D / 4;
#pragma unroll
    for (int c = 0; c < D; c += 16) {
        float a[16];
        tc::tmem_ld16(ta + c, a);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float4* p = xrow_chunk(sX, r, (c >> 2) + i);
            const int o = c + 4 * i;
            *p = resid4(*p, make_float4(a[4 * i], a[4 * i + 1], a[4 * i + 2], a[4 * i + 3]),
                        make_float4(sbias[o], sbias[o + 1], sbias[o + 2], sbias[o + 3]));
        }
    }
    float part[32];
#pragma unroll
    for (int l = 0; l < 32; l++) part[l] = l < nq ? __fadd_rn(0.f, sum4(*xrow_chunk(sX, r, l))) : 0.f;
    const float mean = tree32(part) / (float)D;
#pragma unroll
    for (int l = 0; l < 32; l++) part[l] = l < nq ? __fadd_rn(0.f, sqdev4(*xrow_chunk(sX, r, l), mean)) : 0.f;
    const float rstd = ln_rstd(tree32(part), D);
#pragma unroll
    for (int c = 0; c < D; c += 8) {
        const float4 v0 = *xrow_chunk(sX, r, c >> 2), v1 = *xrow_chunk(sX, r, (c >> 2) + 1);
        const float in[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; i++) o[i] = ln1(in[i], mean, rstd, sg[c + i], sb[c + i]);
        if (lnrow) BfVec<8>::store(lnrow + c, o);
    }
}

__device__ __forceinline__ void row_resid_ln(uint32_t ta, int r, int D, uint8_t* sX, const float* sbias,
                                             const float* sg, const float* sb, bf16* lnrow) {
    if (D == 128) row_resid_ln_t<128>(ta, r, D, sX, sbias, sg, sb, lnrow);
    else row_resid_ln_t<0>(ta, r, D, sX, sbias, sg, sb, lnrow);
}

constexpr int kLnMaxD = 128;  // widest row the row-per-thread LayerNorm serves

// Fused MLP: x += gelu(LN2(x) @ W1 + b1) @ W2 + b2, then LayerNorm of the new
// x (the next block's norm1, or the final norm) into `ln`. Per chunk of NC
// hidden columns, one after the other, S = A @ W1_chunk (TMEM), h = gelu(S +
// b1) written to shared memory as bf16 by all 8 warps (two per TMEM lane
// quarter, one column half each), O += h @ W2_chunk (TMEM); the hidden
// activations never leave the SM. Every summation order is fixed by
// NC-independent K slices of 16, so every chunk width gives the same bits.
// The residual + LayerNorm epilogue stages O through shared memory and runs
// one warp per row.
constexpr int kMlpSerialThreads = 256;

__global__ void __launch_bounds__(kMlpSerialThreads, 2) tc_mlp_serial_kernel(const __grid_constant__ CUtensorMap tmA,
                                                             const bf16* __restrict__ W1, const bf16* __restrict__ W2,
                                                             const float* __restrict__ b1,
                                                             const float* __restrict__ b2, int D, int F, int NC, int R,
                                                             float* __restrict__ x, const float* __restrict__ g,
                                                             const float* __restrict__ b, bf16* __restrict__ ln,
                                                             int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sA = smem;                           // [D/8][128][8]
    uint8_t* sB1 = sA + (size_t)D * 256;          // [D/8][NC][8]
    uint8_t* sB2 = sB1 + (size_t)D * NC * 2;      // [NC/8][D][8]
    uint8_t* sH = sB2 + (size_t)D * NC * 2;       // [NC/8][128][8]
    __shared__ __align__(16) float sb1[1024];
    __shared__ uint64_t bar_a, bar_w1, bar_w2, bar_s, bar_o;
    __shared__ uint32_t tmem_base;
    __shared__ volatile int failed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int quarter = warp & 3, half = warp >> 2;
    const int m0 = blockIdx.x * 128;
    const uint32_t ncols = D <= 128 ? 256 : 512;
    const uint32_t s_col = D <= 128 ? 128 : 256;  // O in [0, D), S in [s_col, s_col + NC)
    if (threadIdx.x == 0) {
        tc::mbar_init(&bar_a, 1);
        tc::mbar_init(&bar_w1, 1);
        tc::mbar_init(&bar_w2, 1);
        tc::mbar_init(&bar_s, 1);
        tc::mbar_init(&bar_o, 1);
        tc::fence_barrier_init();
        failed = 0;
        if (tc::smem_u32(smem) & 1023u) {  // operand tiles need aligned shared memory
            failed = 1;
            atomicExch(err, 2);
        }
    }
    for (int i = threadIdx.x; i < F; i += blockDim.x) sb1[i] = b1[i];
    if (warp == 0) tc::tmem_alloc(&tmem_base, ncols);
    tc::tc_fence_before();
    __syncthreads();
    JC_PDL_ENTRY;
    tc::tc_fence_after();
    const uint32_t tO = tmem_base, tS = tmem_base + s_col;
    const uint64_t dA = tc::sdesc(tc::smem_u32(sA), 2048, 128), dW1 = tc::sdesc(tc::smem_u32(sB1), NC * 16, 128),
                   dW2 = tc::sdesc(tc::smem_u32(sB2), D * 16, 128), dH = tc::sdesc(tc::smem_u32(sH), 2048, 128);
    const int nchunks = F / NC;
    const uint32_t wbytes = (uint32_t)D * NC * 2;
    auto issue_s = [&]() {  // S = A @ W1_chunk into tS
        const uint32_t idesc = tc::idesc_bf16(128, NC);
        for (int k = 0; k < D / 16; k++)
            tc::mma_bf16(tS, tc::sdesc_at(dA, k * 4096), tc::sdesc_at(dW1, k * 2 * NC * 16), idesc, k > 0 ? 1u : 0u);
        tc::mma_commit(&bar_s);
    };
    // Chunk j's critical path is GELU_j then S_{j+1}: W1_{j+1} is loaded as
    // soon as S_j has read W1_j, W2_j once O_{j-1} has read W2_{j-1}, and
    // S_{j+1} is issued right after GELU_j, ahead of O_j. The MMAs and their
    // accumulation order are those of one chunk after another.
    if (warp == 0 && tc::elect_one() && !failed) {
        tc::mbar_expect_tx(&bar_a, (uint32_t)D * 256);
        for (int kc = 0; kc < D / 8; kc++) tc::tma_load_2d(sA + kc * 2048, &tmA, kc * 8, m0, &bar_a);
        tc::mbar_expect_tx(&bar_w1, wbytes);
        tc::bulk_load(sB1, W1, wbytes, &bar_w1);
        tc::mbar_expect_tx(&bar_w2, wbytes);
        tc::bulk_load(sB2, W2, wbytes, &bar_w2);
        if (tc::mbar_wait(&bar_a, 0, err, &failed) && tc::mbar_wait(&bar_w1, 0, err, &failed)) {
            tc::tc_fence_after();
            issue_s();
        }
    }
    __syncwarp();
    bool ok = true;
    for (int j = 0; j < nchunks && ok; j++) {
        ok = __syncthreads_and(tc::mbar_wait(&bar_s, j & 1, err, &failed) ? 1 : 0) != 0;
        tc::tc_fence_after();
        if (!ok) break;
        if (warp == 0 && tc::elect_one() && !failed && j + 1 < nchunks) {  // S_j has read W1_j
            tc::mbar_expect_tx(&bar_w1, wbytes);
            tc::bulk_load(sB1, W1 + (size_t)(j + 1) * D * NC, wbytes, &bar_w1);
        }
        if (j > 0) {  // O_{j-1} has read h_{j-1} and W2_{j-1}
            ok = __syncthreads_and(tc::mbar_wait(&bar_o, (j - 1) & 1, err, &failed) ? 1 : 0) != 0;
            tc::tc_fence_after();
            if (!ok) break;
            if (warp == 0 && tc::elect_one() && !failed) {
                tc::mbar_expect_tx(&bar_w2, wbytes);
                tc::bulk_load(sB2, W2 + (size_t)j * D * NC, wbytes, &bar_w2);
            }
        }
        {
            // h = gelu(S + b1) -> bf16 -> shared memory in the core-matrix layout
            const int r = quarter * 32 + lane;
            const uint32_t ta = lane_addr(tS);
            const int c0 = half * (NC / 2), c1 = c0 + NC / 2;
            for (int c = c0; c < c1; c += 16) {
                float a[16];
                tc::tmem_ld16(ta + c, a);
#pragma unroll
                for (int i = 0; i < 16; i += 2) gelu_fast_pair(a[i], a[i + 1], sb1[j * NC + c + i], sb1[j * NC + c + i + 1]);
                BfVec<8>::store(reinterpret_cast<bf16*>(sH + (size_t)(c / 8) * 2048 + r * 16), a);
                BfVec<8>::store(reinterpret_cast<bf16*>(sH + (size_t)(c / 8 + 1) * 2048 + r * 16), a + 8);
            }
        }
        tc::fence_async_shared();
        tc::tc_fence_before();
        __syncthreads();
        tc::tc_fence_after();
        if (warp == 0 && tc::elect_one() && !failed) {
            // S_{j+1} first (tS was read by every GELU thread), then O_j
            if (j + 1 < nchunks && tc::mbar_wait(&bar_w1, (j + 1) & 1, err, &failed)) {
                tc::tc_fence_after();
                issue_s();
            }
            if (!failed && tc::mbar_wait(&bar_w2, j & 1, err, &failed)) {
                tc::tc_fence_after();
                const uint32_t idesc = tc::idesc_bf16(128, D);
                for (int k = 0; k < NC / 16; k++)
                    tc::mma_bf16(tO, tc::sdesc_at(dH, k * 4096), tc::sdesc_at(dW2, k * 2 * D * 16), idesc,
                                 (j > 0 || k > 0) ? 1u : 0u);
                tc::mma_commit(&bar_o);
            }
        }
        __syncwarp();
    }
    XRows xr2;  // the residual rows, loaded while the last O runs
    if (D == 128) load_xrows(x, m0, R, warp, kMlpSerialThreads / 32, 128, xr2);
    if (ok) {  // the last O
        ok = __syncthreads_and(tc::mbar_wait(&bar_o, (nchunks - 1) & 1, err, &failed) ? 1 : 0) != 0;
        tc::tc_fence_after();
    }
    if (ok) {
        // every MMA is complete: reuse the operand shared memory for the f32 O tile
        float* tile = reinterpret_cast<float*>(smem);
        stage_rows(lane_addr(tO), quarter * 32 + lane, D, half * (D / 2), (half + 1) * (D / 2), tile);
        __syncthreads();
        rows_resid_ln_any<true>(tile, D, m0, R, b2, x, g, b, ln, warp, kMlpSerialThreads / 32, 128,
                                D == 128 ? &xr2 : nullptr);
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem_base, ncols);
}

// The same for dims above 128 that are multiples of 64, one 128-row tile a CTA, its
// stages on separate warps:
//   0-15 the GELUs (16 columns of a chunk and the 32 lanes of a TMEM quarter each)
//        and the residual + LayerNorm;
//   16   (one lane) loads the weights, two chunks of W1 and two of W2 in flight;
//   17   (one lane) loads A (swizzled boxes of 64 columns) and issues the MMAs.
// Chunks of 64 hidden columns go through two TMEM accumulators: S_{j+1} runs while
// the row warps work on S_j; h_j lies packed over S_j's own columns and is O's A
// operand from there. The MMAs' K order is that of the kernel above. That one,
// with one buffer of everything and CTA barriers between its steps, took 44 us
// for 32 tiles of dim 256 with 1024 hidden columns (one tile an SM, 16 chunks in
// a chain); this takes 27.
constexpr int kMWRowWarps = 16, kMWThreads = (kMWRowWarps + 2) * 32, kMWNC = 64;
__host__ __device__ constexpr size_t mlp_wide_smem(int D) { return (size_t)D * 256 + 4 * (size_t)D * kMWNC * 2; }
static bool mlp_wide(int D, int nc) { return D > 128 && D % 64 == 0 && nc == kMWNC; }

__global__ void __launch_bounds__(kMWThreads, 1) tc_mlp_wide_kernel(
    const __grid_constant__ CUtensorMap tmA, const bf16* __restrict__ W1, const bf16* __restrict__ W2,
    const float* __restrict__ b1, const float* __restrict__ b2, int D, int F, int R, float* __restrict__ x,
    const float* __restrict__ g, const float* __restrict__ b, bf16* __restrict__ ln, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int NC = kMWNC;
    const uint32_t wb = (uint32_t)D * NC * 2;
    uint8_t *sA = smem, *sW1 = smem + (size_t)D * 256, *sW2 = sW1 + 2 * (size_t)wb;
    __shared__ __align__(16) float sb1[1024];
    __shared__ uint64_t a_full, w1_full[2], w1_empty[2], w2_full[2], w2_empty[2], s_full[2], h_full[2], o_full;
    __shared__ uint32_t tmem_base;
    __shared__ volatile int failed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * 128, n = F / NC;
    if (threadIdx.x == 0) {
        tc::mbar_init(&a_full, 1);
        tc::mbar_init(&o_full, 1);
        for (int i = 0; i < 2; i++) {
            for (uint64_t* q : {&w1_full[i], &w1_empty[i], &w2_full[i], &w2_empty[i], &s_full[i]}) tc::mbar_init(q, 1);
            tc::mbar_init(&h_full[i], kMWRowWarps);
        }
        tc::fence_barrier_init();
        failed = 0;
        if (tc::smem_u32(smem) & 1023u) {  // operand tiles need aligned shared memory
            failed = 1;
            atomicExch(err, 2);
        }
    }
    for (int i = threadIdx.x; i < F; i += kMWThreads) sb1[i] = b1[i];
    if (warp == 0) tc::tmem_alloc(&tmem_base, 512);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tO = tmem_base, tS = tmem_base + 256;  // O | S_0 | S_1
    if (warp == kMWRowWarps) {
        // the weights never change: their loads do not wait for the previous kernel
        if (tc::elect_one() && !failed) {
            bool ok = true;
            auto put = [&](uint8_t* ring, const bf16* W, uint64_t* full, uint64_t* empty, int j) {
                if (j >= n || !ok) return;
                if (j >= 2) ok = tc::mbar_wait(&empty[j & 1], (uint32_t)(j / 2 - 1) & 1u, err, &failed);
                if (!ok) return;
                tc::mbar_expect_tx(&full[j & 1], wb);
                tc::bulk_load(ring + (j & 1) * (size_t)wb, W + (size_t)j * D * NC, wb, &full[j & 1]);
            };
            put(sW1, W1, w1_full, w1_empty, 0);
            put(sW1, W1, w1_full, w1_empty, 1);
            for (int j = 0; j < n && ok; j++) {
                put(sW2, W2, w2_full, w2_empty, j);
                put(sW1, W1, w1_full, w1_empty, j + 2);
            }
        }
        __syncwarp();
        JC_PDL_ENTRY;
    } else if (warp == kMWRowWarps + 1) {
        JC_PDL_ENTRY;
        if (tc::elect_one() && !failed) {
            tc::mbar_expect_tx(&a_full, (uint32_t)D * 256);
            for (int c = 0; c < D / 64; c++) tc::tma_load_2d(sA + c * 16384, &tmA, 64 * c, m0, &a_full);
            const uint32_t idS = tc::idesc_bf16(128, NC), idO = tc::idesc_bf16(128, D);
            const uint64_t dA = tc::sdesc_sw128(tc::smem_u32(sA)), dW1 = tc::sdesc(tc::smem_u32(sW1), NC * 16, 128),
                           dW2 = tc::sdesc(tc::smem_u32(sW2), D * 16, 128);
            auto issue_s = [&](int j) {  // S_j = A @ W1_j
                const uint64_t w = tc::sdesc_at(dW1, (j & 1) * wb);
                tc::tc_fence_after();
                for (int k = 0; k < D / 16; k++)
                    tc::mma_bf16(tS + (j & 1) * NC, tc::sdesc_at(dA, (k >> 2) * 16384 + (k & 3) * 32),
                                 tc::sdesc_at(w, k * 2 * NC * 16), idS, k > 0 ? 1u : 0u);
                tc::mma_commit(&s_full[j & 1]);
                tc::mma_commit(&w1_empty[j & 1]);
            };
            bool ok = tc::mbar_wait(&a_full, 0, err, &failed);
            for (int j = 0; j < 2 && j < n && ok; j++) {
                ok = tc::mbar_wait(&w1_full[j], 0, err, &failed);
                if (ok) issue_s(j);
            }
            for (int j = 0; j < n && ok; j++) {
                const uint32_t ph = (uint32_t)(j >> 1) & 1u;
                ok = tc::mbar_wait(&w2_full[j & 1], ph, err, &failed) && tc::mbar_wait(&h_full[j & 1], ph, err, &failed);
                if (!ok) break;
                tc::tc_fence_after();
                const uint64_t w = tc::sdesc_at(dW2, (j & 1) * wb);
#pragma unroll
                for (int k = 0; k < NC / 16; k++)  // 16 columns of h lie packed in the first 8 of their own
                    tc::mma_bf16_ta(tO, tS + (j & 1) * NC + 16 * k, tc::sdesc_at(w, k * 2 * D * 16), idO,
                                    (j > 0 || k > 0) ? 1u : 0u);
                tc::mma_commit(j == n - 1 ? &o_full : &w2_empty[j & 1]);
                if (j + 2 < n) {  // after O_j, which reads h_j from S_j's columns
                    ok = tc::mbar_wait(&w1_full[j & 1], ph ^ 1u, err, &failed);
                    if (ok) issue_s(j + 2);
                }
            }
        }
        __syncwarp();
    } else {
        JC_PDL_ENTRY;
        const int sub = warp >> 2;
        for (int j = 0; j < n; j++) {
            // (after a failed wait the later ones fail at once; every warp reaches the barriers below)
            tc::mbar_wait(&s_full[j & 1], (uint32_t)(j >> 1) & 1u, err, &failed);
            __syncwarp();
            tc::tc_fence_after();
            const uint32_t ts = lane_addr(tS + (j & 1) * NC + 16 * sub);
            const float* bj = sb1 + j * NC + 16 * sub;
            float a[16];
            tc::tmem_ld16(ts, a);
            uint32_t h[8];
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                gelu_fast_pair(a[i], a[i + 1], bj[i], bj[i + 1]);
                __nv_bfloat162 p = __floats2bfloat162_rn(a[i], a[i + 1]);
                h[i / 2] = *reinterpret_cast<uint32_t*>(&p);
            }
            tc::tmem_st8(ts, h);
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&h_full[j & 1]);
        }
    }
    const bool ok = __syncthreads_and(tc::mbar_wait(&o_full, 0, err, &failed) ? 1 : 0) != 0;
    tc::tc_fence_after();
    // every MMA is complete: reuse the operand shared memory for the f32 O tile
    float* tile = reinterpret_cast<float*>(smem);
    if (ok && warp < kMWRowWarps) {
        const int sub = warp >> 2, c0 = sub * (D / 4);
        stage_rows(lane_addr(tO), (warp & 3) * 32 + lane, D, c0, c0 + D / 4, tile);
    }
    __syncthreads();
    if (ok && warp < kMWRowWarps)
        rows_resid_ln_any<false>(tile, D, m0, R, b2, x, g, b, ln, warp, kMWRowWarps);
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem_base, 512);
}

// One decision for the `n` threads (whole warps) that meet at named barrier `bar`.
__device__ __forceinline__ bool all_of(bool v, int bar, int n) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbarrier.red.and.pred p, %2, %3, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r)
        : "r"(v ? 1u : 0u), "r"(bar), "r"(n)
        : "memory");
    return r != 0;
}

// Output projection + MLP of one block at dim 128 (cpu.rs:300-313): x += attn @
// Wp + bp, A = LN2(x), x += gelu(A @ W1 + b1) @ W2 + b2, ln = LN(x) for the next
// step. Persistent: one CTA per SM walks 128-row tiles, its stages on separate
// warps:
//   0-15 the row work: both residual + LayerNorms and the GELUs;
//   16   (one lane) loads the weights in 16 KB blocks, in the order the MMAs
//        take them, into a ring of kPMSlots slots, tiles ahead included;
//   17   (one lane) issues every MMA;
//   18   (one lane) loads the attention and residual rows, a tile ahead, and
//        stores each tile's rows.
// The hidden columns go through in chunks of 128: S_c = A @ W1_c into one of two
// TMEM accumulators, h_c = gelu(S_c + b1_c) rounded to bf16 back over S_c's own
// columns (a thread holds all it reads before it writes), O += h_c @ W2_c with
// h_c as the MMA's A operand straight from TMEM. S_{c+1} runs while the row
// warps work on S_c, and the next tile's projection P, in the accumulator that
// chunk n - 2 has left, while they work on the last LayerNorm: they wait for an
// MMA only at the two ends of a tile. A (packed bf16) lies in TMEM too. The
// residual rows stay in the row warps' registers from one LayerNorm to the other;
// they come and go through one shared-memory buffer: each thread takes the next
// tile's values out of the places that it puts this tile's in. That leaves the
// weights 112 KB (with two buffers of rows 48 KB, and a chunk's MMAs waited 650
// cycles for each block). The rows leave by bulk copies (an SM writes about 30
// bytes a cycle: stored by the row warps themselves the 64 KB held them 2500
// cycles a tile).
// The residual + LayerNorm rows are read from TMEM as 16 x 8 fragments: two warps
// share 16 rows, half of the columns each, and a row lies in four lanes of each.
// Wp's and W2's output columns are stored in the order (pm_column) that gives
// lane j of the four the columns 16 m + 4 j .. + 3, m even in one warp and odd in
// the other: it moves its part of a row as float4s, and a row's sum takes one
// exchange between the warps and two shuffles, in tree32's order. The arithmetic
// and its order are those of rows_resid_ln_t (D = 128), so every form gives the
// same bits. The MMAs' K order is that of tc_mlp_serial_kernel.
// What bounds it: the GELUs' MUFU operations (an ex2 at 32 and a reciprocal at 16
// a cycle for each of 65,536 hidden values a tile, 6.1 K cycles) and, while they
// wait, the row work around them, which shared memory's 128 bytes a cycle bound
// (the rows' exchange alone 128 KB). At 64 K rows: 76 us a launch for the form
// before it (two CTAs per SM, one accumulator, the chunk through shared memory,
// CTA barriers around every step), 51 with 8 row warps and two row buffers, 46 for
// this one; a tile alone on its SM 28, 17.5 and 16.5 us. A tile's 18.4 K cycles: the
// four chunks' GELUs 8.9 K, S_0 1.1 K, the last O 1.1 K, the LayerNorms 2.0 K and
// 2.2 K, the rows' exchange 1.4 K.
constexpr int kPMRowWarps = 16, kPMThreads = (kPMRowWarps + 3) * 32;
constexpr int kPMD = 128, kPMNC = 128;       // width; hidden columns per chunk
constexpr int kPMBlock = 64 * kPMD * 2;      // bytes of a weight block: 64 hidden columns (or half of Wp's K)
constexpr int kPMSlots = 7;
constexpr int kPMX = kPMD * 512;             // bytes of a tile's residual rows
constexpr int kPMOffX = kPMD * 256, kPMOffW = kPMOffX + kPMX;
constexpr int kPMSmem = kPMOffW + kPMSlots * kPMBlock;

// The logical output column in column p of the weights arranged for
// tc_proj_mlp_kernel: the even 16-column groups, then the odd ones, and within a
// group the order in which a fragment pair gives lane j of a row's four columns 4 j .. + 3.
__host__ __device__ constexpr int pm_column(int p) {
    return 16 * (2 * ((p >> 4) & 3) + (p >> 6)) + 4 * ((p >> 1) & 3) + 2 * ((p >> 3) & 1) + (p & 1);
}

// A layer's weights as tc_proj_mlp_kernel reads them, from the arrangements the
// other kernels read, in 16-byte pieces (8 K elements of a column): Wp and W2
// with their columns in pm_column's order, W1 in blocks of 64 K x 128 columns
// (its last 64 columns, if F is an odd multiple of 64, as they were).
__global__ void pm_arrange_kernel(const uint4* __restrict__ wp, const uint4* __restrict__ w1,
                                  const uint4* __restrict__ w2, int F, uint4* __restrict__ dst) {
    constexpr int D = kPMD, KC = D / 8;
    const int n_p = KC * D, n_1 = F * KC, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n_p) {
        dst[i] = wp[(i & ~(D - 1)) + pm_column(i % D)];
    } else if (i < n_p + n_1) {
        const int e = i - n_p, c = e / (KC * 128);
        if ((c + 1) * 128 > F) {
            dst[i] = w1[e];
        } else {
            const int kc = e / 128 % KC, col = e % 128;
            dst[i] = w1[((2 * c + col / 64) * KC + kc) * 64 + col % 64];
        }
    } else if (i < n_p + 2 * n_1) {
        const int e = i - n_p - n_1;
        dst[i] = w2[(e & ~(D - 1)) + pm_column(e % D)];
    }
}

// Sums of two rows that lie in four lanes of two warps, in tree32's order: p[k][i]
// is row k's slot 4 (2 i + half) + lane % 4, and the other warp of the pair has the
// other half's. xch: this pair's two blocks of 32 partial sums.
__device__ __forceinline__ float2 frag_row_sums(float (&p)[2][4], int half, float2 (*xch)[32], int pair) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < 2; k++)
        p[k][0] = __fadd_rn(__fadd_rn(p[k][0], p[k][2]), __fadd_rn(p[k][1], p[k][3]));
    xch[half][lane] = make_float2(p[0][0], p[1][0]);
    asm volatile("bar.sync %0, 64;" ::"r"(1 + pair) : "memory");
    const float2 o = xch[half ^ 1][lane];
    float2 t = make_float2(__fadd_rn(p[0][0], o.x), __fadd_rn(p[1][0], o.y));
#pragma unroll
    for (int d = 2; d > 0; d >>= 1) {
        t.x = __fadd_rn(t.x, __shfl_xor_sync(0xffffffffu, t.x, d));
        t.y = __fadd_rn(t.y, __shfl_xor_sync(0xffffffffu, t.y, d));
    }
    return t;
}

// A row warp's place in the residual + LayerNorm work.
struct FragPos {
    int half, pair;       // column half; the two warps of the same rows have one pair number
    float2 (*xch)[2][32]; // their exchange: [sum, squares][half][lane]
};

// x[2 i + k] holds columns 16 (2 i + half) + 4 (lane % 4) .. + 3 of row k (rows
// lane / 4 and lane / 4 + 8 of the warp's 16): x += acc + bias (acc: the warp's 16
// TMEM lanes and 64 columns at tacc), and the rows' mean and 1 / sqrt(variance + eps).
__device__ __forceinline__ void frag_resid(float4 (&x)[8], uint32_t tacc, const float* bias, const FragPos& at,
                                           float (&mean)[2], float (&rstd)[2]) {
    const float4* b4 = reinterpret_cast<const float4*>(bias) + 4 * at.half + (threadIdx.x & 3);
#pragma unroll
    for (int q = 0; q < 2; q++) {
        float a[16];
        tc::tmem_ld_frag32(tacc + 32 * q, a);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float4 bb = b4[8 * (2 * q + i)];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                float4& v = x[2 * (2 * q + i) + k];
                const float2 lo = add_f32x2(make_float2(v.x, v.y), add_f32x2(make_float2(a[8 * i + 2 * k], a[8 * i + 2 * k + 1]),
                                                                             make_float2(bb.x, bb.y)));
                const float2 hi = add_f32x2(make_float2(v.z, v.w),
                                            add_f32x2(make_float2(a[8 * i + 4 + 2 * k], a[8 * i + 5 + 2 * k]),
                                                      make_float2(bb.z, bb.w)));
                v = make_float4(lo.x, lo.y, hi.x, hi.y);
            }
        }
    }
    float p[2][4];
#pragma unroll
    for (int k = 0; k < 2; k++)
#pragma unroll
        for (int i = 0; i < 4; i++) p[k][i] = sum4(x[2 * i + k]);
    const float2 sum = frag_row_sums(p, at.half, at.xch[0], at.pair);
    mean[0] = sum.x / (float)kPMD;
    mean[1] = sum.y / (float)kPMD;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float2 nm = make_float2(-mean[k], -mean[k]);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 v = x[2 * i + k];
            const float2 e = add_f32x2(make_float2(v.x, v.y), nm), f = add_f32x2(make_float2(v.z, v.w), nm);
            p[k][i] = __fadd_rn(__fmaf_rn(e.x, e.x, __fmul_rn(e.y, e.y)), __fmaf_rn(f.x, f.x, __fmul_rn(f.y, f.y)));
        }
    }
    const float2 sq = frag_row_sums(p, at.half, at.xch[1], at.pair);
    rstd[0] = ln_rstd(sq.x, kPMD);
    rstd[1] = ln_rstd(sq.y, kPMD);
}

// LayerNorm(x) of four columns of row k, as two bf16 pairs.
__device__ __forceinline__ uint2 frag_ln4(const float4 v, float mean, float rstd, const float4 g, const float4 b) {
    const float2 nm = make_float2(-mean, -mean), rs = make_float2(rstd, rstd);
    const float2 lo = fma_f32x2(mul_f32x2(add_f32x2(make_float2(v.x, v.y), nm), rs), make_float2(g.x, g.y),
                                make_float2(b.x, b.y));
    const float2 hi = fma_f32x2(mul_f32x2(add_f32x2(make_float2(v.z, v.w), nm), rs), make_float2(g.z, g.w),
                                make_float2(b.z, b.w));
    const __nv_bfloat162 l = __floats2bfloat162_rn(lo.x, lo.y), h = __floats2bfloat162_rn(hi.x, hi.y);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&l), *reinterpret_cast<const uint32_t*>(&h));
}
// Into TMEM as an MMA's A operand: this half's groups of 8 of the 64 packed columns at tA.
__device__ __forceinline__ void frag_ln_tmem(const float4 (&x)[8], const float (&mean)[2], const float (&rstd)[2],
                                             const float* g, const float* b, int half, uint32_t tA) {
    const int at = 4 * half + (threadIdx.x & 3);
    const float4 *g4 = reinterpret_cast<const float4*>(g) + at, *b4 = reinterpret_cast<const float4*>(b) + at;
    uint32_t r[16];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float4 gg = g4[8 * i], be = b4[8 * i];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint2 u = frag_ln4(x[2 * i + k], mean[k], rstd[k], gg, be);
            r[4 * i + 2 * k] = u.x;
            r[4 * i + 2 * k + 1] = u.y;
        }
    }
    tc::tmem_st_frag8x4(tA + 8 * half, r);
}
// Into the swizzled tile sOut (boxes of 64 columns x 128 rows; tr = the tile row
// that lane / 4 falls on).
__device__ __forceinline__ void frag_ln_smem(const float4 (&x)[8], const float (&mean)[2], const float (&rstd)[2],
                                             const float* g, const float* b, int half, uint8_t* sOut, int tr) {
    const int j = threadIdx.x & 3, sw = tr & 7;
    const float4 *g4 = reinterpret_cast<const float4*>(g) + 4 * half + j, *b4 = reinterpret_cast<const float4*>(b) + 4 * half + j;
    uint8_t* row = sOut + (size_t)tr * 128 + (j & 1) * 8;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int m = 2 * i + half;
        const float4 gg = g4[8 * i], be = b4[8 * i];
        uint8_t* to = row + (m >> 2) * 16384 + (((2 * (m & 3) + (j >> 1)) ^ sw) << 4);
#pragma unroll
        for (int k = 0; k < 2; k++)
            *reinterpret_cast<uint2*>(to + k * 8 * 128) = frag_ln4(x[2 * i + k], mean[k], rstd[k], gg, be);
    }
}

// The same to global memory (row: this thread's first row there; those from R on are not written).
__device__ __forceinline__ void frag_ln_global(const float4 (&x)[8], const float (&mean)[2], const float (&rstd)[2],
                                               const float* g, const float* b, int half, bf16* ln, int row, int R) {
    const int at = 4 * half + (threadIdx.x & 3);
    const float4 *g4 = reinterpret_cast<const float4*>(g) + at, *b4 = reinterpret_cast<const float4*>(b) + at;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float4 gg = g4[8 * i], be = b4[8 * i];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint2 u = frag_ln4(x[2 * i + k], mean[k], rstd[k], gg, be);
            if (row + 8 * k < R) reinterpret_cast<uint2*>(ln + (size_t)(row + 8 * k) * kPMD)[8 * i + at] = u;
        }
    }
}

// SPLIT: two CTAs take one tile, each the row work of 16 lanes of every 32
// (blockIdx.x % 2), one tile a CTA; the MMAs, whose time does not depend on the
// rows, they both do (each also loads the other's rows, which may
// change meanwhile, and does not use them). The rows go straight to global memory.
template <bool SPLIT>
__global__ void __launch_bounds__(kPMThreads, 1) tc_proj_mlp_kernel(
    const __grid_constant__ CUtensorMap tmAttn, const __grid_constant__ CUtensorMap tmLn,
    const __grid_constant__ CUtensorMap tmX, const bf16* __restrict__ Wp,
    const bf16* __restrict__ W1, const bf16* __restrict__ W2, const float* __restrict__ bp, const float* __restrict__ g2,
    const float* __restrict__ be2, const float* __restrict__ b1, const float* __restrict__ b2,
    const float* __restrict__ g, const float* __restrict__ b, int F, int R, float* __restrict__ xg, bf16* __restrict__ ln,
    int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int D = kPMD, NC = kPMNC, NS = kPMSlots;
    constexpr uint32_t kB = kPMBlock;
    uint8_t* sAT = smem;            // attention rows, then the tile's LayerNorm rows: 2 x [128][64] swizzled
    uint8_t* sX = smem + kPMOffX;   // residual rows on their way in or out: 8 x [128][16] f32
    uint8_t* sW = smem + kPMOffW;   // weight ring
    __shared__ __align__(16) float sb1[1024], sv[6][D];          // bp, g2, be2, b2, g, b
    __shared__ float2 s_xch[8][2][2][32];                        // the row warps' partial sums, by pair
    __shared__ uint64_t w_full[NS], w_empty[NS], at_full, at_empty, x_full, x_taken, p_full, a_full, s_full[2], h_full[2],
        o_full, out_full;
    __shared__ uint32_t tmem_base;
    __shared__ volatile int failed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tiles = (R + 127) / 128;
    const int first = SPLIT ? blockIdx.x / 2 : blockIdx.x, step = SPLIT ? n_tiles : gridDim.x;
    const int my_tiles = first < n_tiles ? (n_tiles - 1 - first) / step + 1 : 0;
    auto m0_of = [&](int it) { return (first + it * step) * 128; };
    const int n = (F + NC - 1) / NC;  // chunks; the last may have 64 columns
    if (threadIdx.x == 0) {
        for (int i = 0; i < NS; i++) {
            tc::mbar_init(&w_full[i], 1);
            tc::mbar_init(&w_empty[i], 1);
        }
        for (uint64_t* q : {&at_full, &at_empty, &x_full, &p_full, &s_full[0], &s_full[1], &o_full}) tc::mbar_init(q, 1);
        for (uint64_t* q : {&x_taken, &a_full, &h_full[0], &h_full[1], &out_full}) tc::mbar_init(q, kPMRowWarps);  // one arrival per row warp
        tc::fence_barrier_init();
        failed = 0;
        if (tc::smem_u32(smem) & 1023u) {  // operand tiles need aligned shared memory
            failed = 1;
            atomicExch(err, 2);
        }
    }
    for (int i = threadIdx.x; i < F; i += kPMThreads) sb1[i] = b1[i];
    for (int i = threadIdx.x; i < 6 * D; i += kPMThreads) {
        const float* src = i < D ? bp : i < 2 * D ? g2 : i < 3 * D ? be2 : i < 4 * D ? b2 : i < 5 * D ? g : b;
        sv[i / D][i % D] = src[i % D];
    }
    if (warp == 0) tc::tmem_alloc(&tmem_base, 512);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tO = tmem_base, tS = tmem_base + 128, tA = tmem_base + 384;  // O | S_0 | S_1 | A (64 columns)
    const uint32_t tP = tS + (n & 1) * NC;                // P: the accumulator that chunk n - 2 used
    auto blocks_of = [&](int c) { return min(NC, F - c * NC) / 64; };
    if (warp == kPMRowWarps) {
        // the weights never change: their loads do not wait for the previous kernel
        if (tc::elect_one() && !failed) {
            int cnt = 0;
            bool ok = true;
            auto put = [&](const bf16* src) {
                const int sl = cnt % NS;
                if (cnt >= NS) ok = ok && tc::mbar_wait(&w_empty[sl], (uint32_t)(cnt / NS - 1) & 1u, err, &failed);
                if (!ok) return;
                tc::mbar_expect_tx(&w_full[sl], kB);
                tc::bulk_load(sW + sl * kB, src, kB, &w_full[sl]);
                cnt++;
            };
            auto put_chunk = [&](const bf16* W, int c) {
                for (int q = 0; q < blocks_of(c); q++) put(W + (size_t)(2 * c + q) * 64 * D);
            };
            auto put_p = [&]() {
                put(Wp);
                put(Wp + 64 * D);
            };
            if (my_tiles > 0) put_p();
            for (int it = 0; it < my_tiles && ok; it++) {
                for (int c = 0; c < 2 && c < n; c++) put_chunk(W1, c);
                for (int c = 0; c < n && ok; c++) {
                    put_chunk(W2, c);
                    if (c + 2 < n) put_chunk(W1, c + 2);
                    if (c == n - 1 && it + 1 < my_tiles) put_p();
                }
            }
        }
        __syncwarp();
        JC_PDL_ENTRY;
    } else if (warp == kPMRowWarps + 1) {
        JC_PDL_ENTRY;
        if (tc::elect_one() && !failed) {
            constexpr uint32_t id128 = tc::idesc_bf16(128, D), id64 = tc::idesc_bf16(128, 64);
            const uint64_t dAT = tc::sdesc_sw128(tc::smem_u32(sAT));
            const uint64_t dW128 = tc::sdesc(tc::smem_u32(sW), D * 16, 128), dW64 = tc::sdesc(tc::smem_u32(sW), 64 * 16, 128);
            // Weight blocks are waited for (take) ahead of what their MMAs wait for
            // last, and given back after the commit that somebody waits for.
            int t_sl = 0, u_sl = 0, ahead = 0, used = 0;
            uint32_t t_ph = 0;
            bool ok = true;
            auto take = [&](int k) {
                for (; ok && ahead < k; ahead++) {
                    ok = tc::mbar_wait(&w_full[t_sl], t_ph, err, &failed);
                    if (++t_sl == NS) {
                        t_sl = 0;
                        t_ph ^= 1u;
                    }
                }
                tc::tc_fence_after();
            };
            auto slot = [&]() {  // the next taken block's offset
                const int at = u_sl + used++;
                ahead--;
                return (uint32_t)(at < NS ? at : at - NS) * kB;
            };
            auto give_back = [&]() {
                for (; used > 0; used--) {
                    tc::mma_commit(&w_empty[u_sl]);
                    if (++u_sl == NS) u_sl = 0;
                }
            };
            auto issue_p = [&](int it) {  // P = attn @ Wp
                take(2);
                ok = ok && tc::mbar_wait(&at_full, (uint32_t)it & 1u, err, &failed);
                if (!ok) return;
                tc::tc_fence_after();
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const uint64_t w = tc::sdesc_at(dW128, slot()), a = tc::sdesc_at(dAT, q * 16384);
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        tc::mma_bf16(tP, tc::sdesc_at(a, k * 32), tc::sdesc_at(w, k * 2 * D * 16), id128,
                                     k > 0 ? 1u : (uint32_t)q);
                }
                tc::mma_commit(&p_full);
                give_back();
                tc::mma_commit(&at_empty);
            };
            auto issue_s = [&](int c) {  // S_c = A @ W1_c: 128 columns in two K halves, or 64 in one block
                const int nb = blocks_of(c);
                const uint32_t t = tS + (c & 1) * NC;
                take(nb);
                if (!ok) return;
                if (nb == 2) {
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        const uint64_t w = tc::sdesc_at(dW128, slot());
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            tc::mma_bf16_ta(t, tA + q * 32 + k * 8, tc::sdesc_at(w, k * 2 * 128 * 16), id128,
                                            k > 0 ? 1u : (uint32_t)q);
                    }
                } else {
                    const uint64_t w = tc::sdesc_at(dW64, slot());
#pragma unroll
                    for (int k = 0; k < D / 16; k++)
                        tc::mma_bf16_ta(t, tA + k * 8, tc::sdesc_at(w, k * 2 * 64 * 16), id64, k > 0 ? 1u : 0u);
                }
                tc::mma_commit(&s_full[c & 1]);
                give_back();
            };
            auto issue_o = [&](int c) {  // O += h_c @ W2_c; 32 columns of h lie packed in the first 16 of their own
                const int nb = blocks_of(c);
                for (int q = 0; q < nb; q++) {
                    const uint64_t w = tc::sdesc_at(dW128, slot());
                    const uint32_t t = tS + (c & 1) * NC + q * 64;
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        tc::mma_bf16_ta(tO, t + (k >> 1) * 32 + (k & 1) * 8, tc::sdesc_at(w, k * 2 * D * 16), id128,
                                        k > 0 ? 1u : (uint32_t)(c + q > 0));
                }
                if (c == n - 1) tc::mma_commit(&o_full);
                give_back();
            };
            uint32_t ph_h = 0u;  // a bit for each accumulator
            if (my_tiles > 0) issue_p(0);
            for (int it = 0; it < my_tiles && ok; it++) {
                take(blocks_of(0));
                ok = ok && tc::mbar_wait(&a_full, (uint32_t)it & 1u, err, &failed);
                tc::tc_fence_after();
                for (int c = 0; c < 2 && c < n && ok; c++) issue_s(c);
                for (int c = 0; c < n && ok; c++) {
                    take(blocks_of(c));
                    ok = ok && tc::mbar_wait(&h_full[c & 1], ph_h >> (c & 1) & 1u, err, &failed);
                    ph_h ^= 1u << (c & 1);
                    if (!ok) break;
                    tc::tc_fence_after();
                    issue_o(c);
                    if (c + 2 < n && ok) issue_s(c + 2);  // after O_c, which reads h_c from its columns
                    if (c == n - 1 && it + 1 < my_tiles) issue_p(it + 1);
                }
            }
        }
        __syncwarp();
    } else if (warp == kPMRowWarps + 2) {
        JC_PDL_ENTRY;
        if (tc::elect_one() && !failed) {
            auto load_attn = [&](int it) {
                tc::mbar_expect_tx(&at_full, D * 256);
                for (int c = 0; c < 2; c++) tc::tma_load_2d(sAT + c * 16384, &tmAttn, 64 * c, m0_of(it), &at_full);
            };
            auto load_x = [&](int it) {
                tc::mbar_expect_tx(&x_full, kPMX);
                for (int m = 0; m < 8; m++) tc::tma_load_2d(sX + m * 8192, &tmX, 16 * m, m0_of(it), &x_full);
            };
            bool ok = true;
            if (my_tiles > 0) {
                load_attn(0);
                load_x(0);
            }
            if (my_tiles > 1) {
                ok = tc::mbar_wait(&x_taken, 0, err, &failed);
                if (ok) load_x(1);
                ok = ok && tc::mbar_wait(&at_empty, 0, err, &failed);
                if (ok) load_attn(1);
            }
            for (int it = 0; it < my_tiles && ok && !SPLIT; it++) {
                ok = tc::mbar_wait(&out_full, (uint32_t)it & 1u, err, &failed);
                if (!ok) break;
                for (int c = 0; c < 2; c++) tc::tma_store_2d(&tmLn, sAT + c * 16384, 64 * c, m0_of(it));
                for (int m = 0; m < 8; m++) tc::tma_store_2d(&tmX, sX + m * 8192, 16 * m, m0_of(it));
                tc::bulk_commit();
                tc::bulk_wait_read();
                if (it + 2 < my_tiles) {
                    load_attn(it + 2);
                    load_x(it + 2);
                }
            }
        }
        __syncwarp();
    } else {
        JC_PDL_ENTRY;
        // warps 4 s + q on TMEM lanes 32 q ..: 16 of them (s % 2) and half of the
        // columns (s / 2) in the LayerNorms, all 32 and 32 of a chunk's columns in the GELUs
        const int quarter = warp & 3, sub = warp >> 2, half = sub >> 1, pair = warp & 7;
        const FragPos at{half, pair, s_xch[pair]};
        const int tr = 32 * quarter + 16 * (sub & 1) + (lane >> 2);  // tile row of this thread's first row
        const uint32_t trow = (uint32_t)(32 * quarter + 16 * (sub & 1)) << 16;
        const int part = SPLIT ? blockIdx.x & 1 : 0;
        const bool norms = !SPLIT || (sub & 1) == part;  // whether this warp has rows in the LayerNorms
        const uint32_t lane_s = ((uint32_t)(32 * quarter + 16 * part) << 16) + 32 * sub;
        // A failed wait ends no loop here: every later wait fails at once, the other
        // warps issue no more copies and MMAs, and no warp is left alone at a pair's barrier.
        auto warp_wait = [&](uint64_t* bar, uint32_t parity) {
            tc::mbar_wait(bar, parity, err, &failed);
            __syncwarp();
            tc::tc_fence_after();
        };
        auto warp_arrive = [&](uint64_t* bar) {
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(bar);
        };
        uint32_t ph_s = 0u;  // a bit for each accumulator
        // this thread's part of its rows: boxes 2 i + half
        uint8_t* xs = sX + half * 8192 + tr * 64 + (lane & 3) * 16;
        float4 x[8];
        if (my_tiles > 0) {
            warp_wait(&x_full, 0);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int k = 0; k < 2; k++) x[2 * i + k] = *reinterpret_cast<const float4*>(xs + i * 16384 + k * 8 * 64);
            warp_arrive(&x_taken);
        }
        for (int it = 0; it < my_tiles; it++) {
            float mean[2], rstd[2];
            if (it == 0) warp_wait(&p_full, 0);
            if (norms) {
                frag_resid(x, tP + trow + 64 * half, sv[0], at, mean, rstd);
                frag_ln_tmem(x, mean, rstd, sv[1], sv[2], half, tA + trow);
            }
            warp_arrive(&a_full);
            for (int c = 0; c < n; c++) {
                warp_wait(&s_full[c & 1], ph_s >> (c & 1) & 1u);
                ph_s ^= 1u << (c & 1);
                if (sub < 2 * blocks_of(c)) {
                    const float* bj = sb1 + c * NC + sub * 32;
                    const uint32_t ts = tS + (c & 1) * NC + lane_s;
                    if constexpr (SPLIT) {
                        float a[16];
                        tc::tmem_ld_frag32(ts, a);
                        uint32_t h[8];
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const float2 bb = *reinterpret_cast<const float2*>(bj + 8 * i + 2 * (lane & 3));
#pragma unroll
                            for (int k = 0; k < 2; k++) {
                                gelu_fast_pair(a[4 * i + 2 * k], a[4 * i + 2 * k + 1], bb.x, bb.y);
                                __nv_bfloat162 p = __floats2bfloat162_rn(a[4 * i + 2 * k], a[4 * i + 2 * k + 1]);
                                h[2 * i + k] = *reinterpret_cast<uint32_t*>(&p);
                            }
                        }
                        tc::tmem_st_pack16(ts, h);
                    } else {
                        float a[32];
                        tc::tmem_ld32(ts, a);
                        uint32_t h[16];
#pragma unroll
                        for (int i = 0; i < 32; i += 4) {
                            const float4 bb = *reinterpret_cast<const float4*>(bj + i);
                            gelu_fast_pair(a[i], a[i + 1], bb.x, bb.y);
                            gelu_fast_pair(a[i + 2], a[i + 3], bb.z, bb.w);
                            __nv_bfloat162 lo = __floats2bfloat162_rn(a[i], a[i + 1]);
                            __nv_bfloat162 hi = __floats2bfloat162_rn(a[i + 2], a[i + 3]);
                            h[i / 2] = *reinterpret_cast<uint32_t*>(&lo);
                            h[i / 2 + 1] = *reinterpret_cast<uint32_t*>(&hi);
                        }
                        tc::tmem_st16(ts, h);
                    }
                }
                warp_arrive(&h_full[c & 1]);
            }
            warp_wait(&o_full, (uint32_t)it & 1u);
            if constexpr (SPLIT) {
                if (norms) {
                    const int row = m0_of(it) + tr;
                    frag_resid(x, tO + trow + 64 * half, sv[3], at, mean, rstd);
                    frag_ln_global(x, mean, rstd, sv[4], sv[5], half, ln, row, R);
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        if (row + 8 * (i & 1) < R)
                            reinterpret_cast<float4*>(xg + (size_t)(row + 8 * (i & 1)) * D)[4 * (2 * (i >> 1) + half) + (lane & 3)] = x[i];
                }
                continue;
            }
            frag_resid(x, tO + trow + 64 * half, sv[3], at, mean, rstd);
            // the LayerNorm rows go over the next tile's attention rows: its P has read them by now
            if (it + 1 < my_tiles) warp_wait(&p_full, (uint32_t)(it + 1) & 1u);
            frag_ln_smem(x, mean, rstd, sv[4], sv[5], half, sAT, tr);
            // the next tile's rows in, this one's out
            if (it + 1 < my_tiles) warp_wait(&x_full, (uint32_t)(it + 1) & 1u);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    float4* slot = reinterpret_cast<float4*>(xs + i * 16384 + k * 8 * 64);
                    const float4 next = *slot;
                    *slot = x[2 * i + k];
                    x[2 * i + k] = next;
                }
            tc::fence_async_shared();
            warp_arrive(&out_full);
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem_base, 512);
}

// Persistent output projection + residual + LayerNorm (cpu.rs:300-313) for
// dims up to 128: x += attn @ Wp + bp, ln = LayerNorm2(x). One CTA per SM
// walks row tiles with its stages on separate warps:
//   warp 0     (one lane) TMA-loads each tile's attention rows and f32
//              residual rows (128-byte swizzled boxes) into one of two slots;
//   warp 1     (one lane) loads Wp once and issues each tile's MMAs into one
//              of two TMEM accumulators;
//   warps 2-5  thread r owns tile row r: the residual update in place in the
//              slot's x rows, the LayerNorm (row_resid_ln, the shared
//              arithmetic), ln rows straight to global, the new x rows back
//              with a TMA store.
constexpr int kPLThreads = 6 * 32;

struct PLSmem {
    size_t b, a, x, total;
    __host__ __device__ explicit PLSmem(int D) {
        b = 0;                                             // Wp [D/8][D][8]
        a = (size_t)D * D * 2;                             // 2 x [D/8][128][8]
        x = (a + 2 * (size_t)D * 256 + 1023) / 1024 * 1024;  // 2 x D/32 boxes of 32 f32 x 128 rows
        total = x + 2 * (size_t)D * 512;
    }
};

__global__ void __launch_bounds__(kPLThreads, 1) tc_projln_persistent_kernel(
    const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmX, const bf16* __restrict__ Wp,
    const float* __restrict__ bias, const float* __restrict__ gam, const float* __restrict__ bet,
    bf16* __restrict__ ln, int D, int R, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const PLSmem L(D);
    uint8_t* sB = smem + L.b;
    uint8_t* sA = smem + L.a;
    uint8_t* sX = smem + L.x;
    __shared__ uint64_t b_full, in_full[2], in_empty[2], acc_full[2], acc_empty[2];
    __shared__ __align__(16) float sbias[kLnMaxD], sg[kLnMaxD], sb[kLnMaxD];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int failed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tiles = (R + 127) / 128;
    const int my_tiles = (int)blockIdx.x < n_tiles ? (n_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const uint32_t ncols = D <= 32 ? 64 : (D <= 64 ? 128 : 256);  // two accumulators
    if (threadIdx.x == 0) {
        tc::mbar_init(&b_full, 1);
        for (int i = 0; i < 2; i++) {
            tc::mbar_init(&in_full[i], 1);
            tc::mbar_init(&in_empty[i], 2);  // the MMAs have read A, the epilogue's store has read x
            tc::mbar_init(&acc_full[i], 1);
            tc::mbar_init(&acc_empty[i], 4 * 32);
        }
        tc::fence_barrier_init();
        failed = 0;
        if ((tc::smem_u32(smem) & 1023u) || D > kLnMaxD || D % 32) {
            failed = 1;
            atomicExch(err, 2);
        }
    }
    for (int i = threadIdx.x; i < D; i += blockDim.x) {
        sbias[i] = bias[i];
        sg[i] = gam[i];
        sb[i] = bet[i];
    }
    if (warp == 0) tc::tmem_alloc(&tmem_base, ncols);
    tc::tc_fence_before();
    __syncthreads();
    JC_PDL_ENTRY;
    tc::tc_fence_after();
    const uint32_t tmem = tmem_base;
    const size_t a_bytes = (size_t)D * 256, x_bytes = (size_t)D * 512;
    if (warp == 0) {
        if (tc::elect_one() && !failed) {
            for (int it = 0; it < my_tiles; it++) {
                const int s = it & 1;
                if (it >= 2 && !tc::mbar_wait(&in_empty[s], (uint32_t)((it - 2) >> 1) & 1u, err, &failed)) break;
                const int m0 = ((int)blockIdx.x + it * (int)gridDim.x) * 128;
                tc::mbar_expect_tx(&in_full[s], (uint32_t)(a_bytes + x_bytes));
                for (int kc = 0; kc < D / 8; kc++)
                    tc::tma_load_2d(sA + s * a_bytes + kc * 2048, &tmA, kc * 8, m0, &in_full[s]);
                for (int bx = 0; bx < D / 32; bx++)
                    tc::tma_load_2d(sX + s * x_bytes + bx * 16384, &tmX, bx * 32, m0, &in_full[s]);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (tc::elect_one() && !failed) {
            tc::mbar_expect_tx(&b_full, (uint32_t)D * D * 2);
            tc::bulk_load(sB, Wp, (uint32_t)D * D * 2, &b_full);
            bool good = tc::mbar_wait(&b_full, 0, err, &failed);
            const uint32_t idesc = tc::idesc_bf16(128, D);
            const uint64_t dA = tc::sdesc(tc::smem_u32(sA), 2048, 128), dB = tc::sdesc(tc::smem_u32(sB), D * 16, 128);
            for (int it = 0; it < my_tiles && good; it++) {
                const int s = it & 1;
                good = tc::mbar_wait(&in_full[s], (uint32_t)(it >> 1) & 1u, err, &failed) &&
                       (it < 2 || tc::mbar_wait(&acc_empty[s], (uint32_t)((it - 2) >> 1) & 1u, err, &failed));
                if (!good) break;
                tc::tc_fence_after();
                const uint64_t da = tc::sdesc_at(dA, s * (uint32_t)a_bytes);
                const uint32_t acc = tmem + (uint32_t)s * D;
                for (int k = 0; k < D / 16; k++)
                    tc::mma_bf16(acc, tc::sdesc_at(da, k * 4096), tc::sdesc_at(dB, k * 2 * D * 16), idesc, k > 0 ? 1u : 0u);
                tc::mma_commit(&in_empty[s]);
                tc::mma_commit(&acc_full[s]);
            }
        }
        __syncwarp();
    } else {
        const int r = (warp & 3) * 32 + lane;
        for (int it = 0; it < my_tiles; it++) {
            const int s = it & 1;
            const bool ready = tc::mbar_wait(&acc_full[s], (uint32_t)(it >> 1) & 1u, err, &failed) &&
                               tc::mbar_wait(&in_full[s], (uint32_t)(it >> 1) & 1u, err, &failed);
            if (!all_of(ready, 1, 128)) break;
            tc::tc_fence_after();
            const int m0 = ((int)blockIdx.x + it * (int)gridDim.x) * 128;
            const int row = m0 + r;
            row_resid_ln(lane_addr(tmem + (uint32_t)s * D), r, D, sX + s * x_bytes, sbias, sg, sb,
                         row < R ? ln + (size_t)row * D : nullptr);
            tc::tc_fence_before();
            tc::mbar_arrive(&acc_empty[s]);
            tc::fence_async_shared();
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (warp == 2 && tc::elect_one()) {
                for (int bx = 0; bx < D / 32; bx++) tc::tma_store_2d(&tmX, sX + s * x_bytes + bx * 16384, bx * 32, m0);
                tc::bulk_commit();
                tc::bulk_wait_read();
                tc::mbar_arrive(&in_empty[s]);
            }
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, ncols);
}

// q/k/v projection (cpu.rs:291-297, the three linears as one GEMM over the
// concatenated weights), D <= 128. A CTA keeps one N block's weights in shared
// memory and walks row tiles; the N blocks of a tile go to neighbouring CTAs.
//   warp 0     (one lane) loads each tile's LayerNorm rows once the MMAs have
//              read the ones before;
//   warp 1     (one lane) loads the weights (before the previous kernel has
//              finished: they never change) and issues each tile's MMAs into one
//              of two TMEM accumulators;
//   warps 2-5  add the bias, round to bf16 into a 128-byte swizzled staging
//              area and store it with TMA.
// Two CTAs per SM, each with one buffer of rows and one of staged output: the other
// CTA's work covers what a CTA waits for, and few tiles still spread over three times
// the CTAs. (At dim 64, one N block of 192 columns, a CTA's two accumulators take all of
// an SM's tensor memory: the second CTA waits in its allocation until the first has
// walked its tiles. With one CTA per SM instead a launch of 1024 tiles alone takes 21 us,
// not 23, but a tick of 64 x 128 x 128 cells, 2 layers, 592 us and not 584.)
// SW (D a multiple of 64): the rows arrive as 128-byte swizzled boxes of 64
// columns, not as 16-byte columns (2048 pieces a tile, which the TMA unit took
// longer over than the rest of the tile). At 64 K rows: 19 us a launch with all
// N blocks in one CTA per SM and 16-byte columns, 16 this way; three tiles: 9
// and 5 us.
constexpr int kQKVPThreads = 6 * 32;

struct QKVPSmem {
    size_t a, b, stage, total;
    __host__ __device__ QKVPSmem(int D, int BN) {
        a = 0;                                                    // [D/64][128][64] swizzled, or [D/8][128][8]
        b = (size_t)D * 256;                                      // [D/8][BN][8]
        stage = (b + (size_t)D * BN * 2 + 1023) / 1024 * 1024;    // ceil(BN/64) boxes of 16 KB
        total = stage + (size_t)((BN + 63) / 64) * 16384;
    }
};

template <bool SW>
__global__ void __launch_bounds__(kQKVPThreads, 2) tc_qkv_kernel(
    const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmO, const bf16* __restrict__ W,
    const float* __restrict__ bias, int D, int BN, int R, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const QKVPSmem L(D, BN);
    uint8_t* sA = smem + L.a;
    uint8_t* sB = smem + L.b;
    uint8_t* sStage = smem + L.stage;
    __shared__ uint64_t b_full, a_full, a_empty, acc_full[2], acc_empty[2];
    __shared__ __align__(16) float sbias[3 * 128];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int failed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int NB = 3 * D / BN, nb = (int)blockIdx.x % NB;
    const int tile0 = (int)blockIdx.x / NB, tstep = (int)gridDim.x / NB;
    const int n_tiles = (R + 127) / 128;
    const int total = tile0 < n_tiles ? (n_tiles - 1 - tile0) / tstep + 1 : 0;
    uint32_t ncols = 32;
    while (ncols < 2u * BN) ncols <<= 1;
    if (threadIdx.x == 0) {
        tc::mbar_init(&b_full, 1);
        tc::mbar_init(&a_full, 1);
        tc::mbar_init(&a_empty, 1);
        for (int i = 0; i < 2; i++) {
            tc::mbar_init(&acc_full[i], 1);
            tc::mbar_init(&acc_empty[i], 4);
        }
        tc::fence_barrier_init();
        failed = 0;
        if ((tc::smem_u32(smem) & 1023u) || D > 128 || 3 * D % BN || ncols > 512) {
            failed = 1;
            atomicExch(err, 2);
        }
    }
    for (int i = threadIdx.x; i < BN && i < 3 * 128; i += blockDim.x) sbias[i] = bias[nb * BN + i];
    if (warp == 0) tc::tmem_alloc(&tmem_base, ncols);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    if (warp == 1 && tc::elect_one() && !failed) {
        tc::mbar_expect_tx(&b_full, (uint32_t)D * BN * 2);
        tc::bulk_load(sB, W + (size_t)nb * D * BN, (uint32_t)D * BN * 2, &b_full);
    }
    __syncwarp();
    JC_PDL_ENTRY;
    const uint32_t tmem = tmem_base;
    if (warp == 0) {
        if (tc::elect_one() && !failed) {
            for (int it = 0; it < total; it++) {
                if (it > 0 && !tc::mbar_wait(&a_empty, (uint32_t)(it - 1) & 1u, err, &failed)) break;
                const int m0 = (tile0 + it * tstep) * 128;
                tc::mbar_expect_tx(&a_full, (uint32_t)D * 256);
                if (SW)
                    for (int c = 0; c < D / 64; c++) tc::tma_load_2d(sA + c * 16384, &tmA, c * 64, m0, &a_full);
                else
                    for (int kc = 0; kc < D / 8; kc++) tc::tma_load_2d(sA + kc * 2048, &tmA, kc * 8, m0, &a_full);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (tc::elect_one() && !failed) {
            bool good = tc::mbar_wait(&b_full, 0, err, &failed);
            const uint32_t idesc = tc::idesc_bf16(128, BN);
            const uint64_t dA = SW ? tc::sdesc_sw128(tc::smem_u32(sA)) : tc::sdesc(tc::smem_u32(sA), 2048, 128);
            const uint64_t dB = tc::sdesc(tc::smem_u32(sB), BN * 16, 128);
            for (int it = 0; it < total && good; it++) {
                good = tc::mbar_wait(&a_full, (uint32_t)it & 1u, err, &failed) &&
                       (it < 2 || tc::mbar_wait(&acc_empty[it & 1], (uint32_t)((it - 2) >> 1) & 1u, err, &failed));
                if (!good) break;
                tc::tc_fence_after();
                const uint32_t acc = tmem + (uint32_t)(it & 1) * BN;
                for (int k = 0; k < D / 16; k++)
                    tc::mma_bf16(acc, tc::sdesc_at(dA, SW ? (k >> 2) * 16384 + (k & 3) * 32 : k * 4096),
                                 tc::sdesc_at(dB, k * 2 * BN * 16), idesc, k > 0 ? 1u : 0u);
                tc::mma_commit(&a_empty);
                tc::mma_commit(&acc_full[it & 1]);
            }
        }
        __syncwarp();
    } else {
        const int r = (warp & 3) * 32 + lane;
        for (int it = 0; it < total; it++) {
            const bool ready = tc::mbar_wait(&acc_full[it & 1], (uint32_t)(it >> 1) & 1u, err, &failed);
            if (warp == 2 && tc::elect_one()) tc::bulk_wait_read();  // the last store has read the staging area
            if (!all_of(ready, 1, 128)) break;
            tc::tc_fence_after();
            const uint32_t ta = lane_addr(tmem + (uint32_t)(it & 1) * BN);
            // 32 columns per TMEM round trip (BN is a multiple of 32)
            for (int c = 0; c < BN; c += 32) {
                float a[32];
                tc::tmem_ld32(ta + c, a);
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const float4 bv = *reinterpret_cast<const float4*>(sbias + c + i);
                    a[i] += bv.x;
                    a[i + 1] += bv.y;
                    a[i + 2] += bv.z;
                    a[i + 3] += bv.w;
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int cc = c + 16 * h;
                    uint8_t* box = sStage + (size_t)(cc / 64) * 16384 + (size_t)r * 128;
                    const int j0 = (cc % 64) / 8;
                    BfVec<8>::store(reinterpret_cast<bf16*>(box + ((j0 ^ (r & 7)) << 4)), a + 16 * h);
                    BfVec<8>::store(reinterpret_cast<bf16*>(box + (((j0 + 1) ^ (r & 7)) << 4)), a + 16 * h + 8);
                }
            }
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&acc_empty[it & 1]);
            tc::fence_async_shared();
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (warp == 2 && tc::elect_one()) {
                const int m0 = (tile0 + it * tstep) * 128;
                for (int c = 0; c < BN; c += 64) tc::tma_store_2d(&tmO, sStage + (size_t)(c / 64) * 16384, nb * BN + c, m0);
                tc::bulk_commit();
            }
        }
        if (warp == 2 && tc::elect_one()) tc::bulk_wait_read();
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, ncols);
}

// 3x3 zero-padded convolution over each instance's grid as an implicit GEMM
// (cpu.rs:171-205): tile = 8 x 16 positions (M = 128, row r <-> position
// (y0 + r/8, x0 + r%8)); the halo tile [C/8 planes][18][10][8] is loaded by
// TMA (zero fill outside the grid); tap (ky, kx) is the halo addressed from
// offset (ky*10 + kx)*16 bytes. B per tap: [C/8][BN][8] (the N block `nb`).
// Epilogue (token_mix): out = xn + gelu(acc + b) (cpu.rs:326-328), bf16. The
// cell-head convolutions have their own persistent kernel (tc_cellconv_kernel).

// Shared memory of tc_conv3_kernel: the halo planes, then the weight blocks of
// the taps in flight.
constexpr int kConvTaps = 2;
static __host__ __device__ size_t conv3_smem(int C, int BN) {
    return (size_t)(C / 8) * kHaloPlane + (size_t)kConvTaps * C * BN * 2;
}
// Where the epilogue stages its output boxes: after the halo, which it still
// reads (1024-aligned, for the 128-byte swizzle).
static __host__ __device__ size_t conv3_stage_offset(int C) {
    return ((size_t)(C / 8) * kHaloPlane + 1023) / 1024 * 1024;
}
// Dynamic shared memory of a launch: operands, or the staged output boxes
// (64 channels each) if those need more.
static size_t conv3_launch_smem(int C, int BN) {
    return std::max(conv3_smem(C, BN), conv3_stage_offset(C) + (size_t)((BN + 63) / 64) * 16384);
}

__global__ void __launch_bounds__(128) tc_conv3_kernel(const CUtensorMap* __restrict__ maps, int map_slot,
                                                       int store_slot, const bf16* __restrict__ Wt,
                                                       const float* __restrict__ bias, int C, int BN,
                                                       const InstDev* inst, int n_inst, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sHalo = smem;                                   // [C/8][18][10][8]
    uint8_t* sB = smem + (size_t)(C / 8) * kHaloPlane;       // NS x [C/8][BN][8]
    constexpr int NS = kConvTaps;
    __shared__ uint64_t bar_h, bar_b[NS], bar_m[NS], bar_done;
    __shared__ __align__(16) float sbias[256];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int failed;
    const int warp = threadIdx.x >> 5;
    // tile -> instance
    const int tile = blockIdx.x, nb = blockIdx.y;
    const int lo = warp_find_last_le(n_inst, tile, [&](int i) {
        return (long long)inst[i].tt0;
    });
    const InstDev I = inst[lo];
    const int gw = I.tx;
    const int tiles_x = (gw + kConvTX - 1) / kConvTX;
    const int tl = tile - I.tt0;
    const int x0 = (tl % tiles_x) * kConvTX, y0 = (tl / tiles_x) * kConvTY;
    const CUtensorMap* map = maps + kMapsPerInst * lo + map_slot;
    const CUtensorMap* omap = maps + kMapsPerInst * lo + store_slot;
    const uint32_t ncols = BN <= 32 ? 32 : (BN <= 64 ? 64 : (BN <= 128 ? 128 : 256));
    if (threadIdx.x == 0) {
        tc::mbar_init(&bar_h, 1);
        tc::mbar_init(&bar_done, 1);
        for (int i = 0; i < NS; i++) {
            tc::mbar_init(&bar_b[i], 1);
            tc::mbar_init(&bar_m[i], 1);
        }
        tc::fence_barrier_init();
        failed = 0;
        if (tc::smem_u32(smem) & 1023u) {  // aligned operand tiles
            failed = 1;
            atomicExch(err, 2);
        }
    }
    for (int i = threadIdx.x; i < BN; i += blockDim.x) sbias[i] = bias[nb * BN + i];
    if (warp == 0) tc::tmem_alloc(&tmem_base, ncols);
    tc::tc_fence_before();
    __syncthreads();
    JC_PDL_ENTRY;
    tc::tc_fence_after();
    const uint32_t tmem = tmem_base;
    const uint32_t wtap = (uint32_t)C * BN * 2;  // bytes of one tap's B block
    const bf16* Wn = Wt + (size_t)nb * 9 * C * BN;
    if (warp == 0 && tc::elect_one() && !failed) {
        tc::tensormap_acquire(map);
        tc::tensormap_acquire(omap);
        tc::mbar_expect_tx(&bar_h, (uint32_t)(C / 8) * (kHaloW * kHaloH * 16));
        for (int kc = 0; kc < C / 8; kc++)
            tc::tma_load_3d(sHalo + kc * kHaloPlane, map, kc * 8, x0 - 1, y0 - 1, &bar_h);
        for (int t = 0; t < NS; t++) {
            tc::mbar_expect_tx(&bar_b[t], wtap);
            tc::bulk_load(sB + t * wtap, Wn + (size_t)t * C * BN, wtap, &bar_b[t]);
        }
        bool good = tc::mbar_wait(&bar_h, 0, err, &failed);
        const uint32_t idesc = tc::idesc_bf16(128, BN);
        const uint64_t dH = tc::sdesc(tc::smem_u32(sHalo), kHaloPlane, kHaloW * 16), dB = tc::sdesc(tc::smem_u32(sB), BN * 16, 128);
        for (int t = 0; t < 9 && good; t++) {
            const int buf = t % NS;
            good = tc::mbar_wait(&bar_b[buf], (uint32_t)(t / NS) & 1u, err, &failed);
            if (!good) break;
            tc::tc_fence_after();
            const int ky = t / 3, kx = t % 3;
            const uint64_t dh = tc::sdesc_at(dH, (ky * kHaloW + kx) * 16), db = tc::sdesc_at(dB, buf * wtap);
            for (int k = 0; k < C / 16; k++)
                tc::mma_bf16(tmem, tc::sdesc_at(dh, 2 * k * kHaloPlane), tc::sdesc_at(db, 2 * k * BN * 16), idesc,
                             (t > 0 || k > 0) ? 1u : 0u);
            if (t + NS < 9) {
                // the stage is refilled once the MMAs reading it are done
                tc::mma_commit(&bar_m[buf]);
                good = tc::mbar_wait(&bar_m[buf], (uint32_t)(t / NS) & 1u, err, &failed);
                if (!good) break;
                tc::mbar_expect_tx(&bar_b[buf], wtap);
                tc::bulk_load(sB + buf * wtap, Wn + (size_t)(t + NS) * C * BN, wtap, &bar_b[buf]);
            }
        }
        if (good) tc::mma_commit(&bar_done);  // arrives when every MMA above is done
    }
    __syncwarp();
    const bool ok = __syncthreads_and(tc::mbar_wait(&bar_done, 0, err, &failed) ? 1 : 0) != 0;
    tc::tc_fence_after();
    if (ok) {
        // epilogue into 128-byte swizzled boxes of the 128 tile positions
        // (row r = position (y0 + r / 8, x0 + r % 8)), stored with TMA;
        // positions outside the grid are clipped by the store
        const int r = threadIdx.x;
        const uint32_t ta = lane_addr(tmem);
        constexpr int EB = 2;        // bytes per output element (bf16)
        constexpr int PB = 128 / EB;  // elements per box row
        // the epilogue still reads the halo centre, so it stages after the halo
        uint8_t* stage = smem + conv3_stage_offset(C);
        for (int c = 0; c < BN; c += 16) {
            float a[16];
            tc::tmem_ld16(ta + c, a);
            // the centre of the halo tile is xn at this token
            const uint8_t* centre = sHalo + ((r / kConvTX + 1) * kHaloW + (r % kConvTX + 1)) * 16;
            const int n0 = nb * BN;
#pragma unroll
            for (int i = 0; i < 16; i += 2) gelu_fast_pair(a[i], a[i + 1], sbias[c + i], sbias[c + i + 1]);
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const int ch = n0 + c + i;
                const float xn = bf2f(*reinterpret_cast<const bf16*>(centre + (size_t)(ch / 8) * kHaloPlane + (ch % 8) * 2));
                a[i] = xn + a[i];
            }
            uint8_t* box = stage + (size_t)(c / PB) * 16384 + (size_t)r * 128;
            const int j0 = (c % PB) * EB / 16;
            BfVec<8>::store(reinterpret_cast<bf16*>(box + ((j0 ^ (r & 7)) << 4)), a);
            BfVec<8>::store(reinterpret_cast<bf16*>(box + (((j0 + 1) ^ (r & 7)) << 4)), a + 8);
        }
        tc::fence_async_shared();
        __syncthreads();
        if (warp == 0 && tc::elect_one()) {
            for (int c = 0; c < BN; c += PB)
                tc::tma_store_3d(omap, stage + (size_t)(c / PB) * 16384, nb * BN + c, x0, y0);
            tc::bulk_commit();
            tc::bulk_wait_read();
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, ncols);
}

// token_mix and to_cells for dims up to 128 (cpu.rs:326-334): t1 = xn + gelu(
// conv3x3(xn) + b) rounded to bf16, z0 = t1 @ Wtc + b. Persistent, one CTA per SM
// walking 8 x 16 token tiles, its stages on separate warps:
//   0-3  copy each tile's halo (10 x 18 positions of xn) into one of two buffers
//        [C/8 planes][18][10][8], 16 bytes a copy, zeros outside the grid;
//   4    (one lane) loads the tap weights, one after another, into a ring of
//        three, and Wtc once, all before the previous kernel has finished where
//        they can be;
//   5    (one lane) issues the MMAs: 9 taps x C / 16 K steps into one of two TMEM
//        accumulators (tap (ky, kx) is the halo from position (ky, kx)), and
//        to_cells' from t1 in TMEM;
//   6-9  (one TMEM lane quarter each) the GELU and the residual, t1 packed into
//        TMEM, z0 to memory.
// A plane takes kMixPlane bytes, 16 more than its positions, so that a warp's
// copies (16 planes of two positions) fall on different banks. The MMA order is
// that of tc_conv3_kernel and tc_gemm_kernel, which serve wider models.
// At 64 K rows both took 48 us (the halo as 2880 16-byte pieces a tile through
// the TMA unit, two taps in flight, t1 through memory), this takes 33; four
// tiles: 19 and 13.
constexpr int kMixThreads = 10 * 32, kMixTaps = 3;
constexpr int kMixPlane = kHaloW * kHaloH * 16 + 16;

struct MixSmem {
    size_t halo, halo_bytes, w, tap, wtc, total;
    __host__ __device__ explicit MixSmem(int C) {
        halo = 0;
        halo_bytes = ((size_t)(C / 8) * kMixPlane + 127) / 128 * 128;
        w = (2 * halo_bytes + 1023) / 1024 * 1024;
        tap = (size_t)2 * C * C;  // [C/8][C][8]
        wtc = w + kMixTaps * tap;
        total = wtc + (size_t)64 * C;  // [C/8][32][8]
    }
};

__global__ void __launch_bounds__(kMixThreads, 1) tc_mix_cells_kernel(
    const bf16* __restrict__ xn, const bf16* __restrict__ Wt, const float* __restrict__ bias,
    const bf16* __restrict__ Wtc, const float* __restrict__ tc_bias, int C, int n_tiles, const InstDev* inst, int n_inst,
    float* __restrict__ z0, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int HD = 32, NS = kMixTaps;
    const MixSmem L(C);
    const uint32_t tap = (uint32_t)L.tap;
    __shared__ uint64_t h_full[2], h_empty[2], w_full[NS], w_empty[NS], wtc_full, acc_full[2], acc_empty[2], t_full, z_full;
    __shared__ __align__(16) float sbias[128], szb[HD];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int failed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int my_tiles = (int)blockIdx.x < n_tiles ? (n_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; i++) {
            tc::mbar_init(&h_full[i], 128);
            tc::mbar_init(&h_empty[i], 1 + 4);  // the MMAs have read the halo, and the epilogue warps its centre
            tc::mbar_init(&acc_full[i], 1);
            tc::mbar_init(&acc_empty[i], 4);
        }
        for (int i = 0; i < NS; i++) {
            tc::mbar_init(&w_full[i], 1);
            tc::mbar_init(&w_empty[i], 1);
        }
        tc::mbar_init(&wtc_full, 1);
        tc::mbar_init(&t_full, 4);
        tc::mbar_init(&z_full, 1);
        tc::fence_barrier_init();
        failed = 0;
        if ((tc::smem_u32(smem) & 1023u) || C > 128 || C % 32) {
            failed = 1;
            atomicExch(err, 2);
        }
    }
    for (int i = threadIdx.x; i < C && i < 128; i += kMixThreads) sbias[i] = bias[i];
    if (threadIdx.x < HD) szb[threadIdx.x] = tc_bias[threadIdx.x];
    if (warp == 0) tc::tmem_alloc(&tmem_base, 512);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tT = tmem_base + 256, tZ = tmem_base + 320;  // accumulators | t1 (C / 2 columns) | z0
    auto tile_of = [&](int it, int& x0, int& y0) {  // by a whole warp
        const int tile = (int)blockIdx.x + it * (int)gridDim.x;
        const int ii = warp_find_last_le(n_inst, tile, [&](int i) { return (long long)inst[i].tt0; });
        const int tiles_x = (inst[ii].tx + kConvTX - 1) / kConvTX, tl = tile - inst[ii].tt0;
        x0 = (tl % tiles_x) * kConvTX;
        y0 = (tl / tiles_x) * kConvTY;
        return ii;
    };
    if (warp < 4) {
        JC_PDL_ENTRY;
        const int np = C / 8;
        for (int it = 0; it < my_tiles; it++) {
            const int hb = it & 1;
            int x0, y0;
            const InstDev& I = inst[tile_of(it, x0, y0)];
            const int tx = I.tx, ty = I.ty;
            const bf16* base = xn + (size_t)I.row0 * C;
            bool ok = it < 2 || tc::mbar_wait(&h_empty[hb], (uint32_t)((it - 2) >> 1) & 1u, err, &failed);
            if (!__all_sync(0xffffffffu, ok ? 1 : 0)) break;
            uint8_t* dst = smem + L.halo + hb * L.halo_bytes;
            for (int e = threadIdx.x; e < kHaloW * kHaloH * np; e += 128) {
                const int pos = e / np, pl = e - pos * np;
                const int y = y0 + pos / kHaloW - 1, x = x0 + pos % kHaloW - 1;
                const bool in = y >= 0 && x >= 0 && y < ty && x < tx;
                cp_async16(dst + (size_t)pl * kMixPlane + pos * 16, in ? base + ((size_t)y * tx + x) * C + pl * 8 : xn, in);
            }
            cp_async_wait_all();
            tc::fence_async_shared();  // read by the MMAs
            tc::mbar_arrive(&h_full[hb]);
        }
    } else if (warp == 4) {
        if (tc::elect_one() && !failed) {
            bool ok = true;
            tc::mbar_expect_tx(&wtc_full, 64u * C);
            tc::bulk_load(smem + L.wtc, Wtc, 64u * C, &wtc_full);
            for (int g = 0; g < 9 * my_tiles && ok; g++) {
                const int sl = g % NS;
                if (g >= NS) ok = tc::mbar_wait(&w_empty[sl], (uint32_t)(g / NS - 1) & 1u, err, &failed);
                if (!ok) break;
                tc::mbar_expect_tx(&w_full[sl], tap);
                tc::bulk_load(smem + L.w + sl * tap, Wt + (size_t)(g % 9) * C * C, tap, &w_full[sl]);
            }
        }
        __syncwarp();
        JC_PDL_ENTRY;
    } else if (warp == 5) {
        JC_PDL_ENTRY;
        if (tc::elect_one() && !failed) {
            const uint32_t idC = tc::idesc_bf16(128, C), idZ = tc::idesc_bf16(128, HD);
            const uint64_t dH = tc::sdesc(tc::smem_u32(smem + L.halo), kMixPlane, kHaloW * 16);
            const uint64_t dW = tc::sdesc(tc::smem_u32(smem + L.w), C * 16, 128);
            const uint64_t dZ = tc::sdesc(tc::smem_u32(smem + L.wtc), HD * 16, 128);
            int z_done = 0;  // tiles whose to_cells has been issued
            auto issue_z = [&]() {
                tc::tc_fence_after();
                for (int k = 0; k < C / 16; k++)
                    tc::mma_bf16_ta(tZ, tT + k * 8, tc::sdesc_at(dZ, k * 2 * HD * 16), idZ, k > 0 ? 1u : 0u);
                tc::mma_commit(&z_full);
                z_done++;
            };
            bool ok = tc::mbar_wait(&wtc_full, 0, err, &failed);
            int g = 0;
            for (int it = 0; it < my_tiles && ok; it++) {
                const int b = it & 1;
                ok = tc::mbar_wait(&h_full[b], (uint32_t)(it >> 1) & 1u, err, &failed) &&
                     (it < 2 || tc::mbar_wait(&acc_empty[b], (uint32_t)((it - 2) >> 1) & 1u, err, &failed));
                const uint64_t dh = tc::sdesc_at(dH, b * (uint32_t)L.halo_bytes);
                for (int t = 0; t < 9 && ok; t++, g++) {
                    const int sl = g % NS;
                    ok = tc::mbar_wait(&w_full[sl], (uint32_t)(g / NS) & 1u, err, &failed);
                    if (!ok) break;
                    tc::tc_fence_after();
                    const uint64_t a = tc::sdesc_at(dh, ((t / 3) * kHaloW + t % 3) * 16), w = tc::sdesc_at(dW, sl * tap);
                    for (int k = 0; k < C / 16; k++)
                        tc::mma_bf16(tmem_base + b * 128, tc::sdesc_at(a, 2 * k * kMixPlane), tc::sdesc_at(w, 2 * k * C * 16),
                                     idC, (t > 0 || k > 0) ? 1u : 0u);
                    tc::mma_commit(&w_empty[sl]);
                    // the tile before has its t1: its to_cells goes in between
                    if (z_done < it && tc::mbar_try_wait(&t_full, (uint32_t)z_done & 1u)) issue_z();
                }
                if (!ok) break;
                tc::mma_commit(&h_empty[b]);
                tc::mma_commit(&acc_full[b]);
                if (z_done < it) {
                    ok = tc::mbar_wait(&t_full, (uint32_t)z_done & 1u, err, &failed);
                    if (ok) issue_z();
                }
            }
            if (ok && z_done < my_tiles && tc::mbar_wait(&t_full, (uint32_t)z_done & 1u, err, &failed)) issue_z();
        }
        __syncwarp();
    } else {
        JC_PDL_ENTRY;
        const int r = (warp & 3) * 32 + lane;
        auto warp_wait = [&](uint64_t* bar, uint32_t parity) {
            const bool good = __all_sync(0xffffffffu, tc::mbar_wait(bar, parity, err, &failed) ? 1 : 0) != 0;
            tc::tc_fence_after();
            return good;
        };
        for (int it = 0; it < my_tiles; it++) {
            const int b = it & 1;
            int x0, y0;
            const InstDev& I = inst[tile_of(it, x0, y0)];
            const int x = x0 + r % kConvTX, y = y0 + r / kConvTX;
            const bool inside = x < I.tx && y < I.ty;
            float* out = z0 + ((size_t)I.row0 + (inside ? (size_t)y * I.tx + x : 0)) * HD;
            if (!warp_wait(&h_full[b], (uint32_t)(it >> 1) & 1u) || !warp_wait(&acc_full[b], (uint32_t)(it >> 1) & 1u)) break;
            // the centre of the halo is xn at this token
            const uint8_t* centre = smem + L.halo + b * L.halo_bytes + ((r / kConvTX + 1) * kHaloW + r % kConvTX + 1) * 16;
            for (int c = 0; c < C; c += 32) {
                float a[32];
                tc::tmem_ld32(lane_addr(tmem_base + b * 128 + c), a);
                uint32_t h[16];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    float xv[8];
                    BfVec<8>::load(reinterpret_cast<const bf16*>(centre + (size_t)(c / 8 + q) * kMixPlane), xv);
#pragma unroll
                    for (int i = 0; i < 8; i += 2) {
                        float &v0 = a[8 * q + i], &v1 = a[8 * q + i + 1];
                        gelu_fast_pair(v0, v1, sbias[c + 8 * q + i], sbias[c + 8 * q + i + 1]);
                        __nv_bfloat162 t = __floats2bfloat162_rn(xv[i] + v0, xv[i + 1] + v1);
                        h[4 * q + i / 2] = *reinterpret_cast<uint32_t*>(&t);
                    }
                }
                tc::tmem_st16(lane_addr(tT + c / 2), h);
            }
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                tc::mbar_arrive(&acc_empty[b]);
                tc::mbar_arrive(&h_empty[b]);
                tc::mbar_arrive(&t_full);
            }
            if (!warp_wait(&z_full, (uint32_t)it & 1u)) break;
            float z[HD];
            tc::tmem_ld32(lane_addr(tZ), z);
            if (inside) {
#pragma unroll
                for (int i = 0; i < HD; i += 4)
                    *reinterpret_cast<float4*>(out + i) =
                        make_float4(z[i] + szb[i], z[i + 1] + szb[i + 1], z[i + 2] + szb[i + 2], z[i + 3] + szb[i + 3]);
            }
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem_base, 512);
}

// Persistent cell-head convolutions on the tensor cores, each CTA walking
// its run of consecutive cell tiles with its stages on separate warps, so the
// halo loads, the MMAs and the epilogue of consecutive tiles overlap. (With
// tiles gridDim.x apart each one was in another instance: looking that up, and
// fetching another tensor map, took longer than a tile's work. 64 x 128 x 128
// cells: conv1 55 and conv2 38 us, 46 and 32 in runs.)
//   warp 0     (one lane) TMA-loads each tile's halo into one of two slots;
//   warp 1     (one lane) issues a tile's MMAs into one of two TMEM
//              accumulators (the weights stay resident);
//   warps 2-5  (one TMEM lane quarter each) run the epilogue.
// kCellConv1, conv1 (cpu.rs:343-346): the 3x3 conv of the cell-head input zc
// (48 f16 channels) to 32 channels as 9 taps x 3 MMAs (tap (ky, kx) is the
// halo tile addressed from position (ky, kx)), + bias, GELU, stored as f16
// (c1) by each epilogue warp for itself: 128-byte runs of 8 cells in each of the
// four planes. Shared memory's 128 bytes a cycle bound it (the MMAs read 135 KB
// of A and weights a tile, 1080 cycles), so its epilogue stays out of there:
// with staged boxes, barrier arrivals by each thread instead of each warp and two
// CTA barriers a tile, a tick of 64 x 128 x 128 cells took 652 us, not 630.
// The MMA order and the epilogue arithmetic are those of tc_conv3_kernel.
// kCellConv2, conv2 and the step (cpu.rs:347-348, 84-88): 32 -> 3 channels.
// With 3 outputs the per-tap form would re-read the whole halo tile from
// shared memory for 9 tiny MMAs; instead one GEMM gives every halo position
// p its 27 tap contributions Z[p][(ky, kx), co] = c1[p] . W[co][.][ky][kx]
// (M = the 180 halo positions in two 128-row MMAs, N = 32 with 5 zero
// columns, K = 32 f16 channels, f32 sums), the epilogue stages Z in shared
// memory and each output cell adds its nine neighbours' contributions in
// tap order, + bias, + the state when the tick writes the next state, into
// the instance's planar output. Its f16 operands and sum order make it the
// BF16 form's own conv2 (the FP32 path keeps the reference's f32 order).
constexpr int kC1PThreads = 6 * 32;
constexpr int kCellConv1 = 0, kCellConv2 = 1;

// halo tiles in flight per CTA: two, so that three conv1 CTAs (four conv2
// CTAs) fit on an SM, which measured faster than three stages at two (three)
constexpr int kC1PHaloStages = 2;
constexpr int kHaloPos = kHaloW * kHaloH;  // 180 halo positions
constexpr int kZPitch = 33;                // f32 per staged Z row (bank-conflict-free column reads)

// TMEM columns per accumulator, weight bytes and staged bytes (Z) of each kind.
__host__ __device__ constexpr int cellconv_bn(int kind) { return kind == kCellConv1 ? 32 : 64; }
__host__ __device__ constexpr size_t cellconv_wbytes(int kind, int C) {
    return kind == kCellConv1 ? (size_t)9 * C * 32 * 2 : (size_t)C * 32 * 2;
}
__host__ __device__ constexpr size_t cellconv_stage(int kind) {
    return kind == kCellConv1 ? 0 : (size_t)kHaloPos * kZPitch * 4;
}

struct C1PSmem {
    size_t halo, w, stage, total;
    __host__ __device__ C1PSmem(int kind, int C) {
        halo = 0;                                                          // stages x [C/8][18][10][8]
        w = halo + (size_t)kC1PHaloStages * (C / 8) * kCellPlane;          // the weight blocks
        stage = (w + cellconv_wbytes(kind, C) + 1023) / 1024 * 1024;       // conv2's Z
        total = stage + cellconv_stage(kind);
    }
};

template <int KIND>
__global__ void __launch_bounds__(kC1PThreads) tc_cellconv_kernel(const CUtensorMap* __restrict__ maps,
                                                                   const bf16* __restrict__ Wt,
                                                                   const float* __restrict__ bias, int C,
                                                                   int n_tiles, const InstDev* inst, int n_inst,
                                                                   int mode, __half* __restrict__ c1,
                                                                   long long c1_plane, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int BN = cellconv_bn(KIND);
    constexpr int kInSlot = KIND == kCellConv1 ? 1 : 3;  // zc halo | c1 halo
    const C1PSmem L(KIND, C);
    uint8_t* sHalo = smem + L.halo;
    uint8_t* sW = smem + L.w;
    uint8_t* sStage = smem + L.stage;
    const size_t halo_bytes = (size_t)(C / 8) * kCellPlane;
    const uint32_t wbytes = (uint32_t)cellconv_wbytes(KIND, C);
    constexpr int HS = kC1PHaloStages;
    constexpr int kBias = KIND == kCellConv1 ? 32 : 3;
    __shared__ uint64_t w_full, h_full[HS], h_empty[HS], a_full[2], a_empty[2];
    __shared__ __align__(16) float sbias[32];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int failed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile0 = (int)((long long)n_tiles * blockIdx.x / gridDim.x);
    const int my_tiles = (int)((long long)n_tiles * (blockIdx.x + 1) / gridDim.x) - tile0;
    if (threadIdx.x == 0) {
        tc::mbar_init(&w_full, 1);
        for (int i = 0; i < HS; i++) {
            tc::mbar_init(&h_full[i], 1);
            tc::mbar_init(&h_empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            tc::mbar_init(&a_full[i], 1);
            tc::mbar_init(&a_empty[i], 4);  // the epilogue warps
        }
        tc::fence_barrier_init();
        failed = 0;
        if (tc::smem_u32(smem) & 1023u) {
            failed = 1;
            atomicExch(err, 2);
        }
    }
    if (threadIdx.x < 32) sbias[threadIdx.x] = (int)threadIdx.x < kBias ? bias[threadIdx.x] : 0.f;
    if (warp == 0) tc::tmem_alloc(&tmem_base, 2 * BN);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_base;
    // the instance of the CTA's first tile; the tiles are consecutive, so a walk
    // over them looks at the next instance only
    int ii = my_tiles > 0 ? warp_find_last_le(n_inst, tile0, [&](int i) { return (long long)inst[i].ct0; }) : 0;
    auto next_ct0 = [&]() { return ii + 1 < n_inst ? inst[ii + 1].ct0 : INT_MAX; };
    int next = next_ct0();
    JC_PDL_ENTRY;
    if (warp == 0) {
        if (tc::elect_one() && !failed) {
            // halo producer
            int held = -1, ct0 = 0, tiles_x = 1;  // the instance whose map this thread has acquired
            for (int it = 0; it < my_tiles; it++) {
                const int hb = it % HS;
                while (tile0 + it >= next) {
                    ii++;
                    next = next_ct0();
                }
                if (ii != held) {
                    held = ii;
                    ct0 = inst[ii].ct0;
                    tiles_x = (inst[ii].nx + kConvTX - 1) / kConvTX;
                    tc::tensormap_acquire(maps + kMapsPerInst * ii + kInSlot);
                }
                const int tl = tile0 + it - ct0, x0 = tl % tiles_x * kConvTX, y0 = tl / tiles_x * kConvTY;
                const CUtensorMap* map = maps + kMapsPerInst * ii + kInSlot;
                if (it >= HS && !tc::mbar_wait(&h_empty[hb], (uint32_t)((it - HS) / HS) & 1u, err, &failed)) break;
                tc::mbar_expect_tx(&h_full[hb], (uint32_t)halo_bytes);
                tc::tma_load_3d(sHalo + hb * halo_bytes, map, (x0 - 1) * 8, y0 - 1, 0, &h_full[hb]);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (tc::elect_one() && !failed) {
            // MMA issuer: the weights once, then every tile
            tc::mbar_expect_tx(&w_full, wbytes);
            tc::bulk_load(sW, Wt, wbytes, &w_full);
            bool good = tc::mbar_wait(&w_full, 0, err, &failed);
            const uint32_t idesc = tc::idesc_f16(128, 32);  // f16 input and weights, N = 32
            const uint64_t dW = tc::sdesc(tc::smem_u32(sW), 32 * 16, 128);
            const uint64_t dH = tc::sdesc(tc::smem_u32(sHalo), kCellPlane, KIND == kCellConv1 ? kHaloW * 16 : 128);
            for (int it = 0; it < my_tiles && good; it++) {
                const int b = it & 1, hb = it % HS;
                good = tc::mbar_wait(&h_full[hb], (uint32_t)(it / HS) & 1u, err, &failed) &&
                       (it < 2 || tc::mbar_wait(&a_empty[b], (uint32_t)((it - 2) >> 1) & 1u, err, &failed));
                if (!good) break;
                tc::tc_fence_after();
                const uint64_t dh = tc::sdesc_at(dH, hb * (uint32_t)halo_bytes);
                const uint32_t acc = tmem + (uint32_t)b * BN;
                if constexpr (KIND == kCellConv1) {
                    // rows = the 8 x 16 output positions (8-row groups 10 positions apart)
#pragma unroll
                    for (int t = 0; t < 9; t++)
#pragma unroll
                        for (int k = 0; k < kZcCh / 16; k++)
                            tc::mma_bf16(acc, tc::sdesc_at(dh, 2 * k * kCellPlane + ((t / 3) * kHaloW + t % 3) * 16),
                                         tc::sdesc_at(dW, (t * kZcCh / 8 + 2 * k) * 32 * 16), idesc,
                                         (t > 0 || k > 0) ? 1u : 0u);
                } else {
                    // rows = halo positions 0..127 and 128..255 (those past 179,
                    // read past the plane, are never used)
#pragma unroll
                    for (int m = 0; m < 2; m++)
#pragma unroll
                        for (int k = 0; k < 2; k++)
                            tc::mma_bf16(acc + (uint32_t)m * 32, tc::sdesc_at(dh, 2 * k * kCellPlane + m * 128 * 16),
                                         tc::sdesc_at(dW, 2 * k * 32 * 16), idesc, k > 0 ? 1u : 0u);
                }
                tc::mma_commit(&h_empty[hb]);
                tc::mma_commit(&a_full[b]);
            }
        }
        __syncwarp();
    } else {
        // epilogue: thread r = TMEM lane r
        const int r = (warp & 3) * 32 + lane;
        InstDev I;
        int held = -1;
        for (int it = 0; it < my_tiles; it++) {
            const int b = it & 1;
            // the tile's origin and (conv2) state, fetched before the wait so
            // their latency overlaps the MMAs
            const int tile = tile0 + it;
            while (tile >= next) {
                ii++;
                next = next_ct0();
            }
            if (ii != held) {
                held = ii;
                I = inst[ii];
            }
            const int tiles_x = (I.nx + kConvTX - 1) / kConvTX;
            const int x0 = ((tile - I.ct0) % tiles_x) * kConvTX, y0 = ((tile - I.ct0) / tiles_x) * kConvTY;
            const int x = x0 + (r & 7), y = y0 + (r >> 3);
            const bool inside = x < I.nx && y < I.ny;
            const size_t plane = (size_t)I.nx * I.ny, cl = inside ? (size_t)y * I.nx + x : 0;
            float st[3] = {0.f, 0.f, 0.f};
            if (KIND == kCellConv2 && inside && mode == kWriteNextState) {
#pragma unroll
                for (int co = 0; co < 3; co++) st[co] = I.state[co * plane + cl];
            }
            const uint32_t ta = lane_addr(tmem + (uint32_t)b * BN);
            if constexpr (KIND == kCellConv2) {
                const bool ready = tc::mbar_wait(&a_full[b], (uint32_t)(it >> 1) & 1u, err, &failed);
                uint32_t all_ready;
                asm volatile(
                    "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbarrier.red.and.pred p, 1, 128, q;\n\t"
                    "selp.u32 %0, 1, 0, p;\n\t}"
                    : "=r"(all_ready)
                    : "r"(ready ? 1u : 0u)
                    : "memory");
                if (!all_ready) break;
                tc::tc_fence_after();
                // Z rows r and 128 + r -> shared memory, then output cell r
                float* Z = reinterpret_cast<float*>(sStage);
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    float a[32];
                    tc::tmem_ld32(ta + m * 32, a);
                    const int pos = m * 128 + r;
                    if (pos < kHaloPos) {
#pragma unroll
                        for (int c = 0; c < 27; c++) Z[pos * kZPitch + c] = a[c];
                    }
                }
                tc::tc_fence_before();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&a_empty[b]);
                asm volatile("bar.sync 1, 128;" ::: "memory");
                const int lx = r & 7, ly = r >> 3;
                float v[3] = {0.f, 0.f, 0.f};
#pragma unroll
                for (int t = 0; t < 9; t++) {
                    const float* zr = Z + ((ly + t / 3) * kHaloW + lx + t % 3) * kZPitch + 3 * t;
#pragma unroll
                    for (int co = 0; co < 3; co++) v[co] += zr[co];
                }
                if (inside) {
#pragma unroll
                    for (int co = 0; co < 3; co++) {
                        float o = v[co] + sbias[co];
                        if (mode == kWriteNextState) o = o + st[co];
                        I.out[co * plane + cl] = o;
                    }
                }
                // (the next tile's first barrier comes before Z is written again)
            } else {
                // the warps go their own ways: no staging, no barrier
                if (!__all_sync(0xffffffffu, tc::mbar_wait(&a_full[b], (uint32_t)(it >> 1) & 1u, err, &failed) ? 1 : 0)) break;
                tc::tc_fence_after();
                float a[32];
                tc::tmem_ld32(ta, a);
                tc::tc_fence_before();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&a_empty[b]);
                __half* o = c1 + ((size_t)I.cell0 + cl) * 8;
#pragma unroll
                for (int c = 0; c < 32; c += 8) {
                    uint32_t w[4];
#pragma unroll
                    for (int i = 0; i < 8; i += 2) {
                        gelu_fast_pair(a[c + i], a[c + i + 1], sbias[c + i], sbias[c + i + 1]);
                        __half2 h = __floats2half2_rn(a[c + i], a[c + i + 1]);
                        w[i / 2] = *reinterpret_cast<uint32_t*>(&h);
                    }
                    if (inside) *reinterpret_cast<uint4*>(o + (c / 8) * c1_plane) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 2 * BN);
}

// Whether the shared-memory attention tiles apply (radius-1, dilation-1
// stencil; 64-channel boxes; at most 4 heads of width 32 or 64).
static bool attn_tile_ok(const Dims& d) {
    return d.mask_kind == 1 && d.radius == 1 && d.dilation == 1 && d.D % 64 == 0 && d.heads <= 4 &&
           (d.D / d.heads == 32 || d.D / d.heads == 64);
}
static size_t attn_tile_smem(const Dims&) { return (size_t)2 * kAttBoxKVPad + kAttBoxQ; }

// ---------------------------------------------------------------------------
// host

static const bf16* upload_bf16(DeviceArena& a, const std::vector<uint16_t>& v) {
    return static_cast<const bf16*>(a.upload_bytes(v.data(), v.size() * 2));
}

// B[n][k] for n < N, k < K into [N/BN][K/8][BN][8].
static std::vector<uint16_t> blocked(int N, int K, int BN, const std::function<float(int, int)>& f) {
    std::vector<uint16_t> out((size_t)N * K);
    size_t i = 0;
    for (int nb = 0; nb < N / BN; nb++)
        for (int kc = 0; kc < K / 8; kc++)
            for (int n = 0; n < BN; n++)
                for (int e = 0; e < 8; e++) out[i++] = f2bf(f(nb * BN + n, kc * 8 + e));
    return out;
}

static const HostTensor& tget(const TensorMap& t, const std::string& n) {
    auto it = t.find(n);
    if (it == t.end()) throw Error(JC_BAD_CHECKPOINT, "missing tensor `" + n + "`");
    return it->second;
}

template <class K>
static void set_smem(K kernel, size_t bytes) {
    cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes),
               "cudaFuncSetAttribute");
}

void BF16Path::weight_slots(std::vector<const void**>& out) const {
    auto add = [&](const bf16* const& p) { out.push_back(reinterpret_cast<const void**>(const_cast<const bf16**>(&p))); };
    for (int l = 0; l < dims_.L; l++) {
        add(wqkv[l]);
        add(wp[l]);
    }
    for (int v = 0; v < n_nc; v++)
        for (int l = 0; l < dims_.L; l++) {
            add(w1v[v][l]);
            add(w2v[v][l]);
        }
    add(wtm);
    add(wtc);
    add(wc1);
    add(wc2);
}

BF16Path::BF16Path(const Dims& d, const TensorMap* tp, DeviceArena* ap) {
    const int D = d.D, F = d.F, HD = d.HD;
    dims_D_ = D;
    dims_F_ = F;
    dims_ = d;
    if (D % 32 || D > 256 || 32 % d.heads || F % 64 || HD != 32 || d.C != 3 || d.P != 4 || d.C * d.P * d.P > 64)
        throw Error(JC_LIMIT,
                    "the BF16 path needs dim a multiple of 32 and <= 256, heads dividing 32, a cell-head width of 32, "
                    "3 channels and patch 4");
    n_nc = 2;  // MLP weights arranged for chunk widths 32 and 64
    bn_qkv = (3 * D) % 128 == 0 ? 128 : 3 * D;
    bn_tm = D <= 128 ? D : 64;
    if (F > 1024) throw Error(JC_LIMIT, "the BF16 MLP supports a hidden width of at most 1024");
    {
        int dev = 0;
        cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
        cuda_check(cudaDeviceGetAttribute(&n_sms_, cudaDevAttrMultiProcessorCount, dev), "SM count");
    }
    // default: the serial kernel, 64 columns (fits every supported width)
    def_tuning_ = Tuning{64, 256};
    if (!mlp_fits(64)) def_tuning_.nc = 32;
    if (!mlp_fits(def_tuning_.nc)) throw Error(JC_LIMIT, "the BF16 MLP does not fit in shared memory at this width");
    if (attn_tile_ok(d)) def_tuning_.attn_threads = 0;  // shared-memory attention tiles
    for (int l = 0; l < kMaxLayers; l++) {
        wqkv[l] = wp[l] = nullptr;
        w1v[0][l] = w1v[1][l] = w2v[0][l] = w2v[1][l] = nullptr;
    }
    wtm = wtc = wc1 = nullptr;
    if (tp) upload_weights(d, *tp, *ap);
    cache_key_ = "d" + std::to_string(D) + "_l" + std::to_string(d.L) + "_f" + std::to_string(F) + "_r" +
                 std::to_string(d.radius) + "_k" + std::to_string(d.mask_kind) + "_g" + std::to_string(d.dilation);
    load_cache();
    set_kernel_attributes();
}

void BF16Path::upload_weights(const Dims& d, const TensorMap& t, DeviceArena& arena) {
    const int D = d.D, F = d.F, HD = d.HD;
    for (int l = 0; l < d.L; l++) {
        const std::string p = "blocks." + std::to_string(l) + ".";
        const auto &q = tget(t, p + "q.weight").data, &k = tget(t, p + "k.weight").data, &v = tget(t, p + "v.weight").data;
        // B[n][k] = Wqkv[k][n]: q | k | v along n
        wqkv[l] = upload_bf16(arena, blocked(3 * D, D, bn_qkv, [&](int n, int kk) {
                                  const auto& w = n < D ? q : (n < 2 * D ? k : v);
                                  return w[(size_t)kk * D + (n % D)];
                              }));
        const auto& wpr = tget(t, p + "proj.weight").data;
        wp[l] = upload_bf16(arena, blocked(D, D, D, [&](int n, int kk) { return wpr[(size_t)kk * D + n]; }));
        const auto& w1h = tget(t, p + "ff1.weight").data;  // [D, F]
        const auto& w2h = tget(t, p + "ff2.weight").data;  // [F, D]
        for (int v = 0; v < n_nc; v++) {
            const int nc = v == 0 ? 32 : 64;
            w1v[v][l] = upload_bf16(arena, blocked(F, D, nc, [&](int n, int kk) { return w1h[(size_t)kk * F + n]; }));
            // W2 chunk j: B2_j[n][k] = W2[j*nc + k][n] -> [j][nc/8][D][8]
            std::vector<uint16_t> w2b((size_t)F * D);
            size_t i = 0;
            for (int j = 0; j < F / nc; j++)
                for (int kc = 0; kc < nc / 8; kc++)
                    for (int n = 0; n < D; n++)
                        for (int e = 0; e < 8; e++) w2b[i++] = f2bf(w2h[(size_t)(j * nc + kc * 8 + e) * D + n]);
            w2v[v][l] = upload_bf16(arena, w2b);
        }
    }
    {
        // token_mix: per N block of 128 (or D) and tap: [C/8][BN][8] of W[co][ci][ky][kx]
        const auto& w = tget(t, "head.token_mix.weight").data;
        const int BN = bn_tm;
        std::vector<uint16_t> o((size_t)9 * D * D);
        size_t i = 0;
        for (int nb = 0; nb < D / BN; nb++)
            for (int tap = 0; tap < 9; tap++)
                for (int kc = 0; kc < D / 8; kc++)
                    for (int n = 0; n < BN; n++)
                        for (int e = 0; e < 8; e++)
                            o[i++] = f2bf(w[((size_t)(nb * BN + n) * D + kc * 8 + e) * 9 + tap]);
        wtm = upload_bf16(arena, o);
    }
    {
        const auto& w = tget(t, "head.to_cells.weight").data;  // [HD][D]
        wtc = upload_bf16(arena, blocked(HD, D, HD, [&](int n, int kk) { return w[(size_t)n * D + kk]; }));
    }
    {
        // conv1 (f16 operands): per tap [48/8][32][8] over the zc channels: z
        // (32), then the state's [hi, lo, hi] parts with weights [W_hi, W_hi, W_lo]
        const auto& w = tget(t, "head.conv1.weight").data;  // [HD][HD+C][3][3]
        const int cin = HD + d.C;
        auto h_round = [](float v) { return __half2float(__float2half_rn(v)); };
        std::vector<uint16_t> o((size_t)9 * kZcCh * HD);
        size_t i = 0;
        for (int tap = 0; tap < 9; tap++)
            for (int kc = 0; kc < kZcCh / 8; kc++)
                for (int n = 0; n < HD; n++)
                    for (int e = 0; e < 8; e++) {
                        const int ch = kc * 8 + e;
                        float v = 0.0f;
                        if (ch < HD) {
                            v = w[((size_t)n * cin + ch) * 9 + tap];
                        } else if (ch < kZcState + 9) {
                            const int part = (ch - kZcState) / 3, c = (ch - kZcState) % 3;
                            const float full = w[((size_t)n * cin + HD + c) * 9 + tap];
                            const float hi = h_round(full);
                            v = part < 2 ? hi : full - hi;
                        }
                        o[i++] = f2h(v);
                    }
        wc1 = upload_bf16(arena, o);  // f16 bits
    }
    {
        // conv2 (f16 operands): [32/8][32][8] over the c1 channels, column
        // n = 3 tap + co for tap = 3 ky + kx, columns 27..31 zero
        const auto& w = tget(t, "head.conv2.weight").data;  // [C][HD][3][3]
        std::vector<uint16_t> o((size_t)HD * 32);
        size_t i = 0;
        for (int kc = 0; kc < HD / 8; kc++)
            for (int n = 0; n < 32; n++)
                for (int e = 0; e < 8; e++)
                    o[i++] = f2h(n < 9 * d.C ? w[((size_t)(n % 3) * HD + kc * 8 + e) * 9 + n / 3] : 0.0f);
        wc2 = upload_bf16(arena, o);  // f16 bits
    }
}

void BF16Path::set_kernel_attributes() {
    set_smem(tc_gemm_kernel<EPI_BF16>, 200 * 1024);
    set_smem(tc_gemm_kernel<EPI_F32>, 200 * 1024);
    set_smem(tc_gemm_kernel<EPI_RESID_LN>, 200 * 1024);
    set_smem(tc_mlp_serial_kernel, kMlpSmemMax);
    set_smem(tc_mlp_wide_kernel, mlp_wide_smem(256));
    set_smem(tc_proj_mlp_kernel<false>, kPMSmem);
    set_smem(tc_proj_mlp_kernel<true>, kPMSmem);
    set_smem(tc_projln_persistent_kernel, 225 * 1024);  // 227 KB per CTA less the static shared memory
    set_smem(tc_qkv_kernel<false>, 225 * 1024);
    set_smem(tc_qkv_kernel<true>, 225 * 1024);
    set_smem(tc_cellconv_kernel<kCellConv1>, 200 * 1024);
    set_smem(tc_cellconv_kernel<kCellConv2>, 200 * 1024);
    set_smem(bf_attn_tile_kernel<32>, 200 * 1024);
    set_smem(bf_attn_tile_kernel<64>, 200 * 1024);
    set_smem(tc_conv3_kernel, 200 * 1024);
    set_smem(tc_mix_cells_kernel, 225 * 1024);
    set_smem(bf_embed_kernel<1, 2>, 100 * 1024);
    set_smem(bf_embed_kernel<1, 8>, 100 * 1024);
    set_smem(bf_embed_kernel<2, 2>, 100 * 1024);
    set_smem(bf_embed_kernel<2, 8>, 100 * 1024);
    set_smem(bf_embed_kernel<3, 2>, 100 * 1024);
    set_smem(bf_embed_kernel<3, 8>, 100 * 1024);
    set_smem(bf_embed_kernel<4, 2>, 100 * 1024);
    set_smem(bf_embed_kernel<4, 8>, 100 * 1024);
    set_smem(bf_embed_kernel<5, 2>, 100 * 1024);
    set_smem(bf_embed_kernel<5, 8>, 100 * 1024);
    set_smem(bf_embed_kernel<6, 2>, 100 * 1024);
    set_smem(bf_embed_kernel<6, 8>, 100 * 1024);
    set_smem(bf_embed_kernel<7, 2>, 100 * 1024);
    set_smem(bf_embed_kernel<7, 8>, 100 * 1024);
    set_smem(bf_embed_kernel<8, 2>, 100 * 1024);
    set_smem(bf_embed_kernel<8, 8>, 100 * 1024);
}

void BF16Path::arrange(DeviceArena& arena, cudaStream_t s) {
    if (dims_D_ != kPMD) return;
    const size_t pieces = (size_t)(kPMD + 2 * dims_F_) * kPMD / 8;  // 16 bytes each
    for (int l = 0; l < dims_.L; l++) {
        bf16* dst = static_cast<bf16*>(arena.alloc(pieces * 16));
        pm_arrange_kernel<<<(unsigned)((pieces + 255) / 256), 256, 0, s>>>(
            reinterpret_cast<const uint4*>(wp[l]), reinterpret_cast<const uint4*>(w1v[1][l]),
            reinterpret_cast<const uint4*>(w2v[1][l]), dims_F_, reinterpret_cast<uint4*>(dst));
        check_launch("pm_arrange");
        pm_w_[l] = dst;
    }
}

// One thread per (token row, head) in CTAs of `threads` threads (64, 128 or
// 256; the arithmetic of a thread does not depend on it).

static void launch_attention(const Dims& d, const bf16* qkv, const InstDev* inst, int n, int R, bf16* attn,
                             int threads, cudaStream_t s, const Pack* p = nullptr) {
    if (threads == 0) {
        // shared-memory tiles: grid (8 x 16 token tiles, their two 8 x 8 halves)
        const CUtensorMap* maps = reinterpret_cast<const CUtensorMap*>(p->tmaps);
        // one CTA per (token tile, 8 x 8 half, 64-channel box of heads)
        const dim3 grid((unsigned)p->n_ttiles, 2, (unsigned)(d.D / 64));
        if (d.D / d.heads == 32)
            cuda_check(launch_pdl(bf_attn_tile_kernel<32>, grid, 64 * 2, attn_tile_smem(d), s, 1u, d, maps, 4, 5, inst,
                                  n, attn, p->err),
                       "launch");
        else
            cuda_check(launch_pdl(bf_attn_tile_kernel<64>, grid, 64, attn_tile_smem(d), s, 1u, d, maps, 4, 5, inst, n,
                                  attn, p->err),
                       "launch");
        return;
    }
    const bool r1 = d.mask_kind == 1 && d.radius == 1;
    const int hd = d.D / d.heads;
    const unsigned blocks = (unsigned)(((long long)R * d.heads + threads - 1) / threads);
#define JC_ATTN_HEAD(H)                                                                          \
    if (hd == H) {                                                                               \
        if (r1) cuda_check(launch_pdl(bf_attn_head_r1_kernel<H>, blocks, threads, 0, s, 1u, d, qkv, inst, n, R, attn), "launch"); \
        else cuda_check(launch_pdl(bf_attn_head_kernel<H>, blocks, threads, 0, s, 1u, d, qkv, inst, n, R, attn), "launch");       \
        return;                                                                                  \
    }
    JC_ATTN_HEAD(8)
    JC_ATTN_HEAD(16)
    JC_ATTN_HEAD(32)
    JC_ATTN_HEAD(64)
#undef JC_ATTN_HEAD
}

// Before anything is launched: with the other widths the dim is one that no kernel
// here is made for (96 has 288 q/k/v columns, more than an MMA or the tensor memory takes).
static void check_head_width(const Dims& d) {
    const int hd = d.D / d.heads;
    if (hd != 8 && hd != 16 && hd != 32 && hd != 64)
        throw Error(JC_LIMIT, "the BF16 attention supports head widths 8, 16, 32 and 64");
}

static int initial_autotune() {
    const char* e = std::getenv("JC_AUTOTUNE");
    return e && std::atoi(e) == 0 ? 0 : 1;
}
std::atomic<int> g_autotune{initial_autotune()};

static int row_bucket(int R) {
    int b = 128;
    while (b < R && b < (1 << 30)) b <<= 1;
    return b;
}

Tuning BF16Path::tuning_for(int rows) const {
    std::lock_guard<std::mutex> lk(tune_mu_);
    if (g_autotune.load()) {
        auto it = tuned_.find(row_bucket(rows));
        if (it != tuned_.end()) return it->second;
    }
    return def_tuning_;
}

// Shared memory of the serial MLP kernel (one stage, one h buffer).
static size_t mlp_serial_smem(int D, int NC) {
    return std::max((size_t)D * 256 + 2 * (size_t)D * NC * 2 + (size_t)NC * 256, (size_t)128 * D * 4);
}

bool BF16Path::mlp_fits(int nc) const {
    return (nc == 32 || nc == 64) && dims_F_ % nc == 0 && mlp_serial_smem(dims_D_, nc) <= kMlpSmemMax;
}

bool BF16Path::proj_fuses(const Tuning& tu) const { return dims_D_ == kPMD && tu.nc == 64; }

void BF16Path::launch_mlp(const Dims& d, const WeightsF32& w, int l, const Tuning& tu, const CUtensorMap& m_ln,
                          const Pack& p, cudaStream_t s, const CUtensorMap* m_attn, const CUtensorMap* m_x) const {
    const int D = d.D, R = p.R;
    const int v = tu.nc == 64 ? 1 : 0;
    const float* ng = l + 1 < d.L ? w.blk[l + 1].n1g : w.norm_g;
    const float* nbeta = l + 1 < d.L ? w.blk[l + 1].n1b : w.norm_b;
    const auto& B = w.blk[l];
    bf16* ln = reinterpret_cast<bf16*>(p.bt[0]);
    if (m_attn) {
        if (!proj_fuses(tu)) throw Error(JC_LIMIT, "the fused projection needs dim 128 and 64-column MLP chunks");
        // While half of the SMs would stand idle two CTAs share a tile (one CTA | two, us a
        // launch between events: 8 tiles 19.2 | 15.9, 32 tiles 19.6 | 16.4, 72 tiles 19.7 |
        // 16.3); from there on a second CTA waits for an SM (80 tiles 20.2 | 26.6).
        const int tiles = (R + 127) / 128;
        const bool split = 2 * tiles <= n_sms_;
        cuda_check(launch_pdl(split ? tc_proj_mlp_kernel<true> : tc_proj_mlp_kernel<false>,
                              (unsigned)(split ? 2 * tiles : std::min(tiles, n_sms_)), kPMThreads, kPMSmem, s, 1u, *m_attn, m_ln,
                              *m_x, pm_w_[l], pm_w_[l] + D * D, pm_w_[l] + D * D + (size_t)d.F * D, B.bp, B.n2g, B.n2b, B.b1, B.b2, ng,
                              nbeta, d.F, R, p.x, ln, p.err),
                   "launch");
        return;
    }
    if (mlp_wide(D, tu.nc)) {
        cuda_check(launch_pdl(tc_mlp_wide_kernel, (unsigned)((R + 127) / 128), kMWThreads, mlp_wide_smem(D), s, 1u,
                              store_map(ln, D, R, D, false), w1v[v][l], w2v[v][l], B.b1, B.b2, D, d.F, R, p.x, ng, nbeta, ln, p.err),
                   "launch");
        return;
    }
    cuda_check(launch_pdl(tc_mlp_serial_kernel, (unsigned)((R + 127) / 128), kMlpSerialThreads,
                          mlp_serial_smem(D, tu.nc), s, 1u, m_ln, w1v[v][l], w2v[v][l], B.b1, B.b2, D, d.F, tu.nc, R,
                          p.x, ng, nbeta, ln, p.err),
               "launch");
}

// Times `launch` with CUDA events: one warm-up, then `reps` launches.
template <class F>
static float time_launches(F&& launch, int reps, cudaStream_t s) {
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    launch();
    cudaEventRecord(a, s);
    for (int i = 0; i < reps; i++) launch();
    cudaEventRecord(b, s);
    cudaEventSynchronize(b);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    return ms / reps;
}

void BF16Path::tune(const Dims& d, const WeightsF32& w, const Pack& p, cudaStream_t s) const {
    if (!g_autotune.load() || p.R == 0) return;
    check_head_width(d);
    const int bucket = row_bucket(p.R);
    {
        std::lock_guard<std::mutex> lk(tune_mu_);
        if (tuned_.count(bucket)) return;
    }
    cudaStreamCaptureStatus cs;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return;
    const int R = p.R, D = d.D;
    bf16* ln = reinterpret_cast<bf16*>(p.bt[0]);
    bf16* qkv = reinterpret_cast<bf16*>(p.bt[1]);
    bf16* attn = reinterpret_cast<bf16*>(p.bt[2]);
    const CUtensorMap m_ln = rows_map(ln, D, R);
    Tuning best = def_tuning_;
    // the workspace holds transient values; the timed launches may leave
    // anything in it (every forward rewrites it from the state)
    std::string log;
    // A candidate replaces the default only when it is clearly faster (by
    // kTuneMargin): a bucket's choice also serves other mixes of instance
    // sizes with that row count, and single timings vary by a few percent.
    constexpr float kTuneMargin = 0.95f;
    constexpr int kTuneReps = 8;
    float def_ms = 0.f, best_ms = 1e30f;
    for (int nc : {def_tuning_.nc, 96 - def_tuning_.nc}) {  // the default width first, then the other
        // where the default width carries the fused output projection, the
        // MLP alone is not the comparison: keep it
        if (!mlp_fits(nc) || proj_fuses(def_tuning_)) continue;
        Tuning t = best;
        t.nc = nc;
        const float ms = time_launches([&] { launch_mlp(d, w, 0, t, m_ln, p, s); }, kTuneReps, s);
        log += (log.empty() ? "" : ", ") + std::string("\"mlp_nc") + std::to_string(nc) + "_ms\": " + std::to_string(ms);
        if (nc == def_tuning_.nc) {
            def_ms = best_ms = ms;
        } else if (ms < kTuneMargin * def_ms && ms < best_ms) {
            best_ms = ms;
            best.nc = nc;
        }
    }
    const int def_attn = def_tuning_.attn_threads;
    std::vector<int> forms = {def_attn};
    for (int threads : {0, 64, 128, 256})
        if (threads != def_attn && (threads != 0 || attn_tile_ok(d))) forms.push_back(threads);
    for (int threads : forms) {
        const float ms = time_launches([&] { launch_attention(d, qkv, p.inst, p.n_inst, R, attn, threads, s, &p); },
                                       kTuneReps, s);
        log += (log.empty() ? "\"attn_" : ", \"attn_") + std::to_string(threads) + "_ms\": " + std::to_string(ms);
        if (threads == def_attn) {
            def_ms = best_ms = ms;
        } else if (ms < kTuneMargin * def_ms && ms < best_ms) {
            best_ms = ms;
            best.attn_threads = threads;
        }
    }
    cuda_check(cudaGetLastError(), "autotune");
    {
        std::lock_guard<std::mutex> lk(tune_mu_);
        tuned_[bucket] = best;
    }
    save_cache(bucket, best, log);
}

// Tuned schedules persist in the JSON-lines file named by JC_AUTOTUNE_CACHE,
// one object per tuned row bucket:
//   {"model": "d128_l4_f512_r1_k1_g1", "rows": 65536, "nc": 64, "attn_threads": 0}
// keyed by the model shape (dim, layers, MLP width, mask radius, kind and
// dilation), followed by the candidates' measured times. Lines that do not
// parse or name another shape are skipped; later lines override earlier ones.
void BF16Path::load_cache() {
    const char* path = std::getenv("JC_AUTOTUNE_CACHE");
    if (!path) return;
    FILE* f = std::fopen(path, "r");
    if (!f) return;
    char line[512], key[128];
    while (std::fgets(line, sizeof line, f)) {
        int bucket, nc, th;
        if (std::sscanf(line, " {\"model\": \"%127[^\"]\", \"rows\": %d, \"nc\": %d, \"attn_threads\": %d", key,
                        &bucket, &nc, &th) != 4)
            continue;
        if (cache_key_ == key && mlp_fits(nc) && (th == 64 || th == 128 || th == 256 || (th == 0 && attn_tile_ok(dims_))))
            tuned_[bucket] = Tuning{nc, th};
    }
    std::fclose(f);
}

void BF16Path::save_cache(int bucket, const Tuning& t, const std::string& timings) const {
    const char* path = std::getenv("JC_AUTOTUNE_CACHE");
    if (!path) return;
    std::lock_guard<std::mutex> lk(tune_mu_);
    FILE* f = std::fopen(path, "a");
    if (!f) return;
    std::fprintf(f, "{\"model\": \"%s\", \"rows\": %d, \"nc\": %d, \"attn_threads\": %d%s%s}\n", cache_key_.c_str(),
                 bucket, t.nc, t.attn_threads, timings.empty() ? "" : ", ", timings.c_str());
    std::fclose(f);
}

void BF16Path::alloc_workspace(DeviceArena& a, const Dims& d, Pack& p, int rows, long long cells, int max_inst) const {
    const size_t R = (size_t)rows, NC = (size_t)cells;
    const int strides[4] = {d.D * 2, 3 * d.D * 2, d.D * 2, d.D * 2};  // ln, qkv, attn, t1
    for (int i = 0; i < 4; i++) {
        p.bt[i] = static_cast<char*>(a.alloc(R * strides[i] + 256));
        p.bt_stride[i] = strides[i];
    }
    // zc and c1, f16, plane-major: [channels / 8][cells][8]
    const int planes[2] = {kZcCh / 8, d.HD / 8};
    for (int i = 0; i < 2; i++) {
        p.bc[i] = static_cast<char*>(a.alloc(NC * planes[i] * 16 + 256));
        p.bc_stride[i] = 16;
        p.bc_plane[i] = (long long)NC * 16;
    }
    p.tmaps = a.alloc((size_t)max_inst * kMapsPerInst * sizeof(CUtensorMap));
}

void BF16Path::prepare(const Dims& d, const Pack& p, const InstDev* hinst, cudaStream_t s, CUtensorMap* hstage) const {
    std::vector<CUtensorMap> tmp(hstage ? 0 : (size_t)p.n_inst * kMapsPerInst);
    CUtensorMap* maps = hstage ? hstage : tmp.data();
    for (int i = 0; i < p.n_inst; i++) {
        const InstDev& I = hinst[i];
        CUtensorMap* m = &maps[(size_t)kMapsPerInst * i];
        m[0] = halo_map(p.bt[0] + (size_t)I.row0 * p.bt_stride[0], d.D, I.tx, I.ty);
        m[1] = cell_plane_map(p.bc[0] + (size_t)I.cell0 * 16, kZcCh / 8, p.bc_plane[0], I.nx, I.ny);
        m[2] = tile_store_map(p.bt[3] + (size_t)I.row0 * p.bt_stride[3], d.D, I.tx, I.ty, false);
        m[3] = cell_plane_map(p.bc[1] + (size_t)I.cell0 * 16, d.HD / 8, p.bc_plane[1], I.nx, I.ny);
        if (attn_tile_ok(d)) {
            m[4] = att_map(p.bt[1] + (size_t)I.row0 * p.bt_stride[1], d.D, I.tx, I.ty, kAttHalo);
            m[5] = att_map(p.bt[1] + (size_t)I.row0 * p.bt_stride[1], d.D, I.tx, I.ty, kAttTile);
        }
    }
    cuda_check(cudaMemcpyAsync(p.tmaps, maps, (size_t)p.n_inst * kMapsPerInst * sizeof(CUtensorMap),
                               cudaMemcpyHostToDevice, s),
               "tensor maps", JC_MAP);
    // a temporary host array is released on return: wait for the copy
    if (!hstage) cuda_check(cudaStreamSynchronize(s), "tensor maps", JC_POLL);
}

void BF16Path::forward(const Dims& d, const WeightsF32& w, const Pack& p, int mode, cudaStream_t s) const {
    const int R = p.R, D = d.D, n = p.n_inst;
    if (R == 0) return;
    check_head_width(d);
    bf16* ln = reinterpret_cast<bf16*>(p.bt[0]);
    bf16* qkv = reinterpret_cast<bf16*>(p.bt[1]);
    bf16* attn = reinterpret_cast<bf16*>(p.bt[2]);
    bf16* t1 = reinterpret_cast<bf16*>(p.bt[3]);
    const CUtensorMap m_ln = rows_map(ln, D, R), m_attn = rows_map(attn, D, R), m_t1_box = store_map(t1, D, R, D, false);
    const CUtensorMap m_qkv_out = store_map(qkv, 3 * D, R, 3 * D, false), m_z0_out = store_map(p.z0, d.HD, R, d.HD, true);
    const CUtensorMap m_x = store_map(p.x, D, R, D, true);
    // 64-column swizzled boxes (loads and stores of the fused projection + MLP)
    const CUtensorMap m_attn_box = store_map(attn, D, R, D, false), m_ln_box = store_map(ln, D, R, D, false);
    const CUtensorMap m_x_box = resid_map(p.x, D, R);
    const unsigned gm = (unsigned)((R + 127) / 128);
    const Tuning tu = tuning_for(R);
    {
        KScope k("bf_embed", s);
        // persistent: as many CTAs as fit on the SMs at once. While tiles of 16 rows
        // (two a warp) all run at once they are the shorter chain: 375 rows of 128 took
        // 11 us with eight rows a warp and take 7, 4096 rows 11 and 9. With more rows
        // than that eight a warp read the weights less often (four: 48 us for 64 K, 43).
        static int occupancy[2][9] = {};  // CTAs per SM, per rows a warp and D / 32
        auto launch = [&](auto kernel, int rw) {
            const int rows = 8 * rw;
            int& per_sm = occupancy[rw == 8][D / 32];
            if (per_sm == 0)
                cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, embed_smem(D, rows)), "occupancy");
            const int slots = std::max(1, per_sm) * n_sms_;
            if (rw == 2 && (R + rows - 1) / rows > slots) return false;
            cuda_check(launch_pdl(kernel, (unsigned)std::min((R + rows - 1) / rows, slots), 256, embed_smem(D, rows), s, 1u, d,
                                  w.embed_w, w.embed_b, w.meta_w, w.meta_b, w.blk[0].n1g, w.blk[0].n1b, p.inst, n, R, p.x, ln),
                       "launch");
            return true;
        };
#define JC_EMBED(CPL)                                                              \
    case CPL:                                                                      \
        if (!launch(bf_embed_kernel<CPL, 2>, 2)) launch(bf_embed_kernel<CPL, 8>, 8); \
        break;
        switch (D / 32) {
            JC_EMBED(1) JC_EMBED(2) JC_EMBED(3) JC_EMBED(4) JC_EMBED(5) JC_EMBED(6) JC_EMBED(7) JC_EMBED(8)
            default: throw Error(JC_LIMIT, "the BF16 embed supports dim 32..256 in steps of 32");
        }
#undef JC_EMBED
        check_launch("bf_embed");
    }
    for (int l = 0; l < d.L; l++) {
        const auto& B = w.blk[l];
        {
            KScope k("tc_qkv", s);
            const int BN = bn_qkv;
            if (D <= 128) {
                const int NB = 3 * D / BN;
                const unsigned grid = (unsigned)(NB * std::min((int)gm, std::max(1, 2 * n_sms_ / NB)));
                const size_t smem = QKVPSmem(D, BN).total;
                if (D % 64 == 0)
                    cuda_check(launch_pdl(tc_qkv_kernel<true>, grid, kQKVPThreads, smem, s, 1u, m_ln_box, m_qkv_out, wqkv[l],
                                          B.bqkv, D, BN, R, p.err), "launch");
                else
                    cuda_check(launch_pdl(tc_qkv_kernel<false>, grid, kQKVPThreads, smem, s, 1u, m_ln, m_qkv_out, wqkv[l],
                                          B.bqkv, D, BN, R, p.err), "launch");
            } else {
                GemmEpi ep{B.bqkv, qkv, nullptr, nullptr, nullptr, nullptr, 3 * D};
                const size_t smem = std::max((size_t)D * 256 + (size_t)D * BN * 2, (size_t)((BN + 63) / 64) * 16384);
                cuda_check(launch_pdl(tc_gemm_kernel<EPI_BF16>, dim3(gm, 3 * D / BN), gemm_threads(EPI_BF16), smem, s, 1u, m_ln_box, m_qkv_out, wqkv[l], D, BN, R, ep,
                                                                             p.err), "launch");
            }
            check_launch("tc_qkv");
        }
        {
            KScope k("bf_attention", s);
            launch_attention(d, qkv, p.inst, n, R, attn, tu.attn_threads, s, &p);
            check_launch("bf_attention");
        }
        if (proj_fuses(tu)) {
            // output projection + LayerNorm2 inside the MLP kernel
            KScope k("tc_proj_mlp", s);
            launch_mlp(d, w, l, tu, m_ln_box, p, s, &m_attn_box, &m_x_box);
            check_launch("tc_proj_mlp");
            continue;
        }
        {
            KScope k("tc_proj_ln", s);
            if (D <= kLnMaxD) {
                const unsigned grid = (unsigned)std::min((int)gm, n_sms_);
                cuda_check(launch_pdl(tc_projln_persistent_kernel, grid, kPLThreads, PLSmem(D).total, s, 1u, m_attn, m_x, wp[l], B.bp, B.n2g,
                                                                                    B.n2b, ln, D, R, p.err), "launch");
            } else {
                GemmEpi ep{B.bp, ln, nullptr, p.x, B.n2g, B.n2b, D};
                const size_t smem = std::max((size_t)D * 256 + (size_t)D * D * 2, (size_t)128 * D * 4);
                cuda_check(launch_pdl(tc_gemm_kernel<EPI_RESID_LN>, dim3(gm, 1), gemm_threads(EPI_RESID_LN), smem, s, 1u, m_attn_box, m_attn_box, wp[l], D, D, R, ep,
                                                                            p.err), "launch");
            }
            check_launch("tc_proj_ln");
        }
        {
            KScope k("tc_mlp", s);
            launch_mlp(d, w, l, tu, m_ln, p, s);
            check_launch("tc_mlp");
        }
    }
    if (D <= 128) {
        KScope k("tc_mix_cells", s);
        cuda_check(launch_pdl(tc_mix_cells_kernel, (unsigned)std::min(p.n_ttiles, n_sms_), kMixThreads, MixSmem(D).total, s, 1u,
                              ln, wtm, w.tm_b, wtc, w.tc_b, D, p.n_ttiles, p.inst, n, p.z0, p.err), "launch");
        check_launch("tc_mix_cells");
    } else {
        {
            KScope k("tc_token_mix", s);
            const int BN = bn_tm;
            cuda_check(launch_pdl(tc_conv3_kernel, dim3(p.n_ttiles, D / BN), 128, conv3_launch_smem(D, BN), s, 1u,
                reinterpret_cast<const CUtensorMap*>(p.tmaps), 0, 2, wtm, w.tm_b, D, BN, p.inst, n, p.err), "launch");
            check_launch("tc_token_mix");
        }
        {
            KScope k("tc_to_cells", s);
            GemmEpi ep{w.tc_b, nullptr, p.z0, nullptr, nullptr, nullptr, d.HD};
            const size_t smem = std::max((size_t)D * 256 + (size_t)D * d.HD * 2, (size_t)((d.HD + 31) / 32) * 16384);
            cuda_check(launch_pdl(tc_gemm_kernel<EPI_F32>, dim3(gm, 1), gemm_threads(EPI_F32), smem, s, 1u, m_t1_box, m_z0_out, wtc, D, d.HD, R, ep, p.err), "launch");
            check_launch("tc_to_cells");
        }
    }
    {
        KScope k("bf_upsample", s);
        cuda_check(launch_pdl(bf_upsample_kernel<32, 3>, (unsigned)p.n_ctiles, 128, 0, s, 1u, d, p.z0, p.inst, n,
                                                                       reinterpret_cast<__half*>(p.bc[0]), p.bc_plane[0] / 2), "launch");
        check_launch("bf_upsample");
    }
    {
        KScope k("tc_conv1", s);
        const unsigned grid = (unsigned)std::min(p.n_ctiles, 3 * n_sms_);
        cuda_check(launch_pdl(tc_cellconv_kernel<kCellConv1>, grid, kC1PThreads,
                              C1PSmem(kCellConv1, kZcCh).total, s, 1u,
                              reinterpret_cast<const CUtensorMap*>(p.tmaps), wc1, w.c1_b, kZcCh, p.n_ctiles, p.inst, n,
                              mode, reinterpret_cast<__half*>(p.bc[1]), p.bc_plane[1] / 2, p.err),
                   "launch");
        check_launch("tc_conv1");
    }
    {
        KScope k("tc_conv2", s);
        const unsigned grid = (unsigned)std::min(p.n_ctiles, 4 * n_sms_);
        cuda_check(launch_pdl(tc_cellconv_kernel<kCellConv2>, grid, kC1PThreads, C1PSmem(kCellConv2, d.HD).total, s, 1u,
                              reinterpret_cast<const CUtensorMap*>(p.tmaps), wc2, w.c2_b, d.HD, p.n_ctiles, p.inst, n,
                              mode, nullptr, 0, p.err),
                   "launch");
        check_launch("tc_conv2");
    }
}

}  // namespace jc
