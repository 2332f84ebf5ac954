// cl_mlp.cu — the light-response surrogate: a 3 -> 256 -> 256 -> 256 -> 192 SiLU
// MLP trained and evaluated on sm_100a by hand-written kernels.
//
// Everything GEMM-shaped runs on the 5th-generation tensor cores: BF16 operands
// in 128-byte swizzled shared-memory tiles, one thread issuing tcgen05.mma into
// FP32 accumulators in tensor memory, sixteen warps draining them.
//
//   net_forward   all four layers of 128 rows at a time; inference keeps nothing
//                 but the outputs, training also stores the hidden layers, the
//                 pre-activations and the gradient of the loss
//   net_backward  the gradients of the three hidden layers' pre-activations and
//                 those of layer 1's parameters
//   weight_grads  the three 256-wide weight gradients and their biases
//   adam_all      the parameters and their BF16 copies
//
// A training step is these four launches, each starting while the one before
// drains.  The activations stay in shared and tensor memory from layer to layer;
// what a later kernel reads is written out beside that by TMA (H, dZ) or in
// blocks that the same warps read back (Z).  One kernel per layer and direction
// (twelve launches a step) took 113 us a step at a batch of 4,096 rows and
// 244 us at 65,536; these take 64 us and 232 us.  A batch of 65,536 rows is 512
// units of 128 rows over 148 SMs: 4 rounds where 3.46 would do.  A unit that an SM
// has left over takes 17 us forward and 20 us backward by itself, so a batch just
// above 2 or 4 whole rounds gains nothing: 297 units 182.8 us against 181.4, 593
// units 283 against 272 (296: 144 and 168; 592: 246 and 263).
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <new>
#include <vector>

#include <atomic>
#include <mutex>

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/crysplight_cuda.h"
#include "cl_umma.cuh"

namespace cl {
namespace mlp {

using bf16 = __nv_bfloat16;

// Programmatic dependent launch: the kernels of a training step are launched
// so that the next one may be scheduled while the previous one drains; each
// kernel allows that at its start (pdl_trigger) and waits for the previous
// kernel's completion and memory (pdl_wait) before its first global access.
// Without the launch attribute both are no-ops.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launches kernel k with the programmatic-serialization attribute on stream st.
template <typename... P, typename... A>
cudaError_t launch_pdl(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

constexpr int TILE_M = 128;     // rows per CTA tile (TMEM lanes)
constexpr int TILE_K = 64;      // K elements per pipeline stage (one 128-byte swizzle row)
constexpr int EPI_WARPS = 16;                 // epilogue warps: warp w drains TMEM lane quadrant w % 4,
                                             // 32-column chunks c with c % (EPI_WARPS/4) == w / 4
constexpr int PRODUCER_WARP = EPI_WARPS;        // TMA producer
constexpr int MMA_WARP = EPI_WARPS + 1;         // MMA issuer / TMEM owner
constexpr int GEMM_THREADS = 32 * (EPI_WARPS + 2);
constexpr uint32_t TMEM_COLS = 512; // two 256-column FP32 accumulators
constexpr uint32_t WAIT_BUDGET = 1u << 22;   // polls before a wait gives up

enum Epi : int {
    EPI_F32 = 0,         // out_f[m][n] = acc
    EPI_PARTIAL = 1,     // out_f[split][m][n] = acc (split-K partial)
};
constexpr int GEMM_STAGES = 4;
constexpr uint32_t STAGE_TILE_BYTES = 32 * 64;   // 32 rows x 32 BF16

__host__ __device__ constexpr size_t gemm_smem_bytes(int N)
{
    return 1024 + (size_t)GEMM_STAGES * ((size_t)TILE_M * 128 + (size_t)N * 128);
}

struct GemmArgs {
    int M, N, K;                    // M % 128 == 0, N % 32 == 0 && 32 <= N <= 256, K % 64 == 0
    int k_split;                    // K elements per split (gridDim.y splits)
    float* out_f; int64_t ldf;
    unsigned int* err;
};

// SiLU and its derivative with the approximate exponential and reciprocal, results
// below the normal range flushed to zero (they are rounded to BF16 afterwards; for
// a large negative z the exponential is infinite and its reciprocal 0)
__device__ __forceinline__ float silu(float z)
{
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(z * -1.4426950216293335f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return z * r;
}
__device__ __forceinline__ float dsilu(float z)
{
    float e, s;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(z * -1.4426950216293335f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(1.0f + e));
    return s * (1.0f + z * (1.0f - s));
}

// Byte offset of 16-byte piece j (0..3) of row r in a 32-row x 64-byte tile
// with the 64-byte swizzle of the TMA stores (piece index XOR bits 7-8 of the
// offset; the tile is 2 KB aligned).  Sixteen-byte stores of 32 rows by 32
// lanes then touch every bank group equally often (no conflicts).
__device__ __forceinline__ uint32_t sw64(uint32_t r, uint32_t j)
{
    return r * 64u + ((j ^ ((r >> 1) & 3u)) << 4);
}

// This lane's row of 32 BF16 as column `lane` of a transposed staging tile
// (tile row c = column c of the chunk); each store writes one tile row of 64
// bytes across the warp.
__device__ __forceinline__ void stage_col(uint8_t* tile, int lane, const bf16* h)
{
    const uint32_t j = (uint32_t)lane >> 3, e = 2u * ((uint32_t)lane & 7u);
#pragma unroll
    for (int c = 0; c < 32; ++c) *reinterpret_cast<bf16*>(tile + sw64((uint32_t)c, j) + e) = h[c];
}

// Makes this lane's staging writes visible to the TMA unit and joins the warp;
// then lane 0 may issue the stores.
__device__ __forceinline__ void stage_done()
{
    umma::fence_async_smem();
    __syncwarp();
}

// Eight consecutive per-column constants (or row inputs) from shared memory
// (all lanes read the same address: a broadcast).
__device__ __forceinline__ void cst8(const float* c, float* o)
{
    const float4 p = reinterpret_cast<const float4*>(c)[0], q = reinterpret_cast<const float4*>(c)[1];
    o[0] = p.x; o[1] = p.y; o[2] = p.z; o[3] = p.w; o[4] = q.x; o[5] = q.y; o[6] = q.z; o[7] = q.w;
}

// Column sums over the warp's 32 rows, read from the transposed staging tile
// (lane c sums tile row c, rows in order 0..31), added to dst[0..31]; with xs
// (the rows' inputs by component, xs[32 k + r]), also sum g x_k added to
// gw[256 k + c].  dst and gw are the CTA's shared-memory accumulators.
__device__ __forceinline__ void warp_col_sums(const uint8_t* tt, int lane, float* dst, const float* xs, float* gw)
{
    float s = 0.0f, s0 = 0.0f, s1 = 0.0f, s2 = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint4 q = *reinterpret_cast<const uint4*>(tt + sw64((uint32_t)lane, (uint32_t)j));
        const bf16* g8 = reinterpret_cast<const bf16*>(&q);
        float xa[8], xb[8], xc[8];
        if (xs) { cst8(xs + 8 * j, xa); cst8(xs + 32 + 8 * j, xb); cst8(xs + 64 + 8 * j, xc); }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float v = __bfloat162float(g8[e]);
            s += v;
            if (xs) { s0 += v * xa[e]; s1 += v * xb[e]; s2 += v * xc[e]; }
        }
    }
    atomicAdd(dst + lane, s);
    if (xs) {
        atomicAdd(gw + lane, s0);
        atomicAdd(gw + 256 + lane, s1);
        atomicAdd(gw + 512 + lane, s2);
    }
}

// Epilogue of one 128 x N tile of the diagnostic GEMM: the warp owns rows row0 +
// lane (row0 = tile row + 32 (w % 4)) and the 32-column chunks c0 = 32 (half + 4 k).
template <int EPI>
__device__ __forceinline__ void epilogue(const GemmArgs& G, uint32_t tbase, int row0, int lane, int half)
{
    const int row = row0 + lane;
    for (int c0 = 32 * half; c0 < G.N; c0 += 32 * (EPI_WARPS / 4)) {
        float v[32];
        umma::tmem_ld32(tbase + (uint32_t)c0, v);
        float* o = G.out_f + (EPI == EPI_PARTIAL ? (int64_t)blockIdx.y * G.M * G.ldf : 0) + (int64_t)row * G.ldf + c0;
#pragma unroll
        for (int g = 0; g < 8; ++g)
            *reinterpret_cast<float4*>(o + 4 * g) = make_float4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
    }
}

// C = A B^T on the tensor cores.  A [M][K] and B [N][K] BF16, K-major, read
// through TMA tensor maps (128-byte swizzle, boxes of 64 x 128 rows and 64 x N
// rows).  A diagnostic (cl_umma_gemm_bf16) for the descriptors, barriers and
// accumulators that the network kernels below use in the same way.  Persistent
// over 128-row tiles (blockIdx.x, stride gridDim.x), K split over blockIdx.y.
// Roles: lane 0 of warp 16 streams A/B stages (full/empty mbarriers), lane 0 of
// warp 17 issues tcgen05.mma into one of two TMEM accumulators and commits, warps
// 0-15 drain the other accumulator through the epilogue.  Every wait is bounded; a wait that runs out sets bit 0 of *err,
// tells the other roles to stop, and the CTA still waits (bounded) for its
// copies and MMAs in flight before freeing TMEM.
template <int EPI>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ GemmArgs G)
{
    constexpr int STAGES = GEMM_STAGES;
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte aligned in the shared window (the swizzle atom); offset from
    // smem_raw so that the compiler still sees shared-memory accesses
    uint8_t* smem = smem_raw + ((1024u - (umma::smem_u32(smem_raw) & 1023u)) & 1023u);
    const int N = G.N;
    const uint32_t a_bytes = TILE_M * 128, stage_bytes = a_bytes + (uint32_t)N * 128;
    __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;

    const int split = blockIdx.y;
    const int k_begin = split * G.k_split;
    const int k_end = min(G.K, k_begin + G.k_split);
    const int n_chunks = (k_end - k_begin) / TILE_K;
    const int n_tiles = G.M / TILE_M;
    if (n_chunks <= 0 || (int)blockIdx.x >= n_tiles) return;   // uniform over the CTA

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int* abort_v = &abort_flag;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { umma::mbar_init(&full[s], 1); umma::mbar_init(&empty[s], 1); }
        for (int a = 0; a < 2; ++a) { umma::mbar_init(&acc_full[a], 1); umma::mbar_init(&acc_empty[a], EPI_WARPS); }
        abort_flag = 0;
    }
    if (warp == MMA_WARP) umma::tmem_alloc(&tmem_slot, TMEM_COLS);
    if (warp == PRODUCER_WARP && lane == 0) {
        umma::prefetch_tmap(&tmA);
        umma::prefetch_tmap(&tmB);
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = tmem_slot;

    if (warp == PRODUCER_WARP) {
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
                for (int c = 0; c < n_chunks; ++c, ++it) {
                    const uint32_t s = it % STAGES, r = it / STAGES;
                    if (r > 0 && !umma::mbar_wait_or_abort(&empty[s], (r - 1) & 1u, WAIT_BUDGET, abort_v)) {
                        ok = false;
                        break;
                    }
                    uint8_t* st = smem + s * stage_bytes;
                    umma::mbar_arrive_expect_tx(&full[s], stage_bytes);
                    const int k0 = k_begin + c * TILE_K;
                    umma::tma_load_2d(st, &tmA, k0, tile * TILE_M, &full[s]);
                    umma::tma_load_2d(st + a_bytes, &tmB, k0, 0, &full[s]);
                }
            }
            if (!ok) { atomicOr(G.err, 1u); *abort_v = 1; }
            // copies still in flight land before the CTA can exit
            for (uint32_t j = it > (uint32_t)STAGES ? it - STAGES : 0u; j < it; ++j)
                umma::mbar_wait(&full[j % STAGES], (j / STAGES) & 1u, WAIT_BUDGET);
        }
    } else if (warp == MMA_WARP) {
        if (lane == 0) {
            const uint32_t idesc = umma::make_idesc_bf16(TILE_M, N);
            uint32_t it = 0, j = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++j) {
                const uint32_t a = j & 1u, u = j >> 1;
                if (u > 0 && !umma::mbar_wait_or_abort(&acc_empty[a], (u - 1) & 1u, WAIT_BUDGET, abort_v)) {
                    ok = false;
                    break;
                }
                umma::fence_after_sync();
                const uint32_t d = tmem + a * 256u;
                for (int c = 0; c < n_chunks; ++c, ++it) {
                    const uint32_t s = it % STAGES, r = it / STAGES;
                    if (!umma::mbar_wait_or_abort(&full[s], r & 1u, WAIT_BUDGET, abort_v)) { ok = false; break; }
                    umma::fence_after_sync();
                    const uint32_t sa = umma::smem_u32(smem + s * stage_bytes), sb = sa + a_bytes;
#pragma unroll
                    for (int k = 0; k < TILE_K / 16; ++k) {
                        const uint64_t ad = umma::make_desc_sw128(sa + 32u * k);
                        const uint64_t bd = umma::make_desc_sw128(sb + 32u * k);
                        umma::mma_bf16(d, ad, bd, idesc, (c > 0 || k > 0) ? 1u : 0u);
                    }
                    umma::commit(&empty[s]);
                }
                if (!ok) break;
                umma::commit(&acc_full[a]);
            }
            if (!ok) { atomicOr(G.err, 1u); *abort_v = 1; }
            // the last MMAs complete before TMEM is freed
            if (it > 0) umma::mbar_wait(&empty[(it - 1) % STAGES], ((it - 1) / STAGES) & 1u, WAIT_BUDGET);
        }
    } else {
        uint32_t j = 0;
        for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++j) {
            const uint32_t a = j & 1u, u = j >> 1;
            if (!umma::mbar_wait_or_abort(&acc_full[a], u & 1u, WAIT_BUDGET, abort_v)) {
                if (lane == 0) atomicOr(G.err, 1u);
                *abort_v = 1;
                break;
            }
            umma::fence_after_sync();
            const int quad = warp & 3;
            epilogue<EPI>(G, tmem + a * 256u + ((uint32_t)(32 * quad) << 16), tile * TILE_M + 32 * quad, lane, warp >> 2);
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&acc_empty[a]);
        }
    }
    __syncthreads();
    if (warp == MMA_WARP) {
        umma::fence_after_sync();
        umma::tmem_dealloc(tmem, TMEM_COLS);
    }
}

// ---- host side: tensor maps and launches ----
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::once_flag g_encode_once;

bool encoder()
{
    std::call_once(g_encode_once, [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
        cudaGetLastError();
    });
    return g_encode != nullptr;
}

// rows x K BF16 matrix with row stride ld (elements), boxes of 64 x box_rows,
// 128-byte swizzle.
bool make_map(CUtensorMap* m, const bf16* base, int64_t rows, int64_t K, int64_t ld, int box_rows)
{
    if (!encoder() || ((uintptr_t)base & 15) || (ld * 2) % 16 || K % TILE_K) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)(ld * 2)};
    const cuuint32_t box[2] = {(cuuint32_t)TILE_K, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return g_encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// MN-major operand map: a K x MN BF16 matrix stored row by row (row stride ld
// elements), boxes of 64 MN-elements x 64 K-rows with the 128-byte swizzle.
bool make_map_mn(CUtensorMap* m, const bf16* base, int64_t k_rows, int64_t mn, int64_t ld)
{
    if (!encoder() || ((uintptr_t)base & 15) || (ld * 2) % 16 || mn % 64 || k_rows % TILE_K || ld < mn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)mn, (cuuint64_t)k_rows};
    const cuuint64_t strides[1] = {(cuuint64_t)(ld * 2)};
    const cuuint32_t box[2] = {64, 64};
    const cuuint32_t estr[2] = {1, 1};
    return g_encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A [M][K] (row stride lda), B [N][K] (row stride ldb).
template <int EPI>
int launch_gemm(const GemmArgs& g, const bf16* A, int64_t lda, const bf16* B, int64_t ldb, int grid_x,
                int splits, cudaStream_t st)
{
    if (g.M % TILE_M || g.M <= 0 || g.N % 32 || g.N > 256 || g.N < 32 || g.K % TILE_K || g.K <= 0 ||
        splits < 1 || g.k_split % TILE_K || g.k_split <= 0 || (int64_t)(splits - 1) * g.k_split >= g.K ||
        (int64_t)splits * g.k_split < g.K || grid_x < 1)
        return CL_ERR_ARG;
    CUtensorMap ta, tb;
    if (!make_map(&ta, A, g.M, g.K, lda, TILE_M) || !make_map(&tb, B, g.N, g.K, ldb, g.N)) return CL_ERR_ARG;
    // the shared-memory opt-in is a per-device attribute of the kernel: set it
    // once for every device this process launches on
    static std::atomic<uint64_t> attr_devices{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(attr_devices.load() & bit)) {
        if (cudaFuncSetAttribute(gemm_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)gemm_smem_bytes(256)) != cudaSuccess)
            return CL_ERR_CUDA;
        attr_devices.fetch_or(bit);
    }
    const int tiles = g.M / TILE_M;
    dim3 grid((unsigned)(grid_x < tiles ? grid_x : tiles), (unsigned)splits);
    // at least 116 KB so that one CTA holds an SM: each allocates all 512 TMEM columns
    const size_t smem = gemm_smem_bytes(g.N) > 116 * 1024 ? gemm_smem_bytes(g.N) : 116 * 1024;
    gemm_kernel<EPI><<<grid, GEMM_THREADS, smem, st>>>(ta, tb, g);
    return cudaGetLastError() == cudaSuccess ? CL_OK : CL_ERR_CUDA;
}


// ===========================================================================
// The MLP: 3 -> 256 -> 256 -> 256 -> 192, SiLU, BF16 weights/activations,
// FP32 accumulation and FP32 master weights with Adam.
// ===========================================================================
constexpr int D_IN = 3, D_H = 256, D_OUT = 192;
constexpr int WGRAD_MIN_CHUNKS = 4;      // fewest 64-row chunks per CTA of the weight gradients (2, 4 and 8 are
                                         // equally fast at 512 to 4,096 rows)
constexpr int WGRAD_MIN_RUN = 8;         // chunks that any run may have
// Parameter block layout (FP32, contiguous): W1[256][3] b1[256] W2t[256][256]
// b2[256] W3t[256][256] b3[256] W4t[192][256] b4[192].
constexpr int64_t OFF_W1 = 0, OFF_B1 = OFF_W1 + D_H * D_IN, OFF_W2 = OFF_B1 + D_H,
                  OFF_B2 = OFF_W2 + D_H * D_H, OFF_W3 = OFF_B2 + D_H, OFF_B3 = OFF_W3 + D_H * D_H,
                  OFF_W4 = OFF_B3 + D_H, OFF_B4 = OFF_W4 + D_OUT * D_H, N_PARAMS = OFF_B4 + D_OUT;

__device__ __forceinline__ uint32_t hash32(uint32_t a, uint32_t b, uint32_t c)
{
    // Philox4x32-10 with key (c, 0x5eed) on counter (a, b, 0, 0): first word
    uint32_t c0 = a, c1 = b, c2 = 0, c3 = 0, k0 = c, k1 = 0x5eedu;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint64_t p0 = (uint64_t)0xD2511F53u * c0, p1 = (uint64_t)0xCD9E8D57u * c2;
        const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c1 ^ k0, n2 = (uint32_t)(p0 >> 32) ^ c3 ^ k1;
        c1 = (uint32_t)p1; c3 = (uint32_t)p0; c0 = n0; c2 = n2;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
    return c0;
}

// Adam over the whole parameter block in one launch, four parameters per
// thread (FP32 master weights; the gradient is zeroed as it is read); the three
// weight matrices of the tensor-core layers also get their BF16 copies.  All
// offsets in the block are multiples of 4.  One parameter per thread, with a
// 64-bit division per matrix and a second, transposed copy, took 16.5 us, this
// 6.0 (181,000 parameters).
struct AdamCopies {
    bf16 *w2t, *w3t, *w4t;
};
__global__ void __launch_bounds__(128) adam_all(float* __restrict__ w, float* __restrict__ g, float* __restrict__ m,
                                                float* __restrict__ v, float lr, float b1, float b2, float eps,
                                                float bc1, float bc2, const AdamCopies C)
{
    pdl_trigger();
    const int i = 4 * (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= (int)N_PARAMS) return;
    pdl_wait();
    const float4 g4 = *reinterpret_cast<const float4*>(g + i);
    float4 m4 = *reinterpret_cast<const float4*>(m + i), v4 = *reinterpret_cast<const float4*>(v + i),
           w4 = *reinterpret_cast<const float4*>(w + i);
    *reinterpret_cast<float4*>(g + i) = make_float4(0.f, 0.f, 0.f, 0.f);   // for the next step's accumulation
    auto step = [&](float gi, float& mo, float& vo, float& wo) {
        const float mi = b1 * mo + (1.0f - b1) * gi;
        const float vi = b2 * vo + (1.0f - b2) * gi * gi;
        mo = mi; vo = vi;
        wo = wo - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    };
    step(g4.x, m4.x, v4.x, w4.x);
    step(g4.y, m4.y, v4.y, w4.y);
    step(g4.z, m4.z, v4.z, w4.z);
    step(g4.w, m4.w, v4.w, w4.w);
    *reinterpret_cast<float4*>(m + i) = m4;
    *reinterpret_cast<float4*>(v + i) = v4;
    *reinterpret_cast<float4*>(w + i) = w4;
    bf16* copy = nullptr;
    if (i >= OFF_W2 && i < OFF_B2) copy = C.w2t + (i - OFF_W2);
    else if (i >= OFF_W3 && i < OFF_B3) copy = C.w3t + (i - OFF_W3);
    else if (i >= OFF_W4 && i < OFF_B4) copy = C.w4t + (i - OFF_W4);
    if (copy) {
        __nv_bfloat162 q[2] = {__floats2bfloat162_rn(w4.x, w4.y), __floats2bfloat162_rn(w4.z, w4.w)};
        *reinterpret_cast<uint2*>(copy) = *reinterpret_cast<uint2*>(q);
    }
}

__global__ void to_bf16(const float* w, int n, bf16* o)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) o[i] = __float2bfloat16_rn(w[i]);
}

// ===========================================================================
// Inference: the whole network in one kernel
// ===========================================================================
// One CTA per SM walks units of 128 rows (of one member of an ensemble) through
// all four layers.  A unit's activations never leave the SM: layer 1 and each
// epilogue write the next layer's A operand (128 x 256 BF16, 128-byte swizzle)
// into the unit's 64 KB of shared memory, the accumulators stay in tensor
// memory, and only the inputs, the weights (streamed from L2 by TMA in stages
// of 64 K-elements) and the outputs (stored from registers, 64 bytes of a row per
// lane) move.  Layer by layer the same network went through global memory: H written
// and read three times, the outputs copied once more.
//
// Two units are in flight per CTA: while the sixteen epilogue warps work on one
// unit's layer, the tensor cores run the other unit's.  The bound is the
// special-function unit: SiLU takes an exponential and a reciprocal, 2 x 256 x 3
// per row at 16 per clock and SM, 96 cycles per row (the tensor cores need 43).
// 200,001 rows through MLP.forward: 355 -> 154 us.
constexpr int NET_MAX = 8;               // members one launch evaluates
constexpr int NET_STAGES = 2;            // weight stages of 256 x 64 BF16
constexpr uint32_t NET_A_BYTES = TILE_M * 512;           // a unit's A operand: 4 K-blocks of 16 KB
constexpr uint32_t NET_STAGE_BYTES = 256 * 128;
constexpr int NET_CST_W1 = 2 * D_H + D_OUT;              // b2, b3, b4, then (W1 row, b1) per feature
constexpr int NET_CST = NET_CST_W1 + 4 * D_H;
constexpr size_t NET_SMEM = 1024 + 2 * (size_t)NET_A_BYTES + NET_STAGES * (size_t)NET_STAGE_BYTES;

struct NetArgs {
    CUtensorMap w[NET_MAX][3];           // W2^T, W3^T, W4^T: boxes of 64 x 256 (192)
    const float* params[NET_MAX];        // FP32 parameter blocks
    const float* x;                      // [n][3]
    float* out;                          // [members][n][192]
    int64_t n;
    int members, tiles;                  // units: members x tiles
    unsigned int* err;
};

// Byte offset of 16-byte piece j (0..7) of row r in a K-block (128-byte rows, 128-byte swizzle).
__device__ __forceinline__ uint32_t sw128(uint32_t r, uint32_t j) { return r * 128u + ((j ^ (r & 7u)) << 4); }

// 32 BF16 (columns c0 .. c0 + 31 of row r) into an A operand.
__device__ __forceinline__ void store_a(uint8_t* A, int r, int c0, const bf16* h)
{
    uint8_t* blk = A + (c0 >> 6) * (TILE_M * 128);
#pragma unroll
    for (int j = 0; j < 4; ++j)
        *reinterpret_cast<uint4*>(blk + sw128((uint32_t)r, (uint32_t)(((c0 & 63) >> 3) + j))) =
            reinterpret_cast<const uint4*>(h)[j];
}

// 16 consecutive floats of this lane's row: two whole 32-byte sectors.
__device__ __forceinline__ void store_row16(float* o, const float* v, bool wide)
{
    if (wide) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
            asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(o + 8 * i), "f"(v[8 * i]),
                         "f"(v[8 * i + 1]), "f"(v[8 * i + 2]), "f"(v[8 * i + 3]), "f"(v[8 * i + 4]), "f"(v[8 * i + 5]),
                         "f"(v[8 * i + 6]), "f"(v[8 * i + 7]) : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) o[i] = v[i];
    }
}

// The pre-activations only pass between the two training kernels, whose warps
// read back exactly the 32 x 32 blocks that the same warps wrote: a block is
// kept as four 512-byte pieces [j][lane] of 16 bytes, so that an instruction
// touches 4 lines (row by row, 32).
__device__ __forceinline__ int64_t z_block(int tile, int quad, int chunk)
{
    return (((int64_t)tile * (D_H / 32) + chunk) * 4 + quad) * 1024;     // BF16 elements
}
__device__ __forceinline__ void store_block(bf16* o, int lane, const bf16* z)
{
#pragma unroll
    for (int j = 0; j < 4; ++j)
        reinterpret_cast<uint4*>(o)[32 * j + lane] = reinterpret_cast<const uint4*>(z)[j];
}
__device__ __forceinline__ void load_block(const bf16* o, int lane, bf16* z)
{
#pragma unroll
    for (int j = 0; j < 4; ++j)
        reinterpret_cast<uint4*>(z)[j] = __ldg(reinterpret_cast<const uint4*>(o) + 32 * j + lane);
}

// 8 consecutive floats, one whole 32-byte sector per lane (32-byte aligned).
__device__ __forceinline__ void load8(const float* p, float* v)
{
    asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}

// Row of the training set that minibatch row b is (random with replacement), or
// b itself where the batch is given (n_all == 0).
struct BatchRows {
    uint32_t n_all, step, seed;
};
__device__ __forceinline__ int64_t batch_row(const BatchRows& r, int64_t b)
{
    return r.n_all ? (int64_t)(hash32((uint32_t)b, r.step, r.seed) % r.n_all) : b;
}

// Training keeps what the backward pass and the weight gradients read: H of the
// three hidden layers and the loss gradient dO (stored by TMA from the unit's
// operand memory) and Z of layers 2 and 3 (before SiLU, BF16, z_block layout).
// 65,536 rows: 89 us (92 us as four kernels, a gather and layer 1 among them);
// an SM writes 368 KB per unit at about 32 bytes per cycle, 11,500 cycles,
// beside 12,300 of SiLU and the gathered targets (98 KB).
struct NetTrain {
    CUtensorMap h[4];                    // H1, H2, H3, dO: boxes of 64 x 128
    bf16 *z2, *z3;
    const float* target;                 // [training set rows][192]
    BatchRows rows;
    int32_t* brow;                       // training-set row of each batch row (written here)
    bool wide;                           // targets 32-byte aligned
    float scale;
    float* loss;
    int whole;                           // tiles below this add four sums per 32 rows to the loss, the others six
};

constexpr int STORE_WARP = EPI_WARPS + 2;        // training: issues the TMA stores of the operands
constexpr int NET_TRAIN_THREADS = GEMM_THREADS + 32;

template <bool TRAIN>
__global__ void __launch_bounds__(TRAIN ? NET_TRAIN_THREADS : GEMM_THREADS, 1)
    net_forward(const __grid_constant__ NetArgs G, const __grid_constant__ NetTrain T)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (umma::smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* ring = smem + 2 * NET_A_BYTES;
    __shared__ __align__(8) uint64_t full[NET_STAGES], empty[NET_STAGES], a_ready[2], acc_full[2], stored[2], o_ready[2], epi_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    __shared__ __align__(16) float s_cst[2][NET_CST];
    __shared__ float4 s_x[EPI_WARPS][16];
    __shared__ float2 s_sq[2][4][4];         // training: squared errors by slot, 32 rows and column group

    if (TRAIN) pdl_trigger();

    const int n_units = G.members * G.tiles;
    const int my_units = ((int)blockIdx.x < n_units) ? (n_units - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    if (my_units == 0) return;               // uniform over the CTA
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int* abort_v = &abort_flag;
    if (threadIdx.x == 0) {
        for (int s = 0; s < NET_STAGES; ++s) { umma::mbar_init(&full[s], 1); umma::mbar_init(&empty[s], 1); }
        for (int s = 0; s < 2; ++s) {
            umma::mbar_init(&a_ready[s], EPI_WARPS);
            umma::mbar_init(&acc_full[s], 1);
            umma::mbar_init(&stored[s], 1);
            umma::mbar_init(&o_ready[s], EPI_WARPS);
        }
        umma::mbar_init(&epi_bar, EPI_WARPS);
        abort_flag = 0;
    }
    if (warp == MMA_WARP) umma::tmem_alloc(&tmem_slot, TMEM_COLS);
    if (TRAIN) {
        pdl_wait();
        // the rows of this CTA's units
        for (int i = threadIdx.x; i < my_units * TILE_M; i += blockDim.x) {
            const int64_t b = (int64_t)((int)blockIdx.x + (i / TILE_M) * (int)gridDim.x) * TILE_M + i % TILE_M;
            T.brow[b] = (int32_t)batch_row(T.rows, b);
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = tmem_slot;

    if (warp == PRODUCER_WARP) {
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int u0 = 0; u0 < my_units && ok; u0 += 2)
                for (int l = 0; l < 3 && ok; ++l)
                    for (int s = 0; s < 2 && u0 + s < my_units && ok; ++s) {
                        const int member = ((int)blockIdx.x + (u0 + s) * (int)gridDim.x) / G.tiles;
                        const uint32_t bytes = (l == 2 ? D_OUT : D_H) * 128u;
                        for (int c = 0; c < D_H / TILE_K; ++c, ++it) {
                            const uint32_t st = it % NET_STAGES, r = it / NET_STAGES;
                            if (r > 0 && !umma::mbar_wait_or_abort(&empty[st], (r - 1) & 1u, WAIT_BUDGET, abort_v)) {
                                ok = false;
                                break;
                            }
                            umma::mbar_arrive_expect_tx(&full[st], bytes);
                            umma::tma_load_2d(ring + st * NET_STAGE_BYTES, &G.w[member][l], c * TILE_K, 0, &full[st]);
                        }
                    }
            if (!ok) { atomicOr(G.err, 1u); *abort_v = 1; }
            // copies still in flight land before the CTA can exit
            for (uint32_t j = it > (uint32_t)NET_STAGES ? it - NET_STAGES : 0u; j < it; ++j)
                umma::mbar_wait(&full[j % NET_STAGES], (j / NET_STAGES) & 1u, WAIT_BUDGET);
        }
    } else if (warp == MMA_WARP) {
        if (lane == 0) {
            uint32_t it = 0, job[2] = {0, 0};
            bool ok = true;
            for (int u0 = 0; u0 < my_units && ok; u0 += 2)
                for (int l = 0; l < 3 && ok; ++l)
                    for (int s = 0; s < 2 && u0 + s < my_units && ok; ++s) {
                        if (!umma::mbar_wait_or_abort(&a_ready[s], job[s]++ & 1u, WAIT_BUDGET, abort_v)) { ok = false; break; }
                        umma::fence_after_sync();
                        const uint32_t idesc = umma::make_idesc_bf16(TILE_M, l == 2 ? D_OUT : D_H, false, false);
                        const uint32_t a0 = umma::smem_u32(smem + s * NET_A_BYTES), d = tmem + s * 256u;
                        for (int c = 0; c < D_H / TILE_K; ++c, ++it) {
                            const uint32_t st = it % NET_STAGES, r = it / NET_STAGES;
                            if (!umma::mbar_wait_or_abort(&full[st], r & 1u, WAIT_BUDGET, abort_v)) { ok = false; break; }
                            umma::fence_after_sync();
                            const uint32_t sb = umma::smem_u32(ring + st * NET_STAGE_BYTES);
#pragma unroll
                            for (int k = 0; k < TILE_K / 16; ++k)
                                umma::mma_bf16(d, umma::make_desc_sw128(a0 + c * (TILE_M * 128u) + 32u * k),
                                               umma::make_desc_sw128(sb + 32u * k), idesc, (c > 0 || k > 0) ? 1u : 0u);
                            umma::commit(&empty[st]);
                        }
                        if (ok) umma::commit(&acc_full[s]);
                    }
            if (!ok) { atomicOr(G.err, 1u); *abort_v = 1; }
            // the last MMAs complete before TMEM is freed
            if (it > 0) umma::mbar_wait(&empty[(it - 1) % NET_STAGES], ((it - 1) / NET_STAGES) & 1u, WAIT_BUDGET);
        }
    } else if (TRAIN && warp == STORE_WARP) {
        // a unit's operands are H1, H2, H3; dO follows in the same memory.  The
        // target rows, which the loss reads three layers later, are brought into
        // L2 while the first layers run.
        uint32_t job[2] = {0, 0};
        bool ok = true;
        auto fetch_targets = [&](int u) {
            if (u >= my_units) return;
            // plain prefetches of the lines: the copy engine would take the row-sized
            // ones in turn with the operands' stores
            const int64_t b0 = (int64_t)((int)blockIdx.x + u * (int)gridDim.x) * TILE_M;
            int32_t r[TILE_M / 32];
#pragma unroll
            for (int i = 0; i < TILE_M / 32; ++i) r[i] = T.brow[b0 + 32 * i + lane];
#pragma unroll
            for (int i = 0; i < TILE_M / 32; ++i)
#pragma unroll
                for (int j = 0; j < D_OUT / 32; ++j)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(T.target + (int64_t)r[i] * D_OUT + 32 * j));
        };
        // The loss is one FP32 sum over all steps, and the rounding of its additions
        // (about 1e-5 of it) depends on what is added at a time, not on the order.
        // So that losses stay comparable with those of the kernel per layer, its
        // sums are added: per 32 rows the columns 0-31 and 128-159, 32-63 and
        // 160-191, 64-95, 96-127, and in the tiles of a short last round each 32
        // columns by themselves.  The column groups' sums are [.x: 32 columns of
        // one chunk, .y: 16 columns of the chunk shared with the neighbour].
        auto add_loss = [&](int s, int tile) {
            const int j = lane >> 2;
            if (j >= (tile < T.whole ? 4 : 6)) return;
            const float2* q = s_sq[s][lane & 3];
            auto chunk = [&](int c) {
                return c == 1 ? q[0].y + q[1].y : c == 4 ? q[2].y + q[3].y : q[(c + 1) >> 1].x;
            };
            float d = chunk(j);
            if (tile < T.whole && j < 2) d += chunk(j + 4);
            atomicAdd(T.loss, d * T.scale);
        };
        fetch_targets(0);
        fetch_targets(1);
        for (int u0 = 0; u0 < my_units && ok; u0 += 2)
            for (int l = 0; l < 4 && ok; ++l) {
                for (int s = 0; s < 2 && u0 + s < my_units && ok; ++s) {
                    if (lane == 0) {
                        ok = l < 3 ? umma::mbar_wait_or_abort(&a_ready[s], job[s]++ & 1u, WAIT_BUDGET, abort_v)
                                   : umma::mbar_wait_or_abort(&o_ready[s], (uint32_t)(u0 >> 1) & 1u, WAIT_BUDGET, abort_v);
                        if (ok) {
                            const int tile = (int)blockIdx.x + (u0 + s) * (int)gridDim.x;
                            for (int c = 0; c < (l < 3 ? D_H : D_OUT) / TILE_K; ++c)
                                umma::tma_store_2d(&T.h[l], c * TILE_K, tile * TILE_M,
                                                   smem + s * NET_A_BYTES + c * (TILE_M * 128));
                            umma::bulk_commit();
                        } else {
                            atomicOr(G.err, 1u);
                            *abort_v = 1;
                        }
                    }
                    ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
                    if (!ok) break;
                    if (l == 3) {
                        __syncwarp();
                        add_loss(s, (int)blockIdx.x + (u0 + s) * (int)gridDim.x);
                        __syncwarp();
                    }
                    if (lane == 0) {
                        umma::bulk_wait_read0();
                        umma::mbar_arrive(&stored[s]);
                    }
                }
                if (ok && l == 2) {
                    fetch_targets(u0 + 2);
                    fetch_targets(u0 + 3);
                }
            }
        if (lane == 0) umma::bulk_wait0();
    } else {
        const int quad = warp & 3, group = warp >> 2;
        const int row = 32 * quad + lane;                 // of the unit
        const uint32_t tlane = (uint32_t)(32 * quad) << 16;
        const bool wide = ((uintptr_t)G.out & 31) == 0;   // 32-byte stores
        float4* const xs = s_x[warp];
        int loaded[2] = {-1, -1};                         // member whose constants a slot holds
        uint32_t job[2] = {0, 0}, met = 0;
        bool ok = true;
        auto give_up = [&] {
            if (lane == 0) atomicOr(G.err, 1u);
            *abort_v = 1;
            ok = false;
        };
        // the epilogue warps meet, bounded like every wait
        auto meet = [&] {
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&epi_bar);
            if (!umma::mbar_wait_or_abort(&epi_bar, met++ & 1u, WAIT_BUDGET, abort_v)) give_up();
        };
        // training: the last operand has been stored and may be overwritten
        uint32_t n_stored[2] = {0, 0};
        auto wait_stored = [&](int s) {
            if (!umma::mbar_wait_or_abort(&stored[s], n_stored[s]++ & 1u, WAIT_BUDGET, abort_v)) give_up();
        };
        auto wait_acc = [&](int s) {
            if (TRAIN) wait_stored(s);
            if (!umma::mbar_wait_or_abort(&acc_full[s], job[s]++ & 1u, WAIT_BUDGET, abort_v)) give_up();
            umma::fence_after_sync();
        };
        auto operand_ready = [&](int s) {
            umma::fence_before_sync();
            stage_done();
            if (lane == 0) umma::mbar_arrive(&a_ready[s]);
        };
        // inputs of the 16 rows whose layer 1 this warp computes, one per lane,
        // requested a unit ahead
        const int row1 = 16 * (warp >> 1) + (lane & 15), col1 = 128 * (warp & 1) + 4 * lane;
        float xn[2][3];
        auto fetch_x = [&](int s, int u) {
            const int64_t gr = (int64_t)(((int)blockIdx.x + u * (int)gridDim.x) % G.tiles) * TILE_M + row1;
            const bool in = u < my_units && gr < G.n;
            const int64_t xr = TRAIN && in ? (int64_t)T.brow[gr] : gr;
#pragma unroll
            for (int k = 0; k < 3; ++k) xn[s][k] = in ? G.x[xr * 3 + k] : 0.f;
        };
        // layer 1 of unit `u` into slot s's operand: 16 rows x 128 columns, four
        // columns per lane (their weights in registers), the rows' inputs broadcast;
        // between(k), k = 0..3, runs before each four rows
        auto first_layer = [&](int s, int u, auto&& between) {
            const int member = ((int)blockIdx.x + u * (int)gridDim.x) / G.tiles;
            float* cst = s_cst[s];
            if (loaded[s] != member) {
                meet();                      // no warp reads the last member's constants any more
                const float* p = G.params[member];
                // one network: both slots at once
                for (int q = s; q < (G.members == 1 ? 2 : s + 1); ++q) {
                    float* o = s_cst[q];
                    for (int i = threadIdx.x; i < D_H; i += 32 * EPI_WARPS) {
                        o[i] = p[OFF_B2 + i];
                        o[D_H + i] = p[OFF_B3 + i];
                        if (i < D_OUT) o[2 * D_H + i] = p[OFF_B4 + i];
                        reinterpret_cast<float4*>(o + NET_CST_W1)[i] =
                            make_float4(p[OFF_W1 + 3 * i], p[OFF_W1 + 3 * i + 1], p[OFF_W1 + 3 * i + 2], p[OFF_B1 + i]);
                    }
                    loaded[q] = member;
                }
                meet();
                if (!ok) return;
            }
            __syncwarp();
            if (lane < 16) xs[lane] = make_float4(xn[s][0], xn[s][1], xn[s][2], 0.f);
            __syncwarp();
            fetch_x(s, u + 2);
            const float4* w = reinterpret_cast<const float4*>(cst + NET_CST_W1) + col1;
            const float4 w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3];
            uint8_t* blk = smem + s * NET_A_BYTES + (col1 >> 6) * (TILE_M * 128);
            const uint32_t j = (uint32_t)((col1 & 63) >> 3), e = (uint32_t)(col1 & 7) * 2u;
            for (int k = 0; k < 4; ++k) {
                between(k);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int r = 4 * k + i;
                    const float4 x = xs[r];
                    auto z = [&](const float4& v) { return __fmaf_rn(x.z, v.z, __fmaf_rn(x.y, v.y, __fmaf_rn(x.x, v.x, v.w))); };
                    __nv_bfloat162 h[2] = {__floats2bfloat162_rn(silu(z(w0)), silu(z(w1))),
                                           __floats2bfloat162_rn(silu(z(w2)), silu(z(w3)))};
                    *reinterpret_cast<uint2*>(blk + sw128((uint32_t)(16 * (warp >> 1) + r), j) + e) =
                        *reinterpret_cast<uint2*>(h);
                }
            }
            operand_ready(s);
        };

        fetch_x(0, 0);
        fetch_x(1, 1);
        for (int s = 0; s < 2 && s < my_units && ok; ++s) first_layer(s, s, [](int) {});
        for (int u0 = 0; u0 < my_units && ok; u0 += 2) {
            // layers 2 and 3: accumulator -> bias, SiLU -> next operand
            for (int l = 0; l < 2 && ok; ++l)
                for (int s = 0; s < 2 && u0 + s < my_units; ++s) {
                    wait_acc(s);
                    if (!ok) break;
                    for (int c0 = 32 * group; c0 < D_H; c0 += 8 * EPI_WARPS) {
                        float v[32];
                        umma::tmem_ld32(tmem + s * 256u + tlane + (uint32_t)c0, v);
                        __align__(16) bf16 h[32];
                        __align__(16) bf16 zz[32];
                        (void)zz;
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            float b[8];
                            cst8(s_cst[s] + l * D_H + c0 + 8 * g, b);
#pragma unroll
                            for (int q = 0; q < 8; ++q) {
                                const float z = v[8 * g + q] + b[q];
                                if (TRAIN) zz[8 * g + q] = __float2bfloat16_rn(z);
                                h[8 * g + q] = __float2bfloat16_rn(silu(z));
                            }
                        }
                        if (TRAIN) {
                            const int tile = (int)blockIdx.x + (u0 + s) * (int)gridDim.x;
                            store_block((l ? T.z3 : T.z2) + z_block(tile, quad, c0 >> 5), lane, zz);
                        }
                        store_a(smem + s * NET_A_BYTES, row, c0, h);
                    }
                    operand_ready(s);
                }
            // outputs, then layer 1 of the slot's next unit: the stores drain
            // under its special functions
            for (int s = 0; s < 2 && u0 + s < my_units && ok; ++s) {
                // training: the row's targets, two pieces of 16 columns ahead of their use
                float tg[3][TRAIN ? 16 : 1];
                const float* trow = nullptr;
                auto fetch_t = [&](int k) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        if (T.wide) load8(trow + 16 * k + 8 * i, &tg[k][8 * i]);
                        else cst8(trow + 16 * k + 8 * i, &tg[k][8 * i]);
                    }
                };
                if (TRAIN) {
                    const int64_t b = (int64_t)((int)blockIdx.x + (u0 + s) * (int)gridDim.x) * TILE_M + row;
                    trow = T.target + (int64_t)T.brow[b] * D_OUT + 48 * group;
                    fetch_t(0);
                    fetch_t(1);
                }
                wait_acc(s);
                if (!ok) break;
                const int unit = (int)blockIdx.x + (u0 + s) * (int)gridDim.x;
                const int member = unit / G.tiles, tile = unit - member * G.tiles;
                const int64_t gr = (int64_t)tile * TILE_M + row;
                float* o = TRAIN ? nullptr : G.out + ((int64_t)member * G.n + gr) * D_OUT;
                const float* b4 = s_cst[s] + 2 * D_H;
                if (TRAIN) {
                    // loss: dO into the (consumed) operand memory for the store warp
                    float2 sq = make_float2(0.f, 0.f);   // squared errors, see add_loss
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const int c0 = 48 * group + 16 * k;
                        float sk = 0.0f;
                        if (k == 0) fetch_t(2);
                        float v[16];
                        umma::tmem_ld16(tmem + s * 256u + tlane + (uint32_t)c0, v);
                        __align__(16) bf16 g[16];
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            float b[8];
                            cst8(b4 + c0 + 8 * i, b);
#pragma unroll
                            for (int q = 0; q < 8; ++q) {
                                const float d = (v[8 * i + q] + b[q]) - tg[k][8 * i + q];
                                sk += d * d;
                                g[8 * i + q] = __float2bfloat16_rn(2.0f * d * T.scale);
                            }
                        }
                        uint8_t* blk = smem + s * NET_A_BYTES + (c0 >> 6) * (TILE_M * 128);
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            *reinterpret_cast<uint4*>(blk + sw128((uint32_t)row, (uint32_t)(((c0 & 63) >> 3) + i))) =
                                reinterpret_cast<const uint4*>(g)[i];
                        if (k == (group & 1 ? 0 : 2)) sq.y += sk;
                        else sq.x += sk;
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        sq.x += __shfl_xor_sync(0xffffffffu, sq.x, o);
                        sq.y += __shfl_xor_sync(0xffffffffu, sq.y, o);
                    }
                    if (lane == 0) s_sq[s][quad][group] = sq;
                    umma::fence_before_sync();
                    stage_done();
                    if (lane == 0) umma::mbar_arrive(&o_ready[s]);
                    continue;
                }
                auto out16 = [&](int k) {
                    const int c0 = 48 * group + 16 * k;
                    float v[16];
                    umma::tmem_ld16(tmem + s * 256u + tlane + (uint32_t)c0, v);
#pragma unroll
                    for (int g = 0; g < 2; ++g) {
                        float b[8];
                        cst8(b4 + c0 + 8 * g, b);
#pragma unroll
                        for (int q = 0; q < 8; ++q) v[8 * g + q] += b[q];
                    }
                    if (gr < G.n) store_row16(o + c0, v, wide);
                };
                const int nu = u0 + s + 2;
                if (nu < my_units && ((int)blockIdx.x + nu * (int)gridDim.x) / G.tiles == member) {
                    // every other warp starts a piece later, so that the stores
                    // (32 bytes per clock and SM) come evenly
                    first_layer(s, nu, [&](int k) {
                        const int c = k - (warp & 1);
                        if (c >= 0 && c < 3) out16(c);
                    });
                } else {
                    for (int k = 0; k < 3; ++k) out16(k);
                    if (nu < my_units) first_layer(s, nu, [](int) {});
                }
            }
            if (TRAIN)
                for (int s = 0; s < 2 && u0 + s + 2 < my_units && ok; ++s) {
                    wait_stored(s);
                    if (ok) first_layer(s, u0 + s + 2, [](int) {});
                }
        }
    }
    __syncthreads();
    if (warp == MMA_WARP) {
        umma::fence_after_sync();
        umma::tmem_dealloc(tmem, TMEM_COLS);
    }
}

// Backward through the activations in one kernel, on the same two slots:
//   dZ3 = (dO W4) silu'(Z3),  dZ2 = (dZ3 W3) silu'(Z2),  dZ1 = (dZ2 W2) silu'(Z1)
// with Z1 recomputed from the inputs.  dO comes in by TMA as the first operand;
// each epilogue writes the next operand, which the store warp also writes out
// (dZ3, dZ2, for the weight and bias gradients); the last one forms the layer-1
// gradients.  The bound is that last epilogue, 256 columns x 4 sums over the
// unit's rows through transposed staging tiles (11,000 to 17,000 cycles of the
// 40,000 a unit takes), beside the SiLU derivatives (an exponential and a
// reciprocal each) and, for 65,536 rows, 92 MB to read (Z3, Z2, dO) and 67 MB to
// write (dZ3, dZ2); at DRAM 126 and 34 MB.  65,536 rows: 82 us, 87 us as three
// kernels.
struct NetBack {
    CUtensorMap dO;                      // boxes of 64 x 128
    CUtensorMap w[3];                    // W4^T, W3^T, W2^T as stored [out][in] (MN-major operands): boxes of 64 x 64
    CUtensorMap dz[2];                   // dZ3, dZ2: boxes of 64 x 128
    const bf16 *z3, *z2;
    const float* x;
    const float* params;
    float* grad;                         // parameter block of gradients (accumulated)
    const int32_t* brow;                 // training-set row of each batch row
    int tiles;
    unsigned int* err;
};

__global__ void __launch_bounds__(NET_TRAIN_THREADS, 1) net_backward(const __grid_constant__ NetBack G)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (umma::smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* ring = smem + 2 * NET_A_BYTES;
    __shared__ __align__(8) uint64_t full[NET_STAGES], empty[NET_STAGES], a_ready[2], acc_full[2], stored[2], a_free[2], a_full[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    __shared__ __align__(16) float s_cst[4 * D_H];       // b1, W1 by input component
    __shared__ float s_acc[4 * D_H];                     // b1 gradient, W1 gradient by component

    pdl_trigger();
    const int my_units = ((int)blockIdx.x < G.tiles) ? (G.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    if (my_units == 0) return;               // uniform over the CTA
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int* abort_v = &abort_flag;
    if (threadIdx.x == 0) {
        for (int s = 0; s < NET_STAGES; ++s) { umma::mbar_init(&full[s], 1); umma::mbar_init(&empty[s], 1); }
        for (int s = 0; s < 2; ++s) {
            umma::mbar_init(&a_ready[s], EPI_WARPS);
            umma::mbar_init(&acc_full[s], 1);
            umma::mbar_init(&stored[s], 1);
            umma::mbar_init(&a_free[s], EPI_WARPS);
            umma::mbar_init(&a_full[s], 1);
        }
        abort_flag = 0;
    }
    for (int i = threadIdx.x; i < 4 * D_H; i += blockDim.x) s_acc[i] = 0.0f;
    if (warp == MMA_WARP) umma::tmem_alloc(&tmem_slot, TMEM_COLS);
    pdl_wait();
    for (int i = threadIdx.x; i < D_H; i += blockDim.x) s_cst[i] = G.params[OFF_B1 + i];
    for (int i = threadIdx.x; i < 3 * D_H; i += blockDim.x) s_cst[D_H * (1 + i % 3) + i / 3] = G.params[OFF_W1 + i];
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = tmem_slot;

    if (warp == PRODUCER_WARP) {
        if (lane == 0) {
            uint32_t it = 0, loads[2] = {0, 0};
            bool ok = true;
            auto fetch_z = [&](int l, int u) {
                umma::prefetch_l2((l ? G.z2 : G.z3) + z_block((int)blockIdx.x + u * (int)gridDim.x, 0, 0), TILE_M * D_H * 2);
            };
            for (int l = 0; l < 2; ++l)
                for (int u = 0; u < 2 && u < my_units; ++u) fetch_z(l, u);
            for (int u0 = 0; u0 < my_units && ok; u0 += 2)
                for (int l = 0; l < 3 && ok; ++l)
                    for (int s = 0; s < 2 && u0 + s < my_units && ok; ++s) {
                        // the pre-activations of the units two ahead into L2 (64 KB in a row)
                        if (l < 2 && u0 + s + 2 < my_units) fetch_z(l, u0 + s + 2);
                        if (l == 0) {
                            // the unit's dO into the slot once the last unit's epilogues are through with it
                            if (loads[s] > 0 && !umma::mbar_wait_or_abort(&a_free[s], (loads[s] - 1) & 1u, WAIT_BUDGET, abort_v)) {
                                ok = false;
                                break;
                            }
                            loads[s] += 1;
                            umma::mbar_arrive_expect_tx(&a_full[s], (D_OUT / TILE_K) * TILE_M * 128u);
                            const int tile = (int)blockIdx.x + (u0 + s) * (int)gridDim.x;
                            for (int c = 0; c < D_OUT / TILE_K; ++c)
                                umma::tma_load_2d(smem + s * NET_A_BYTES + c * (TILE_M * 128), &G.dO, c * TILE_K, tile * TILE_M,
                                                  &a_full[s]);
                        }
                        for (int c = 0; c < (l ? D_H : D_OUT) / TILE_K; ++c, ++it) {
                            const uint32_t st = it % NET_STAGES, r = it / NET_STAGES;
                            if (r > 0 && !umma::mbar_wait_or_abort(&empty[st], (r - 1) & 1u, WAIT_BUDGET, abort_v)) {
                                ok = false;
                                break;
                            }
                            umma::mbar_arrive_expect_tx(&full[st], NET_STAGE_BYTES);
                            for (int q = 0; q < D_H / 64; ++q)
                                umma::tma_load_2d(ring + st * NET_STAGE_BYTES + 8192 * q, &G.w[l], 64 * q, c * TILE_K, &full[st]);
                        }
                    }
            if (!ok) { atomicOr(G.err, 1u); *abort_v = 1; }
            // copies still in flight land before the CTA can exit
            for (uint32_t j = it > (uint32_t)NET_STAGES ? it - NET_STAGES : 0u; j < it; ++j)
                umma::mbar_wait(&full[j % NET_STAGES], (j / NET_STAGES) & 1u, WAIT_BUDGET);
            for (int s = 0; s < 2; ++s)
                if (loads[s] > 0) umma::mbar_wait(&a_full[s], (loads[s] - 1) & 1u, WAIT_BUDGET);
        }
    } else if (warp == MMA_WARP) {
        if (lane == 0) {
            uint32_t it = 0, job[2] = {0, 0}, loads[2] = {0, 0};
            bool ok = true;
            const uint32_t idesc = umma::make_idesc_bf16(TILE_M, D_H, false, true);
            for (int u0 = 0; u0 < my_units && ok; u0 += 2)
                for (int l = 0; l < 3 && ok; ++l)
                    for (int s = 0; s < 2 && u0 + s < my_units && ok; ++s) {
                        const bool there = l == 0
                            ? umma::mbar_wait_or_abort(&a_full[s], loads[s]++ & 1u, WAIT_BUDGET, abort_v)
                            : umma::mbar_wait_or_abort(&a_ready[s], job[s]++ & 1u, WAIT_BUDGET, abort_v);
                        if (!there) { ok = false; break; }
                        umma::fence_after_sync();
                        const uint32_t a0 = umma::smem_u32(smem + s * NET_A_BYTES), d = tmem + s * 256u;
                        for (int c = 0; c < (l ? D_H : D_OUT) / TILE_K; ++c, ++it) {
                            const uint32_t st = it % NET_STAGES, r = it / NET_STAGES;
                            if (!umma::mbar_wait_or_abort(&full[st], r & 1u, WAIT_BUDGET, abort_v)) { ok = false; break; }
                            umma::fence_after_sync();
                            const uint32_t sb = umma::smem_u32(ring + st * NET_STAGE_BYTES);
#pragma unroll
                            for (int k = 0; k < TILE_K / 16; ++k)
                                umma::mma_bf16(d, umma::make_desc_sw128(a0 + c * (TILE_M * 128u) + 32u * k),
                                               umma::make_desc_sw128_mn(sb + 2048u * k, 8192u), idesc, (c > 0 || k > 0) ? 1u : 0u);
                            umma::commit(&empty[st]);
                        }
                        if (ok) umma::commit(&acc_full[s]);
                    }
            if (!ok) { atomicOr(G.err, 1u); *abort_v = 1; }
            // the last MMAs complete before TMEM is freed
            if (it > 0) umma::mbar_wait(&empty[(it - 1) % NET_STAGES], ((it - 1) / NET_STAGES) & 1u, WAIT_BUDGET);
        }
    } else if (warp == STORE_WARP) {
        if (lane == 0) {
            uint32_t job[2] = {0, 0};
            bool ok = true;
            for (int u0 = 0; u0 < my_units && ok; u0 += 2)
                for (int l = 0; l < 2 && ok; ++l)
                    for (int s = 0; s < 2 && u0 + s < my_units && ok; ++s) {
                        if (!umma::mbar_wait_or_abort(&a_ready[s], job[s]++ & 1u, WAIT_BUDGET, abort_v)) { ok = false; break; }
                        const int tile = (int)blockIdx.x + (u0 + s) * (int)gridDim.x;
                        for (int c = 0; c < 4; ++c)
                            umma::tma_store_2d(&G.dz[l], c * TILE_K, tile * TILE_M, smem + s * NET_A_BYTES + c * (TILE_M * 128));
                        umma::bulk_commit();
                        umma::bulk_wait_read0();
                        umma::mbar_arrive(&stored[s]);
                    }
            if (!ok) { atomicOr(G.err, 1u); *abort_v = 1; }
            umma::bulk_wait0();
        }
    } else {
        const int quad = warp & 3, group = warp >> 2;
        const int row = 32 * quad + lane;                 // of the unit
        const uint32_t tlane = (uint32_t)(32 * quad) << 16;
        uint32_t job[2] = {0, 0}, written[2] = {0, 0};
        bool ok = true;
        auto give_up = [&] {
            if (lane == 0) atomicOr(G.err, 1u);
            *abort_v = 1;
            ok = false;
        };
        auto wait_acc = [&](int s) {
            if (!umma::mbar_wait_or_abort(&acc_full[s], job[s]++ & 1u, WAIT_BUDGET, abort_v)) give_up();
            umma::fence_after_sync();
        };
        for (int u0 = 0; u0 < my_units && ok; u0 += 2) {
            float xb[2][3];                               // the rows' inputs, used after two layers
#pragma unroll
            for (int s = 0; s < 2; ++s)
                if (u0 + s < my_units) {
                    const float* xr = G.x + (int64_t)G.brow[(int64_t)((int)blockIdx.x + (u0 + s) * (int)gridDim.x) * TILE_M + row] * 3;
                    xb[s][0] = xr[0]; xb[s][1] = xr[1]; xb[s][2] = xr[2];
                }
            // dZ3, dZ2: the next operand
            for (int l = 0; l < 2 && ok; ++l)
                for (int s = 0; s < 2 && u0 + s < my_units; ++s) {
                    const int tile = (int)blockIdx.x + (u0 + s) * (int)gridDim.x;
                    __align__(16) bf16 z[2][32];         // requested before the accumulator is waited for
#pragma unroll
                    for (int k = 0; k < 2; ++k) load_block((l ? G.z2 : G.z3) + z_block(tile, quad, group + 4 * k), lane, z[k]);
                    wait_acc(s);
                    // dZ3 has been stored from the operand that dZ2 overwrites
                    if (l && !umma::mbar_wait_or_abort(&stored[s], written[s] & 1u, WAIT_BUDGET, abort_v)) give_up();
                    if (l) written[s] += 1;
                    if (!ok) break;
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const int c0 = 32 * group + 128 * k;
                        float v[32];
                        umma::tmem_ld32(tmem + s * 256u + tlane + (uint32_t)c0, v);
                        __align__(16) __nv_bfloat162 g[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float2 zq = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(z[k])[i]);
                            g[i] = __floats2bfloat162_rn(v[2 * i] * dsilu(zq.x), v[2 * i + 1] * dsilu(zq.y));
                        }
                        store_a(smem + s * NET_A_BYTES, row, c0, reinterpret_cast<const bf16*>(g));
                    }
                    umma::fence_before_sync();
                    stage_done();
                    if (lane == 0) umma::mbar_arrive(&a_ready[s]);
                }
            // dZ1 and the layer-1 gradients; its tiles are staged in the operand,
            // which is consumed, and stored (dZ2)
            for (int s = 0; s < 2 && u0 + s < my_units && ok; ++s) {
                const float x0 = xb[s][0], x1 = xb[s][1], x2 = xb[s][2];
                wait_acc(s);
                if (!umma::mbar_wait_or_abort(&stored[s], written[s]++ & 1u, WAIT_BUDGET, abort_v)) give_up();
                if (!ok) break;
                uint8_t* tt = smem + s * NET_A_BYTES + warp * 4096;
                float* xs = reinterpret_cast<float*>(tt + STAGE_TILE_BYTES);
                xs[lane] = x0; xs[32 + lane] = x1; xs[64 + lane] = x2;
                for (int c0 = 32 * group; c0 < D_H; c0 += 8 * EPI_WARPS) {
                    float v[32];
                    umma::tmem_ld32(tmem + s * 256u + tlane + (uint32_t)c0, v);
                    __align__(16) __nv_bfloat162 g[16];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float b[8], w0[8], w1[8], w2[8];
                        cst8(s_cst + c0 + 8 * i, b);
                        cst8(s_cst + D_H + c0 + 8 * i, w0);
                        cst8(s_cst + 2 * D_H + c0 + 8 * i, w1);
                        cst8(s_cst + 3 * D_H + c0 + 8 * i, w2);
#pragma unroll
                        for (int q = 0; q < 8; q += 2) {
                            // the forward's pre-activation, same operations in the same
                            // order; two at a time: a single conversion to BF16 is a
                            // special-function-unit operation, a packed one is not
                            auto z = [&](int e) { return __fmaf_rn(x2, w2[e], __fmaf_rn(x1, w1[e], __fmaf_rn(x0, w0[e], b[e]))); };
                            const float2 zq = __bfloat1622float2(__floats2bfloat162_rn(z(q), z(q + 1)));
                            g[4 * i + q / 2] = __floats2bfloat162_rn(v[8 * i + q] * dsilu(zq.x), v[8 * i + q + 1] * dsilu(zq.y));
                        }
                    }
                    stage_col(tt, lane, reinterpret_cast<const bf16*>(g));
                    __syncwarp();
                    warp_col_sums(tt, lane, s_acc + c0, xs, s_acc + D_H + c0);
                    __syncwarp();
                }
                umma::fence_before_sync();
                stage_done();
                if (lane == 0) umma::mbar_arrive(&a_free[s]);
            }
        }
    }
    __syncthreads();
    if (warp == MMA_WARP) {
        umma::fence_after_sync();
        umma::tmem_dealloc(tmem, TMEM_COLS);
    }
    for (int i = threadIdx.x; i < D_H; i += blockDim.x) atomicAdd(G.grad + OFF_B1 + i, s_acc[i]);
    for (int i = threadIdx.x; i < 3 * D_H; i += blockDim.x) atomicAdd(G.grad + OFF_W1 + i, s_acc[D_H * (1 + i % 3) + i / 3]);
}

// The three weight gradients dW^T[out][in] = sum over rows dZ[row][out] H[row][in]
// in one launch.  Their K dimension, the batch, is cut into 64-row chunks; the
// chunks of the 3 layers make one line that is shared out evenly over pairs of
// CTAs (one per tile of 128 inputs: the second reads the same dZ while it is in
// L2).  A CTA's share is cut into runs, each summed in tensor memory and added
// to the FP32 gradient in place.  The tensor cores' adder truncates (a sum of
// 2,656 rows came out 1.7e-6 smaller than three of 896), so a run is no longer
// than a layer's share of all pairs, or 8 chunks where that is more: 65,536 rows
// take 232.6 us a step so, 227.9 with one run per CTA and layer.  One launch per
// layer (a start-up and a drain of the pipeline each) took 51.7 us at 65,536
// rows, this one 46.6 (194 MB read: 4.2 TB/s).  Both operands are MN-major (the activations and
// gradients as stored).  The bias gradients, the column sums of dZ, come from
// the same stages: the epilogue warps, which have little else to do, add up the
// dZ operand of the first tile's runs.
struct WeightGrads {
    CUtensorMap h[3], dz[3];             // H3, H2, H1 and dO, dZ3, dZ2: boxes of 64 x 64
    float* out[3];                       // gradients of W4^T, W3^T, W2^T, row stride 256
    float* bias[3];                      // gradients of b4, b3, b2
    int chunks;                          // batch / 64
    int longest;                         // chunks of one run at most
    unsigned int* err;
};
constexpr int WG_STAGES = 4;
constexpr uint32_t WG_A_BYTES = TILE_M * 128, WG_STAGE_BYTES = WG_A_BYTES + D_H * 128;
constexpr size_t WG_SMEM = 1024 + (size_t)WG_STAGES * WG_STAGE_BYTES;

// The run of chunks that starts at chunk c of the line: its layer, tile, first
// chunk in the batch and length (up to `end` and the longest run).
struct WgRun {
    int layer, tile, first, count;
};
__device__ __forceinline__ WgRun wg_run(int c, int end, const WeightGrads& G)
{
    const int layer = c / G.chunks, first = c - layer * G.chunks;
    return WgRun{layer, (int)(blockIdx.x & 1), first, min(G.longest, min(end - c, G.chunks - first))};
}

__global__ void __launch_bounds__(GEMM_THREADS, 1) weight_grads(const __grid_constant__ WeightGrads G)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (umma::smem_u32(smem_raw) & 1023u)) & 1023u);
    __shared__ __align__(8) uint64_t full[WG_STAGES], empty[WG_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;

    pdl_trigger();
    const int64_t line = 3 * (int64_t)G.chunks;
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int c_begin = (int)(line * pair / pairs), c_end = (int)(line * (pair + 1) / pairs);
    if (c_begin >= c_end) return;            // uniform over the CTA
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int* abort_v = &abort_flag;
    if (threadIdx.x == 0) {
        for (int s = 0; s < WG_STAGES; ++s) { umma::mbar_init(&full[s], 1); umma::mbar_init(&empty[s], 1 + EPI_WARPS); }
        for (int a = 0; a < 2; ++a) { umma::mbar_init(&acc_full[a], 1); umma::mbar_init(&acc_empty[a], EPI_WARPS); }
        abort_flag = 0;
    }
    if (warp == MMA_WARP) umma::tmem_alloc(&tmem_slot, TMEM_COLS);
    pdl_wait();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = tmem_slot;

    if (warp == PRODUCER_WARP) {
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int c = c_begin; c < c_end && ok;) {
                const WgRun r = wg_run(c, c_end, G);
                const int boxes = (r.layer ? D_H : D_OUT) / 64;
                for (int k = 0; k < r.count; ++k, ++it) {
                    const uint32_t s = it % WG_STAGES, n = it / WG_STAGES;
                    if (n > 0 && !umma::mbar_wait_or_abort(&empty[s], (n - 1) & 1u, WAIT_BUDGET, abort_v)) { ok = false; break; }
                    uint8_t* st = smem + s * WG_STAGE_BYTES;
                    const int k0 = (r.first + k) * TILE_K;
                    umma::mbar_arrive_expect_tx(&full[s], WG_A_BYTES + 8192u * boxes);
                    for (int q = 0; q < 2; ++q)
                        umma::tma_load_2d(st + 8192 * q, &G.h[r.layer], r.tile * TILE_M + 64 * q, k0, &full[s]);
                    for (int q = 0; q < boxes; ++q)
                        umma::tma_load_2d(st + WG_A_BYTES + 8192 * q, &G.dz[r.layer], 64 * q, k0, &full[s]);
                }
                c += r.count;
            }
            if (!ok) { atomicOr(G.err, 1u); *abort_v = 1; }
            // copies still in flight land before the CTA can exit
            for (uint32_t j = it > (uint32_t)WG_STAGES ? it - WG_STAGES : 0u; j < it; ++j)
                umma::mbar_wait(&full[j % WG_STAGES], (j / WG_STAGES) & 1u, WAIT_BUDGET);
        }
    } else if (warp == MMA_WARP) {
        if (lane == 0) {
            uint32_t it = 0, j = 0;
            bool ok = true;
            for (int c = c_begin; c < c_end && ok; ++j) {
                const WgRun r = wg_run(c, c_end, G);
                const uint32_t idesc = umma::make_idesc_bf16(TILE_M, r.layer ? D_H : D_OUT, true, true);
                const uint32_t a = j & 1u, u = j >> 1;
                if (u > 0 && !umma::mbar_wait_or_abort(&acc_empty[a], (u - 1) & 1u, WAIT_BUDGET, abort_v)) { ok = false; break; }
                umma::fence_after_sync();
                const uint32_t d = tmem + a * 256u;
                for (int k = 0; k < r.count; ++k, ++it) {
                    const uint32_t s = it % WG_STAGES, n = it / WG_STAGES;
                    if (!umma::mbar_wait_or_abort(&full[s], n & 1u, WAIT_BUDGET, abort_v)) { ok = false; break; }
                    umma::fence_after_sync();
                    const uint32_t sa = umma::smem_u32(smem + s * WG_STAGE_BYTES), sb = sa + WG_A_BYTES;
#pragma unroll
                    for (int q = 0; q < TILE_K / 16; ++q)
                        umma::mma_bf16(d, umma::make_desc_sw128_mn(sa + 2048u * q, 8192u),
                                       umma::make_desc_sw128_mn(sb + 2048u * q, 8192u), idesc, (k > 0 || q > 0) ? 1u : 0u);
                    umma::commit(&empty[s]);
                }
                if (!ok) break;
                umma::commit(&acc_full[a]);
                c += r.count;
            }
            if (!ok) { atomicOr(G.err, 1u); *abort_v = 1; }
            // the last MMAs complete before TMEM is freed
            if (it > 0) umma::mbar_wait(&empty[(it - 1) % WG_STAGES], ((it - 1) / WG_STAGES) & 1u, WAIT_BUDGET);
        }
    } else {
        const int quad = warp & 3;
        uint32_t j = 0, it = 0;
        bool ok = true;
        for (int c = c_begin; c < c_end && ok; ++j) {
            const WgRun r = wg_run(c, c_end, G);
            const uint32_t a = j & 1u, u = j >> 1;
            const int N = r.layer ? D_H : D_OUT;
            // column sums of the stages' dZ (first tile): a lane takes the 8 columns
            // of piece `piece` in every 16th row (8 lanes on 8 different bank groups)
            const int piece = 2 * warp + (lane >> 4);
            const bool sums = r.tile == 0 && 8 * piece < N;
            float cs[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int k = 0; k < r.count && ok; ++k, ++it) {
                const uint32_t s = it % WG_STAGES, n = it / WG_STAGES;
                if (!umma::mbar_wait_or_abort(&full[s], n & 1u, WAIT_BUDGET, abort_v)) { ok = false; break; }
                if (sums) {
                    const uint8_t* blk = smem + s * WG_STAGE_BYTES + WG_A_BYTES + 8192 * (piece >> 3);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint4 g4 = *reinterpret_cast<const uint4*>(blk + sw128((uint32_t)(16 * q + (lane & 15)), (uint32_t)(piece & 7)));
                        const bf16* g8 = reinterpret_cast<const bf16*>(&g4);
#pragma unroll
                        for (int e = 0; e < 8; ++e) cs[e] += __bfloat162float(g8[e]);
                    }
                }
                __syncwarp();
                if (lane == 0) umma::mbar_arrive(&empty[s]);
            }
            if (r.tile == 0) {
#pragma unroll
                for (int e = 0; e < 8; ++e)
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) cs[e] += __shfl_xor_sync(0xffffffffu, cs[e], o);
                if (sums && (lane & 15) < 8) {
                    float v = cs[0];
#pragma unroll
                    for (int e = 1; e < 8; ++e) v = (lane & 7) == e ? cs[e] : v;
                    atomicAdd(G.bias[r.layer] + 8 * piece + (lane & 7), v);
                }
            }
            if (!ok || !umma::mbar_wait_or_abort(&acc_full[a], u & 1u, WAIT_BUDGET, abort_v)) {
                if (lane == 0) atomicOr(G.err, 1u);
                *abort_v = 1;
                break;
            }
            umma::fence_after_sync();
            for (int c0 = 32 * (warp >> 2); c0 < N; c0 += 8 * EPI_WARPS) {
                float v[32];
                umma::tmem_ld32(tmem + a * 256u + ((uint32_t)(32 * quad) << 16) + (uint32_t)c0, v);
                // column n of the tile is row n of the gradient: the warp's 32 inputs
                // are 32 consecutive floats there (one coalesced reduction)
                float* o = G.out[r.layer] + (int64_t)c0 * D_H + r.tile * TILE_M + 32 * quad + lane;
#pragma unroll
                for (int i = 0; i < 32; ++i) atomicAdd(o + i * D_H, v[i]);
            }
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&acc_empty[a]);
            c += r.count;
        }
    }
    __syncthreads();
    if (warp == MMA_WARP) {
        umma::fence_after_sync();
        umma::tmem_dealloc(tmem, TMEM_COLS);
    }
}

}  // namespace mlp
}  // namespace cl

using namespace cl::mlp;

struct cl_mlp {
    int device = 0;
    int max_batch = 0;
    int num_sms = 0;
    int max_ctas = 0;               // cap on the GEMM grid (0: one CTA per SM)
    cudaStream_t stream = nullptr;
    char err[256] = {0};
    // FP32 master parameters, gradients, Adam moments
    float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
    int64_t adam_t = 0;
    // BF16 weight copies
    bf16 *w2t = nullptr, *w3t = nullptr, *w4t = nullptr;
    // activations and gradients (max_batch rows)
    int32_t* brow = nullptr;        // training-set row of each minibatch row
    bf16 *h1 = nullptr, *h2 = nullptr, *z2 = nullptr, *h3 = nullptr, *z3 = nullptr;
    bf16 *dO = nullptr, *dz3 = nullptr, *dz2 = nullptr;
    float* loss = nullptr;          // device accumulator
    unsigned int* derr = nullptr;
    // training set (device pointers owned by the caller)
    const float* data_x = nullptr;
    const float* data_t = nullptr;
    int64_t n_data = 0;
    std::vector<void*> allocs;
};

namespace {

int mlp_fail(cl_mlp* m, int code, const char* fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(m->err, sizeof m->err, fmt, ap);
    va_end(ap);
    return code;
}

template <typename T>
bool dalloc(cl_mlp* m, T** p, size_t count)
{
    void* q = nullptr;
    if (cudaMalloc(&q, count * sizeof(T)) != cudaSuccess) { cudaGetLastError(); return false; }
    m->allocs.push_back(q);
    *p = (T*)q;
    return true;
}

void refresh_bf16(cl_mlp* m, cudaStream_t st)
{
    to_bf16<<<(D_H * D_H + 255) / 256, 256, 0, st>>>(m->p + OFF_W2, D_H * D_H, m->w2t);
    to_bf16<<<(D_H * D_H + 255) / 256, 256, 0, st>>>(m->p + OFF_W3, D_H * D_H, m->w3t);
    to_bf16<<<(D_OUT * D_H + 255) / 256, 256, 0, st>>>(m->p + OFF_W4, D_OUT * D_H, m->w4t);
}

// Rows of targets are read 16 bytes at a time at least.
int check_targets(cl_mlp* m, const float* target)
{
    return (uintptr_t)target & 15 ? mlp_fail(m, CL_ERR_ARG, "the training targets must start on a 16-byte boundary") : CL_OK;
}

int grid_for(const cl_mlp* m, int B)
{
    const int tiles = B / TILE_M;
    const int cap = m->max_ctas > 0 && m->max_ctas < m->num_sms ? m->max_ctas : m->num_sms;
    return tiles < cap ? tiles : cap;
}

// The shared-memory opt-in is a per-device attribute of a kernel: set once for
// every device this process launches on.
int net_attributes(int device)
{
    static std::atomic<uint64_t> done{0};
    const uint64_t bit = 1ull << (device & 63);
    if (done.load() & bit) return CL_OK;
    for (const void* k : {(const void*)net_forward<false>, (const void*)net_forward<true>, (const void*)net_backward,
                          (const void*)weight_grads})
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(k == (const void*)weight_grads ? WG_SMEM : NET_SMEM)) != cudaSuccess)
            return CL_ERR_CUDA;
    done.fetch_or(bit);
    return CL_OK;
}

// Tensor maps of a network's W2^T, W3^T, W4^T.
bool net_weight_maps(const cl_mlp* m, CUtensorMap* w)
{
    return make_map(&w[0], m->w2t, D_H, D_H, D_H, D_H) && make_map(&w[1], m->w3t, D_H, D_H, D_H, D_H) &&
           make_map(&w[2], m->w4t, D_OUT, D_H, D_H, D_OUT);
}

// Forward and backward passes over a batch of B rows (B % 128 == 0) of the
// training set (x, target), m->g accumulating: two kernels for the activations,
// then the weight gradients.  rows.n_all == 0: the batch is the set's first B rows.
int forward_backward(cl_mlp* m, int B, const float* x, const float* target, const BatchRows& rows, cudaStream_t st)
{
    if (int rc = net_attributes(m->device)) return rc;
    const int grid = grid_for(m, B);
    NetArgs f;
    NetTrain t;
    NetBack k;
    memset(&f, 0, sizeof f);
    memset(&t, 0, sizeof t);
    memset(&k, 0, sizeof k);
    if (!net_weight_maps(m, f.w[0]) || !make_map(&t.h[0], m->h1, B, D_H, D_H, TILE_M) ||
        !make_map(&t.h[1], m->h2, B, D_H, D_H, TILE_M) || !make_map(&t.h[2], m->h3, B, D_H, D_H, TILE_M) || !make_map(&t.h[3], m->dO, B, D_OUT, D_OUT, TILE_M) ||
        !make_map(&k.dO, m->dO, B, D_OUT, D_OUT, TILE_M) || !make_map_mn(&k.w[0], m->w4t, D_OUT, D_H, D_H) ||
        !make_map_mn(&k.w[1], m->w3t, D_H, D_H, D_H) || !make_map_mn(&k.w[2], m->w2t, D_H, D_H, D_H) ||
        !make_map(&k.dz[0], m->dz3, B, D_H, D_H, TILE_M) || !make_map(&k.dz[1], m->dz2, B, D_H, D_H, TILE_M))
        return CL_ERR_ARG;
    f.params[0] = m->p; f.x = x; f.n = B; f.members = 1; f.tiles = B / TILE_M; f.err = m->derr;
    t.z2 = m->z2; t.z3 = m->z3; t.target = target; t.rows = rows; t.brow = m->brow;
    t.wide = ((uintptr_t)target & 31) == 0;
    t.scale = 1.0f / ((float)B * (float)D_OUT); t.loss = m->loss;
    const int tail = f.tiles % grid;
    t.whole = 2 * tail <= grid ? f.tiles - tail : f.tiles;
    if (launch_pdl(net_forward<true>, dim3((unsigned)grid), dim3(NET_TRAIN_THREADS), NET_SMEM, st, f, t) != cudaSuccess)
        return CL_ERR_CUDA;
    k.z3 = m->z3; k.z2 = m->z2; k.x = x; k.params = m->p; k.grad = m->g; k.brow = m->brow; k.tiles = B / TILE_M; k.err = m->derr;
    if (launch_pdl(net_backward, dim3((unsigned)grid), dim3(NET_TRAIN_THREADS), NET_SMEM, st, k) != cudaSuccess)
        return CL_ERR_CUDA;
    WeightGrads w;
    memset(&w, 0, sizeof w);
    const bf16* hs[3] = {m->h3, m->h2, m->h1};
    const bf16* dzs[3] = {m->dO, m->dz3, m->dz2};
    const int64_t offs[3] = {OFF_W4, OFF_W3, OFF_W2};
    for (int l = 0; l < 3; ++l) {
        const int N = l ? D_H : D_OUT;
        if (!make_map_mn(&w.h[l], hs[l], B, D_H, D_H) || !make_map_mn(&w.dz[l], dzs[l], B, N, N)) return CL_ERR_ARG;
        w.out[l] = m->g + offs[l];
        w.bias[l] = m->g + offs[l] + (int64_t)N * D_H;      // b follows its W in the block
    }
    w.chunks = B / TILE_K;
    w.err = m->derr;
    // enough chunks per CTA that a run's additions (128 KB) stay small beside it
    const int most = m->num_sms / 2, pairs = std::min(std::max(3 * w.chunks / WGRAD_MIN_CHUNKS, 3), most);
    w.longest = std::max((w.chunks + pairs - 1) / pairs, WGRAD_MIN_RUN);
    if (launch_pdl(weight_grads, dim3(2u * (unsigned)pairs), dim3(GEMM_THREADS),
                   WG_SMEM, st, w) != cudaSuccess)
        return CL_ERR_CUDA;
    return CL_OK;
}

// net_forward over members x n rows, NET_MAX members and 2^24 rows per launch
// (the tensor maps' and tile indices' range).
int net_forward_enqueue(cl_mlp* const* nets, int members, const float* d_x, float* d_out, int64_t n, cudaStream_t st)
{
    cl_mlp* const m = nets[0];
    if (int rc = net_attributes(m->device)) return rc;
    for (int k0 = 0; k0 < members; k0 += NET_MAX) {
        const int K = members - k0 < NET_MAX ? members - k0 : NET_MAX;
        NetArgs g;
        memset(&g, 0, sizeof g);
        for (int k = 0; k < K; ++k) {
            if (!net_weight_maps(nets[k0 + k], g.w[k])) return CL_ERR_ARG;
            g.params[k] = nets[k0 + k]->p;
        }
        g.members = K;
        g.err = m->derr;
        constexpr int64_t ROWS = 1 << 24;
        for (int64_t r0 = 0; r0 < n; r0 += ROWS) {
            const int64_t rows = n - r0 < ROWS ? n - r0 : ROWS;
            // a member's block of rows is n rows from the next one's
            for (int k = 0; k < (rows < n ? K : 1); ++k) {
                const int Kl = rows < n ? 1 : K;
                NetArgs a = g;
                float* out = d_out + ((int64_t)(k0 + k) * n + r0) * D_OUT;
                if (rows < n) {
                    for (int l = 0; l < 3; ++l) a.w[0][l] = g.w[k][l];
                    a.params[0] = g.params[k];
                }
                a.members = Kl;
                a.x = d_x + r0 * D_IN;
                a.n = rows;
                a.tiles = (int)((rows + TILE_M - 1) / TILE_M);
                a.out = out;
                const int units = Kl * a.tiles;
                const int cap = m->max_ctas > 0 && m->max_ctas < m->num_sms ? m->max_ctas : m->num_sms;
                net_forward<false><<<(unsigned)(units < cap ? units : cap), GEMM_THREADS, NET_SMEM, st>>>(a, NetTrain());
                if (cudaPeekAtLastError() != cudaSuccess) return CL_ERR_CUDA;     // the caller reports it
            }
        }
    }
    return CL_OK;
}

cudaError_t adam(cl_mlp* m, float lr, cudaStream_t st)
{
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    m->adam_t += 1;
    const float bc1 = 1.0f - powf(b1, (float)m->adam_t), bc2 = 1.0f - powf(b2, (float)m->adam_t);
    const AdamCopies c = {m->w2t, m->w3t, m->w4t};
    return launch_pdl(adam_all, dim3((unsigned)((N_PARAMS / 4 + 127) / 128)), dim3(128), 0, st, m->p, m->g, m->m, m->v, lr, b1,
                      b2, eps, bc1, bc2, c);
}

}  // namespace

extern "C" {

int cl_mlp_param_count(void) { return (int)N_PARAMS; }

int cl_mlp_create(cl_mlp** out, int device, int max_batch)
{
    if (!out || max_batch < TILE_M || max_batch % TILE_M) return CL_ERR_ARG;
    *out = nullptr;
    cl_mlp* m = new (std::nothrow) cl_mlp();
    if (!m) return CL_ERR_OOM;
    m->device = device;
    m->max_batch = max_batch;
    if (cudaSetDevice(device) != cudaSuccess ||
        cudaDeviceGetAttribute(&m->num_sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        delete m;
        return CL_ERR_CUDA;
    }
    const size_t B = (size_t)max_batch;
    bool ok = dalloc(m, &m->p, N_PARAMS) && dalloc(m, &m->g, N_PARAMS) && dalloc(m, &m->m, N_PARAMS) &&
              dalloc(m, &m->v, N_PARAMS) &&
              dalloc(m, &m->w2t, (size_t)D_H * D_H) && dalloc(m, &m->w3t, (size_t)D_H * D_H) &&
              dalloc(m, &m->w4t, (size_t)D_OUT * D_H) && dalloc(m, &m->brow, B) &&
              dalloc(m, &m->h1, B * D_H) &&
              dalloc(m, &m->h2, B * D_H) && dalloc(m, &m->z2, B * D_H) &&
              dalloc(m, &m->h3, B * D_H) && dalloc(m, &m->z3, B * D_H) &&
              dalloc(m, &m->dO, B * D_OUT) && dalloc(m, &m->dz3, B * D_H) && dalloc(m, &m->dz2, B * D_H) &&
              dalloc(m, &m->loss, 1) &&
              dalloc(m, &m->derr, 1);
    if (!ok) {
        for (void* q : m->allocs) cudaFree(q);
        delete m;
        return CL_ERR_OOM;
    }
    cudaMemsetAsync(m->m, 0, N_PARAMS * sizeof(float), m->stream);
    cudaMemsetAsync(m->v, 0, N_PARAMS * sizeof(float), m->stream);
    cudaMemsetAsync(m->g, 0, N_PARAMS * sizeof(float), m->stream);
    cudaMemsetAsync(m->derr, 0, sizeof(unsigned int), m->stream);
    cudaMemsetAsync(m->p, 0, N_PARAMS * sizeof(float), m->stream);
    refresh_bf16(m, m->stream);
    cudaStreamSynchronize(m->stream);
    *out = m;
    return CL_OK;
}

void cl_mlp_destroy(cl_mlp* m)
{
    if (!m) return;
    cudaSetDevice(m->device);
    cudaStreamSynchronize(m->stream);
    for (void* q : m->allocs) cudaFree(q);
    cudaStreamDestroy(m->stream);
    delete m;
}

const char* cl_mlp_last_error(const cl_mlp* m) { return m ? m->err : ""; }

// Cap the number of CTAs of the forward and backward passes (0 = one per SM); with few
// CTAs each one walks many tiles (tests of the persistent pipeline).
int cl_mlp_set_max_ctas(cl_mlp* m, int n)
{
    if (!m || n < 0) return CL_ERR_ARG;
    m->max_ctas = n;
    return CL_OK;
}

// Parameters in the FP32 block layout above (host buffers of cl_mlp_param_count()).
// Setting parameters resets the Adam state.
int cl_mlp_set_params(cl_mlp* m, const float* host)
{
    if (!m || !host) return CL_ERR_ARG;
    cudaSetDevice(m->device);
    cudaMemcpyAsync(m->p, host, N_PARAMS * sizeof(float), cudaMemcpyHostToDevice, m->stream);
    cudaMemsetAsync(m->m, 0, N_PARAMS * sizeof(float), m->stream);
    cudaMemsetAsync(m->v, 0, N_PARAMS * sizeof(float), m->stream);
    m->adam_t = 0;
    refresh_bf16(m, m->stream);
    return cudaStreamSynchronize(m->stream) == cudaSuccess ? CL_OK : CL_ERR_CUDA;
}

int cl_mlp_get_params(cl_mlp* m, float* host)
{
    if (!m || !host) return CL_ERR_ARG;
    cudaSetDevice(m->device);
    cudaMemcpyAsync(host, m->p, N_PARAMS * sizeof(float), cudaMemcpyDeviceToHost, m->stream);
    return cudaStreamSynchronize(m->stream) == cudaSuccess ? CL_OK : CL_ERR_CUDA;
}

// Training set: n rows of inputs x [n][3] and targets t [n][192], FP32 device
// arrays that stay owned by the caller and must outlive the training calls.
int cl_mlp_set_data(cl_mlp* m, const float* d_x, const float* d_t, int64_t n)
{
    if (!m || !d_x || !d_t || n < 1 || n > 0x7fffffff) return CL_ERR_ARG;
    m->data_x = d_x; m->data_t = d_t; m->n_data = n;
    return CL_OK;
}

// `steps` Adam steps on random minibatches of `batch` rows (batch % 128 == 0,
// batch <= max_batch); *loss_out = mean loss over the steps.
int cl_mlp_train(cl_mlp* m, int steps, int batch, float lr, uint32_t seed, uint32_t step0, float* loss_out)
{
    if (!m || steps < 0 || batch < TILE_M || batch % TILE_M || batch > m->max_batch || !m->data_x)
        return CL_ERR_ARG;
    if (const int rc = steps > 0 ? check_targets(m, m->data_t) : CL_OK) return rc;
    cudaSetDevice(m->device);
    cudaStream_t st = m->stream;
    cudaMemsetAsync(m->loss, 0, sizeof(float), st);
    // the gradient is zeroed once here and then by each Adam step, so that a
    // step is an unbroken chain of kernels
    cudaMemsetAsync(m->g, 0, N_PARAMS * sizeof(float), st);
    for (int s = 0; s < steps; ++s) {
        int rc = forward_backward(m, batch, m->data_x, m->data_t,
                                  BatchRows{(uint32_t)m->n_data, step0 + (uint32_t)s, seed}, st);
        if (!rc && adam(m, lr, st) != cudaSuccess) rc = CL_ERR_CUDA;
        if (rc) return mlp_fail(m, rc, "kernel launch failed: %s", cudaGetErrorString(cudaGetLastError()));
    }
    float loss = 0.0f;
    unsigned int e = 0;
    cudaMemcpyAsync(&loss, m->loss, sizeof loss, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&e, m->derr, sizeof e, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return mlp_fail(m, CL_ERR_CUDA, "%s", cudaGetErrorString(cudaGetLastError()));
    if (e) return mlp_fail(m, CL_ERR_TIMEOUT, "tensor-core completion wait ran out");
    if (loss_out) *loss_out = steps > 0 ? loss / (float)steps : 0.0f;
    return CL_OK;
}

// Inference of `members` networks on one GPU: out[members][n][192] (FP32,
// device) for x[n][3] (FP32, device), enqueued on `stream` (NULL: the first
// network's own); cl_mlp_sync waits and reports.
int cl_mlp_forward_ensemble(cl_mlp* const* nets, int members, const float* d_x, float* d_out, int64_t n, void* stream)
{
    if (!nets || members < 1 || !nets[0]) return CL_ERR_ARG;
    cl_mlp* const m = nets[0];
    m->err[0] = 0;
    if (n < 0) return mlp_fail(m, CL_ERR_ARG, "the number of rows must be >= 0");
    for (int k = 1; k < members; ++k)
        if (!nets[k] || nets[k]->device != m->device)
            return mlp_fail(m, CL_ERR_ARG, "network %d of the ensemble is missing or on another device", k);
    if (n == 0) return CL_OK;
    if (!d_x || !d_out) return mlp_fail(m, CL_ERR_ARG, "null input or output");
    cudaSetDevice(m->device);
    const int rc = net_forward_enqueue(nets, members, d_x, d_out, n, stream ? (cudaStream_t)stream : m->stream);
    return rc ? mlp_fail(m, rc, "forward launch failed: %s", cudaGetErrorString(cudaGetLastError())) : CL_OK;
}

// Wait for the work on `stream` (NULL: the network's own) and report a
// tensor-core wait that ran out.
int cl_mlp_sync(cl_mlp* m, void* stream)
{
    if (!m) return CL_ERR_ARG;
    cudaSetDevice(m->device);
    cudaStream_t st = stream ? (cudaStream_t)stream : m->stream;
    unsigned int e = 0;
    cudaMemcpyAsync(&e, m->derr, sizeof e, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return mlp_fail(m, CL_ERR_CUDA, "%s", cudaGetErrorString(cudaGetLastError()));
    return e ? mlp_fail(m, CL_ERR_TIMEOUT, "tensor-core completion wait ran out") : CL_OK;
}

// Inference: out[n][192] (FP32, device) for x[n][3] (FP32, device).
int cl_mlp_forward(cl_mlp* m, const float* d_x, float* d_out, int64_t n)
{
    if (!m || !d_x || !d_out || n < 0) return CL_ERR_ARG;
    cudaSetDevice(m->device);
    const int rc = n > 0 ? net_forward_enqueue(&m, 1, d_x, d_out, n, m->stream) : CL_OK;
    if (rc) return mlp_fail(m, rc, "forward launch failed: %s", cudaGetErrorString(cudaGetLastError()));
    return cl_mlp_sync(m, nullptr);
}

// Gradient of the loss for one given batch (x [B][3], t [B][192] FP32 device;
// B % 128 == 0): host grad[cl_mlp_param_count()] and the loss.  For tests.
int cl_mlp_gradient(cl_mlp* m, const float* d_x, const float* d_t, int B, float* host_grad, float* loss_out)
{
    if (!m || !d_x || !d_t || !host_grad || B < TILE_M || B % TILE_M || B > m->max_batch) return CL_ERR_ARG;
    if (const int rc = check_targets(m, d_t)) return rc;
    cudaSetDevice(m->device);
    cudaStream_t st = m->stream;
    cudaMemsetAsync(m->loss, 0, sizeof(float), st);
    cudaMemsetAsync(m->g, 0, N_PARAMS * sizeof(float), st);
    const int rc = forward_backward(m, B, d_x, d_t, BatchRows{0u, 0u, 0u}, st);
    if (rc) return mlp_fail(m, rc, "launch failed");
    float loss = 0.0f;
    cudaMemcpyAsync(host_grad, m->g, N_PARAMS * sizeof(float), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&loss, m->loss, sizeof loss, cudaMemcpyDeviceToHost, st);
    unsigned int e = 0;
    cudaMemcpyAsync(&e, m->derr, sizeof e, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return mlp_fail(m, CL_ERR_CUDA, "%s", cudaGetErrorString(cudaGetLastError()));
    if (loss_out) *loss_out = loss;
    return e ? mlp_fail(m, CL_ERR_TIMEOUT, "tensor-core completion wait ran out") : CL_OK;
}

}  // extern "C"


extern "C" {

// Diagnostic: C[M][N] (fp32) = A[M][K] * B[N][K]^T with BF16 device operands,
// on the tensor cores (grid_x CTAs in x, `splits` K splits written as partials
// C[split][M][N] when splits > 1).  Returns CL_ERR_TIMEOUT if an mbarrier wait
// ran out.
int cl_umma_gemm_bf16(const void* A, const void* B, float* C, int M, int N, int K, int grid_x,
                      int splits, unsigned int* d_err, void* stream)
{
    if (!A || !B || !C || !d_err || M <= 0 || N <= 0 || K <= 0 || grid_x <= 0 || splits < 1) return CL_ERR_ARG;
    GemmArgs g;
    memset(&g, 0, sizeof g);
    g.M = M; g.N = N; g.K = K;
    g.out_f = C; g.ldf = N;
    g.err = d_err;
    if (splits > 1) {
        g.k_split = ((K / splits + TILE_K - 1) / TILE_K) * TILE_K;
        return launch_gemm<EPI_PARTIAL>(g, (const bf16*)A, K, (const bf16*)B, K, grid_x, splits,
                                        (cudaStream_t)stream);
    }
    g.k_split = K;
    return launch_gemm<EPI_F32>(g, (const bf16*)A, K, (const bf16*)B, K, grid_x, 1, (cudaStream_t)stream);
}

}  // extern "C"
