// y = x W^T for the products of steps of few rows (decode steps of up to 8 sequences, short prompts), bfloat16
// operands, float sums.
//
// What bounds it: the weights, each byte of which crosses the memory bus once, and the chain of dependent kernels that a
// decode step is. So a block owns 16 output features and the whole of K: the sum is complete inside the block, and whatever
// reads the product next, the activation, the residual add and the weight half of the norm behind it, happens here instead
// of in a kernel of its own over split sums. 16 features a tile, not the 128 of a tcgen05 tile, because no split of K is then
// needed to give every SM work: 2,048 features are 128 tiles, and a wide product leaves the SMs at most one small tile apart.
// With 1 to 8 rows the tensor pipe has nothing to win: mma.sync m16n8k16 takes the weights as its 16-row operand and the
// step's rows as its 8 columns.
//
// The weights do not depend on the kernel before: a ring of six stages (16 weight rows x 512 columns by one TMA copy) is
// filled ahead of the dependency wait, 96 KB a block and two blocks an SM, so that a product's first weights arrive while
// the kernel before still runs. The eight warps work on a stage together, each on 64 of its columns, with the step's rows
// of those columns in registers: all their loads are in flight at once behind the wait, and the rows serve every tile of
// the block. That holds for up to 2,048 columns; a longer K is split over blocks whose float sums the reader adds. (Measured
// before, 2,048 features of K = 8,192, one row and eight: rows of x fetched again four stages ahead 8.2 and 9.3 us; copied
// ahead through shared memory 9.5 and 17; a warp a stage, so that a place of the ring stays taken while one warp reads it,
// 8.3 and 9.3, and 16,384 features of K = 2,048 14.7 against 11.1; the blocks of a cluster adding up over distributed shared
// memory 11.6 and 12.6. A stage's place asked full again by the working warps in turn instead of a producer: 17 against 11.1.)
// A lane takes 16 columns in a row of both operands, so the order of the columns inside 64 differs from the instruction's
// own, alike on both sides; the swizzle then puts the eight lanes that read two rows together on different banks.
//
// In a chain of one product, 8 rows: 16,384 x 2,048 11.3 us (6.0 TB/s; the transposed tcgen05 product 14.1), 8,192 x 2,048 6.4 (8.1), 2,048 x 8,192
// 6.5 (7.8), 128,256 x 2,048 78 (86).
//
// It stands where the reference runs q8_gemv (src/cuda_resident.rs:230, :1494).
//
// Every wait on an mbarrier is bounded: when a bound is hit the block sets *err, stops waiting (all its warps still pass
// the same barriers) and writes nothing more; it leaves after its copies have had time to land.
#define CML_HAS_GATE_ACT
#include "common.cuh"
#include "activations.cuh"
#include <cuda.h>

#define FEW_WARPS 8
#define FEW_THREADS (32 * FEW_WARPS + 32)
#define FEW_KB 512                        // columns of a stage
#define FEW_STAGE (16 * FEW_KB * 2)       // eight boxes of 16 rows x 64 columns, 128-byte swizzle
#define FEW_STAGES 6                      // at most: two blocks fit an SM
#define FEW_WAIT_CYCLES 2000000000ll

enum { FEW_F32 = 0, FEW_BF16 = 1, FEW_GATED = 2, FEW_ADD = 3, FEW_ADD_NORM = 4 };

struct FewParams {
    const bf16* w; long ldw; int n;       // weights [n, k]
    const bf16* x; long ldx; int rows, k; // the step's rows
    void* out; long ldo;                  // FEW_F32 float, FEW_BF16 / FEW_GATED bfloat16, FEW_ADD(_NORM) the float residual stream
    const float* bias; int act;           // FEW_BF16
    GateAct gate;                         // FEW_GATED: w holds 16 gate rows, the 16 up rows of the same outputs, and so on
    const float* in_sumsq; int in_parts; float in_inv_hidden, in_eps;   // the scale the rows of x still lack, or null
    const void* norm_w; int norm_w_dtype; bf16* x_out; long ldxo; float* out_sumsq;   // FEW_ADD_NORM
    int tiles, blocks;                    // blocks a share of K
    int share, part;                      // blocks that share K, stages of K a block
    long split_stride;                    // from one share's outputs to the next one's (elements)
    // Routed products: the shares are (row, choice) pairs instead, pair i multiplies row i / top of x with the matrix of expert
    // ids[i] (its rows in w from ids[i] * n on; a choice beyond the experts is left alone). Written by an earlier kernel.
    const int* ids; int top, experts;
    int stages;                           // of the ring
    int whole;                            // K is a multiple of 64: a stage is one copy
    int* err;
};

__device__ __forceinline__ uint32_t few_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool few_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool few_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (few_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (true) {
        if (few_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > FEW_WAIT_CYCLES) {
            *abort_flag = 1;
            return false;
        }
    }
}
__device__ __forceinline__ void few_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

#define FEW_X_STAGES 4                    // stages of K whose rows of x a block keeps in registers

template <int EPI>
__global__ void __launch_bounds__(FEW_THREADS, 2) gemm_few_kernel(const __grid_constant__ CUtensorMap map, const FewParams p) {
    extern __shared__ uint8_t smem_raw[];
    // the warps' sums of a tile: features g and g + 8, rows 2t and 2t + 1 of a lane side by side, the lanes of one g 20 floats
    // from the next one's, so that the reads of 16 features meet on no bank (the writes of a lane's four do, two by two: once a tile)
    __shared__ __align__(16) float red[2][FEW_WARPS][8 * 20];
    __shared__ float row_scale[8];
    __shared__ __align__(8) uint64_t bars[2 * FEW_STAGES];
    __shared__ int abort_word;
    volatile int* abort_flag = &abort_word;
    const uint32_t ring = (few_smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint8_t* ring_ptr = smem_raw + (ring - few_smem_u32(smem_raw));
    const uint32_t bar0 = few_smem_u32(bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (FEW_STAGES + s); };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int share = p.share, rank = (int)blockIdx.x % share;
    if (threadIdx.x == 32) asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&map) : "memory");
    if (threadIdx.x == 0) {
        for (int s = 0; s < FEW_STAGES; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(full_bar(s)), "r"(1));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty_bar(s)), "r"(FEW_WARPS));
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    pdl_launch_dependents();

    const int first = (int)blockIdx.x / share, step = (int)gridDim.x / share;      // this block's first tile, and to its next one
    int my_tiles = (p.tiles - first + step - 1) / step, expert = 0;
    if (p.ids != nullptr) {                                      // (which weights is known behind the wait only)
        pdl_wait();
        expert = p.ids[rank];
        if (expert < 0 || expert >= p.experts) my_tiles = 0;
    }
    const int k0 = p.ids != nullptr ? 0 : rank * p.part * FEW_KB, k1 = min(p.k, k0 + p.part * FEW_KB);    // this block's columns
    const int kblocks = max(0, (k1 - k0 + FEW_KB - 1) / FEW_KB);
    const int stages = p.stages;

    // Asks for a stage, by all lanes of one warp: one copy where the map can cut K into pieces of 64 columns (a copy of 2 KB
    // costs the copy engine nearly what one of 16 KB does: 5.2 TB/s of weights against 6.9), else a lane copies a piece.
    // FEW_GATED: rows 0 to 7 of a tile are gate rows, 8 to 15 the up rows of the same eight outputs.
    auto ask = [&](int tile, int k, int s) {
        constexpr int BOXES = EPI == FEW_GATED ? 2 : 1, BOX_BYTES = 16 * 128 / BOXES;
        const uint32_t to = ring + (uint32_t)(s * FEW_STAGE);
        const int pieces = p.whole ? FEW_KB / 64 : min(FEW_KB / 64, (k1 - k + 63) / 64);       // boxes that hold any column of K
        if (lane == 0) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full_bar(s)), "r"(pieces * 16 * 128) : "memory");
            if (p.whole && EPI == FEW_GATED)
                asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
                             ::"r"(to), "l"((uint64_t)&map), "r"(full_bar(s)), "r"(0), "r"(8 * (tile & 1)), "r"(0), "r"(expert * (p.n / 32) + (tile >> 1)),
                             "r"(k / 64) : "memory");
            else if (p.whole)
                asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                             ::"r"(to), "l"((uint64_t)&map), "r"(full_bar(s)), "r"(0), "r"(expert * p.n + 16 * tile), "r"(k / 64) : "memory");
        }
        if (p.whole) return;
        __syncwarp();
        const int piece = lane & 7, half = lane >> 3;
        if (half < BOXES && piece < pieces)
            asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                         ::"r"(to + (uint32_t)(piece * 16 * 128 + half * BOX_BYTES)), "l"((uint64_t)&map), "r"(full_bar(s)),
                         "r"(k + piece * 64), "r"(expert * p.n + (EPI == FEW_GATED ? 32 * (tile >> 1) + 8 * (tile & 1) + 16 * half : 16 * tile)) : "memory");
    };
    if (warp == FEW_WARPS) {                                     // the producer: its first stages ahead of everything that waits
        // (counters, no divisions: what lies between a place's last read and its next copy is taken from the bytes in flight;
        // 16,384 features of K = 2,048: 13.1 us with four divisions a stage)
        int s = 0;
        uint32_t phase = 1;                                      // (a ring's first round waits for nothing)
        bool ok = true;
        for (int tile = first; tile < first + my_tiles * step && ok; tile += step)
            for (int k = k0; k < k1; k += FEW_KB) {
                ok = __all_sync(0xffffffffu, few_wait(empty_bar(s), phase, abort_flag));
                if (!ok) break;
                ask(tile, k, s);
                if (++s == stages) s = 0, phase ^= 1u;
            }
        if (*abort_flag) {
            const long long t0 = clock64();
            while (clock64() - t0 < 20000000ll) {}               // (copies that are in flight land before the block leaves)
        }
        return;
    }

    const int g = lane >> 2, t = lane & 3;
    uint4 x[FEW_X_STAGES][2];
    pdl_wait();
    {
        const bf16* x_lane = p.x + (size_t)(p.ids != nullptr ? rank / p.top : min(g, p.rows - 1)) * p.ldx;
#pragma unroll
        for (int u = 0; u < FEW_X_STAGES; ++u)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int k = k0 + u * FEW_KB + warp * 64 + t * 16 + 8 * j;
                x[u][j] = (g < p.rows && k < k1) ? *reinterpret_cast<const uint4*>(x_lane + k) : make_uint4(0u, 0u, 0u, 0u);
            }
    }
    if (p.in_sumsq != nullptr && warp < p.rows) {
        // the rows' scale: a warp a row, beside the loads of the rows themselves (the first barrier below hands it over)
        float ssq = 0.f;
        for (int q0 = 0; q0 < p.in_parts; q0 += 128) {
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int q = q0 + 32 * j + lane;
                v[j] = p.in_sumsq[(size_t)min(q, p.in_parts - 1) * p.rows + warp];
                if (q >= p.in_parts) v[j] = 0.f;
            }
            ssq += (v[0] + v[1]) + (v[2] + v[3]);
        }
        ssq = warp_sum(ssq);
        if (lane == 0) row_scale[warp] = 1.0f / sqrtf(ssq * p.in_inv_hidden + p.in_eps);
    }

    // The epilogue of a tile: four warps (the first and the last four take turns), half a warp a row of the step, a lane an
    // output feature.
    const int r = 2 * (warp & 3) + (lane >> 4);
    const int at = (lane & 7) * 20 + (r >> 1) * 4 + ((lane >> 3) & 1) * 2 + (r & 1);
    bool ok = true;
    int s = 0;
    uint32_t phase = 0;                                          // the stage's place in the ring, and how often that was used, odd or even
    for (int it = 0; it < my_tiles; ++it) {
        const int tile = first + it * step, f = 16 * tile + (lane & 15);
        const bool last_half = (warp >> 2) == (it & 1) && 2 * (warp & 3) < p.rows, mine = r < p.rows && f < p.n;
        float old = 0.f, mul = 0.f;                              // (on their way before the sums are there)
        if (last_half && mine) {
            if (EPI == FEW_ADD || EPI == FEW_ADD_NORM) old = ((const float*)p.out)[(size_t)r * p.ldo + f];
            if (EPI == FEW_ADD_NORM) mul = p.norm_w_dtype == CML_DTYPE_F32 ? ((const float*)p.norm_w)[f] : __bfloat162float(((const bf16*)p.norm_w)[f]);
            if (EPI == FEW_BF16 && p.bias != nullptr) old = p.bias[f];
        }
        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int u = 0; u < FEW_X_STAGES; ++u) {
            if (u >= kblocks) break;
            if (ok) ok = few_wait(full_bar(s), phase, abort_flag);
            if (k0 + u * FEW_KB + warp * 64 < k1) {              // (beyond K nothing was copied)
                // rows g and g + 8 of the warp's box; the swizzle exchanges a row's 16-byte pieces by the row's number
                const uint8_t* row = ring_ptr + s * FEW_STAGE + warp * 16 * 128 + g * 128;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const uint4 lo = *reinterpret_cast<const uint4*>(row + (((2 * t + j) ^ g) << 4));
                    const uint4 hi = *reinterpret_cast<const uint4*>(row + 8 * 128 + (((2 * t + j) ^ g) << 4));
                    few_mma(acc[j], lo.x, hi.x, lo.y, hi.y, x[u][j].x, x[u][j].y);
                    few_mma(acc[j], lo.z, hi.z, lo.w, hi.w, x[u][j].z, x[u][j].w);
                }
            }
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty_bar(s)) : "memory");
            if (++s == stages) s = 0, phase ^= 1u;
        }
        *reinterpret_cast<float4*>(&red[it & 1][warp][g * 20 + t * 4]) =
            make_float4(acc[0][0] + acc[1][0], acc[0][1] + acc[1][1], acc[0][2] + acc[1][2], acc[0][3] + acc[1][3]);
        // the warps' sums are there (and those of two tiles before have been read)
        asm volatile("bar.sync 1, %0;" ::"n"(32 * FEW_WARPS) : "memory");
        if (!last_half) continue;                                // (whole warps)
        float v = 0.f;
#pragma unroll
        for (int wp = 0; wp < FEW_WARPS; ++wp) v += red[it & 1][wp][at];
        const bool write = mine && *abort_flag == 0;
        if (p.in_sumsq != nullptr) v *= row_scale[min(r, p.rows - 1)];
        if (EPI == FEW_GATED) {
            const float up = __shfl_xor_sync(0xffffffffu, v, 8);
            if (write && (lane & 8) == 0)
                ((bf16*)p.out)[(size_t)rank * p.split_stride + (size_t)r * p.ldo + 8 * tile + (lane & 7)] = __float2bfloat16_rn(gate_act_fast(v, up, p.gate));
        } else if (EPI == FEW_F32) {
            if (write) ((float*)p.out)[(size_t)rank * p.split_stride + (size_t)r * p.ldo + f] = v;
        } else if (EPI == FEW_BF16) {
            if (write) ((bf16*)p.out)[(size_t)r * p.ldo + f] = __float2bfloat16_rn(apply_act(v + old, p.act));
        } else {
            v += old;
            if (write) ((float*)p.out)[(size_t)r * p.ldo + f] = v;
            if (EPI == FEW_ADD_NORM) {
                if (write) p.x_out[(size_t)r * p.ldxo + f] = __float2bfloat16_rn(v * mul);
                float ssq = write ? v * v : 0.f;
#pragma unroll
                for (int o = 1; o < 16; o <<= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, o);
                if (write && (lane & 15) == 0) p.out_sumsq[(size_t)tile * p.rows + r] = ssq;
            }
        }
    }
    if (threadIdx.x == 0 && *abort_flag) atomicExch(p.err, 2);
}

typedef CUresult (*FewEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                CUtensorMapFloatOOBfill);
static FewEncodeFn few_encode() {
    static FewEncodeFn fn = nullptr;
    if (!fn) {
        void* q = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &q, cudaEnableDefault, &r) == cudaSuccess && r == cudaDriverEntryPointSuccess)
            fn = (FewEncodeFn)q;
    }
    return fn;
}

template <int EPI>
static int few_launch(const FewParams& p, cudaStream_t s) {
    FewEncodeFn encode = few_encode();
    if (!encode) return CML_ERR_BAD_SIZE;
    CUtensorMap map;
    const cuuint64_t k = (cuuint64_t)p.k, n = (cuuint64_t)p.n * (p.ids != nullptr ? p.experts : 1), ld = (cuuint64_t)p.ldw * 2;
    const cuuint32_t one[5] = {1, 1, 1, 1, 1};
    // whole: columns in pieces of 64 are a dimension of their own; FEW_GATED: its rows as 16 rows of (gate, up) of every 16 outputs
    const cuuint64_t dims2[2] = {k, n}, dims3[3] = {64, n, k / 64}, dims5[5] = {64, 16, 2, n / 32, k / 64};
    const cuuint64_t strides2[1] = {ld}, strides3[2] = {ld, 128}, strides5[4] = {ld, 16 * ld, 32 * ld, 128};
    const cuuint32_t box2[2] = {64, EPI == FEW_GATED ? 8u : 16u}, box3[3] = {64, 16, FEW_KB / 64}, box5[5] = {64, 8, 2, 1, FEW_KB / 64};
    const int rank = !p.whole ? 2 : (EPI == FEW_GATED ? 5 : 3);
    if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<bf16*>(p.w), rank == 2 ? dims2 : (rank == 3 ? dims3 : dims5),
               rank == 2 ? strides2 : (rank == 3 ? strides3 : strides5), rank == 2 ? box2 : (rank == 3 ? box3 : box5), one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return CML_ERR_BAD_SIZE;
    const size_t smem = 1024 + (size_t)p.stages * FEW_STAGE;
    cudaError_t e = cml_allow_smem<gemm_few_kernel<EPI>>(smem);
    if (e != cudaSuccess) return (int)e;
    e = launch_pdl(gemm_few_kernel<EPI>, dim3((unsigned)(p.blocks * p.share)), dim3(FEW_THREADS), smem, s, map, p);
    return e != cudaSuccess ? (int)e : cml_launch_status();
}

// x [rows, k] (rows ldx apart), W [n, k] (rows ldw apart): bases on 16 bytes, k and the row strides multiples of 8, rows 1 to 8;
// k is shared by `splits` blocks of at most 2,048 columns each, none of them empty. epilogue: FEW_F32 out float = x W^T (split s of several writes
// its sums at out + s * split_stride; all else takes k in one); FEW_BF16 out = act(x W^T + bias) (the codes of apply_act; bias float or null);
// FEW_GATED out [rows, n / 2] = gated activation of W's interleaved gate and up rows (n a multiple of 32); FEW_ADD out (the
// float residual stream) += x W^T; FEW_ADD_NORM also x_out = bfloat16(out * norm_w) and out_sumsq [ceil(n / 16)][rows] = each
// row's sum of squares of a tile's 16 columns. in_sumsq (or null): [in_parts][rows]; the rows of x lack the scale
// rsqrt(sum of their parts / in_hidden + in_eps), which the sums are multiplied with.
extern "C" int cml_gemm_few(const void* x, long ldx, int rows, const void* w, long ldw, int n, int k, void* out, long ldo,
                            int epilogue, const float* bias, int act, const float* in_sumsq, int in_parts, int in_hidden,
                            float in_eps, const void* norm_w, int norm_w_dtype, void* x_out, long ldxo, float* out_sumsq, int splits,
                            long split_stride, int* err, void* stream) {
    if (rows <= 0 || n <= 0) return 0;
    if (rows > 8 || k <= 0 || (k & 7) || (ldx & 7) || (ldw & 7)) return CML_ERR_BAD_SIZE;
    if ((((uintptr_t)x | (uintptr_t)w) & 15)) return CML_ERR_BAD_ALIGN;
    if (epilogue == FEW_GATED && (n & 31)) return CML_ERR_BAD_SIZE;
    if (in_sumsq && (in_parts < 1 || in_hidden < 1)) return CML_ERR_BAD_SIZE;
    if (epilogue == FEW_ADD_NORM) {
        if (!norm_w || !x_out || !out_sumsq) return CML_ERR_BAD_SIZE;
        if (norm_w_dtype != CML_DTYPE_F32 && norm_w_dtype != CML_DTYPE_BF16) return CML_ERR_BAD_DTYPE;
    }
    FewParams p;
    p.w = (const bf16*)w; p.ldw = ldw; p.n = n;
    p.x = (const bf16*)x; p.ldx = ldx; p.rows = rows; p.k = k;
    p.out = out; p.ldo = ldo;
    p.bias = bias; p.act = act;
    p.gate = cml_gate_act_now;
    p.in_sumsq = in_sumsq; p.in_parts = in_parts; p.in_inv_hidden = in_hidden > 0 ? 1.0f / (float)in_hidden : 0.f; p.in_eps = in_eps;
    p.norm_w = norm_w; p.norm_w_dtype = norm_w_dtype; p.x_out = (bf16*)x_out; p.ldxo = ldxo; p.out_sumsq = out_sumsq;
    p.tiles = (n + 15) / 16;
    const int kblocks = (k + FEW_KB - 1) / FEW_KB;
    if (splits < 1) return CML_ERR_BAD_SIZE;
    p.part = (kblocks + splits - 1) / splits;
    if (p.part > FEW_X_STAGES || (splits - 1) * p.part >= kblocks || (splits > 1 && epilogue != FEW_F32)) return CML_ERR_BAD_SIZE;
    p.share = splits;
    p.split_stride = split_stride;
    p.ids = nullptr; p.top = 1; p.experts = 0;
    const int most = cml_sm_count() / splits;
    p.blocks = p.tiles < most ? p.tiles : (most > 0 ? most : 1);
    // A block that has one tile keeps a ring of it: what it leaves free lets the blocks of the kernel behind it start early. One of
    // two keeps both, so that the second is asked for at once (4,096 features, 8 rows, ring of one tile / of two: K = 512 2.7 us / 2.0,
    // 1,024 3.3 / 2.6, 1,536 3.7 / 3.1; the tcgen05 product 2.6, 3.7, 4.5), where they fit; four stages of a tile and six 4.2 / 4.0 alone,
    // but 6.3 / 6.4 with the norm behind.
    const int rounds = (p.tiles + p.blocks - 1) / p.blocks;
    p.stages = rounds > 2 ? FEW_STAGES : rounds == 2 && 2 * p.part <= FEW_STAGES ? 2 * p.part : p.part;
    p.whole = (k & 63) == 0;
    p.err = err;
    cudaStream_t s = (cudaStream_t)stream;
#define FEW_CASE(E) case E: return few_launch<E>(p, s)
    switch (epilogue) {
        FEW_CASE(FEW_F32);
        FEW_CASE(FEW_BF16);
        FEW_CASE(FEW_GATED);
        FEW_CASE(FEW_ADD);
        FEW_CASE(FEW_ADD_NORM);
    }
#undef FEW_CASE
    return CML_ERR_BAD_SIZE;
}

// The routed products of few rows: pair i of `pairs` (row i / top of x, its choice i % top) times the matrix of expert ids[i]:
// w [experts * n, k] (expert e's rows from e * n on), out [pairs, ldo]: FEW_F32 float, FEW_GATED bfloat16 [pairs, n / 2]. A
// choice beyond the experts leaves its output as it is. k up to 2,048.
//
// A pair is the share of some blocks, which stream its expert's matrix for one row, twice where two pairs chose one expert (the
// second time from L2). The grouped tcgen05 product sorts the rows by expert and takes a tile of 128 rows for each expert that
// has any: for 4 pairs of 1,024 x 2,048 and 1,024 x 1,024 28 us with the sorting, against 9 here.
extern "C" int cml_gemm_few_experts(const void* x, long ldx, int pairs, int top, const void* w, long ldw, int experts, int n, int k,
                                    void* out, long ldo, int epilogue, const int* ids, int* err, void* stream) {
    if (pairs <= 0 || n <= 0) return 0;
    if (pairs > 64 || top < 1 || experts < 1 || k <= 0 || k > FEW_X_STAGES * FEW_KB || (k & 7) || (ldx & 7) || (ldw & 7)) return CML_ERR_BAD_SIZE;
    if ((((uintptr_t)x | (uintptr_t)w) & 15)) return CML_ERR_BAD_ALIGN;
    if (!ids || (epilogue != FEW_F32 && epilogue != FEW_GATED) || (epilogue == FEW_GATED && (n & 31))) return CML_ERR_BAD_SIZE;
    FewParams p = {};
    p.w = (const bf16*)w; p.ldw = ldw; p.n = n;
    p.x = (const bf16*)x; p.ldx = ldx; p.rows = 1; p.k = k;
    p.out = out; p.ldo = ldo; p.split_stride = ldo;
    p.gate = cml_gate_act_now;
    p.tiles = (n + 15) / 16;
    p.share = pairs;
    p.part = (k + FEW_KB - 1) / FEW_KB;
    p.ids = ids; p.top = top; p.experts = experts;
    const int most = cml_sm_count() / pairs;
    p.blocks = p.tiles < most ? p.tiles : (most > 0 ? most : 1);
    p.stages = FEW_STAGES;
    p.whole = (k & 63) == 0;
    p.err = err;
    return epilogue == FEW_F32 ? few_launch<FEW_F32>(p, (cudaStream_t)stream) : few_launch<FEW_GATED>(p, (cudaStream_t)stream);
}
