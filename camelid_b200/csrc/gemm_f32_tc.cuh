// Float matrix products of many rows on the tensor cores without losing a bit of the operands: D[M, N] = A[M, K] W[N, K]^T.
//
// A float times 2^16 is the exact sum of three bfloat16 numbers h + m + l (each the rounding of what the ones before it left; |m| <= 2^-9,
// |l| <= 2^-18 of the whole), whatever its size: a float is a multiple of 2^-149, so 2^16 of it of 2^-133, bfloat16's own smallest step. (Unscaled,
// floats below 2^-109 would lose their last bits.) A product of two bfloat16 numbers is exact in float. Of the nine products of pieces the six of
// at least 2^-18 of the whole are taken (h h, h m, m h, m m, h l, l h); the three left out lie below 2^-26 of it, a quarter of a float's
// half unit. The tensor core adds in float but cuts instead of rounding, which over a whole K would be a drift of the sum: so
// the h h products of 64 k's are summed there and each such sum is then added, rounded, to the thread's own in registers, and the five small
// ones have an accumulator of their own, where what is cut is 2^-9 of that. The finished sum is multiplied by 2^-32. Against 64 bits the result is closer than plain
// float multiply-adds in order of k: normal operands 1.3e-7 (K = 2,048) and 2.4e-7 (8,192) against their 8.1e-7 and 1.6e-6, all positive 1.1e-7
// against 6.3e-7, sizes over e^(2 normal) 1.6e-7 against 8.1e-7 (2-norms, at 65 to 2,048 rows).
//
// A block computes 128 x 128 outputs in steps of 64 k's. Warps 0-7 hold the next step's floats of both operands in registers, split them
// and store the pieces as 128-byte swizzled rows (16 KB a piece and operand, 96 KB a step, two steps), then add up the h h sums of the step
// before. One thread of warp 8 issues the 24 products of a step, h h first, so that its sums are collected while the
// other 20 run. Shared memory is what it uses most (70 % busy, the tensor pipe 53 %, of active cycles): a product of 128 x 128 x 16 reads 8 KB
// in the 64 cycles it takes, all that a multiprocessor can read, and the pieces have to be written beside it. Measured at 673 rows, against 128 x 128 tiles of packed float
// multiply-adds: 16,384 x 2,048 318 us (142 TFLOP/s) against 1,113; 3,072 x 2,048 62 against 224; 2,048 x 8,192 214 against 882; 2,048 x 2,048 60
// against 222; 65 rows of that 54 against 215. (Floats by cp.async in steps of 32, three ahead, were 1.5 to 2.5 times slower than in
// registers: they cross shared memory twice more.)
//
// An output that is not finite is made again by plain multiply-adds: an operand that is infinite or of 2^111 and more has no pieces, and
// sums of 2^95 and more do not fit while they are scaled.
// Waits are bounded as in the other tensor-core kernels: one that runs out sets *err to 8, and every warp leaves.
#pragma once
#include "common.cuh"

#define FT_ROWS 128
#define FT_K 64
#define FT_THREADS 288
#define FT_WAIT_CYCLES 2000000000ll
#define FT_PIECE (FT_ROWS * FT_K * 2)                   // bytes of a piece of an operand in a step
#define FT_STEP (6 * FT_PIECE)                          // h, m, l of A, then of W
#define FT_SMEM (2 * FT_STEP)

__device__ __forceinline__ uint32_t ft_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool ft_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool ft_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (ft_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (true) {
        if (ft_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > FT_WAIT_CYCLES) {
            *abort_flag = 1;
            return false;
        }
    }
}
__device__ __forceinline__ void ft_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void ft_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void ft_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void ft_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
// adds 64 columns of the accumulator at `taddr` to sum
__device__ __forceinline__ void ft_collect(uint32_t taddr, float (&sum)[64]) {
#pragma unroll
    for (int c = 0; c < 64; c += 32) {
        uint32_t r[16], u[16];
        ft_ld16(taddr + c, r);
        ft_ld16(taddr + c + 16, u);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 16; ++i) { sum[c + i] += __uint_as_float(r[i]); sum[c + 16 + i] += __uint_as_float(u[i]); }
    }
}
// K-major tile of 128-byte rows, 128-byte swizzle, 1,024 bytes between groups of 8 rows
__device__ __forceinline__ uint64_t ft_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
__device__ __forceinline__ uint32_t ft_pack(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}
#define FT_SCALE 65536.0f                               // what both operands are multiplied by, and the sum divided by twice
#define FT_UNSCALE (1.0f / 4294967296.0f)
// two floats side by side: x * f, and x - h, each rounded as by itself
__device__ __forceinline__ float2 ft_mul2(float2 x, float f) { return __fmul2_rn(x, make_float2(f, f)); }
__device__ __forceinline__ float2 ft_sub2(float2 x, float2 h) { return __ffma2_rn(h, make_float2(-1.f, -1.f), x); }
// eight neighbouring floats -> the three pieces of each, scaled, 16 bytes a piece
__device__ __forceinline__ void ft_split(const float4& a, const float4& b, uint4& h, uint4& m, uint4& l) {
    float2 x[4] = {make_float2(a.x, a.y), make_float2(a.z, a.w), make_float2(b.x, b.y), make_float2(b.z, b.w)};
    uint32_t p[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = ft_mul2(x[i], FT_SCALE);
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            p[q][i] = ft_pack(x[i].x, x[i].y);
            x[i] = ft_sub2(x[i], make_float2(__uint_as_float(p[q][i] << 16), __uint_as_float(p[q][i] & 0xffff0000u)));
        }
    h = make_uint4(p[0][0], p[0][1], p[0][2], p[0][3]);
    m = make_uint4(p[1][0], p[1][1], p[1][2], p[1][3]);
    l = make_uint4(p[2][0], p[2][1], p[2][2], p[2][3]);
}
__device__ __forceinline__ void ft_store16(uint32_t at, const uint4& v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// those of n outputs that are not finite again, by plain multiply-adds
__device__ __noinline__ void ft_plain_sums(float* out, const float* x, const float* w, int ldw, int n, int K) {
    for (int i = 0; i < n; ++i) {
        if (fabsf(out[i]) <= 3.402823466e38f) continue;
        float v = 0.f;
        for (int k = 0; k < K; ++k) v = fmaf(x[k], w[(size_t)i * ldw + k], v);
        out[i] = v;
    }
}

template <int EPI>
__global__ void __launch_bounds__(FT_THREADS, 1)
gemm_f32_tc_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ C, int ldc, int M,
                   int n_wrows, int K, int tiles_m, int* err, const GateAct act) {
    extern __shared__ uint8_t ft_raw[];
    __shared__ __align__(8) uint64_t bar_store[9];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_store;
    volatile int* abort_flag = &abort_store;
    const uint32_t base = (ft_smem(ft_raw) + 1023u) & ~1023u, bars = ft_smem(bar_store);
    // per step: pieces there, pieces read, h h sums there, h h sums collected; then all small sums there
    auto full = [&](int s) { return bars + 8u * s; };
    auto empty = [&](int s) { return bars + 16u + 8u * s; };
    auto sums = [&](int s) { return bars + 32u + 8u * s; };
    auto taken = [&](int s) { return bars + 48u + 8u * s; };
    const uint32_t done = bars + 64u;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = (int)(blockIdx.x % tiles_m) * FT_ROWS, n0 = (int)(blockIdx.x / tiles_m) * FT_ROWS;
    const int steps = (K + FT_K - 1) / FT_K;
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(full(s)), "r"(256));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty(s)), "r"(1));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sums(s)), "r"(1));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(taken(s)), "r"(256));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(done), "r"(1));
        abort_store = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ft_smem(&tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;                    // columns: h h of even steps, of odd steps, the small products
    pdl_launch_dependents();
    if (warp == 8) {
        if (lane == 0) {
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(FT_ROWS >> 3) << 17) | ((uint32_t)(FT_ROWS >> 4) << 24);
            bool ok = true;
            for (int i = 0; i < steps && ok; ++i) {
                const int s = i & 1;
                const uint32_t ph = (uint32_t)(i >> 1) & 1u;
                ok = ft_wait(full(s), ph, abort_flag) && ft_wait(taken(s), ph ^ 1u, abort_flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t at = base + s * FT_STEP;
                const uint64_t a[3] = {ft_desc(at), ft_desc(at + FT_PIECE), ft_desc(at + 2 * FT_PIECE)};
                const uint64_t w[3] = {ft_desc(at + 3 * FT_PIECE), ft_desc(at + 4 * FT_PIECE), ft_desc(at + 5 * FT_PIECE)};
#pragma unroll
                for (int k = 0; k < FT_K / 16; ++k) ft_mma(tmem + s * FT_ROWS, a[0] + 2 * k, w[0] + 2 * k, idesc, k ? 1u : 0u);
                ft_commit(sums(s));
#pragma unroll
                for (int x = 0; x < 5; ++x) {           // the smallest products first
                    const int pa = x == 0 ? 0 : x == 1 ? 2 : x == 2 ? 1 : x == 3 ? 0 : 1, pw = x == 0 ? 2 : x == 1 ? 0 : x == 2 ? 1 : x == 3 ? 1 : 0;
#pragma unroll
                    for (int k = 0; k < FT_K / 16; ++k)
                        ft_mma(tmem + 2 * FT_ROWS, a[pa] + 2 * k, w[pw] + 2 * k, idesc, (i | x | k) ? 1u : 0u);
                }
                ft_commit(empty(s));
            }
            if (ok) ft_commit(done);
        }
    } else {
        // A thread has four rows of each operand, 32 apart, and of each of them the columns 4 c .. 4 c + 3 and 32 + 4 c .. 32 + 4 c + 3 of a
        // step (whole sectors for neighbouring lanes). They are stored as columns 8 c .. 8 c + 7: the order of k is the same in both operands.
        const int r = tid >> 3, c = tid & 7;
        const float* ap[4];
        const float* wp[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {                   // (rows beyond a matrix repeat its last one: their outputs are never stored)
            ap[p] = A + (size_t)min(m0 + r + 32 * p, M - 1) * lda + c * 4;
            wp[p] = W + (size_t)min(n0 + r + 32 * p, n_wrows - 1) * ldw + c * 4;
        }
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        float4 ra[4][2], rw[4][2];
        auto fetch = [&](const float* const (&from)[4], float4 (&to)[4][2], int k0) {
            const bool in0 = k0 + c * 4 < K, in1 = k0 + 32 + c * 4 < K;
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                to[p][0] = in0 ? *reinterpret_cast<const float4*>(from[p] + k0) : zero;
                to[p][1] = in1 ? *reinterpret_cast<const float4*>(from[p] + k0 + 32) : zero;
            }
        };
        const uint32_t mine = (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4));       // (row r + 32 p has the same swizzle)
        auto store = [&](uint32_t at, const float4 (&from)[4][2]) {
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                uint4 h, m, l;
                ft_split(from[p][0], from[p][1], h, m, l);
                const uint32_t o = at + mine + p * 32 * 128;
                ft_store16(o, h);
                ft_store16(o + FT_PIECE, m);
                ft_store16(o + 2 * FT_PIECE, l);
            }
        };
        auto wait_all = [&](uint32_t bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, ft_wait(bar, parity, abort_flag)); };
        const uint32_t my_cols = tmem + (uint32_t)((warp >> 2) * 64) + ((uint32_t)((warp & 3) * 32) << 16);
        float sum[64];
#pragma unroll
        for (int i = 0; i < 64; ++i) sum[i] = 0.f;
        auto collect = [&](int i) -> bool {
            if (!wait_all(sums(i & 1), (uint32_t)(i >> 1) & 1u)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            ft_collect(my_cols + (i & 1) * FT_ROWS, sum);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            ft_arrive(taken(i & 1));
            return true;
        };
        pdl_wait();                                     // for both operands: the second may be a kernel's output as well
        fetch(wp, rw, 0);
        fetch(ap, ra, 0);
        bool ok = true;
        for (int i = 0; i < steps && ok; ++i) {
            const int s = i & 1;
            ok = wait_all(empty(s), ((uint32_t)(i >> 1) & 1u) ^ 1u);
            if (!ok) break;
            store(base + s * FT_STEP, ra);
            store(base + s * FT_STEP + 3 * FT_PIECE, rw);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            ft_arrive(full(s));
            if (i + 1 < steps) {
                fetch(ap, ra, (i + 1) * FT_K);
                fetch(wp, rw, (i + 1) * FT_K);
            }
            if (i > 0) ok = collect(i - 1);
        }
        ok = ok && collect(steps - 1) && wait_all(done, 0);
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            ft_collect(my_cols + 2 * FT_ROWS, sum);
            const int row = m0 + (warp & 3) * 32 + lane, col0 = n0 + (warp >> 2) * 64;
            if (row < M) {
                bool all_finite = true;
#pragma unroll
                for (int i = 0; i < 64; ++i) { all_finite &= fabsf(sum[i]) <= 3.402823466e38f; sum[i] *= FT_UNSCALE; }
                if (!all_finite) {                      // through 256 bytes of the thread's own in the pieces' place, which nothing reads any more
                    float* out = reinterpret_cast<float*>(ft_raw + (base - ft_smem(ft_raw))) + tid * 64;
#pragma unroll
                    for (int i = 0; i < 64; ++i) out[i] = sum[i];
                    ft_plain_sums(out, A + (size_t)row * lda, W + (size_t)col0 * ldw, ldw, min(64, n_wrows - col0), K);
#pragma unroll
                    for (int i = 0; i < 64; ++i) sum[i] = out[i];
                }
                if (EPI == EPI_SWIGLU) {                // groups of 16 gate rows and the 16 up rows of the same outputs
#pragma unroll
                    for (int g = 0; g < 64; g += 32) {
                        const int out = (col0 + g) / 2;
                        float* o = C + (size_t)row * ldc + out;
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (2 * out < n_wrows) o[i] = gate_act(sum[g + i], sum[g + 16 + i], act);
                    }
                } else {
                    float* o = C + (size_t)row * ldc + col0;
                    const bool vec = (((uintptr_t)o) & 15) == 0;
#pragma unroll
                    for (int i = 0; i < 64; i += 4) {
                        if (vec && col0 + i + 4 <= n_wrows) {
                            float4 v = make_float4(sum[i], sum[i + 1], sum[i + 2], sum[i + 3]);
                            if (EPI == EPI_ADD_F32) {
                                const float4 t = *reinterpret_cast<const float4*>(o + i);
                                v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
                            }
                            *reinterpret_cast<float4*>(o + i) = v;
                        } else {
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                if (col0 + i + j < n_wrows) o[i + j] = EPI == EPI_ADD_F32 ? o[i + j] + sum[i + j] : sum[i + j];
                        }
                    }
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    if (warp == 8) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
    if (tid == 0 && abort_store && err) atomicExch(err, 8);
}

// A: [M, K], W: [n_wrows, K], both 16-byte aligned with K and the row strides in multiples of 4; SwiGLU: W packed in groups of 16.
static int launch_gemm_f32_tc(const void* A, int lda, const void* W, int ldw, void* C, int ldc, int M, int N, int K, int epilogue, int* err,
                              cudaStream_t s) {
    const int n_wrows = epilogue == EPI_SWIGLU ? 2 * N : N;
    const int tiles_m = (M + FT_ROWS - 1) / FT_ROWS;
    const long tiles = (long)tiles_m * ((n_wrows + FT_ROWS - 1) / FT_ROWS);
    if (tiles > 0x7fffffffL) return CML_ERR_BAD_SIZE;
    constexpr size_t smem = FT_SMEM + 1024;
    cudaError_t e;
#define CML_GEMMF(E)                                                                                                             \
    e = cml_allow_smem<gemm_f32_tc_kernel<E>>(smem);                                                                             \
    if (e != cudaSuccess) return (int)e;                                                                                         \
    launch_pdl(gemm_f32_tc_kernel<E>, dim3((unsigned)tiles), dim3(FT_THREADS), smem, s, (const float*)A, lda, (const float*)W, ldw, \
               (float*)C, ldc, M, n_wrows, K, tiles_m, err, cml_gate_act_now)
    switch (epilogue) {
        case EPI_STORE:
        case EPI_STORE_F32: CML_GEMMF(EPI_STORE_F32); break;
        case EPI_ADD_F32: CML_GEMMF(EPI_ADD_F32); break;
        case EPI_SWIGLU: CML_GEMMF(EPI_SWIGLU); break;
        default: return CML_ERR_BAD_SIZE;
    }
#undef CML_GEMMF
    return cml_launch_status();
}
