// Recurrent mixers with a matrix state per head: S [key_dim, value_dim] in float, carried from
// token to token for each sequence.
//
//   gated delta rule (one decay per key channel, or one per head):  S <- diag(g) S;  u = beta (v - S^T k);
//                                                  S <- S + k u^T;  o = S^T q
//   matrix memory with exponential gates:          m' = max(f + m, i);
//                                                  S <- e^(f + m - m') S + e^(i - m') k v^T  (n likewise with k alone);
//                                                  o = S^T q / (max(|n . q|, e^(-m')) + 1e-6)
//
//   retention (a fixed decay per head):            S <- d S + k v^T;  o = S^T q
//   state-space recurrence (decay e^(-e^A dt) and step dt per head and token, k and q shared by groups of heads):
//                                                  S <- e^(-e^A dt) S + dt k v^T;  o = S^T q + D v
//   generalized delta rule (decay w and removal rate a per key channel, u = k / |k|):
//                                                  S <- diag(w) S - (a * u)(u^T S) + k v^T;  o = S^T r
//
// All are independent per column of S: eight threads of a warp share one column (a slice of
// the key axis each, in registers) of one (sequence, head) and walk the sequence's new tokens
// in order, so a prompt's rows and the same rows fed one by one are summed in the same order.
// The matrix memory keeps n as one more column (whose v is 1) and a copy of m per column, so
// that no thread reads what another writes. q, k, gates of a few tokens at a time are staged
// in shared memory by the whole block.
//
// Before them: the short causal convolution with SiLU and the unit norm of q and k for the
// delta rule. After them: the per-head RMS norm with weight and sigmoid gate.
#include "common.cuh"

__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float logsigmoid_f(float x) { return x < 0.f ? x - log1pf(expf(x)) : -log1pf(expf(-x)); }
__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float split_sum(const float* p, int n, long stride) {
    float v = p[0];
    for (int s0 = 1; s0 < n; s0 += 8) {                        // eight splits' loads in flight, added in split order
        float t[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) t[k] = p[(size_t)min(s0 + k, n - 1) * stride];
#pragma unroll
        for (int k = 0; k < 8; ++k) v += s0 + k < n ? t[k] : 0.f;
    }
    return v;
}

// ------------------------------------------------------------------------------------
// Short convolution + SiLU (+ unit norm). `proj` [rows, ld] holds, from column 0, the q
// channels (qk_heads x key_dim), the k channels (the same) and the v channels (heads x
// value_dim) before the convolution; `conv_w` [channels, taps] float, the last tap the current
// token's; `state` [slots, taps - 1, channels] the inputs of the tokens before the step.
// A warp owns one (row, head of q | k | v). q and k become x / sqrt(sum x^2 + 1e-6), q times
// q_scale. out [rows, channels] float. With `update_state` (steps in which every sequence brings
// one row) the warp also moves its channels of the state on by that row; otherwise a later
// launch replaces the state. `early`: the step's integers stood in place before the kernel ahead of this one began; they are
// read ahead of the wait.
__global__ void conv_unit_kernel(const float* __restrict__ proj, long ld, const float* __restrict__ conv_w,
                                 float* __restrict__ state, int update_state, const int* __restrict__ row_seq,
                                 const int* __restrict__ row_pos, const int* __restrict__ seq_row0,
                                 const int* __restrict__ seq_slot, float* __restrict__ out, int rows, int qk_heads,
                                 int heads, int key_dim, int value_dim, int taps, float q_scale,
                                 const float* __restrict__ decay_in, long ldd, const float* __restrict__ a_log,
                                 const float* __restrict__ dt_bias, float* __restrict__ decay_out, int decay_dim, int early) {
    if (!early) pdl_wait();
    const int units = 2 * qk_heads + heads + (decay_in ? heads : 0);
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int r = min(warp / units, rows - 1), u = warp % units;
    const int s = row_seq[r], pos = row_pos[r], inside = r - seq_row0[s], slot = seq_slot[s];
    pdl_wait();
    pdl_launch_dependents();
    if (warp >= rows * units) return;
    if (u >= 2 * qk_heads + heads) {
        // the decays of one (row, head), once for all the scan's blocks of that head:
        // g = exp(-exp(a_log[head]) softplus(x + dt_bias))
        const int hd = u - 2 * qk_heads - heads;
        const float rate = expf(a_log[hd]);
        for (int d = lane; d < decay_dim; d += 32) {            // decay_dim: key_dim (a decay per channel) or 1 (per head)
            const float x = decay_in[(size_t)r * ldd + hd * decay_dim + d] + dt_bias[hd * decay_dim + d];
            decay_out[((size_t)r * heads + hd) * decay_dim + d] = expf(-rate * softplus_f(x));
        }
        return;
    }
    const int channels = 2 * qk_heads * key_dim + heads * value_dim;
    int c0, n;
    if (u < 2 * qk_heads) { c0 = u * key_dim; n = key_dim; }
    else { c0 = 2 * qk_heads * key_dim + (u - 2 * qk_heads) * value_dim; n = value_dim; }
    float* st = state + (size_t)slot * (taps - 1) * channels;
    float ss = 0.f;
    if (taps == 4 && n > 0 && n <= 128 && update_state) {
        // Single-token steps, four taps and heads of up to 128 channels: the tokens before are all in the state, and its three rows, the
        // new one and the taps are asked for at once (tap by tap, then the state again to move it on: five trips to memory; 5.8 us -> 3.1).
        // The same numbers: taps in order, a tap before the sequence's start left out.
        float x[4][4], w[4][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int c = c0 + min(lane + 32 * e, n - 1);
#pragma unroll
            for (int j = 0; j < 3; ++j) x[j][e] = st[(size_t)j * channels + c];
            x[3][e] = proj[(size_t)r * ld + c];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j][e] = conv_w[(size_t)c * 4 + j];
        }
        float a[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int c = c0 + lane + 32 * e;
            float acc = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (3 - j <= pos) acc = fmaf(w[j][e], x[j][e], acc);
            a[e] = silu_f(acc);
            if (lane + 32 * e >= n) continue;
            ss = fmaf(a[e], a[e], ss);
            st[c] = pos >= 2 ? x[1][e] : 0.f;
            st[(size_t)channels + c] = pos >= 1 ? x[2][e] : 0.f;
            st[(size_t)2 * channels + c] = x[3][e];
        }
        float scale = 1.0f;
        if (u < 2 * qk_heads) {
            ss = warp_sum(ss);
            scale = (u < qk_heads ? q_scale : 1.0f) / sqrtf(ss + 1e-6f);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (lane + 32 * e < n) out[(size_t)r * channels + c0 + lane + 32 * e] = u < 2 * qk_heads ? a[e] * scale : a[e];
        return;
    }
    // A lane's channels eight at a time, tap by tap: the eight loads of a tap are unconditional (of a valid
    // place) and in flight together; nothing is stored until every tap has been read.
    for (int base = c0; base < c0 + n; base += 256) {
        float acc[8];
        int cc[8];
        bool ok[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int c = base + lane + 32 * e;
            ok[e] = c < c0 + n;
            cc[e] = ok[e] ? c : c0;
            acc[e] = 0.f;
        }
        const int ne = min(8, (c0 + n - base + 31) / 32);  // groups of 32 channels that are there at all (the same for the warp)
        for (int j = 0; j < taps; ++j) {
            const int back = taps - 1 - j;                 // tokens before this one
            if (back > pos) continue;                      // before the sequence's start
            const float* src = back <= inside ? proj + (size_t)(r - back) * ld : st + (size_t)(taps - 1 + inside - back) * channels;
            float x[8], w[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (e < ne) { x[e] = src[cc[e]]; w[e] = conv_w[(size_t)cc[e] * taps + j]; }
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (e < ne) acc[e] = fmaf(w[e], x[e], acc[e]);
        }
        if (update_state && taps > 1) {                    // one row per sequence: drop the oldest input, keep this one
            for (int j = 0; j + 2 < taps; ++j) {
                float t[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) t[e] = st[(size_t)(j + 1) * channels + cc[e]];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (ok[e]) st[(size_t)j * channels + cc[e]] = pos + j + 2 >= taps ? t[e] : 0.f;
            }
            float t[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) t[e] = proj[(size_t)r * ld + cc[e]];
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (ok[e]) st[(size_t)(taps - 2) * channels + cc[e]] = t[e];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            if (!ok[e]) continue;
            const float a = silu_f(acc[e]);
            out[(size_t)r * channels + cc[e]] = a;
            ss = fmaf(a, a, ss);
        }
    }
    if (u < 2 * qk_heads) {
        ss = warp_sum(ss);
        const float scale = (u < qk_heads ? q_scale : 1.0f) / sqrtf(ss + 1e-6f);
        __syncwarp();
        for (int c = c0 + lane; c < c0 + n; c += 32) out[(size_t)r * channels + c] *= scale;
    }
}

// The same, number for number, for steps of many rows, with four taps and heads of up to 128 channels in whole 16-byte pieces: a warp takes CU_ROWS
// rows of one head, a lane four channels, whose taps (16 bytes a channel) are read once and whose last three inputs stay in registers from row
// to row; all rows' inputs are asked for together. The kernel above reads the taps again for every row, a channel's 16 bytes from those of its
// neighbour, and each input four times. 2,048 rows, 48 heads of 128 and 16 of decays: 134 us -> 50 (134 MB, 21 us at the copy bandwidth; 44 with
// the squares added in the cheapest order); 512 rows 31.6 -> 14.8; 2,048 rows of 24 heads of 128 with a decay per head 57 -> 19.5.
#define CU_ROWS 8
#define CU_MIN_WARPS 592        // a block of four on every multiprocessor: 512 warps took 6.8 us where those of one row each take 6.4 and 5.9, 768 7.0 against 8.5
// The sum of a head's squares as conv_unit_kernel adds it, where lane v has channels v, v + 32, v + 64, v + 96: their chain, then a butterfly over
// 16, 8, 4, 2 and 1. Here lane l = 8 e + j has channels 4 l + m, that is channel 32 e of the lanes v = 4 j + m there: the chain runs over the
// lanes j, 8 + j, 16 + j, 24 + j, the butterfly over the bits of j (each lane keeping half of its sums), then of m.
__device__ __forceinline__ float conv_squares(const float4& a, bool mine, int lane) {
    const float v[4] = {a.x, a.y, a.z, a.w};
    float s[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) s[m] = mine ? fmaf(v[m], v[m], 0.f) : 0.f;
#pragma unroll
    for (int e = 1; e < 4; ++e)
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const float t = __shfl_up_sync(0xffffffffu, s[m], 8);
            if ((lane >> 3) == e) s[m] = mine ? fmaf(v[m], v[m], t) : t;
        }
    // lanes 24 + j have the sums of the lanes v = 4 j + m
    float p[2];
#pragma unroll
    for (int m = 0; m < 2; ++m) {                               // bit 2 of j (16 of v): a lane keeps m or m + 2
        const bool up = (lane & 4) != 0;
        p[m] = (up ? s[m + 2] : s[m]) + __shfl_xor_sync(0xffffffffu, up ? s[m] : s[m + 2], 4);
    }
    const bool up = (lane & 2) != 0;                            // bit 1 of j (8 of v)
    float q = (up ? p[1] : p[0]) + __shfl_xor_sync(0xffffffffu, up ? p[0] : p[1], 2);
    q += __shfl_xor_sync(0xffffffffu, q, 1);                    // bit 0 of j (4 of v)
    q += __shfl_xor_sync(0xffffffffu, q, 4);                    // m's bit 1 (which the lane's bit 2 chose)
    q += __shfl_xor_sync(0xffffffffu, q, 2);                    // m's bit 0
    return __shfl_sync(0xffffffffu, q, 24);
}
__global__ void __launch_bounds__(128) conv_unit_rows_kernel(const float* __restrict__ proj, long ld, const float* __restrict__ conv_w,
                                                             const float* __restrict__ state, const int* __restrict__ row_seq,
                                                             const int* __restrict__ row_pos, const int* __restrict__ seq_row0,
                                                             const int* __restrict__ seq_slot, float* __restrict__ out, int rows, int qk_heads,
                                                             int heads, int key_dim, int value_dim, float q_scale,
                                                             const float* __restrict__ decay_in, long ldd, const float* __restrict__ a_log,
                                                             const float* __restrict__ dt_bias, float* __restrict__ decay_out, int decay_dim) {
    pdl_wait();
    pdl_launch_dependents();
    const int units = 2 * qk_heads + heads + (decay_in ? heads : 0);
    const long warp = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31, u = (int)(warp % units);
    const long first = warp / units * CU_ROWS;
    if (first >= rows) return;
    const int r0 = (int)first, nr = min(CU_ROWS, rows - r0);
    auto at4 = [](const float* p) -> float4 { return *reinterpret_cast<const float4*>(p); };
    if (u >= 2 * qk_heads + heads) {                            // the decays of one head: g = exp(-exp(a_log[head]) softplus(x + dt_bias))
        const int hd = u - 2 * qk_heads - heads, d = lane * 4;
        const float rate = expf(a_log[hd]);
        if (decay_dim == 1) {                                   // a lane per row
            if (lane < nr) decay_out[(size_t)(r0 + lane) * heads + hd] = expf(-rate * softplus_f(decay_in[(size_t)(r0 + lane) * ldd + hd] + dt_bias[hd]));
            return;
        }
        if (d >= decay_dim) return;
        const float4 b = at4(dt_bias + hd * decay_dim + d);
        float4 x[CU_ROWS];
#pragma unroll
        for (int i = 0; i < CU_ROWS; ++i) x[i] = at4(decay_in + (size_t)(r0 + min(i, nr - 1)) * ldd + hd * decay_dim + d);
#pragma unroll
        for (int i = 0; i < CU_ROWS; ++i)
            if (i < nr)
                *reinterpret_cast<float4*>(decay_out + ((size_t)(r0 + i) * heads + hd) * decay_dim + d) =
                    make_float4(expf(-rate * softplus_f(x[i].x + b.x)), expf(-rate * softplus_f(x[i].y + b.y)),
                                expf(-rate * softplus_f(x[i].z + b.z)), expf(-rate * softplus_f(x[i].w + b.w)));
        return;
    }
    const int channels = 2 * qk_heads * key_dim + heads * value_dim;
    const int n = u < 2 * qk_heads ? key_dim : value_dim;
    const int c = (u < 2 * qk_heads ? u * key_dim : 2 * qk_heads * key_dim + (u - 2 * qk_heads) * value_dim) + (lane * 4 < n ? lane * 4 : 0);
    const bool mine = lane * 4 < n;
    float4 w[4];                                                // by channel: its four taps, the last one the current token's
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = at4(conv_w + (size_t)(c + e) * 4);
    float4 x[CU_ROWS];
#pragma unroll
    for (int i = 0; i < CU_ROWS; ++i) x[i] = at4(proj + (size_t)(r0 + min(i, nr - 1)) * ld + c);
    float4 b3, b2, b1;                                          // the inputs three, two and one tokens before
    int before = -1;
#pragma unroll
    for (int i = 0; i < CU_ROWS; ++i) {
        if (i >= nr) break;
        const int r = r0 + i, s = row_seq[r];
        if (s != before) {                                      // the group's first row, or a sequence's
            before = s;
            const int pos = row_pos[r], inside = r - seq_row0[s];
            const float* st = state + (size_t)seq_slot[s] * 3 * channels + c;
            auto earlier = [&](int back) -> float4 {
                if (back > pos) return make_float4(0.f, 0.f, 0.f, 0.f);
                return back <= inside ? at4(proj + (size_t)(r - back) * ld + c) : at4(st + (size_t)(3 + inside - back) * channels);
            };
            b3 = earlier(3); b2 = earlier(2); b1 = earlier(1);
        }
        float4 a;
        a.x = silu_f(fmaf(w[0].w, x[i].x, fmaf(w[0].z, b1.x, fmaf(w[0].y, b2.x, fmaf(w[0].x, b3.x, 0.f)))));
        a.y = silu_f(fmaf(w[1].w, x[i].y, fmaf(w[1].z, b1.y, fmaf(w[1].y, b2.y, fmaf(w[1].x, b3.y, 0.f)))));
        a.z = silu_f(fmaf(w[2].w, x[i].z, fmaf(w[2].z, b1.z, fmaf(w[2].y, b2.z, fmaf(w[2].x, b3.z, 0.f)))));
        a.w = silu_f(fmaf(w[3].w, x[i].w, fmaf(w[3].z, b1.w, fmaf(w[3].y, b2.w, fmaf(w[3].x, b3.w, 0.f)))));
        b3 = b2; b2 = b1; b1 = x[i];
        if (u < 2 * qk_heads) {
            const float scale = (u < qk_heads ? q_scale : 1.0f) / sqrtf(conv_squares(a, mine, lane) + 1e-6f);
            a.x *= scale; a.y *= scale; a.z *= scale; a.w *= scale;
        }
        if (mine) *reinterpret_cast<float4*>(out + (size_t)r * channels + c) = a;
    }
}

// decay_in (may be null) [rows, ldd] (heads x decay_dim, decay_dim = key_dim or 1): the decays' inputs; decay_out [rows, heads x decay_dim] gets
// g = exp(-exp(a_log[head]) softplus(x + dt_bias)), what the delta-rule scan multiplies its state by.
extern "C" int cml_conv_unit(const float* proj, long ld, const float* conv_w, float* state, int update_state, const int* row_seq,
                             const int* row_pos, const int* seq_row0, const int* seq_slot, float* out, int rows, int qk_heads,
                             int heads, int key_dim, int value_dim, int taps, float q_scale, const float* decay_in, long ldd,
                             const float* a_log, const float* dt_bias, float* decay_out, int decay_dim, int early, void* stream) {
    if (rows <= 0) return 0;
    if (taps < 1 || (decay_in && decay_dim != 1 && decay_dim != key_dim)) return CML_ERR_BAD_SIZE;
    const int units = 2 * qk_heads + heads + (decay_in ? heads : 0);
    const bool pieces = !((key_dim | value_dim) & 3) && key_dim <= 128 && value_dim <= 128 && !(ld & 3) &&
                        !((((uintptr_t)proj) | ((uintptr_t)conv_w) | ((uintptr_t)state) | ((uintptr_t)out)) & 15) &&
                        (!decay_in || decay_dim == 1 || (!(ldd & 3) && !((((uintptr_t)decay_in) | ((uintptr_t)dt_bias) | ((uintptr_t)decay_out)) & 15)));
    const long row_warps = ((long)rows + CU_ROWS - 1) / CU_ROWS * units;
    if (taps == 4 && row_warps >= CU_MIN_WARPS && !update_state && pieces) {    // (fewer: the warps of one row each are needed to fill the device)
        launch_pdl(conv_unit_rows_kernel, dim3((unsigned)((row_warps + 3) / 4)), dim3(128), 0, (cudaStream_t)stream, proj, ld, conv_w,
                   (const float*)state, row_seq, row_pos, seq_row0, seq_slot, out, rows, qk_heads, heads, key_dim, value_dim, q_scale, decay_in,
                   ldd, a_log, dt_bias, decay_out, decay_dim);
        return cml_launch_status();
    }
    const long warps = (long)rows * units;
    launch_pdl(conv_unit_kernel, dim3((unsigned)((warps + 3) / 4)), dim3(128), 0, (cudaStream_t)stream, proj, ld, conv_w, state,
               update_state, row_seq, row_pos, seq_row0, seq_slot, out, rows, qk_heads, heads, key_dim, value_dim, taps, q_scale, decay_in, ldd,
               a_log, dt_bias, decay_out, decay_dim, early);
    return cml_launch_status();
}

// ------------------------------------------------------------------------------------
// The scans. A block of 128 threads owns 128 / NS columns of one (sequence, head); the key axis of a
// column is cut into NS slices (a power of two up to 32) of DS channels, one thread each, the NS
// threads of a column in one warp (lane = NS * column + slice), so that a dot product over the key
// axis is DS multiply-adds and a butterfly of log2 NS shuffles, always in the same order, whatever
// the step or the batch. The delta rule takes its two products
// (with k for the write, with q for the read-out) from the decayed state at once and adds the
// write's share u (k . q) to the read-out, so a token waits only for the write of the one before. The state lies column by column
// ([.., column, key channel]): a warp reads and writes whole rows of it with 16-byte accesses.
// q, k and the decays of SCAN_TOKENS tokens at a time stand in shared memory (slices padded by
// four floats against bank conflicts); the next tokens' values are fetched into registers
// while these are worked on.
//
// MODE 0, gated delta rule. in_a = qkv [rows, lda]: unit q (qk_heads x D), unit k, v (heads x Dv)
// from conv_unit_kernel; in_b [rows, ldb]: beta before the sigmoid at column b_col + head;
// in_c [rows, ldc] (heads x D, or heads with one decay per head): the decays g (decay_ready), or their input:
// g = exp(-exp(a_log[head]) softplus(x + dt_bias)).
// state [slots, heads, Dv, D]. out [rows, heads x Dv] = S^T q.
// MODE 1, matrix memory. in_a = proj [rows, lda] with q at q_col (heads x D), k at k_col, v at
// v_col (heads x Dv), gate inputs at i_col + head and f_col + head (before bias and cap).
// state [slots, heads, Dv + 1, D] (column Dv is n), state_m [slots, heads, Dv + 1] (m, one copy
// per column, so that no thread reads what another writes). out [rows, heads, Dv + 2]: S^T q per
// column, then n . q, then m after the token.
// MODE 2, retention. in_a = proj [rows, lda] with q at q_col (heads x D), k at k_col, v at v_col (heads x Dv), q and k
// turned and scaled already; vec_a [heads]: the heads' decays. state [slots, heads, Dv, D]. out [rows, heads x Dv].
// MODE 3, state-space recurrence. in_a [rows, lda] from ssm_inputs_kernel: v at v_col (heads x Dv), k and q at k_col and q_col
// (qk_heads x D, each shared by heads / qk_heads heads); in_b [rows, ldb]: the steps dt (heads), then the decays
// (heads); vec_a [heads]: D. state [slots, heads, Dv, D]. out [rows, heads x Dv].
#define SCAN_TOKENS 8

struct ScanParams {
    const float* in_a; long lda;
    const float* in_b; long ldb; int b_col;
    const float* in_c; long ldc;
    const float* vec_a;           // a_log [heads]            | input-gate bias [heads]
    const float* vec_b;           // dt_bias [heads x D]      | forget-gate bias [heads]
    float* state; float* state_m;
    const int* seq_row0; const int* seq_new; const int* seq_start; const int* seq_slot;
    float* out;
    int heads, qk_heads, D, Dv;
    int q_col, k_col, v_col, i_col, f_col;
    float cap, q_scale;
    int decay_ready;              // in_c holds the decays themselves (conv_unit_kernel made them)
    int decay_dim;                // D: one decay per key channel; 1: one per head (in_c and vec_b are heads x decay_dim)
    int below;                    // greater than zero: sequences with as many new rows or more are left alone (they run by chunks)
};

template <int NS>
__device__ __forceinline__ float slices_sum(float v) {
#pragma unroll
    for (int sh = 1; sh < NS; sh <<= 1) v += __shfl_xor_sync(0xffffffffu, v, sh);
    return v;
}

template <int DS, int MODE, int NS>
__global__ void __launch_bounds__(128) scan_kernel(const ScanParams p) {
    constexpr int SCAN_COLS = 128 / NS;                // columns of a block
    constexpr int DPAD = NS * DS;                      // key channels a block can take
    constexpr int SL = DS == 4 ? 4 : DS + 4;           // floats of a slice in shared memory (padded against bank conflicts)
    constexpr int PER = SCAN_TOKENS * DPAD / 128;      // staged values per thread and array
    __shared__ __align__(16) float sq[SCAN_TOKENS][NS * SL], sk[SCAN_TOKENS][NS * SL], sg[MODE == 0 ? SCAN_TOKENS : 1][NS * SL];
    __shared__ float sv[SCAN_TOKENS][SCAN_COLS], s1[SCAN_TOKENS], s2[SCAN_TOKENS], skq[SCAN_TOKENS];
    pdl_wait();
    pdl_launch_dependents();
    const int s = blockIdx.x, hd = blockIdx.y;
    const int D = p.D, Dv = p.Dv, heads = p.heads;
    const int cols = MODE == 1 ? Dv + 1 : Dv;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int slice = lane % NS;
    const int wcol = warp * (32 / NS) + lane / NS;       // this thread's column within the block
    const int c = blockIdx.z * SCAN_COLS + wcol;
    const bool live = c < cols;
    const int d0 = slice * DS;
    const int row0 = p.seq_row0[s], n = p.seq_new[s];
    if (p.below > 0 && n >= p.below) return;
    const bool fresh = p.seq_start[s] == 0;
    const size_t cell = ((size_t)p.seq_slot[s] * heads + hd) * cols + (live ? c : 0);
    float* st = p.state + cell * D;
    const bool vec = (D & 3) == 0;
    float S[DS];
#pragma unroll
    for (int i = 0; i < DS; i += 4) {
        if (live && !fresh && vec && d0 + i < D) {
            const float4 t = *reinterpret_cast<const float4*>(st + d0 + i);
            S[i] = t.x; S[i + 1] = t.y; S[i + 2] = t.z; S[i + 3] = t.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) S[i + j] = (live && !fresh && d0 + i + j < D) ? st[d0 + i + j] : 0.f;
        }
    }
    float m = 0.f;
    if (MODE == 1 && live && !fresh) m = p.state_m[cell];
    const float keep = MODE >= 2 ? p.vec_a[hd] : 0.f;          // retention: the head's decay; state space: its D
    const int g = (MODE == 0 || MODE == 3) ? hd / (heads / p.qk_heads) : hd;
    const int qc = MODE == 0 ? g * D : p.q_col + g * D;
    const int kc = MODE == 0 ? (p.qk_heads + g) * D : p.k_col + g * D;
    const int vc = MODE == 0 ? 2 * p.qk_heads * D + hd * Dv : p.v_col + hd * Dv;
    const float a_rate = (MODE == 0 && !p.decay_ready) ? expf(p.vec_a[hd]) : 0.f;
    const bool head_decay = MODE == 0 && p.decay_dim == 1;      // one decay per head: a number per token (s2), not a row of sg
    // staging: thread -> (token, key channel) of each array, one value of v, and the scalars
    // Nothing uses a fetched value before `stage`: a use right behind its load would hold the warp until the
    // load is back, once per round, instead of behind the tokens in between.
    float rq[PER], rk[PER], rg[MODE == 0 ? PER : 1], rv = 0.f, r1 = 0.f, r2 = 0.f;
    float bias[MODE == 0 ? PER : 1];                   // dt_bias of the channels this thread stages (the same every round)
    if (MODE == 0 && !p.decay_ready) {
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const int d = (threadIdx.x + 128 * e) % DPAD;
            bias[e] = p.vec_b[head_decay ? hd : hd * D + (d < D ? d : 0)];
        }
    }
    auto fetch = [&](int t0) {
        const int nt = min(SCAN_TOKENS, n - t0);
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const int idx = threadIdx.x + 128 * e, t = idx / DPAD, d = idx % DPAD;
            const bool ok = t < nt && d < D;
            const size_t r = (size_t)(row0 + t0 + (ok ? t : 0));
            const int dd = ok ? d : 0;
            rq[e] = p.in_a[r * p.lda + qc + dd];
            rk[e] = p.in_a[r * p.lda + kc + dd];
            if (MODE == 0 && !head_decay) rg[e] = p.in_c[r * p.ldc + hd * D + dd];
        }
        if (threadIdx.x < SCAN_TOKENS * SCAN_COLS) {
            const int t = threadIdx.x / SCAN_COLS, cc = blockIdx.z * SCAN_COLS + threadIdx.x % SCAN_COLS;
            const bool ok = t < nt && cc < Dv;
            rv = p.in_a[(size_t)(row0 + t0 + (ok ? t : 0)) * p.lda + vc + (ok ? cc : 0)];
        }
        if (threadIdx.x < SCAN_TOKENS) {
            const size_t r = (size_t)(row0 + t0 + (threadIdx.x < nt ? threadIdx.x : 0));
            if (MODE == 0) {
                r1 = p.in_b[r * p.ldb + p.b_col + hd];
                if (head_decay) r2 = p.in_c[r * p.ldc + hd];
            } else if (MODE == 1) { r1 = p.in_a[r * p.lda + p.i_col + hd]; r2 = p.in_a[r * p.lda + p.f_col + hd]; }
            else if (MODE == 3) { r1 = p.in_b[r * p.ldb + hd]; r2 = p.in_b[r * p.ldb + heads + hd]; }
        }
        // The loads stay here, ahead of the tokens that are worked on meanwhile: without this the compiler moves
        // them down to their first use, where the warp would wait for them. (No instruction is emitted.)
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            asm volatile("" : "+f"(rq[e]), "+f"(rk[e]));
            if (MODE == 0) asm volatile("" : "+f"(rg[e]));
        }
        asm volatile("" : "+f"(rv), "+f"(r1), "+f"(r2));
    };
    auto stage = [&]() {
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const int idx = threadIdx.x + 128 * e, t = idx / DPAD, d = idx % DPAD;
            const int at = (d / DS) * SL + d % DS;
            const bool in = d < D;                     // channels beyond D stay out of every sum
            sq[t][at] = in ? (MODE == 1 ? rq[e] * p.q_scale : rq[e]) : 0.f;
            sk[t][at] = in ? rk[e] : 0.f;
            if (MODE == 0 && !head_decay) sg[t][at] = p.decay_ready ? rg[e] : expf(-a_rate * softplus_f(rg[e] + bias[e]));
        }
        if (threadIdx.x < SCAN_TOKENS * SCAN_COLS) {
            const int cc = blockIdx.z * SCAN_COLS + threadIdx.x % SCAN_COLS;
            sv[threadIdx.x / SCAN_COLS][threadIdx.x % SCAN_COLS] = cc < Dv ? rv : ((MODE == 1 && cc == Dv) ? 1.0f : 0.f);   // the column of n has v = 1
        }
        if (threadIdx.x < SCAN_TOKENS) {
            if (MODE == 0) {
                s1[threadIdx.x] = sigmoid_f(r1);
                if (head_decay) s2[threadIdx.x] = p.decay_ready ? r2 : expf(-a_rate * softplus_f(r2 + p.vec_b[hd]));
            } else if (MODE == 1) {
                s1[threadIdx.x] = p.cap * tanhf((r1 + p.vec_a[hd]) / p.cap);
                s2[threadIdx.x] = logsigmoid_f(p.cap * tanhf((r2 + p.vec_b[hd]) / p.cap));
            } else if (MODE == 3) { s1[threadIdx.x] = r1; s2[threadIdx.x] = r2; }
        }
    };
    fetch(0);
    for (int t0 = 0; t0 < n; t0 += SCAN_TOKENS) {
        const int nt = min(SCAN_TOKENS, n - t0);
        __syncthreads();                               // the tokens before are done with the staged values
        stage();
        __syncthreads();
        if (MODE == 0) {
            // k . q of every staged token, the same for all columns: warp w takes tokens 2w and 2w + 1
#pragma unroll
            for (int tt = 0; tt < SCAN_TOKENS / 4; ++tt) {
                const int t = warp * (SCAN_TOKENS / 4) + tt;
                float a = 0.f;
                for (int d = lane; d < DPAD; d += 32) {
                    const int at = (d / DS) * SL + d % DS;
                    a = fmaf(sk[t][at], sq[t][at], a);
                }
                a = warp_sum(a);
                if (lane == 0) skq[t] = a;
            }
            __syncthreads();
        }
        if (t0 + SCAN_TOKENS < n) fetch(t0 + SCAN_TOKENS);
        // Gated delta rule, one token. With S' = diag(g) S both products S'^T k and S'^T q are taken at once (two
        // butterflies side by side), and since the state after the write is S' + k u^T, the read-out is
        // S'^T q + u (k . q): the only thing the next token waits for is the write itself.
        auto delta_token = [&](int t) {
            const float* kq = &sk[t][slice * SL];
            const float* qq = &sq[t][slice * SL];
            const float* gg = &sg[t][slice * SL];
            const float vcol = sv[t][wcol];
            float kr[DS];
            float d4[4] = {0.f, 0.f, 0.f, 0.f}, o4[4] = {0.f, 0.f, 0.f, 0.f};       // four chains each, always in this order
            if (head_decay) {
                const float gh = s2[t];
#pragma unroll
                for (int i = 0; i < DS; ++i) S[i] *= gh;
            } else {
#pragma unroll
                for (int i = 0; i < DS; i += 4) {
                    const float4 gv = *reinterpret_cast<const float4*>(gg + i);
                    S[i] *= gv.x; S[i + 1] *= gv.y; S[i + 2] *= gv.z; S[i + 3] *= gv.w;
                }
            }
#pragma unroll
            for (int i = 0; i < DS; i += 4) {
                const float4 kv = *reinterpret_cast<const float4*>(kq + i);
                const float4 qv = *reinterpret_cast<const float4*>(qq + i);
                kr[i] = kv.x; kr[i + 1] = kv.y; kr[i + 2] = kv.z; kr[i + 3] = kv.w;
                d4[0] = fmaf(S[i], kv.x, d4[0]); d4[1] = fmaf(S[i + 1], kv.y, d4[1]);
                d4[2] = fmaf(S[i + 2], kv.z, d4[2]); d4[3] = fmaf(S[i + 3], kv.w, d4[3]);
                o4[0] = fmaf(S[i], qv.x, o4[0]); o4[1] = fmaf(S[i + 1], qv.y, o4[1]);
                o4[2] = fmaf(S[i + 2], qv.z, o4[2]); o4[3] = fmaf(S[i + 3], qv.w, o4[3]);
            }
            float dk = (d4[0] + d4[1]) + (d4[2] + d4[3]), dq = (o4[0] + o4[1]) + (o4[2] + o4[3]);
#pragma unroll
            for (int sh = 1; sh < NS; sh <<= 1) {
                const float a = __shfl_xor_sync(0xffffffffu, dk, sh), b = __shfl_xor_sync(0xffffffffu, dq, sh);
                dk += a;
                dq += b;
            }
            const float u = s1[t] * (vcol - dk);
#pragma unroll
            for (int i = 0; i < DS; ++i) S[i] = fmaf(kr[i], u, S[i]);
            if (live && slice == 0) p.out[(size_t)(row0 + t0 + t) * heads * Dv + hd * Dv + c] = fmaf(u, skq[t], dq);
        };
        if constexpr (MODE == 0) {
            if (nt == SCAN_TOKENS) {        // a whole round unrolled: the next tokens' loads and this one's read-out overlap
#pragma unroll
                for (int t = 0; t < SCAN_TOKENS; ++t) delta_token(t);
            } else {
                for (int t = 0; t < nt; ++t) delta_token(t);
            }
        } else if constexpr (MODE == 2 || MODE == 3) {
            // Retention, one token: S = d S + k v, then the read-out from the new state; four chains, always in this order.
            // The state-space recurrence is the same with a decay and a step of the token's own, and D v beside the read-out.
            auto retention_token = [&](int t) {
                const float* kq = &sk[t][slice * SL];
                const float* qq = &sq[t][slice * SL];
                const float raw = sv[t][wcol];
                const float vcol = MODE == 3 ? raw * s1[t] : raw, fade = MODE == 3 ? s2[t] : keep;
                float o4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int i = 0; i < DS; i += 4) {
                    const float4 kv = *reinterpret_cast<const float4*>(kq + i), qv = *reinterpret_cast<const float4*>(qq + i);
                    S[i] = fmaf(fade, S[i], vcol * kv.x); S[i + 1] = fmaf(fade, S[i + 1], vcol * kv.y);
                    S[i + 2] = fmaf(fade, S[i + 2], vcol * kv.z); S[i + 3] = fmaf(fade, S[i + 3], vcol * kv.w);
                    o4[0] = fmaf(S[i], qv.x, o4[0]); o4[1] = fmaf(S[i + 1], qv.y, o4[1]);
                    o4[2] = fmaf(S[i + 2], qv.z, o4[2]); o4[3] = fmaf(S[i + 3], qv.w, o4[3]);
                }
                float o = slices_sum<NS>((o4[0] + o4[1]) + (o4[2] + o4[3]));
                if (MODE == 3) o = fmaf(keep, raw, o);
                if (live && slice == 0) p.out[(size_t)(row0 + t0 + t) * heads * Dv + hd * Dv + c] = o;
            };
            if (nt == SCAN_TOKENS) {
#pragma unroll
                for (int t = 0; t < SCAN_TOKENS; ++t) retention_token(t);
            } else {
                for (int t = 0; t < nt; ++t) retention_token(t);
            }
        } else {
            for (int t = 0; t < nt; ++t) {
                const float* kq = &sk[t][slice * SL];
                const float* qq = &sq[t][slice * SL];
                const float vcol = sv[t][wcol];
                float o = 0.f;
                const float fm = s2[t] + m;
                const float m_new = fmaxf(fm, s1[t]);
                const float a = expf(fm - m_new);
                const float bv = expf(s1[t] - m_new) * vcol;
                m = m_new;
                float o4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int i = 0; i < DS; i += 4) {
                    const float4 kv = *reinterpret_cast<const float4*>(kq + i), qv = *reinterpret_cast<const float4*>(qq + i);
                    S[i] = fmaf(a, S[i], bv * kv.x); S[i + 1] = fmaf(a, S[i + 1], bv * kv.y);
                    S[i + 2] = fmaf(a, S[i + 2], bv * kv.z); S[i + 3] = fmaf(a, S[i + 3], bv * kv.w);
                    o4[0] = fmaf(S[i], qv.x, o4[0]); o4[1] = fmaf(S[i + 1], qv.y, o4[1]);
                    o4[2] = fmaf(S[i + 2], qv.z, o4[2]); o4[3] = fmaf(S[i + 3], qv.w, o4[3]);
                }
                o = slices_sum<NS>((o4[0] + o4[1]) + (o4[2] + o4[3]));
                if (live && slice == 0) {
                    float* orow = p.out + ((size_t)(row0 + t0 + t) * heads + hd) * (Dv + 2);
                    orow[c] = o;
                    if (c == Dv) orow[Dv + 1] = m;
                }
            }
        }
    }
    if (live) {
#pragma unroll
        for (int i = 0; i < DS; i += 4) {
            if (vec && d0 + i < D) {
                *reinterpret_cast<float4*>(st + d0 + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (d0 + i + j < D) st[d0 + i + j] = S[i + j];
            }
        }
        if (MODE == 1 && slice == 0) p.state_m[cell] = m;
    }
}

// Eight slices per column: with 16 or 32 (more and lighter warps for a lone prompt) the staging of q and k, which every
// block repeats, weighs as much as the shorter sums save, and a prompt ran no faster.
#define SCAN_SLICES 8

template <int MODE>
static int launch_scan(const ScanParams& p, int n_seqs, cudaStream_t s) {
    if (n_seqs <= 0) return 0;
    if (p.D < 1 || p.D > 256 || p.Dv < 1) return CML_ERR_BAD_SIZE;
    const int cols = MODE == 1 ? p.Dv + 1 : p.Dv;
    constexpr int block_cols = 128 / SCAN_SLICES;
    dim3 grid(n_seqs, p.heads, (cols + block_cols - 1) / block_cols);
#define SCAN_CASE(DS_)                                                                    \
    if (p.D <= SCAN_SLICES * DS_) {                                                       \
        launch_pdl(scan_kernel<DS_, MODE, SCAN_SLICES>, grid, dim3(128), 0, s, p);        \
        return cml_launch_status();                                                       \
    }
    SCAN_CASE(4) SCAN_CASE(8) SCAN_CASE(16) SCAN_CASE(32)
#undef SCAN_CASE
    return CML_ERR_BAD_SIZE;
}

extern "C" int cml_delta_scan(const float* qkv, long ldq, const float* beta_in, long ldb, int beta_col, const float* decay_in,
                              long ldd, const float* a_log, const float* dt_bias, float* state, const int* seq_row0,
                              const int* seq_new, const int* seq_start, const int* seq_slot, float* out, int n_seqs, int heads,
                              int qk_heads, int D, int Dv, int decay_ready, int decay_dim, int below, void* stream) {
    if (qk_heads < 1 || heads % qk_heads || (decay_dim != 1 && decay_dim != D)) return CML_ERR_BAD_SIZE;
    ScanParams p = {};
    p.in_a = qkv; p.lda = ldq; p.in_b = beta_in; p.ldb = ldb; p.b_col = beta_col; p.in_c = decay_in; p.ldc = ldd;
    p.vec_a = a_log; p.vec_b = dt_bias; p.state = state; p.state_m = nullptr;
    p.seq_row0 = seq_row0; p.seq_new = seq_new; p.seq_start = seq_start; p.seq_slot = seq_slot; p.out = out;
    p.heads = heads; p.qk_heads = qk_heads; p.D = D; p.Dv = Dv; p.decay_ready = decay_ready; p.decay_dim = decay_dim; p.below = below;
    return launch_scan<0>(p, n_seqs, (cudaStream_t)stream);
}

extern "C" int cml_memory_scan(const float* proj, long ld, int q_col, int k_col, int v_col, int i_col, int f_col,
                               const float* i_bias, const float* f_bias, float cap, float q_scale, float* state,
                               float* state_m, const int* seq_row0, const int* seq_new, const int* seq_start,
                               const int* seq_slot, float* out, int n_seqs, int heads, int D, int Dv, int below, void* stream) {
    ScanParams p = {};
    p.below = below;
    p.in_a = proj; p.lda = ld; p.vec_a = i_bias; p.vec_b = f_bias; p.state = state; p.state_m = state_m;
    p.seq_row0 = seq_row0; p.seq_new = seq_new; p.seq_start = seq_start; p.seq_slot = seq_slot; p.out = out;
    p.heads = heads; p.qk_heads = heads; p.D = D; p.Dv = Dv;
    p.q_col = q_col; p.k_col = k_col; p.v_col = v_col; p.i_col = i_col; p.f_col = f_col; p.cap = cap; p.q_scale = q_scale;
    return launch_scan<1>(p, n_seqs, (cudaStream_t)stream);
}

extern "C" int cml_retention_scan(const float* proj, long ld, int q_col, int k_col, int v_col, const float* decay, float* state,
                                  const int* seq_row0, const int* seq_new, const int* seq_start, const int* seq_slot,
                                  float* out, int n_seqs, int heads, int D, int Dv, int below, void* stream) {
    ScanParams p = {};
    p.below = below;
    p.in_a = proj; p.lda = ld; p.vec_a = decay; p.state = state; p.state_m = nullptr;
    p.seq_row0 = seq_row0; p.seq_new = seq_new; p.seq_start = seq_start; p.seq_slot = seq_slot; p.out = out;
    p.heads = heads; p.qk_heads = heads; p.D = D; p.Dv = Dv;
    p.q_col = q_col; p.k_col = k_col; p.v_col = v_col; p.q_scale = 1.0f;
    return launch_scan<2>(p, n_seqs, (cudaStream_t)stream);
}

extern "C" int cml_ssm_scan(const float* rows_in, long ld, int x_col, int b_col, int c_col, const float* gates, long ldg,
                            const float* d_skip, float* state, const int* seq_row0, const int* seq_new, const int* seq_start,
                            const int* seq_slot, float* out, int n_seqs, int heads, int groups, int D, int Dv, int below, void* stream) {
    if (groups < 1 || heads % groups) return CML_ERR_BAD_SIZE;
    ScanParams p = {};
    p.below = below;
    p.in_a = rows_in; p.lda = ld; p.in_b = gates; p.ldb = ldg; p.vec_a = d_skip; p.state = state; p.state_m = nullptr;
    p.seq_row0 = seq_row0; p.seq_new = seq_new; p.seq_start = seq_start; p.seq_slot = seq_slot; p.out = out;
    p.heads = heads; p.qk_heads = groups; p.D = D; p.Dv = Dv;
    p.q_col = c_col; p.k_col = b_col; p.v_col = x_col; p.q_scale = 1.0f;
    return launch_scan<3>(p, n_seqs, (cudaStream_t)stream);
}

// ------------------------------------------------------------------------------------
// What the state-space recurrence reads. proj [rows, ld] (n_splits matrices split_stride apart, added in split order):
// z (inner), then the convolved channels (x, B, C), then one step-size input per head. Every channel passes a causal
// convolution (conv_w [taps, channels], the last tap the current token's; `state` [slots, max(taps - 1, 1), channels] holds
// the inputs of the tokens before the step) with bias, then SiLU: out [rows, channels]. The steps: dt = softplus(in +
// dt_bias), gates [rows, 2 heads] = dt, then exp(-exp(a_log) dt). z_out (may be null) gets z [rows, inner]. With
// update_state (every sequence of the step brings one row) the state moves on by that row here. A thread takes VEC
// neighbouring columns of up to `rows_per` rows.
struct SsmInputs {
    const float* proj; long ld; int n_splits; long split_stride;
    const float* conv_w; const float* conv_b; const float* dt_bias; const float* a_log;
    float* state; int update_state;
    const int* row_seq; const int* row_pos; const int* seq_row0; const int* seq_slot;
    float* out; float* gates; float* z_out;
    int rows, rows_per, inner, channels, heads, taps;
};

template <int VEC> struct SsmPiece { float v[VEC]; };
template <int VEC> __device__ __forceinline__ SsmPiece<VEC> ssm_load(const float* p) {
    SsmPiece<VEC> r;
    if constexpr (VEC == 4) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w;
    } else {
        r.v[0] = p[0];
    }
    return r;
}
template <int VEC> __device__ __forceinline__ void ssm_store(float* p, const SsmPiece<VEC>& r) {
    if constexpr (VEC == 4) *reinterpret_cast<float4*>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
    else p[0] = r.v[0];
}
template <int VEC> __device__ __forceinline__ SsmPiece<VEC> ssm_sum(const float* p, int n, long stride) {
    SsmPiece<VEC> r = ssm_load<VEC>(p);
    for (int s0 = 1; s0 < n; s0 += 8) {                        // eight splits' loads in flight, added in split order
        SsmPiece<VEC> t[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) t[k] = ssm_load<VEC>(p + (size_t)min(s0 + k, n - 1) * stride);
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (s0 + k < n)
#pragma unroll
                for (int e = 0; e < VEC; ++e) r.v[e] += t[k].v[e];
    }
    return r;
}

template <int VEC>
__global__ void __launch_bounds__(128) ssm_inputs_kernel(const SsmInputs p) {
    pdl_wait();
    pdl_launch_dependents();
    const int nz = p.z_out ? p.inner / VEC : 0, nc = p.channels / VEC;
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    const int r0 = blockIdx.y * p.rows_per, r1 = min(p.rows, r0 + p.rows_per);
    if (u >= nc + nz) {                                        // a head's steps and decays
        const int h = u - nc - nz;
        if (h >= p.heads) return;
        const float bias = p.dt_bias[h], rate = expf(p.a_log[h]);
        for (int r = r0; r < r1; ++r) {
            const float dt = softplus_f(split_sum(p.proj + (size_t)r * p.ld + p.inner + p.channels + h, p.n_splits, p.split_stride) + bias);
            p.gates[(size_t)r * 2 * p.heads + h] = dt;
            p.gates[(size_t)r * 2 * p.heads + p.heads + h] = expf(-rate * dt);
        }
        return;
    }
    if (u >= nc) {                                             // z
        const int c = (u - nc) * VEC;
        for (int r = r0; r < r1; ++r)
            ssm_store<VEC>(p.z_out + (size_t)r * p.inner + c, ssm_sum<VEC>(p.proj + (size_t)r * p.ld + c, p.n_splits, p.split_stride));
        return;
    }
    const int c = u * VEC, taps = p.taps, keep = max(taps - 1, 1);
    const float* col = p.proj + p.inner + c;
    const SsmPiece<VEC> bias = ssm_load<VEC>(p.conv_b + c);
    SsmPiece<VEC> w[4];                                        // the taps of the token and of the three before it
#pragma unroll
    for (int back = 0; back < 4; ++back) w[back] = ssm_load<VEC>(p.conv_w + (size_t)max(taps - 1 - back, 0) * p.channels + c);
    for (int r = r0; r < r1; ++r) {
        const int s = p.row_seq[r], pos = p.row_pos[r], inside = r - p.seq_row0[s];
        float* st = p.state + (size_t)p.seq_slot[s] * keep * p.channels + c;
        auto input = [&](int back) -> SsmPiece<VEC> {
            return back <= inside ? ssm_sum<VEC>(col + (size_t)(r - back) * p.ld, p.n_splits, p.split_stride)
                                  : ssm_load<VEC>(st + (size_t)(taps - 1 + inside - back) * p.channels);
        };
        SsmPiece<VEC> acc = bias, own = input(0), before[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const bool there = k + 1 < taps && k + 1 <= pos;   // (a token before the sequence's start counts as zero)
            before[k] = there ? input(k + 1) : own;
            if (!there)
#pragma unroll
                for (int e = 0; e < VEC; ++e) before[k].v[e] = 0.f;
        }
#pragma unroll
        for (int e = 0; e < VEC; ++e)
            acc.v[e] = fmaf(w[3].v[e], before[2].v[e], fmaf(w[2].v[e], before[1].v[e], fmaf(w[1].v[e], before[0].v[e], fmaf(w[0].v[e], own.v[e], acc.v[e]))));
        for (int back = 4; back < taps && back <= pos; ++back) {
            const SsmPiece<VEC> x = input(back), wb = ssm_load<VEC>(p.conv_w + (size_t)(taps - 1 - back) * p.channels + c);
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc.v[e] = fmaf(wb.v[e], x.v[e], acc.v[e]);
        }
        if (p.update_state && taps > 1) {
            for (int j = 0; j + 2 < taps; ++j) {
                SsmPiece<VEC> t = ssm_load<VEC>(st + (size_t)(j + 1) * p.channels);
                if (pos + j + 2 < taps)
#pragma unroll
                    for (int e = 0; e < VEC; ++e) t.v[e] = 0.f;
                ssm_store<VEC>(st + (size_t)j * p.channels, t);
            }
            ssm_store<VEC>(st + (size_t)(taps - 2) * p.channels, own);
        }
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc.v[e] = silu_f(acc.v[e]);
        ssm_store<VEC>(p.out + (size_t)r * p.channels + c, acc);
    }
}

// The same for prompts (complete rows, up to four taps): a thread asks for the inputs of SSI_ROWS neighbouring rows and of the three
// before them at once and keeps them in registers; what a row lacks within the step comes from the state.
#define SSI_ROWS 8
template <int VEC>
__global__ void __launch_bounds__(128) ssm_inputs_rows_kernel(const SsmInputs p) {
    pdl_wait();
    pdl_launch_dependents();
    const int nc = p.channels / VEC, u = blockIdx.x * blockDim.x + threadIdx.x;
    const int r0 = blockIdx.y * SSI_ROWS, r1 = min(p.rows, r0 + SSI_ROWS);
    if (u >= nc) {                                             // a head's steps and decays
        const int h = u - nc;
        if (h >= p.heads) return;
        const float bias = p.dt_bias[h], rate = expf(p.a_log[h]);
        float x[SSI_ROWS];
#pragma unroll
        for (int i = 0; i < SSI_ROWS; ++i) x[i] = p.proj[(size_t)min(r0 + i, p.rows - 1) * p.ld + p.inner + p.channels + h];
        for (int i = 0; i < r1 - r0; ++i) {
            float* o = p.gates + (size_t)(r0 + i) * 2 * p.heads + h;
            const float dt = softplus_f(x[i] + bias);
            o[0] = dt;
            o[p.heads] = expf(-rate * dt);
        }
        return;
    }
    const int c = u * VEC, taps = p.taps;
    const float* col = p.proj + p.inner + c;
    SsmPiece<VEC> x[SSI_ROWS + 3], w[4];
#pragma unroll
    for (int i = 0; i < SSI_ROWS + 3; ++i) x[i] = ssm_load<VEC>(col + (size_t)min(max(r0 + i - 3, 0), p.rows - 1) * p.ld);
    const SsmPiece<VEC> bias = ssm_load<VEC>(p.conv_b + c);
#pragma unroll
    for (int back = 0; back < 4; ++back) w[back] = ssm_load<VEC>(p.conv_w + (size_t)max(taps - 1 - back, 0) * p.channels + c);
#pragma unroll
    for (int i = 0; i < SSI_ROWS; ++i) {
        const int r = r0 + i;
        if (r >= r1) break;
        const int s = p.row_seq[r], pos = p.row_pos[r], inside = r - p.seq_row0[s];
        SsmPiece<VEC> acc = bias;
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc.v[e] = fmaf(w[0].v[e], x[i + 3].v[e], acc.v[e]);
#pragma unroll
        for (int back = 1; back < 4; ++back) {
            if (back >= taps || back > pos) break;             // (a token before the sequence's start counts as zero)
            SsmPiece<VEC> b = x[i + 3 - back];
            if (back > inside) b = ssm_load<VEC>(p.state + ((size_t)p.seq_slot[s] * (taps - 1) + taps - 1 + inside - back) * p.channels + c);
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc.v[e] = fmaf(w[back].v[e], b.v[e], acc.v[e]);
        }
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc.v[e] = silu_f(acc.v[e]);
        ssm_store<VEC>(p.out + (size_t)r * p.channels + c, acc);
    }
}

extern "C" int cml_ssm_inputs(const float* proj, long ld, int n_splits, long split_stride, const float* conv_w, const float* conv_b,
                              const float* dt_bias, const float* a_log, float* state, int update_state, const int* row_seq,
                              const int* row_pos, const int* seq_row0, const int* seq_slot, float* out, float* gates, float* z_out,
                              int rows, int inner, int channels, int heads, int taps, void* stream) {
    if (rows <= 0) return 0;
    if (n_splits < 1 || inner < 1 || channels < 1 || heads < 1 || taps < 1) return CML_ERR_BAD_SIZE;
    SsmInputs p = {proj, ld, n_splits, split_stride, conv_w, conv_b, dt_bias, a_log, state, update_state, row_seq, row_pos, seq_row0,
                   seq_slot, out, gates, z_out, rows, 1, inner, channels, heads, taps};
    const bool vec = (((long)inner | (long)channels | ld | split_stride) & 3) == 0 &&
                     ((((uintptr_t)proj) | ((uintptr_t)conv_w) | ((uintptr_t)conv_b) | ((uintptr_t)state) | ((uintptr_t)out) | ((uintptr_t)z_out)) & 15) == 0;
    const int per = vec ? 4 : 1;
    const long units = (long)channels / per + (z_out ? inner / per : 0) + heads;
    if (!update_state && !z_out && n_splits == 1 && taps <= 4 && rows > 64 && rows <= 65535 * SSI_ROWS) {
        const dim3 grid((unsigned)((units + 127) / 128), (unsigned)((rows + SSI_ROWS - 1) / SSI_ROWS));
        if (vec) launch_pdl(ssm_inputs_rows_kernel<4>, grid, dim3(128), 0, (cudaStream_t)stream, p);
        else launch_pdl(ssm_inputs_rows_kernel<1>, grid, dim3(128), 0, (cudaStream_t)stream, p);
        return cml_launch_status();
    }
    if (((long)rows + p.rows_per - 1) / p.rows_per > 65535) p.rows_per = (int)((rows + 65534L) / 65535);
    const dim3 grid((unsigned)((units + 127) / 128), (unsigned)((rows + p.rows_per - 1) / p.rows_per));
    if (vec) launch_pdl(ssm_inputs_kernel<4>, grid, dim3(128), 0, (cudaStream_t)stream, p);
    else launch_pdl(ssm_inputs_kernel<1>, grid, dim3(128), 0, (cudaStream_t)stream, p);
    return cml_launch_status();
}

// After the state-space scan: v = y * silu(z), a row's `groups` equal parts each divided by its own root mean square
// (eps inside), times w, in the compute type. y [rows, width] float; z [rows, ldz] float; w [width] float; out rows ldo
// apart. A block owns one (row, part), whose values stay in shared memory between the two passes.
template <typename TO>
__global__ void __launch_bounds__(256) gated_group_norm_kernel(const float* __restrict__ y, const float* __restrict__ z, long ldz,
                                                               const float* __restrict__ w, TO* __restrict__ out, long ldo, int width,
                                                               int part, float eps) {
    extern __shared__ __align__(16) float gg_row[];
    __shared__ float red[32];
    pdl_wait();
    pdl_launch_dependents();
    const int r = blockIdx.x, c0 = blockIdx.y * part;
    const float* yr = y + (size_t)r * width + c0;
    const float* zr = z + (size_t)r * ldz + c0;
    float ss = 0.f;
    const bool vec = (((long)part | (long)width | ldz) & 3) == 0 && ((((uintptr_t)y) | ((uintptr_t)z)) & 15) == 0;
    if (vec) {
        for (int c = threadIdx.x * 4; c < part; c += blockDim.x * 4) {
            const float4 a = *reinterpret_cast<const float4*>(yr + c), g = *reinterpret_cast<const float4*>(zr + c);
            const float4 v = make_float4(a.x * silu_f(g.x), a.y * silu_f(g.y), a.z * silu_f(g.z), a.w * silu_f(g.w));
            *reinterpret_cast<float4*>(gg_row + c) = v;
            ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
        }
    } else {
        for (int c = threadIdx.x; c < part; c += blockDim.x) {
            const float v = yr[c] * silu_f(zr[c]);
            gg_row[c] = v;
            ss = fmaf(v, v, ss);
        }
    }
    const float scale = 1.0f / sqrtf(block_sum(ss, red) / (float)part + eps);
    TO* o = out + (size_t)r * ldo + c0;
    if (vec) {                                                 // each thread reads back what it wrote itself
        for (int c = threadIdx.x * 4; c < part; c += blockDim.x * 4)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[c + e] = from_f32<TO>(gg_row[c + e] * scale * w[c0 + c + e]);
    } else {
        for (int c = threadIdx.x; c < part; c += blockDim.x) o[c] = from_f32<TO>(gg_row[c] * scale * w[c0 + c]);
    }
}

extern "C" int cml_gated_group_norm(const float* y, const float* z, long ldz, const float* w, void* out, long ldo, int out_dtype, int rows,
                                    int width, int groups, float eps, void* stream) {
    if (rows <= 0) return 0;
    if (groups < 1 || groups > 65535 || width % groups) return CML_ERR_BAD_SIZE;
    const int part = width / groups;
    const size_t smem = (size_t)part * sizeof(float);
    if (smem > 200 * 1024) return CML_ERR_BAD_SIZE;
    const int block = part >= 1024 ? 256 : part >= 256 ? 128 : part >= 64 ? 64 : 32;
#define GG_CASE(T_, D_)                                                                                                   \
    if (out_dtype == D_) {                                                                                                \
        if (smem > 48 * 1024 && cml_allow_smem<gated_group_norm_kernel<T_>>(smem) != cudaSuccess) return CML_ERR_BAD_SIZE; \
        launch_pdl(gated_group_norm_kernel<T_>, dim3(rows, groups), dim3(block), smem, (cudaStream_t)stream, y, z, ldz, w, \
                   (T_*)out, ldo, width, part, eps);                                                                      \
        return cml_launch_status();                                                                                       \
    }
    GG_CASE(float, CML_DTYPE_F32)
    GG_CASE(bf16, CML_DTYPE_BF16)
#undef GG_CASE
    return CML_ERR_BAD_DTYPE;
}

// ------------------------------------------------------------------------------------
// Generalized delta rule. Both terms of the write read the old state, so with p = k^T S (S before the token), q = (r * w)^T S,
// n2 = 1 / (sum k^2 + 1e-6) the token is
//
//   S' = diag(w) S + k (v - a * (n2 p))^T,     o = q - n2 (sum r a k) p + (sum r k) v
//
// and the two products over the state, p and q, are taken side by side. What does not depend on the state is made
// beforehand, once per (row, head), by the kernel below: `packed` [rows, heads, 4 D + Dv] = k, r * w, w, a, v and `scal`
// [rows, heads, 4] = n2, n2 sum r a k, sum r k, 0.
//
// proj (n_splits matrices split_stride apart, added in split order) [rows, ld]: columns r, k (heads x D each), v
// (heads x Dv), the removal rates' inputs (heads x D), the gate's (heads x Dv), then `rank` columns of the decays' narrow
// inputs. a = sigmoid(in + a_bias). The decays' inputs z come as a product of their own (`high`, n_high matrices
// high_stride apart [rows, heads x D]) or, where `high` is null, are made here: z = W2 tanh(narrow), W2 [heads x D, rank].
// w = exp(-rate * sigmoid(z + w0)). gate_out (may be null) gets the gate's summed inputs [rows, heads x Dv].
struct DeltaInputs {
    const float* proj; long ld; int n_splits; long split_stride;
    const float* high; int n_high; long high_stride;
    const void* w2; int rank;
    const float* a_bias; const float* w0;
    float rate;
    float* packed; float* scal; float* gate_out;
    int heads, D, Dv;
    int early;                          // w2 stood in place before the kernel ahead of this one began
};

template <typename T>
__global__ void __launch_bounds__(256) delta_inputs_kernel(const DeltaInputs p) {
    extern __shared__ __align__(16) float di_low[];            // tanh of the narrow inputs
    __shared__ float red0[32], red1[32], red2[32];
    if (!p.early) pdl_wait();
    const int r = blockIdx.x, hd = blockIdx.y, D = p.D, Dv = p.Dv, HD = p.heads * p.D, HV = p.heads * p.Dv;
    const float* row = p.proj + (size_t)r * p.ld;
    // Ahead of the wait: the first 128 bytes of this thread's row of W2, which for narrow inputs of up to 128 / sizeof(T) are all
    // (asked for behind the narrow inputs, piece by piece, they were most of the kernel's 7.6 us in a step's chain; now 4.0).
    constexpr int PIECE = 16 / (int)sizeof(T), PRE = 8;
    const bool pieces = p.high == nullptr && p.rank >= PIECE && p.rank % PIECE == 0 && (((uintptr_t)p.w2) & 15) == 0;
    uint4 pre[PRE];
    if (pieces && (int)threadIdx.x < D) {
        const T* w = (const T*)p.w2 + (size_t)(hd * D + threadIdx.x) * p.rank;
#pragma unroll
        for (int j = 0; j < PRE; ++j) pre[j] = *reinterpret_cast<const uint4*>(w + min(j * PIECE, p.rank - PIECE));
    }
    pdl_wait();
    pdl_launch_dependents();
    if (p.high == nullptr) {
        const float* narrow = row + 3 * HD + 2 * HV;
        for (int j = threadIdx.x; j < p.rank; j += blockDim.x) di_low[j] = tanhf(split_sum(narrow + j, p.n_splits, p.split_stride));
        __syncthreads();
    }
    float* pk = p.packed + ((size_t)r * p.heads + hd) * (4 * D + Dv);
    float k2 = 0.f, rak = 0.f, rk = 0.f;
    for (int d = threadIdx.x; d < D; d += blockDim.x) {
        const int c = hd * D + d;
        const float rr = split_sum(row + c, p.n_splits, p.split_stride);
        const float kk = split_sum(row + HD + c, p.n_splits, p.split_stride);
        const float aa = sigmoid_f(split_sum(row + 2 * HD + HV + c, p.n_splits, p.split_stride) + p.a_bias[c]);
        float z = 0.f;
        if (p.high != nullptr) {
            z = split_sum(p.high + (size_t)r * HD + c, p.n_high, p.high_stride);
        } else {
            const T* w = (const T*)p.w2 + (size_t)c * p.rank;
            int j = 0;
            if (pieces) {
                if (d == (int)threadIdx.x) {
#pragma unroll
                    for (int q = 0; q < PRE; ++q) {
                        if (j >= p.rank) break;
                        union { uint4 raw; T e[PIECE]; } v;
                        v.raw = pre[q];
#pragma unroll
                        for (int e = 0; e < PIECE; ++e) z = fmaf(to_f32(v.e[e]), di_low[j + e], z);
                        j += PIECE;
                    }
                }
                for (; j < p.rank; j += PIECE) {
                    union { uint4 raw; T e[PIECE]; } v;
                    v.raw = *reinterpret_cast<const uint4*>(w + j);
#pragma unroll
                    for (int e = 0; e < PIECE; ++e) z = fmaf(to_f32(v.e[e]), di_low[j + e], z);
                }
            } else {
                for (; j < p.rank; ++j) z = fmaf(to_f32(w[j]), di_low[j], z);
            }
        }
        const float ww = expf(-p.rate * sigmoid_f(z + p.w0[c]));
        pk[d] = kk;
        pk[D + d] = rr * ww;
        pk[2 * D + d] = ww;
        pk[3 * D + d] = aa;
        k2 = fmaf(kk, kk, k2);
        rak = fmaf(rr * aa, kk, rak);
        rk = fmaf(rr, kk, rk);
    }
    for (int c = threadIdx.x; c < Dv; c += blockDim.x) {
        pk[4 * D + c] = split_sum(row + 2 * HD + hd * Dv + c, p.n_splits, p.split_stride);
        if (p.gate_out) p.gate_out[(size_t)r * HV + hd * Dv + c] = split_sum(row + 3 * HD + HV + hd * Dv + c, p.n_splits, p.split_stride);
    }
    k2 = block_sum(k2, red0);
    rak = block_sum(rak, red1);
    rk = block_sum(rk, red2);
    if (threadIdx.x == 0) {
        const float n2 = 1.0f / (k2 + 1e-6f);
        float4* out = reinterpret_cast<float4*>(p.scal + ((size_t)r * p.heads + hd) * 4);
        *out = make_float4(n2, n2 * rak, rk, 0.f);
    }
}

extern "C" int cml_delta_inputs(const float* proj, long ld, int n_splits, long split_stride, const float* high, int n_high,
                                long high_stride, const void* w2, int dtype, int rank, const float* a_bias, const float* w0,
                                float rate, float* packed, float* scal, float* gate_out, int rows, int heads, int D, int Dv,
                                int early, void* stream) {
    if (rows <= 0) return 0;
    if (heads < 1 || heads > 65535 || D < 1 || Dv < 1 || n_splits < 1 || rank < 0 || rank > 8192) return CML_ERR_BAD_SIZE;
    if (high == nullptr ? w2 == nullptr : n_high < 1) return CML_ERR_BAD_SIZE;
    if (((uintptr_t)scal) & 15) return CML_ERR_BAD_ALIGN;
    DeltaInputs p = {proj, ld, n_splits, split_stride, high, n_high, high_stride, w2, rank, a_bias, w0, rate, packed, scal, gate_out,
                     heads, D, Dv, early};
    const int most = D > Dv ? D : Dv;
    const int block = most >= 256 ? 256 : (most + 31) / 32 * 32;
    const size_t smem = high == nullptr ? (size_t)rank * sizeof(float) : 0;
    if (dtype == CML_DTYPE_F32)
        launch_pdl(delta_inputs_kernel<float>, dim3(rows, heads), dim3(block), smem, (cudaStream_t)stream, p);
    else if (dtype == CML_DTYPE_BF16)
        launch_pdl(delta_inputs_kernel<bf16>, dim3(rows, heads), dim3(block), smem, (cudaStream_t)stream, p);
    else
        return CML_ERR_BAD_DTYPE;
    return cml_launch_status();
}

// The scan: like the scans above a block of 128 threads owns 128 / NS columns of one (sequence, head), NS threads of a warp
// share a column (a slice of DS key channels each) and walk the new tokens in order. The prepared rows of
// GD_TOKENS tokens come by cp.async into one of two buffers of shared memory while the other one's are worked on.
#define GD_TOKENS 8
struct GeneralDelta {
    const float* packed; const float* scal; float* state;
    const int* seq_row0; const int* seq_new; const int* seq_start; const int* seq_slot;
    float* out;
    int heads, D, Dv;
};

template <int BYTES>
__device__ __forceinline__ void gd_copy(float* smem, const float* gmem) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}

template <int DS, int NS>
__global__ void __launch_bounds__(128) general_delta_kernel(const GeneralDelta p) {
    constexpr int COLS = 128 / NS;
    constexpr int SL = DS == 4 ? 4 : DS + 4;               // floats of a slice in shared memory (padded against bank conflicts)
    constexpr int ROW = NS * SL;                           // floats of one array of a token
    constexpr int TOKEN = 4 * ROW + COLS + 4;              // k, r * w, w, a; the block's values; the scalars
    extern __shared__ __align__(16) float gd_sh[];         // [2][GD_TOKENS][TOKEN]
    pdl_wait();
    pdl_launch_dependents();
    const int s = blockIdx.x, hd = blockIdx.y;
    const int D = p.D, Dv = p.Dv, heads = p.heads;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, slice = lane % NS;
    const int wcol = warp * (32 / NS) + lane / NS;
    const int col0 = blockIdx.z * COLS, c = col0 + wcol;
    const bool live = c < Dv;
    const int d0 = slice * DS;
    const int row0 = p.seq_row0[s], n = p.seq_new[s];
    const bool fresh = p.seq_start[s] == 0, vec = ((D | Dv) & 3) == 0;     // whole heads of `packed` start on 16 bytes
    const size_t per_head = 4 * D + Dv, per_row = per_head * heads;
    float* st = p.state + (((size_t)p.seq_slot[s] * heads + hd) * Dv + (live ? c : 0)) * D;
    auto fetch = [&](int t0, int buf) {
        const int nt = min(GD_TOKENS, n - t0);
        float* dst = gd_sh + (size_t)buf * GD_TOKENS * TOKEN;
        const float* src = p.packed + (size_t)(row0 + t0) * per_row + (size_t)hd * per_head;
        if (vec) {
            const int q = D / 4;                           // 16-byte pieces of an array; a warp takes every fourth (token, array)
            for (int ta = warp; ta < 4 * nt; ta += 4)
                for (int i = lane; i < q; i += 32) {
                    const int d = 4 * i;
                    gd_copy<16>(dst + (ta >> 2) * TOKEN + (ta & 3) * ROW + (d / DS) * SL + d % DS, src + (size_t)(ta >> 2) * per_row + (ta & 3) * D + d);
                }
        } else {
            for (int ta = warp; ta < 4 * nt; ta += 4)
                for (int d = lane; d < D; d += 32)
                    gd_copy<4>(dst + (ta >> 2) * TOKEN + (ta & 3) * ROW + (d / DS) * SL + d % DS, src + (size_t)(ta >> 2) * per_row + (ta & 3) * D + d);
        }
        for (int i = threadIdx.x; i < nt * COLS; i += 128) {
            const int t = i / COLS, cc = i % COLS;
            if (col0 + cc < Dv) gd_copy<4>(dst + t * TOKEN + 4 * ROW + cc, src + (size_t)t * per_row + 4 * D + col0 + cc);
        }
        if (threadIdx.x < nt)
            gd_copy<16>(dst + threadIdx.x * TOKEN + 4 * ROW + COLS, p.scal + ((size_t)(row0 + t0 + threadIdx.x) * heads + hd) * 4);
    };
    if (D < NS * DS || Dv - col0 < COLS) {                 // channels and columns that are not there stay zero
        for (int i = threadIdx.x; i < 2 * GD_TOKENS * TOKEN; i += 128) gd_sh[i] = 0.f;
        __syncthreads();
    }
    fetch(0, 0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    float S[DS];
#pragma unroll
    for (int i = 0; i < DS; i += 4) {
        if (live && !fresh && vec && d0 + i < D) {
            const float4 t = *reinterpret_cast<const float4*>(st + d0 + i);
            S[i] = t.x; S[i + 1] = t.y; S[i + 2] = t.z; S[i + 3] = t.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) S[i + j] = (live && !fresh && d0 + i + j < D) ? st[d0 + i + j] : 0.f;
        }
    }
    for (int t0 = 0, buf = 0; t0 < n; t0 += GD_TOKENS, buf ^= 1) {
        if (t0 + GD_TOKENS < n) fetch(t0 + GD_TOKENS, buf ^ 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");           // all but the newest group: this round's tokens are here
        __syncthreads();
        const float* base = gd_sh + (size_t)buf * GD_TOKENS * TOKEN;
        auto token = [&](int t) {
            const float* tk = base + t * TOKEN + slice * SL;
            const float vcol = base[t * TOKEN + 4 * ROW + wcol];
            const float4 sc = *reinterpret_cast<const float4*>(base + t * TOKEN + 4 * ROW + COLS);
            float kr[DS], p4[4] = {0.f, 0.f, 0.f, 0.f}, q4[4] = {0.f, 0.f, 0.f, 0.f};      // four chains each, always in this order
#pragma unroll
            for (int i = 0; i < DS; i += 4) {
                const float4 kv = *reinterpret_cast<const float4*>(tk + i), rv = *reinterpret_cast<const float4*>(tk + ROW + i);
                kr[i] = kv.x; kr[i + 1] = kv.y; kr[i + 2] = kv.z; kr[i + 3] = kv.w;
                p4[0] = fmaf(S[i], kv.x, p4[0]); p4[1] = fmaf(S[i + 1], kv.y, p4[1]);
                p4[2] = fmaf(S[i + 2], kv.z, p4[2]); p4[3] = fmaf(S[i + 3], kv.w, p4[3]);
                q4[0] = fmaf(S[i], rv.x, q4[0]); q4[1] = fmaf(S[i + 1], rv.y, q4[1]);
                q4[2] = fmaf(S[i + 2], rv.z, q4[2]); q4[3] = fmaf(S[i + 3], rv.w, q4[3]);
            }
            float pk = (p4[0] + p4[1]) + (p4[2] + p4[3]), qr = (q4[0] + q4[1]) + (q4[2] + q4[3]);
#pragma unroll
            for (int sh = 1; sh < NS; sh <<= 1) {
                const float x = __shfl_xor_sync(0xffffffffu, pk, sh), y = __shfl_xor_sync(0xffffffffu, qr, sh);
                pk += x;
                qr += y;
            }
            const float rem = -sc.x * pk;
#pragma unroll
            for (int i = 0; i < DS; i += 4) {
                const float4 wv = *reinterpret_cast<const float4*>(tk + 2 * ROW + i), av = *reinterpret_cast<const float4*>(tk + 3 * ROW + i);
                S[i] = fmaf(kr[i], fmaf(av.x, rem, vcol), wv.x * S[i]);
                S[i + 1] = fmaf(kr[i + 1], fmaf(av.y, rem, vcol), wv.y * S[i + 1]);
                S[i + 2] = fmaf(kr[i + 2], fmaf(av.z, rem, vcol), wv.z * S[i + 2]);
                S[i + 3] = fmaf(kr[i + 3], fmaf(av.w, rem, vcol), wv.w * S[i + 3]);
            }
            // (a plain store might alias the buffers in shared memory as far as the compiler knows, and hold back the next token's loads)
            if (live && slice == 0)
                asm volatile("st.global.f32 [%0], %1;" ::"l"(p.out + ((size_t)(row0 + t0 + t) * heads + hd) * Dv + c), "f"(fmaf(sc.z, vcol, fmaf(-sc.y, pk, qr))));
        };
        const int nt = min(GD_TOKENS, n - t0);
        if (nt == GD_TOKENS) {                             // a whole round unrolled: the next tokens' loads and this one's read-out overlap
#pragma unroll
            for (int t = 0; t < GD_TOKENS; ++t) token(t);
        } else {
            for (int t = 0; t < nt; ++t) token(t);
        }
        __syncthreads();                                   // before the next fetch overwrites this buffer
    }
    if (live) {
#pragma unroll
        for (int i = 0; i < DS; i += 4) {
            if (vec && d0 + i < D) {
                *reinterpret_cast<float4*>(st + d0 + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (d0 + i + j < D) st[d0 + i + j] = S[i + j];
            }
        }
    }
}

extern "C" int cml_general_delta_scan(const float* packed, const float* scal, float* state, const int* seq_row0, const int* seq_new,
                                      const int* seq_start, const int* seq_slot, float* out, int n_seqs, int heads, int D, int Dv,
                                      void* stream) {
    if (n_seqs <= 0) return 0;
    if (D < 1 || D > 256 || Dv < 1 || heads < 1 || heads > 65535) return CML_ERR_BAD_SIZE;
    if ((((uintptr_t)packed) | ((uintptr_t)scal) | ((uintptr_t)state)) & 15) return CML_ERR_BAD_ALIGN;
    GeneralDelta p = {packed, scal, state, seq_row0, seq_new, seq_start, seq_slot, out, heads, D, Dv};
    constexpr int NS = SCAN_SLICES, COLS = 128 / NS;
    dim3 grid(n_seqs, heads, (Dv + COLS - 1) / COLS);
#define GD_CASE(DS_)                                                                                                     \
    if (D <= NS * DS_) {                                                                                                 \
        constexpr size_t smem = (size_t)2 * GD_TOKENS * (4 * NS * (DS_ == 4 ? 4 : DS_ + 4) + COLS + 4) * sizeof(float);  \
        if (smem > 48 * 1024 && cml_allow_smem<general_delta_kernel<DS_, NS>>(smem) != cudaSuccess) return CML_ERR_BAD_SIZE; \
        launch_pdl(general_delta_kernel<DS_, NS>, grid, dim3(128), smem, (cudaStream_t)stream, p);                       \
        return cml_launch_status();                                                                                      \
    }
    GD_CASE(4) GD_CASE(8) GD_CASE(16) GD_CASE(32)
#undef GD_CASE
    return CML_ERR_BAD_SIZE;
}

// ------------------------------------------------------------------------------------
// The state-space recurrence by chunks of SSQ = 64 tokens, for steps that bring many tokens per sequence. With a = -exp(A_log) dt,
// c_t the sum of a over the chunk's tokens up to t and S the state before the chunk, a token of the chunk reads
//
//   y_t = e^(c_t) S^T C_t + sum over s <= t of e^(c_t - c_s) dt_s (C_t . B_s) x_s + D x_t
//
// and the state after the chunk is e^(c_last) S + sum over s of e^(c_last - c_s) dt_s B_s x_s^T. Three kernels: the products
// C_t . B_s of every (chunk, group) and the steps of its heads side by side; the states, each block walking a sequence's chunks with a tile of one head's
// state in registers and leaving the state before every chunk; the outputs of every (chunk, head) side by side. All float (every
// exponent is at most 0). Tokens that a chunk does not have count as zero steps.
//
// Retention and the matrix memory are the same sums with other decays and steps: retention has c_t = (t + 1) ln(decay) and steps of 1;
// the matrix memory, whose state is scaled by e^-m with a running maximum m, has c_t = sum of f over the chunk's tokens up to t, plus m
// before the chunk, minus m_t, and steps of e^(i_t - m_t), and n is one more value whose x is 1. A kernel of its own makes these from
// the gates (MODE 2). A prompt of 2,048 tokens inside a decoder: retention, 16 heads of 128 x 128: 670 us by the scan -> 215 (scores 21,
// states 124, outputs 60); matrix memory, 8 heads of 128 x 129: 1,107 us -> 210 (states 135, outputs 46). The scan's time is its
// serial chain, one token after the other; by chunks it is the walk over the states, then the products. Distance from 64 bits (2-norms, 2,048
// tokens) beside the scan's: retention with a decay of 0.999 3.0e-7 (4.8e-7), 0.98 1.5e-7 (1.5e-7), 0.5 1.0e-7 (0.8e-7); matrix memory 2.5e-7 (2.4e-7).
#define SSQ 64
enum { CH_SSM = 0, CH_RETENTION = 1, CH_MEMORY = 2 };

struct SsmChunks {
    const float* rows; long ld; int x_col, b_col, c_col;       // x (heads x P), B, C (groups x N) of ssm_inputs_kernel
    const float* gates; long ldg;                              // dt at column head
    const float* a_log; const float* d_skip;
    const int* tile_seq; const int* tile_q0;                   // chunks: sequence and first of its new rows
    const int* seq_row0; const int* seq_new; const int* seq_start; const int* seq_slot;
    float* state;                                              // [slots, heads, P, N]
    float* scores;                                             // [chunks, groups, SSQ, SSQ]
    float* steps;                                              // [chunks, heads, n_steps, SSQ]: c_t, dt_t, e^(c_last - c_t) dt_t
    int n_steps;                                               // 3; 4 where c_t is a sum of two floats (its lower part the fourth)
    float* prev;                                               // [chunks, heads, P, N]: the state before the chunk
    float* out;                                                // [rows, heads x P]; matrix memory: [rows, heads, Pv + 2], the last one m
    int heads, groups, N, P;
    int Pv;                                                    // values that lie in the rows; P, or P - 1 (the last value is 1)
    const float* decay;                                        // retention: [heads]
    const float* i_bias; const float* f_bias; int i_col, f_col;        // matrix memory: the gates' biases and columns
    float cap, q_scale;
    float* state_m;                                            // matrix memory: [slots, heads, P], copies of m
    int least;                                                 // sequences with fewer new rows have no tiles and are left alone
};

// the number of the first tile of sequence s: the tiles of the sequences before it, those with fewer than `least` new rows having none
__device__ __forceinline__ int first_tile_of(const int* seq_new, int s, int size, int least) {
    int first = 0;
    for (int q = 0; q < s; ++q) first += seq_new[q] >= least ? (seq_new[q] + size - 1) / size : 0;
    return first;
}

// two products and sums in one instruction, each rounded as by itself
__device__ __forceinline__ void ssm_fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
struct SsmQuad { unsigned long long lo, hi; };                 // four floats as two pairs
__device__ __forceinline__ SsmQuad ssm_quad(const float* p) {
    const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(p);
    return {t.x, t.y};
}
__device__ __forceinline__ float ssm_pair_sum(unsigned long long v) { return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32)); }

// rows [row0 + min(i, nt - 1)] of `cols` floats at column col into shared rows of `pitch` floats; cp.async, 16 bytes a copy
__device__ __forceinline__ void ssm_stage(float* dst, int pitch, const float* src, long ld, int nt, int cols, int tid, int threads) {
    const int q = cols / 4;
    for (int i = tid; i < SSQ * q; i += threads) {
        const int t = i / q, c = (i - t * q) * 4;
        gd_copy<16>(dst + t * pitch + c, src + (size_t)min(t, nt - 1) * ld + c);
    }
}

// 64 x 64 products of rows of A and rows of B over N channels: thread (ty, px) of 8 x 16 takes rows ty + 8 i of A and rows
// 16 j + px of B; even and odd channels of 32 are summed side by side, and the sums of 32 channels added in order (one chain over
// all channels would round each of its sums at the size of the whole)
__device__ __forceinline__ void ssm_dot_tile(const float* a, const float* b, int pitch, int N, int ty, int px, float (&out)[8][4]) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) out[i][j] = 0.f;
    for (int n0 = 0; n0 < N; n0 += 32) {
        unsigned long long acc[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
        const int n1 = min(n0 + 32, N);
        for (int n = n0; n < n1; n += 4) {
            SsmQuad bq[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) bq[j] = ssm_quad(b + (16 * j + px) * pitch + n);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const SsmQuad aq = ssm_quad(a + (ty + 8 * i) * pitch + n);
#pragma unroll
                for (int j = 0; j < 4; ++j) { ssm_fma2(acc[i][j], aq.lo, bq[j].lo); ssm_fma2(acc[i][j], aq.hi, bq[j].hi); }
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) out[i][j] += ssm_pair_sum(acc[i][j]);
    }
}

// a warp: the running sums c_t of a chunk's 64 tokens (two a lane), their steps, and what their B count in the state after the chunk
__device__ __forceinline__ void ssm_steps(const SsmChunks& p, int tile, int row, int nt, int hd, int lane) {
    const float rate = expf(p.a_log[hd]);
    float dt[2], c[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int t = 2 * lane + e;
        const float v = p.gates[(size_t)(row + min(t, nt - 1)) * p.ldg + hd];
        dt[e] = t < nt ? v : 0.f;
    }
    c[0] = -rate * dt[0];
    c[1] = c[0] - rate * dt[1];
    float before = c[1];
#pragma unroll
    for (int sh = 1; sh < 32; sh <<= 1) {
        const float o = __shfl_up_sync(0xffffffffu, before, sh);
        if (lane >= sh) before += o;
    }
    before -= c[1];                                            // the sum before this lane's two tokens
    c[0] += before;
    c[1] += before;
    const float last = __shfl_sync(0xffffffffu, c[1], 31);
    float2* o = reinterpret_cast<float2*>(p.steps + ((size_t)tile * p.heads + hd) * p.n_steps * SSQ) + lane;
    o[0] = make_float2(c[0], c[1]);
    o[SSQ / 2] = make_float2(dt[0], dt[1]);
    o[SSQ] = make_float2(dt[0] * expf(last - c[0]), dt[1] * expf(last - c[1]));
}

// The same for retention: c_t = (number of tokens there up to t) ln(decay), steps of 1.
__device__ __forceinline__ void retention_steps(const SsmChunks& p, int tile, int nt, int hd, int lane) {
    const double fade = log((double)p.decay[hd]);
    float* o = p.steps + ((size_t)tile * p.heads + hd) * p.n_steps * SSQ;
    for (int t = lane; t < SSQ; t += 32) {
        const double c = fade * min(t + 1, nt);
        o[t] = (float)c;
        o[3 * SSQ + t] = (float)(c - (double)(float)c);
        o[SSQ + t] = t < nt ? 1.f : 0.f;
        o[2 * SSQ + t] = t < nt ? (float)exp(fade * (nt - 1 - t)) : 0.f;
    }
}

// The matrix memory's steps: a block per (sequence, head), MS_TOKENS tokens (a thread each) at a time. m_t = max(f_t + m_(t-1), i_t) is
// a scan of pairs (a, b), m -> max(a + m, b): by shuffles in a warp, then over the warps' pairs in order. The sums of f are double: c_t can
// be hundreds where a difference of two of them is a few, and that difference is an exponent.
#define MS_TOKENS 512
__global__ void __launch_bounds__(MS_TOKENS) memory_steps_kernel(const SsmChunks p) {
    __shared__ double s_sum[MS_TOKENS / 32], s_c[MS_TOKENS];
    __shared__ float s_top[MS_TOKENS / 32], s_m[MS_TOKENS];
    pdl_wait();
    pdl_launch_dependents();
    const int s = blockIdx.x, hd = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row0 = p.seq_row0[s], n = p.seq_new[s];
    if (n < p.least) return;
    const int first = first_tile_of(p.seq_new, s, SSQ, p.least);
    float* ms = p.state_m + ((size_t)p.seq_slot[s] * p.heads + hd) * p.P;
    float m0 = p.seq_start[s] == 0 ? 0.f : ms[0];
    __syncthreads();                                           // everyone has read it
    const float bi = p.i_bias[hd], bf = p.f_bias[hd];
    for (int t0 = 0; t0 < n; t0 += MS_TOKENS) {
        const int t = t0 + tid;
        const bool there = t < n;
        const float* row = p.rows + (size_t)(row0 + min(t, n - 1)) * p.ld;
        const float gi = p.cap * tanhf((row[p.i_col + hd] + bi) / p.cap), gf = logsigmoid_f(p.cap * tanhf((row[p.f_col + hd] + bf) / p.cap));
        const float f = there ? gf : 0.f, in = there ? gi : -INFINITY;       // tokens that are not there change nothing
        double a = f;
        float b = in;
#pragma unroll
        for (int sh = 1; sh < 32; sh <<= 1) {
            const double a1 = __shfl_up_sync(0xffffffffu, a, sh);
            const float b1 = __shfl_up_sync(0xffffffffu, b, sh);
            if (lane >= sh) { b = fmaxf((float)(a + b1), b); a += a1; }
        }
        if (lane == 31) { s_sum[warp] = a; s_top[warp] = b; }
        __syncthreads();
        float before = m0;                                     // m before this warp's tokens
        for (int w = 0; w < warp; ++w) before = fmaxf((float)(s_sum[w] + before), s_top[w]);
        const float m = fmaxf((float)(a + before), b);
        s_m[tid] = m;
        __syncthreads();
        // the chunk (two warps): the sum of f from its first token on, m before it
        const int head = tid & ~(SSQ - 1);
        const double c = a + ((warp & 1) ? s_sum[warp - 1] : 0.0) + ((double)(head ? s_m[head - 1] : m0) - m);
        s_c[tid] = c;
        __syncthreads();
        if (t0 + head < n) {
            const float step = expf(in - m);
            float* o = p.steps + ((size_t)(first + (t0 + head) / SSQ) * p.heads + hd) * p.n_steps * SSQ + (tid - head);
            o[0] = (float)c;
            o[SSQ] = step;
            o[2 * SSQ] = step * expf((float)(s_c[head + SSQ - 1] - c));
            o[3 * SSQ] = (float)(c - (double)(float)c);
            if (there) p.out[((size_t)(row0 + t) * p.heads + hd) * (p.Pv + 2) + p.Pv + 1] = m;
        }
        m0 = s_m[MS_TOKENS - 1];
        __syncthreads();                                       // before the next tokens' values
    }
    for (int c = tid; c < p.P; c += MS_TOKENS) ms[c] = m0;
}

template <int MODE>
__global__ void __launch_bounds__(128, 3) ssm_scores_kernel(const SsmChunks p) {
    extern __shared__ __align__(16) float ss_sh[];
    pdl_wait();
    pdl_launch_dependents();
    const int tile = blockIdx.x, g = blockIdx.y, tid = threadIdx.x, N = p.N, pitch = N + 4;
    const int seq = p.tile_seq[tile], q0 = p.tile_q0[tile], nt = min(SSQ, p.seq_new[seq] - q0);
    const float* base = p.rows + (size_t)(p.seq_row0[seq] + q0) * p.ld + g * N;
    float* sC = ss_sh;
    float* sB = sC + SSQ * pitch;
    ssm_stage(sC, pitch, base + p.c_col, p.ld, nt, N, tid, 128);
    ssm_stage(sB, pitch, base + p.b_col, p.ld, nt, N, tid, 128);
    const int per = p.heads / p.groups;                        // meanwhile the steps of the group's heads
    if (MODE == CH_SSM)
        for (int h = tid >> 5; h < per; h += 4) ssm_steps(p, tile, p.seq_row0[seq] + q0, nt, g * per + h, tid & 31);
    else if (MODE == CH_RETENTION)
        for (int h = tid >> 5; h < per; h += 4) retention_steps(p, tile, nt, g * per + h, tid & 31);
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int px = tid & 15, ty = tid >> 4;
    float acc[8][4];
    ssm_dot_tile(sC, sB, pitch, N, ty, px, acc);
    float* o = p.scores + ((size_t)tile * p.groups + g) * SSQ * SSQ;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[(ty + 8 * i) * SSQ + 16 * j + px] = acc[i][j];
}

// A block of 128 threads owns 64 values x 32 channels of one (sequence, head)'s state, four by four a thread.
#define SST_P 64
#define SST_N 32
__global__ void __launch_bounds__(128) ssm_states_kernel(const SsmChunks p) {
    extern __shared__ __align__(16) float st_sh[];             // two buffers of x, B, the tokens' weights, c_t
    pdl_wait();
    pdl_launch_dependents();
    const int s = blockIdx.x, hd = blockIdx.y, N = p.N, P = p.P, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n_tiles_n = (N + SST_N - 1) / SST_N;
    const int p0 = (int)(blockIdx.z / n_tiles_n) * SST_P, n0 = (int)(blockIdx.z % n_tiles_n) * SST_N;
    const int g = hd / (p.heads / p.groups), row0 = p.seq_row0[s], n = p.seq_new[s], n_chunks = (n + SSQ - 1) / SSQ;
    const bool fresh = p.seq_start[s] == 0;
    constexpr int BUF = SSQ * (SST_P + SST_N + 2);
    if (n < p.least) return;
    const int first = first_tile_of(p.seq_new, s, SSQ, p.least);
    const int pc = (warp * 4 + (lane >> 3)) * 4, nc = (lane & 7) * 4;          // this thread's values and channels within the tile
    const bool live_n = n0 + nc < N;
    float* st = p.state + ((size_t)p.seq_slot[s] * p.heads + hd) * P * N;
    float4 S[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const bool ok = live_n && p0 + pc + e < P && !fresh;
        S[e] = ok ? *reinterpret_cast<const float4*>(st + (size_t)(p0 + pc + e) * N + n0 + nc) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const int wp = min(SST_P, p.Pv - p0), wn = min(SST_N, N - n0);     // (no value of the last tile need lie in the rows)
    if (wp < SST_P || wn < SST_N) {                            // values and channels that are not there stay zero
        for (int i = tid; i < 2 * BUF; i += 128) st_sh[i] = 0.f;
        __syncthreads();
        if (p.Pv < P && wp < SST_P) st_sh[(tid >> 6) * BUF + (tid & 63) * SST_P + wp] = 1.f;     // the value that is 1 (SSQ tokens, two buffers)
    }
    auto fetch = [&](int ch, int buf) {
        const int nt = min(SSQ, n - ch * SSQ);
        const float* base = p.rows + (size_t)(row0 + ch * SSQ) * p.ld;
        const float* xs = base + p.x_col + hd * p.Pv + p0;
        const float* bs = base + p.b_col + g * N + n0;
        float* dst = st_sh + buf * BUF;
        if (wp == SST_P) {                                     // whole tiles: places known when compiled
#pragma unroll
            for (int i = 0; i < SSQ * SST_P / 512; ++i) {
                const int t = (tid >> 4) + 8 * i, c = (tid & 15) * 4;
                gd_copy<16>(dst + t * SST_P + c, xs + (size_t)min(t, nt - 1) * p.ld + c);
            }
        } else ssm_stage(dst, SST_P, xs, p.ld, nt, wp, tid, 128);
        if (wn == SST_N) {
#pragma unroll
            for (int i = 0; i < SSQ * SST_N / 512; ++i) {
                const int t = (tid >> 3) + 16 * i, c = (tid & 7) * 4;
                gd_copy<16>(dst + SSQ * SST_P + t * SST_N + c, bs + (size_t)min(t, nt - 1) * p.ld + c);
            }
        } else ssm_stage(dst + SSQ * SST_P, SST_N, bs, p.ld, nt, wn, tid, 128);
        // the tokens' weights, then c_t
        const float* steps = p.steps + ((size_t)(first + ch) * p.heads + hd) * p.n_steps * SSQ;
        if (tid < 32) gd_copy<16>(dst + SSQ * (SST_P + SST_N) + tid * 4, steps + (tid < 16 ? 2 * SSQ + tid * 4 : (tid - 16) * 4));
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0, 0);
    for (int ch = 0; ch < n_chunks; ++ch) {
        const float* sx = st_sh + (ch & 1) * BUF;
        const float* sb = sx + SSQ * SST_P;
        const float* sw = sb + SSQ * SST_N;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                       // this chunk is here, the other buffer is free
        if (ch + 1 < n_chunks) fetch(ch + 1, (ch + 1) & 1);
        // the state before the chunk, for the outputs
        float* pv = p.prev + ((size_t)(first + ch) * p.heads + hd) * P * N;
        const float keep = expf(sw[2 * SSQ - 1]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (live_n && p0 + pc + e < P) *reinterpret_cast<float4*>(pv + (size_t)(p0 + pc + e) * N + n0 + nc) = S[e];
        }
        float4 L[4];                                           // the chunk's own sum, added to the state at once: 64 terms one by one would each round at its size
#pragma unroll
        for (int e = 0; e < 4; ++e) L[e] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int t = 0; t < SSQ; ++t) {
            const float w = sw[t];
            const float4 x = *reinterpret_cast<const float4*>(sx + t * SST_P + pc);
            float4 b = *reinterpret_cast<const float4*>(sb + t * SST_N + nc);
            b.x *= w; b.y *= w; b.z *= w; b.w *= w;
            L[0].x = fmaf(x.x, b.x, L[0].x); L[0].y = fmaf(x.x, b.y, L[0].y); L[0].z = fmaf(x.x, b.z, L[0].z); L[0].w = fmaf(x.x, b.w, L[0].w);
            L[1].x = fmaf(x.y, b.x, L[1].x); L[1].y = fmaf(x.y, b.y, L[1].y); L[1].z = fmaf(x.y, b.z, L[1].z); L[1].w = fmaf(x.y, b.w, L[1].w);
            L[2].x = fmaf(x.z, b.x, L[2].x); L[2].y = fmaf(x.z, b.y, L[2].y); L[2].z = fmaf(x.z, b.z, L[2].z); L[2].w = fmaf(x.z, b.w, L[2].w);
            L[3].x = fmaf(x.w, b.x, L[3].x); L[3].y = fmaf(x.w, b.y, L[3].y); L[3].z = fmaf(x.w, b.z, L[3].z); L[3].w = fmaf(x.w, b.w, L[3].w);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            S[e].x = fmaf(S[e].x, keep, L[e].x); S[e].y = fmaf(S[e].y, keep, L[e].y);
            S[e].z = fmaf(S[e].z, keep, L[e].z); S[e].w = fmaf(S[e].w, keep, L[e].w);
        }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
        if (live_n && p0 + pc + e < P) *reinterpret_cast<float4*>(st + (size_t)(p0 + pc + e) * N + n0 + nc) = S[e];
}

// One block per (chunk, head, 64 values): 64 tokens x 64 values, thread (ty, px) of 8 x 16 takes tokens ty + 8 i and values
// 4 px .. 4 px + 3. The state's rows lie in shared memory so that the rows 4 px + j of neighbouring threads are neighbours.
#define SSM_PITCH 68                                           // floats of a row of the weights and of x in shared memory
template <int MODE>
__global__ void __launch_bounds__(128, 3) ssm_outputs_kernel(const SsmChunks p) {
    extern __shared__ __align__(16) float so_sh[];
    __shared__ float s_dt[SSQ], s_c[SSQ], s_low[MODE == CH_SSM ? 1 : SSQ];
    pdl_wait();
    pdl_launch_dependents();
    const int tile = blockIdx.x, hd = blockIdx.y, p0 = blockIdx.z * 64, tid = threadIdx.x, N = p.N, P = p.P, pitch = N + 4;
    const int seq = p.tile_seq[tile], q0 = p.tile_q0[tile], nt = min(SSQ, p.seq_new[seq] - q0), row0 = p.seq_row0[seq] + q0;
    const int g = hd / (p.heads / p.groups), wp = min(64, P - p0), wv = min(64, p.Pv - p0);     // values of the tile; those in the rows
    const float* base = p.rows + (size_t)row0 * p.ld;
    const int area = SSQ * max(pitch, SSM_PITCH);              // each of the two areas serves twice
    float* sC = so_sh;
    float* sS = so_sh + area;
    ssm_stage(sC, pitch, base + p.c_col + g * N, p.ld, nt, N, tid, 128);
    const float* pv = p.prev + (((size_t)tile * p.heads + hd) * P + p0) * N;
    for (int i = tid; i < 64 * (N / 4); i += 128) {
        const int r = i / (N / 4), c = (i - r * (N / 4)) * 4;
        gd_copy<16>(sS + ((r & 3) * 16 + (r >> 2)) * pitch + c, pv + (size_t)min(r, wp - 1) * N + c);      // (rows beyond P: never stored)
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* steps = p.steps + ((size_t)tile * p.heads + hd) * p.n_steps * SSQ;
    if (tid < SSQ) { s_c[tid] = steps[tid]; s_dt[tid] = steps[SSQ + tid]; }
    if (MODE != CH_SSM && tid < SSQ) s_low[tid] = steps[3 * SSQ + tid];
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int px = tid & 15, ty = tid >> 4;
    float acc[8][4];
    ssm_dot_tile(sC, sS, pitch, N, ty, px, acc);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float f = expf(s_c[ty + 8 * i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] *= f;
    }
    __syncthreads();                                           // both areas are free
    float* sM = so_sh;
    float* sX = so_sh + area;
    if (wv > 0) ssm_stage(sX, SSM_PITCH, base + p.x_col + hd * p.Pv + p0, p.ld, nt, wv, tid, 128);
    if (MODE == CH_MEMORY && wv < wp && tid < SSQ) sX[tid * SSM_PITCH + wv] = 1.f;               // the value that is 1
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* sc = p.scores + ((size_t)tile * p.groups + g) * SSQ * SSQ;
    for (int i = tid; i < SSQ * SSQ / 4; i += 128) {           // the weights of the chunk's own tokens
        const int t = i >> 4, s = (i & 15) * 4;
        float4 v = *reinterpret_cast<const float4*>(sc + i * 4);
        const float ct = s_c[t], low = MODE == CH_SSM ? 0.f : s_low[t];
        auto faded = [&](int j) -> float { return expf(MODE == CH_SSM ? ct - s_c[j] : (ct - s_c[j]) + (low - s_low[j])); };
        v.x = s <= t ? v.x * s_dt[s] * faded(s) : 0.f;
        v.y = s + 1 <= t ? v.y * s_dt[s + 1] * faded(s + 1) : 0.f;
        v.z = s + 2 <= t ? v.z * s_dt[s + 2] * faded(s + 2) : 0.f;
        v.w = s + 3 <= t ? v.w * s_dt[s + 3] * faded(s + 3) : 0.f;
        *reinterpret_cast<float4*>(sM + t * SSM_PITCH + s) = v;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int pc = 4 * px;
    float own[8][4];                                           // the chunk's own tokens, added to what the state gives at the end
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) own[i][j] = 0.f;
    // Rows of tokens before s are left out of s's sums, not multiplied by their zero weights: a value that is not finite stays
    // with its token and the later ones, as in the scan. (Half of the products are none, besides.)
#pragma unroll
    for (int s = 0; s < SSQ; s += 4) {
        float4 x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = *reinterpret_cast<const float4*>(sX + (s + k) * SSM_PITCH + pc);
#pragma unroll
        for (int i = 7; i >= s / 8; --i) {                     // the eight tokens with s among them last: of their x only what they see is left
            if (i == s / 8) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (s % 8 + k > ty) x[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            const float4 m = *reinterpret_cast<const float4*>(sM + (ty + 8 * i) * SSM_PITCH + s);
            own[i][0] = fmaf(m.x, x[0].x, fmaf(m.y, x[1].x, fmaf(m.z, x[2].x, fmaf(m.w, x[3].x, own[i][0]))));
            own[i][1] = fmaf(m.x, x[0].y, fmaf(m.y, x[1].y, fmaf(m.z, x[2].y, fmaf(m.w, x[3].y, own[i][1]))));
            own[i][2] = fmaf(m.x, x[0].z, fmaf(m.y, x[1].z, fmaf(m.z, x[2].z, fmaf(m.w, x[3].z, own[i][2]))));
            own[i][3] = fmaf(m.x, x[0].w, fmaf(m.y, x[1].w, fmaf(m.z, x[2].w, fmaf(m.w, x[3].w, own[i][3]))));
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += own[i][j];
    if (pc >= wp) return;
    const float d = MODE == CH_SSM ? p.d_skip[hd] : 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = ty + 8 * i;
        if (t >= nt) continue;
        if (MODE == CH_MEMORY) {                               // rows of Pv + 2 numbers
            float* o = p.out + ((size_t)(row0 + t) * p.heads + hd) * (p.Pv + 2) + p0 + pc;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (pc + j < wp) o[j] = acc[i][j] * p.q_scale;
            continue;
        }
        if (MODE == CH_RETENTION) {
            *reinterpret_cast<float4*>(p.out + (size_t)(row0 + t) * p.heads * P + hd * P + p0 + pc) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
            continue;
        }
        const float4 x = *reinterpret_cast<const float4*>(sX + t * SSM_PITCH + pc);
        *reinterpret_cast<float4*>(p.out + (size_t)(row0 + t) * p.heads * P + hd * P + p0 + pc) =
            make_float4(fmaf(d, x.x, acc[i][0]), fmaf(d, x.y, acc[i][1]), fmaf(d, x.z, acc[i][2]), fmaf(d, x.w, acc[i][3]));
    }
}

template <int MODE>
static int launch_chunks(const SsmChunks& p, int n_tiles, int n_seqs, cudaStream_t s) {
    const int N = p.N, P = p.P;
    if (n_tiles <= 0 || n_seqs <= 0) return 0;
    if (p.heads < 1 || p.heads > 65535 || p.groups < 1 || p.heads % p.groups || N < 4 || N > 256 || (N & 3) || p.Pv < 4 || (p.Pv & 3)) return CML_ERR_BAD_SIZE;
    if (((p.x_col | p.b_col | p.c_col) & 3) || (p.ld & 3)) return CML_ERR_BAD_ALIGN;
    if ((((uintptr_t)p.rows) | ((uintptr_t)p.state) | ((uintptr_t)p.scores) | ((uintptr_t)p.steps) | ((uintptr_t)p.prev) | ((uintptr_t)p.out)) & 15) return CML_ERR_BAD_ALIGN;
    const size_t smem_dot = (size_t)2 * SSQ * (N + 4) * sizeof(float);
    const size_t smem_out = (size_t)2 * SSQ * (N + 4 > SSM_PITCH ? N + 4 : SSM_PITCH) * sizeof(float);
    if (smem_dot > 48 * 1024 && cml_allow_smem<ssm_scores_kernel<MODE>>(smem_dot) != cudaSuccess) return CML_ERR_BAD_SIZE;
    if (smem_out > 48 * 1024 && cml_allow_smem<ssm_outputs_kernel<MODE>>(smem_out) != cudaSuccess) return CML_ERR_BAD_SIZE;
    constexpr size_t smem_states = (size_t)2 * SSQ * (SST_P + SST_N + 2) * sizeof(float);
    if (cml_allow_smem<ssm_states_kernel>(smem_states) != cudaSuccess) return CML_ERR_BAD_SIZE;
    if (MODE == CH_MEMORY) launch_pdl(memory_steps_kernel, dim3(n_seqs, p.heads), dim3(MS_TOKENS), 0, s, p);
    launch_pdl(ssm_scores_kernel<MODE>, dim3(n_tiles, p.groups), dim3(128), smem_dot, s, p);
    launch_pdl(ssm_states_kernel, dim3(n_seqs, p.heads, ((P + SST_P - 1) / SST_P) * ((N + SST_N - 1) / SST_N)), dim3(128), smem_states, s, p);
    launch_pdl(ssm_outputs_kernel<MODE>, dim3(n_tiles, p.heads, (P + 63) / 64), dim3(128), smem_out, s, p);
    return cml_launch_status();
}

// Retention by chunks: proj as for cml_retention_scan, decays > 0.
extern "C" int cml_retention_chunks(const float* proj, long ld, int q_col, int k_col, int v_col, const float* decay, const int* tile_seq,
                                    const int* tile_q0, int n_tiles, const int* seq_row0, const int* seq_new, const int* seq_start,
                                    const int* seq_slot, float* state, float* scores, float* steps, float* prev, float* out, int n_seqs,
                                    int heads, int D, int Dv, int least, void* stream) {
    SsmChunks p = {};
    p.least = least;
    p.rows = proj; p.ld = ld; p.x_col = v_col; p.b_col = k_col; p.c_col = q_col; p.decay = decay; p.tile_seq = tile_seq; p.tile_q0 = tile_q0;
    p.seq_row0 = seq_row0; p.seq_new = seq_new; p.seq_start = seq_start; p.seq_slot = seq_slot; p.state = state; p.scores = scores;
    p.steps = steps; p.prev = prev; p.out = out; p.heads = heads; p.groups = heads; p.N = D; p.P = Dv; p.Pv = Dv; p.n_steps = 4;
    return launch_chunks<CH_RETENTION>(p, n_tiles, n_seqs, (cudaStream_t)stream);
}

// The matrix memory by chunks: arguments as for cml_memory_scan; prev [tiles, heads, Dv + 1, D].
extern "C" int cml_memory_chunks(const float* proj, long ld, int q_col, int k_col, int v_col, int i_col, int f_col, const float* i_bias,
                                 const float* f_bias, float cap, float q_scale, const int* tile_seq, const int* tile_q0, int n_tiles,
                                 const int* seq_row0, const int* seq_new, const int* seq_start, const int* seq_slot, float* state,
                                 float* state_m, float* scores, float* steps, float* prev, float* out, int n_seqs, int heads, int D, int Dv,
                                 int least, void* stream) {
    SsmChunks p = {};
    p.least = least;
    p.rows = proj; p.ld = ld; p.x_col = v_col; p.b_col = k_col; p.c_col = q_col; p.i_col = i_col; p.f_col = f_col; p.i_bias = i_bias; p.f_bias = f_bias;
    p.cap = cap; p.q_scale = q_scale; p.tile_seq = tile_seq; p.tile_q0 = tile_q0; p.seq_row0 = seq_row0; p.seq_new = seq_new;
    p.seq_start = seq_start; p.seq_slot = seq_slot; p.state = state; p.state_m = state_m; p.scores = scores; p.steps = steps; p.prev = prev;
    p.out = out; p.heads = heads; p.groups = heads; p.N = D; p.P = Dv + 1; p.Pv = Dv; p.n_steps = 4;
    return launch_chunks<CH_MEMORY>(p, n_tiles, n_seqs, (cudaStream_t)stream);
}

extern "C" int cml_ssm_chunks(const float* rows, long ld, int x_col, int b_col, int c_col, const float* gates, long ldg, const float* a_log,
                              const float* d_skip, const int* tile_seq, const int* tile_q0, int n_tiles, const int* seq_row0,
                              const int* seq_new, const int* seq_start, const int* seq_slot, float* state, float* scores, float* steps,
                              float* prev, float* out, int n_seqs, int heads, int groups, int N, int P, int least, void* stream) {
    SsmChunks p = {};
    p.least = least;
    p.rows = rows; p.ld = ld; p.x_col = x_col; p.b_col = b_col; p.c_col = c_col; p.gates = gates; p.ldg = ldg; p.a_log = a_log; p.d_skip = d_skip;
    p.tile_seq = tile_seq; p.tile_q0 = tile_q0; p.seq_row0 = seq_row0; p.seq_new = seq_new; p.seq_start = seq_start; p.seq_slot = seq_slot;
    p.state = state; p.scores = scores; p.steps = steps; p.prev = prev; p.out = out; p.heads = heads; p.groups = groups; p.N = N; p.P = P; p.Pv = P; p.n_steps = 3;
    return launch_chunks<CH_SSM>(p, n_tiles, n_seqs, (cudaStream_t)stream);
}

// ------------------------------------------------------------------------------------
// The generalized delta rule by chunks of GDC = 16 tokens, for steps that bring several tokens per sequence. With
// W_t the product of the decays of the chunk's tokens up to t (per key channel; W_0 = 1) and S_t = diag(W_t) Z_t the rule is
//
//   Z_t = Z_(t-1) - al_t (be_t^T Z_(t-1)) + ka_t v_t^T,     al = a * u / W_t,  be = u * W_(t-1),  ka = k / W_t,  rh = r * W_t
//
// so with M = be al^T, N = be ka^T (strictly lower triangles), Qa = rh al^T, Qk = rh ka^T (with the diagonal), S the state
// before the chunk and P = be^T Z row by row:
//
//   (I + M) P = be S + N V     =>  P = B' S + N' V,    B' = (I + M)^-1 be,  N' = (I + M)^-1 N
//   O = rh S + Qk V - Qa P     =  R' S + E V,          R' = rh - Qa B',     E = Qk - Qa N'
//   S <- diag(W) (S + ka^T V - al^T P) = diag(W) S + G^T V - A'^T (B' S),   A' = al * W,  G = (ka - N'^T al) * W
//
// Everything but the three products with S and V is made by the first kernel for all chunks side by side; the
// second walks a sequence's chunks with the state in registers. All in float: a decay is at least exp(-rate), so W stays
// above exp(-16 rate), and every al, ka meets the be, rh of a later token, so no product grows.
#define GDC 16
#define GDC_FLOATS(D, Dv) ((size_t)(4 * GDC + 1) * (D) + GDC * GDC + GDC * (Dv))      // B', R', G, A', W, E, V of a (chunk, head)

struct DeltaChunks {
    const float* proj; long ld; int n_splits; long split_stride;
    const float* high; int n_high; long high_stride;
    const float* a_bias; const float* w0;
    float rate;
    const int* tile_seq; const int* tile_q0; const int* seq_row0; const int* seq_new;
    float* chunks; float* gate_out;
    int heads, D, Dv;
};

#define GDP 20               // floats of a row of a 16 x 16 matrix in shared memory (16-byte rows, read four at a time)

// One block per (chunk, head); THREADS >= D, a thread owns a key channel. All of a thread's inputs are asked for before
// any of them is used.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) delta_chunks_kernel(const DeltaChunks p) {
    constexpr int NT = 256 / THREADS;                      // pairs of tokens (t, j) of a thread
    extern __shared__ __align__(16) float dc_sh[];
    __shared__ __align__(16) float sM[GDC][GDP], sN[GDC][GDP], sQk[GDC][GDP], sQa[GDC][GDP], sNt[GDC][GDP];
    __shared__ float s_inv[GDC];
    pdl_wait();
    pdl_launch_dependents();
    const int tile = blockIdx.x, hd = blockIdx.y, D = p.D, Dv = p.Dv, HD = p.heads * D, HV = p.heads * Dv;
    const int seq = p.tile_seq[tile], q0 = p.tile_q0[tile];
    const int nt = min(GDC, p.seq_new[seq] - q0), row0 = p.seq_row0[seq] + q0;
    const int pitch = D + 4, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float* be = dc_sh;
    float* al = be + GDC * pitch;
    float* ka = al + GDC * pitch;
    float* rh = ka + GDC * pitch;
    float* out = p.chunks + ((size_t)tile * p.heads + hd) * GDC_FLOATS(D, Dv);
    const int d = min(tid, D - 1), c = hd * D + d;
    const bool mine = tid < D;
    float kk[GDC], rr[GDC], aa[GDC], zz[GDC];
#pragma unroll
    for (int t = 0; t < GDC; ++t) {
        const float* row = p.proj + (size_t)(row0 + min(t, nt - 1)) * p.ld + c;
        kk[t] = row[HD];
        rr[t] = row[0];
        aa[t] = row[2 * HD + HV];
        zz[t] = p.high[(size_t)(row0 + min(t, nt - 1)) * HD + c];
    }
    for (int sp = 1; sp < p.n_splits; ++sp)                // (products of few rows come as split sums)
#pragma unroll
        for (int t = 0; t < GDC; ++t) {
            const float* row = p.proj + (size_t)sp * p.split_stride + (size_t)(row0 + min(t, nt - 1)) * p.ld + c;
            kk[t] += row[HD];
            rr[t] += row[0];
            aa[t] += row[2 * HD + HV];
        }
    for (int sp = 1; sp < p.n_high; ++sp)
#pragma unroll
        for (int t = 0; t < GDC; ++t) zz[t] += p.high[(size_t)sp * p.high_stride + (size_t)(row0 + min(t, nt - 1)) * HD + c];
    const float ab = p.a_bias[c], w0 = p.w0[c];
    if (mine) {
#pragma unroll
        for (int t = 0; t < GDC; ++t) {
            if (t >= nt) kk[t] = 0.f;
            ka[t * pitch + d] = kk[t];
        }
    }
    for (int e = tid; e < Dv; e += THREADS) {              // the values, and the gate's inputs
        float v[GDC];
        const float* col = p.proj + (size_t)row0 * p.ld + 2 * HD + hd * Dv + e;
#pragma unroll
        for (int t = 0; t < GDC; ++t) v[t] = split_sum(col + (size_t)min(t, nt - 1) * p.ld, p.n_splits, p.split_stride);
#pragma unroll
        for (int t = 0; t < GDC; ++t) out[(4 * GDC + 1) * D + GDC * GDC + t * Dv + e] = t < nt ? v[t] : 0.f;
        if (p.gate_out)
            for (int t = 0; t < nt; ++t)
                p.gate_out[(size_t)(row0 + t) * HV + hd * Dv + e] = split_sum(col + (size_t)t * p.ld + HD + HV, p.n_splits, p.split_stride);
    }
    __syncthreads();
    for (int t = warp; t < GDC; t += THREADS / 32) {
        float ss = 0.f;
        for (int i = lane; i < D; i += 32) ss = fmaf(ka[t * pitch + i], ka[t * pitch + i], ss);
        ss = warp_sum(ss);
        if (lane == 0) s_inv[t] = 1.0f / sqrtf(ss + 1e-6f);
    }
    __syncthreads();
    float W = 1.0f;
    if (mine) {
#pragma unroll
        for (int t = 0; t < GDC; ++t) {
            const bool there = t < nt;                     // tokens that are not there change nothing
            const float w = there ? expf(-p.rate * sigmoid_f(zz[t] + w0)) : 1.0f;
            const float u = kk[t] * s_inv[t];
            be[t * pitch + d] = u * W;
            W *= w;
            const float inv = 1.0f / W;
            al[t * pitch + d] = there ? sigmoid_f(aa[t] + ab) * u * inv : 0.f;
            ka[t * pitch + d] = kk[t] * inv;
            rh[t * pitch + d] = there ? rr[t] * W : 0.f;
        }
        out[4 * GDC * D + d] = W;
    }
    __syncthreads();
    {   // the four products of a pair of tokens (t, j); a thread's pairs share j
        const int j = tid & 15;
        float m[NT], n[NT], qk[NT], qa[NT];
#pragma unroll
        for (int u = 0; u < NT; ++u) m[u] = n[u] = qk[u] = qa[u] = 0.f;
        for (int i = 0; i < D; i += 4) {
            const float4 a = *reinterpret_cast<const float4*>(al + j * pitch + i), k = *reinterpret_cast<const float4*>(ka + j * pitch + i);
#pragma unroll
            for (int u = 0; u < NT; ++u) {
                const int t = (tid >> 4) + u * (THREADS / 16);
                const float4 b = *reinterpret_cast<const float4*>(be + t * pitch + i), r = *reinterpret_cast<const float4*>(rh + t * pitch + i);
                m[u] = fmaf(b.x, a.x, fmaf(b.y, a.y, fmaf(b.z, a.z, fmaf(b.w, a.w, m[u]))));
                n[u] = fmaf(b.x, k.x, fmaf(b.y, k.y, fmaf(b.z, k.z, fmaf(b.w, k.w, n[u]))));
                qk[u] = fmaf(r.x, k.x, fmaf(r.y, k.y, fmaf(r.z, k.z, fmaf(r.w, k.w, qk[u]))));
                qa[u] = fmaf(r.x, a.x, fmaf(r.y, a.y, fmaf(r.z, a.z, fmaf(r.w, a.w, qa[u]))));
            }
        }
#pragma unroll
        for (int u = 0; u < NT; ++u) {
            const int t = (tid >> 4) + u * (THREADS / 16);
            sM[t][j] = j < t ? m[u] : 0.f;
            sN[t][j] = j < t ? n[u] : 0.f;
            sQk[t][j] = j <= t ? qk[u] : 0.f;
            sQa[t][j] = j <= t ? qa[u] : 0.f;
        }
    }
    __syncthreads();
    // x <- (I + M)^-1 x for a column x
    auto solve = [&](float (&x)[GDC]) {
#pragma unroll
        for (int t = 1; t < GDC; ++t)
#pragma unroll
            for (int j = 0; j < t; j += 4) {
                const float4 v = *reinterpret_cast<const float4*>(&sM[t][j]);
                x[t] = fmaf(-v.x, x[j], x[t]);
                if (j + 1 < t) x[t] = fmaf(-v.y, x[j + 1], x[t]);
                if (j + 2 < t) x[t] = fmaf(-v.z, x[j + 2], x[t]);
                if (j + 3 < t) x[t] = fmaf(-v.w, x[j + 3], x[t]);
            }
    };
    float x[GDC];
    if (mine) {                                            // B', then R', column by column
#pragma unroll
        for (int t = 0; t < GDC; ++t) x[t] = be[t * pitch + d];
        solve(x);
#pragma unroll
        for (int t = 0; t < GDC; ++t) {
            float v = rh[t * pitch + d];
#pragma unroll
            for (int j = 0; j <= t; j += 4) {
                const float4 q = *reinterpret_cast<const float4*>(&sQa[t][j]);
                v = fmaf(-q.x, x[j], v);
                if (j + 1 <= t) v = fmaf(-q.y, x[j + 1], v);
                if (j + 2 <= t) v = fmaf(-q.z, x[j + 2], v);
                if (j + 3 <= t) v = fmaf(-q.w, x[j + 3], v);
            }
            out[t * D + d] = x[t];
            out[(GDC + t) * D + d] = v;
        }
    }
    if (tid >= THREADS - 32 && lane < GDC) {               // the last warp: N' column by column, both ways round
#pragma unroll
        for (int t = 0; t < GDC; ++t) x[t] = sN[t][lane];
        solve(x);
        __syncwarp(0xffff);
#pragma unroll
        for (int t = 0; t < GDC; ++t) { sN[t][lane] = x[t]; sNt[lane][t] = x[t]; }
    }
    __syncthreads();
    if (mine) {
#pragma unroll
        for (int t = 0; t < GDC; ++t) x[t] = al[t * pitch + d];
#pragma unroll
        for (int j = 0; j < GDC; ++j) {
            float v = ka[j * pitch + d];
#pragma unroll
            for (int t0 = (j + 1) & ~3; t0 < GDC; t0 += 4) {
                const float4 q = *reinterpret_cast<const float4*>(&sNt[j][t0]);
                if (t0 > j) v = fmaf(-q.x, x[t0], v);
                if (t0 + 1 > j) v = fmaf(-q.y, x[t0 + 1], v);
                if (t0 + 2 > j) v = fmaf(-q.z, x[t0 + 2], v);
                if (t0 + 3 > j) v = fmaf(-q.w, x[t0 + 3], v);
            }
            out[(2 * GDC + j) * D + d] = v * W;
            out[(3 * GDC + j) * D + d] = x[j] * W;
        }
    }
    for (int i = tid; i < GDC * GDC; i += THREADS) {
        const int t = i >> 4, j = i & 15;
        float v = sQk[t][j];
        for (int q = j + 1; q <= t; ++q) v = fmaf(-sQa[t][q], sN[q][j], v);
        out[(4 * GDC + 1) * D + i] = v;
    }
}

extern "C" int cml_delta_chunks(const float* proj, long ld, int n_splits, long split_stride, const float* high, int n_high,
                                long high_stride, const float* a_bias, const float* w0, float rate, const int* tile_seq,
                                const int* tile_q0, int n_tiles, const int* seq_row0, const int* seq_new, float* chunks,
                                float* gate_out, int heads, int D, int Dv, void* stream) {
    if (n_tiles <= 0) return 0;
    if (heads < 1 || heads > 65535 || D < 4 || D > 256 || (D & 3) || Dv < 4 || (Dv & 3) || n_splits < 1 || n_high < 1 || rate < 0.f || rate > 2.f)
        return CML_ERR_BAD_SIZE;
    DeltaChunks p = {proj, ld, n_splits, split_stride, high, n_high, high_stride, a_bias, w0, rate, tile_seq, tile_q0, seq_row0, seq_new,
                     chunks, gate_out, heads, D, Dv};
    const size_t smem = (size_t)4 * GDC * (D + 4) * sizeof(float);
    if (D <= 128) {
        launch_pdl(delta_chunks_kernel<128>, dim3(n_tiles, heads), dim3(128), smem, (cudaStream_t)stream, p);
    } else {
        if (smem > 32 * 1024 && cml_allow_smem<delta_chunks_kernel<256>>(smem) != cudaSuccess) return CML_ERR_BAD_SIZE;
        launch_pdl(delta_chunks_kernel<256>, dim3(n_tiles, heads), dim3(256), smem, (cudaStream_t)stream, p);
    }
    return cml_launch_status();
}

// The walk over a sequence's chunks. A warp owns COLS columns of the state of one (sequence, head): NS lanes of DS key
// channels each hold CPT columns, and 32 / NS such groups stand side by side. The products with the state give every lane
// partial sums over its channels for 32 / CPT rows at a time; they are added over the lanes by halving (each step
// hands half of the values over, so a lane ends with sums of its own), in a fixed order. The chunk's matrices come by
// cp.async into one of two buffers while the other one's chunk is worked on.
struct ChunkScan {
    const float* chunks; float* state;
    const int* seq_new; const int* seq_row0; const int* seq_start; const int* seq_slot;
    float* out;
    int heads, D, Dv;
};

template <int DS, int NS, int CPT, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) delta_chunk_scan_kernel(const ChunkScan p) {
    constexpr int G = 32 / NS, WCOLS = G * CPT, COLS = WARPS * WCOLS;
    constexpr int RG = NS / CPT;                           // rows of a group: its RG x CPT sums end in its NS lanes
    constexpr int DP = NS * DS;
    constexpr int THREADS = WARPS * 32;
    extern __shared__ __align__(16) float cs_sh[];
    const int D = p.D, Dv = p.Dv, heads = p.heads;
    constexpr int BUF = (4 * GDC + 1) * DP + GDC * GDC + GDC * COLS;
    float* sP = cs_sh + 2 * BUF;                           // [GDC][COLS]: B' S
    pdl_wait();
    pdl_launch_dependents();
    const int s = blockIdx.x, hd = blockIdx.y, col0 = blockIdx.z * COLS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int group = lane / NS, slice = lane % NS, d0 = slice * DS;
    const int n = p.seq_new[s], row0 = p.seq_row0[s];
    const bool fresh = p.seq_start[s] == 0;
    int first = 0;                                         // chunks of the sequences before this one
    for (int q = 0; q < s; ++q) first += (p.seq_new[q] + GDC - 1) / GDC;
    const int n_chunks = (n + GDC - 1) / GDC;
    const int wc = warp * WCOLS + group * CPT;             // this lane's first column within the block
    float S[CPT][DS];
    size_t cell[CPT];
    bool live[CPT];
#pragma unroll
    for (int e = 0; e < CPT; ++e) {
        live[e] = col0 + wc + e < Dv && d0 < D;
        cell[e] = (((size_t)p.seq_slot[s] * heads + hd) * Dv + (col0 + wc + e < Dv ? col0 + wc + e : 0)) * D + (d0 < D ? d0 : 0);
#pragma unroll
        for (int i = 0; i < DS; i += 4) {
            const bool ok = live[e] && d0 + i < D && !fresh;
            const float4 t = *reinterpret_cast<const float4*>(p.state + cell[e] + (ok ? i : 0));
            S[e][i] = ok ? t.x : 0.f; S[e][i + 1] = ok ? t.y : 0.f; S[e][i + 2] = ok ? t.z : 0.f; S[e][i + 3] = ok ? t.w : 0.f;
        }
    }
    if (D < DP || Dv - col0 < COLS) {                      // channels and columns that are not there stay zero
        for (int i = tid; i < 2 * BUF; i += THREADS) cs_sh[i] = 0.f;
        __syncthreads();
    }
    auto fetch = [&](int ch, int buf) {
        const float* src = p.chunks + ((size_t)(first + ch) * heads + hd) * GDC_FLOATS(D, Dv);
        float* dst = cs_sh + buf * BUF;
        if (D == DP) {                                     // all matrices and E in one run of memory
            for (int i = tid * 4; i < (4 * GDC + 1) * DP + GDC * GDC; i += THREADS * 4) gd_copy<16>(dst + i, src + i);
        } else {
            for (int r = warp; r < 4 * GDC + 1; r += WARPS)
                for (int i = lane * 4; i < D; i += 128) gd_copy<16>(dst + r * DP + i, src + (size_t)r * D + i);
            for (int i = tid * 4; i < GDC * GDC; i += THREADS * 4) gd_copy<16>(dst + (4 * GDC + 1) * DP + i, src + (size_t)(4 * GDC + 1) * D + i);
        }
        const float* v = src + (size_t)(4 * GDC + 1) * D + GDC * GDC + col0;
        for (int i = tid; i < GDC * COLS / 4; i += THREADS) {
            const int t = i / (COLS / 4), e = (i % (COLS / 4)) * 4;
            if (col0 + e < Dv) gd_copy<16>(dst + (4 * GDC + 1) * DP + GDC * GDC + t * COLS + e, v + (size_t)t * Dv + e);
        }
    };
    fetch(0, 0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int ch = 0; ch < n_chunks; ++ch) {
        if (ch + 1 < n_chunks) fetch(ch + 1, (ch + 1) & 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");       // all but the newest group: this chunk is here
        __syncthreads();
        const float* m = cs_sh + (ch & 1) * BUF;
        const float* sE = m + (4 * GDC + 1) * DP;
        const float* sV = sE + GDC * GDC;
        const int nt = min(GDC, n - ch * GDC);
        // B' S and R' S, RG rows at a time
#pragma unroll
        for (int rg = 0; rg < 2 * GDC; rg += RG) {
            float acc[NS];                                 // value r * CPT + e: row rg + r, column e
#pragma unroll
            for (int r = 0; r < RG; ++r) {
#pragma unroll
                for (int e = 0; e < CPT; ++e) acc[r * CPT + e] = 0.f;
#pragma unroll
                for (int i = 0; i < DS; i += 4) {
                    const float4 b = *reinterpret_cast<const float4*>(m + (rg + r) * DP + d0 + i);
#pragma unroll
                    for (int e = 0; e < CPT; ++e)
                        acc[r * CPT + e] = fmaf(b.x, S[e][i], fmaf(b.y, S[e][i + 1], fmaf(b.z, S[e][i + 2], fmaf(b.w, S[e][i + 3], acc[r * CPT + e]))));
                }
            }
#pragma unroll
            for (int h = NS / 2; h > 0; h >>= 1) {         // lane bit h keeps the upper half of what is left
                const bool up = (slice & h) != 0;
#pragma unroll
                for (int i = 0; i < h; ++i) {
                    const float give = up ? acc[i] : acc[i + h], keep = up ? acc[i + h] : acc[i];
                    acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, h);
                }
            }
            const int row = rg + slice / CPT, e = slice % CPT;     // the sum this lane ended with
            if (row < GDC) {
                sP[row * COLS + wc + e] = acc[0];
            } else {
                const int t = row - GDC;
                float o = acc[0];
#pragma unroll
                for (int j = 0; j < GDC; j += 4) {
                    const float4 w = *reinterpret_cast<const float4*>(sE + t * GDC + j);
                    o = fmaf(w.x, sV[j * COLS + wc + e], o);
                    o = fmaf(w.y, sV[(j + 1) * COLS + wc + e], o);
                    o = fmaf(w.z, sV[(j + 2) * COLS + wc + e], o);
                    o = fmaf(w.w, sV[(j + 3) * COLS + wc + e], o);
                }
                if (t < nt && col0 + wc + e < Dv)
                    asm volatile("st.global.f32 [%0], %1;" ::"l"(p.out + ((size_t)(row0 + ch * GDC + t) * heads + hd) * Dv + col0 + wc + e), "f"(o));
            }
        }
        __syncwarp();                                      // a warp reads back its own columns of sP
        // S <- diag(W) S + G^T V - A'^T (B' S)
#pragma unroll
        for (int i = 0; i < DS; i += 4) {
            const float4 w = *reinterpret_cast<const float4*>(m + 4 * GDC * DP + d0 + i);
#pragma unroll
            for (int e = 0; e < CPT; ++e) { S[e][i] *= w.x; S[e][i + 1] *= w.y; S[e][i + 2] *= w.z; S[e][i + 3] *= w.w; }
        }
#pragma unroll
        for (int j = 0; j < GDC; ++j) {
            float v[CPT], q[CPT];
            if constexpr (CPT == 4) {                      // (wc is a multiple of 4)
                const float4 vv = *reinterpret_cast<const float4*>(sV + j * COLS + wc), qq = *reinterpret_cast<const float4*>(sP + j * COLS + wc);
                v[0] = vv.x; v[1] = vv.y; v[2] = vv.z; v[3] = vv.w;
                q[0] = -qq.x; q[1] = -qq.y; q[2] = -qq.z; q[3] = -qq.w;
            } else {
#pragma unroll
                for (int e = 0; e < CPT; ++e) { v[e] = sV[j * COLS + wc + e]; q[e] = -sP[j * COLS + wc + e]; }
            }
#pragma unroll
            for (int i = 0; i < DS; i += 4) {
                const float4 g = *reinterpret_cast<const float4*>(m + (2 * GDC + j) * DP + d0 + i), a = *reinterpret_cast<const float4*>(m + (3 * GDC + j) * DP + d0 + i);
#pragma unroll
                for (int e = 0; e < CPT; ++e) {
                    S[e][i] = fmaf(g.x, v[e], fmaf(a.x, q[e], S[e][i]));
                    S[e][i + 1] = fmaf(g.y, v[e], fmaf(a.y, q[e], S[e][i + 1]));
                    S[e][i + 2] = fmaf(g.z, v[e], fmaf(a.z, q[e], S[e][i + 2]));
                    S[e][i + 3] = fmaf(g.w, v[e], fmaf(a.w, q[e], S[e][i + 3]));
                }
            }
        }
        __syncthreads();                                   // before the next fetch overwrites this buffer
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int e = 0; e < CPT; ++e)
#pragma unroll
        for (int i = 0; i < DS; i += 4)
            if (live[e] && d0 + i < D)
                *reinterpret_cast<float4*>(p.state + cell[e] + i) = make_float4(S[e][i], S[e][i + 1], S[e][i + 2], S[e][i + 3]);
}

extern "C" int cml_delta_chunk_scan(const float* chunks, float* state, const int* seq_row0, const int* seq_new, const int* seq_start,
                                    const int* seq_slot, float* out, int n_seqs, int heads, int D, int Dv, void* stream) {
    if (n_seqs <= 0) return 0;
    if (heads < 1 || heads > 65535 || D < 4 || D > 256 || (D & 3) || Dv < 4 || (Dv & 3)) return CML_ERR_BAD_SIZE;
    if ((((uintptr_t)chunks) | ((uintptr_t)state)) & 15) return CML_ERR_BAD_ALIGN;
    ChunkScan p = {chunks, state, seq_new, seq_row0, seq_start, seq_slot, out, heads, D, Dv};
#define CS_CASE(DS_, NS_, CPT_, WARPS_)                                                                                            \
    if (D <= NS_ * DS_) {                                                                                                          \
        constexpr int COLS = WARPS_ * (32 / NS_) * CPT_;                                                                           \
        constexpr size_t smem = (size_t)(2 * ((4 * GDC + 1) * NS_ * DS_ + GDC * GDC + GDC * COLS) + GDC * COLS) * sizeof(float);   \
        if (smem > 48 * 1024 && cml_allow_smem<delta_chunk_scan_kernel<DS_, NS_, CPT_, WARPS_>>(smem) != cudaSuccess) return CML_ERR_BAD_SIZE; \
        launch_pdl(delta_chunk_scan_kernel<DS_, NS_, CPT_, WARPS_>, dim3(n_seqs, heads, (Dv + COLS - 1) / COLS), dim3(WARPS_ * 32), smem, \
                   (cudaStream_t)stream, p);                                                                                       \
        return cml_launch_status();                                                                                                \
    }
    CS_CASE(4, 8, 2, 2) CS_CASE(4, 16, 2, 4) CS_CASE(4, 32, 4, 4) CS_CASE(8, 32, 4, 4)
#undef CS_CASE
    return CML_ERR_BAD_SIZE;
}

// ------------------------------------------------------------------------------------
// The gated delta rule (unit keys k, decays g per key channel or per head, beta) by chunks of GDL = 32 tokens. With W_t the product of the
// chunk's decays up to t, S the state before the chunk and z_t = beta_t (v_t - k_t^T of the decayed state) what token t writes,
//
//   A[t][j] = sum_d k_t k_j g_(j+1) .. g_t  (j < t),    B[t][j] likewise with q_t  (j <= t)
//   z_t = beta_t (v_t - (k_t W_t)^T S - sum over j < t of A[t][j] z_j)       =>  Z = U - Y S
//   o_t = (q_t W_t)^T S + sum over j <= t of B[t][j] z_j                     =>  O = B U + R S,   R = q W - B Y
//   S <- diag(W) S + sum over j of (k_j g_(j+1) .. g_last) z_j^T
//
// where U and Y solve (I + diag(beta) A) X = diag(beta) (V | k W). No decay is ever divided by: products of decays run from j + 1 on
// forward (or backward from the last), so that none overflows however fast the state fades. The first kernel makes Y, R, the faded keys, W, U
// and B U of all (chunk, head) side by side; the second walks a sequence's chunks with the state in registers. All in float.
// 16 heads of 128 x 128, a prompt of 2,048 tokens: 770 us a layer by the scan inside a decoder (700 alone) -> 303: chunks 101, walk 202.
// Distance from 64 bits beside the scan's: 1.2e-7 to 1.5e-7 (0.9e-7 to 1.25e-7).
#define GDL 32
#define GDL_PITCH 36         // floats of a row of a 32 x 32 matrix in shared memory
#define GDL_FLOATS(D, Dv) ((size_t)(3 * GDL + 1) * (D) + 2 * GDL * (Dv))      // Y and R channel by channel (2 GDL rows each), faded keys, W, U, B U of a (chunk, head)

struct GatedChunks {
    const float* qkv; long ld;                             // unit q (qk_heads x D), unit k, v (heads x Dv)
    const float* beta; long ldb; int beta_col;             // before the sigmoid
    const float* decay; int decay_dim;                     // [rows, heads x decay_dim]
    const int* tile_seq; const int* tile_q0; const int* seq_row0; const int* seq_new; const int* seq_start; const int* seq_slot;
    float* chunks; float* state; float* out;
    int heads, qk_heads, D, Dv;
    int least;                                             // as in SsmChunks
};

// 128 threads; D <= 128: a lane has four channels where a warp works on a pair of tokens, a thread one channel or value elsewhere
__global__ void __launch_bounds__(128) gated_chunks_kernel(const GatedChunks p) {
    constexpr int DP = 128;
    extern __shared__ __align__(16) float gc_sh[];
    __shared__ __align__(16) float sA[GDL][GDL_PITCH], sB[GDL][GDL_PITCH];
    __shared__ float s_beta[GDL];
    pdl_wait();
    pdl_launch_dependents();
    const int tile = blockIdx.x, hd = blockIdx.y, D = p.D, Dv = p.Dv, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int seq = p.tile_seq[tile], q0 = p.tile_q0[tile], nt = min(GDL, p.seq_new[seq] - q0), row0 = p.seq_row0[seq] + q0;
    const int g = hd / (p.heads / p.qk_heads);
    float* sq = gc_sh;                                     // [GDL][DP]: q, k, the decays; zero (one) where there is no token or channel
    float* sk = sq + GDL * DP;
    float* sg = sk + GDL * DP;
    const float* qkv = p.qkv + (size_t)row0 * p.ld;
    float* out = p.chunks + ((size_t)tile * p.heads + hd) * GDL_FLOATS(D, Dv);
    {
        const int d = tid;
        const bool in = d < D;
#pragma unroll 8
        for (int t = 0; t < GDL; ++t) {
            const size_t r = min(t, nt - 1);
            const bool ok = in && t < nt;
            const float q = qkv[r * p.ld + g * D + (in ? d : 0)], k = qkv[r * p.ld + (p.qk_heads + g) * D + (in ? d : 0)];
            const float w = p.decay[(row0 + r) * p.heads * p.decay_dim + hd * p.decay_dim + (in && p.decay_dim > 1 ? d : 0)];
            sq[t * DP + d] = ok ? q : 0.f;
            sk[t * DP + d] = ok ? k : 0.f;
            sg[t * DP + d] = ok ? w : 1.f;
        }
        if (tid < GDL) s_beta[tid] = tid < nt ? sigmoid_f(p.beta[(size_t)(row0 + tid) * p.ldb + p.beta_col + hd]) : 0.f;
        for (int i = tid; i < GDL * GDL_PITCH; i += 128) { (&sA[0][0])[i] = 0.f; (&sB[0][0])[i] = 0.f; }
    }
    __syncthreads();
    // A and B column by column: a warp takes j and walks t, eight tokens' sums at a time
    for (int j = warp; j < GDL; j += 4) {
        float4 x = *reinterpret_cast<const float4*>(sk + j * DP + lane * 4);
        for (int t0 = j & ~7; t0 < GDL; t0 += 8) {
            float acc[16];                                 // A of the eight tokens, then B
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int t = t0 + u;
                const float4 w = *reinterpret_cast<const float4*>(sg + t * DP + lane * 4), k = *reinterpret_cast<const float4*>(sk + t * DP + lane * 4),
                             q = *reinterpret_cast<const float4*>(sq + t * DP + lane * 4);
                if (t > j) { x.x *= w.x; x.y *= w.y; x.z *= w.z; x.w *= w.w; }
                acc[u] = t > j ? fmaf(k.x, x.x, fmaf(k.y, x.y, fmaf(k.z, x.z, k.w * x.w))) : 0.f;
                acc[8 + u] = t >= j ? fmaf(q.x, x.x, fmaf(q.y, x.y, fmaf(q.z, x.z, q.w * x.w))) : 0.f;
            }
#pragma unroll
            for (int h = 8; h > 0; h >>= 1) {              // lane bit h keeps the upper half of what is left
                const bool up = (lane & h) != 0;
#pragma unroll
                for (int i = 0; i < h; ++i) {
                    const float give = up ? acc[i] : acc[i + h], keep = up ? acc[i + h] : acc[i];
                    acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, h);
                }
            }
            const float v = acc[0] + __shfl_xor_sync(0xffffffffu, acc[0], 16);
            if (lane < 8) sA[t0 + lane][j] = v;
            else if (lane < 16) sB[t0 + lane - 8][j] = v;
        }
    }
    __syncthreads();
    // x <- (I + diag(beta) A)^-1 diag(beta) x for a column x, and sums of a row of B with it
    float x[GDL];
    auto solve = [&]() {
#pragma unroll
        for (int t = 0; t < GDL; ++t) {
            float v[4] = {x[t], 0.f, 0.f, 0.f};            // four chains, always in this order
#pragma unroll
            for (int j = 0; j < t; j += 4) {
                const float4 a = *reinterpret_cast<const float4*>(&sA[t][j]);          // (zero from t on)
                v[0] = fmaf(-a.x, x[j], v[0]);
                if (j + 1 < t) v[1] = fmaf(-a.y, x[j + 1], v[1]);
                if (j + 2 < t) v[2] = fmaf(-a.z, x[j + 2], v[2]);
                if (j + 3 < t) v[3] = fmaf(-a.w, x[j + 3], v[3]);
            }
            x[t] = s_beta[t] * ((v[0] + v[1]) + (v[2] + v[3]));
            asm volatile("" ::: "memory");                 // a row's loads stay with their row: all rows' at once would not fit the registers
        }
    };
    auto read = [&](int t) -> float {
        float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < GDL; j += 4) {
            if (j > t) break;
            const float4 b = *reinterpret_cast<const float4*>(&sB[t][j]);
            v[0] = fmaf(b.x, x[j], v[0]);                  // (later tokens are left out, not multiplied by zero: theirs may be no numbers)
            if (j + 1 <= t) v[1] = fmaf(b.y, x[j + 1], v[1]);
            if (j + 2 <= t) v[2] = fmaf(b.z, x[j + 2], v[2]);
            if (j + 3 <= t) v[3] = fmaf(b.w, x[j + 3], v[3]);
        }
        if ((t & 3) == 3) asm volatile("" ::: "memory");
        return (v[0] + v[1]) + (v[2] + v[3]);
    };
    if (tid < D) {
        const int d = tid;
        float w = 1.f;
#pragma unroll
        for (int t = 0; t < GDL; ++t) {
            w *= sg[t * DP + d];
            x[t] = sk[t * DP + d] * w;
        }
        out[3 * GDL * D + d] = w;
        solve();
        w = 1.f;
        float4* o = reinterpret_cast<float4*>(out + (size_t)d * 2 * GDL);
#pragma unroll
        for (int t = 0; t < GDL; t += 4) {
            float r[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                w *= sg[(t + u) * DP + d];
                r[u] = fmaf(sq[(t + u) * DP + d], w, -read(t + u));
            }
            o[t / 4] = make_float4(x[t], x[t + 1], x[t + 2], x[t + 3]);
            o[(GDL + t) / 4] = make_float4(r[0], r[1], r[2], r[3]);
        }
        w = 1.f;
#pragma unroll 8
        for (int t = GDL - 1; t >= 0; --t) {
            out[(2 * GDL + t) * D + d] = sk[t * DP + d] * w;
            w *= sg[t * DP + d];
        }
    }
    for (int e = tid; e < Dv; e += 128) {
        const float* v = qkv + 2 * p.qk_heads * D + hd * Dv + e;
#pragma unroll
        for (int t = 0; t < GDL; ++t) {
            const float u = v[(size_t)min(t, nt - 1) * p.ld];
            x[t] = t < nt ? u : 0.f;
        }
        solve();
        float* o = out + (3 * GDL + 1) * D + e;
#pragma unroll
        for (int t = 0; t < GDL; ++t) {
            o[t * Dv] = x[t];
            o[(GDL + t) * Dv] = read(t);
        }
    }
}

// The walk: a block has 16 columns of the state of one (sequence, head) and takes two products a chunk, both as tiles of registers over
// operands in shared memory: Y and R times the state (four rows by two columns a thread, 128 channels deep), and the faded keys times Z (four
// channels by four columns, 32 tokens deep), whose sums are the state itself. Between the two the state and Z pass through shared memory,
// every number twice, as the packed multiply-adds want one operand. The next chunk comes by cp.async into the other buffer meanwhile.
// One warp a scheduler has to hide the latency of shared memory by itself: the operands of the next channels (tokens) are asked for, in
// so many words, while the ones before are multiplied (202 us; 325 with the loads left to the compiler, which put each right before
// its use; 330 to 377 with the state in a warp's lanes and sums added over the lanes by shuffles).
#define GDW_COLS 16
#define GDW_BUF ((3 * GDL + 1) * 128 + 2 * GDL * GDW_COLS)
#define GDW_SP 36                                          // floats of a channel's columns in shared memory, padded
__device__ __forceinline__ unsigned long long gdw_mul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long gdw_add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// 16 bytes of shared memory; the loads stay in the order and the place in which they are written
__device__ __forceinline__ SsmQuad gdw_load(uint32_t at) {
    SsmQuad v;
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.lo), "=l"(v.hi) : "r"(at));
    return v;
}
__device__ __forceinline__ float gdw_lo(unsigned long long v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float gdw_hi(unsigned long long v) { return __uint_as_float((unsigned)(v >> 32)); }
__global__ void __launch_bounds__(128) gated_walk_kernel(const GatedChunks p) {
    constexpr int DP = 128;
    extern __shared__ __align__(16) float gw_sh[];
    const int D = p.D, Dv = p.Dv, heads = p.heads;
    float* sS = gw_sh + 2 * GDW_BUF;                       // [DP][GDW_SP]: the state, channel by channel, each value twice
    float* sZ = sS + DP * GDW_SP;                          // [GDL][2 GDW_COLS]: Z, each value twice
    pdl_wait();
    pdl_launch_dependents();
    const int s = blockIdx.x, hd = blockIdx.y, col0 = blockIdx.z * GDW_COLS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n = p.seq_new[s], row0 = p.seq_row0[s], n_chunks = (n + GDL - 1) / GDL;
    const bool fresh = p.seq_start[s] == 0;
    if (n < p.least) return;
    const int first = first_tile_of(p.seq_new, s, GDL, p.least);
    const int r0 = (warp * 4 + (lane >> 3)) * 4, cp = (lane & 7) * 2;          // the first product: rows of Y | R, columns
    const int d0 = (warp * 8 + (lane & 7)) * 4, cq = (lane >> 3) * 4;          // the second: channels, columns
    SsmQuad S[4];                                          // by column: four channels
    float* st = p.state + (((size_t)p.seq_slot[s] * heads + hd) * Dv + col0 + cq) * D + d0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        S[c] = {0ull, 0ull};
        if (!fresh && d0 < D && col0 + cq + c < Dv) S[c] = ssm_quad(st + (size_t)c * D);
    }
    if (D < DP || Dv - col0 < GDW_COLS) {                  // channels and columns that are not there stay zero
        for (int i = tid; i < 2 * GDW_BUF; i += 128) gw_sh[i] = 0.f;
        __syncthreads();
    }
    auto fetch = [&](int ch) {
        const float* src = p.chunks + ((size_t)(first + ch) * heads + hd) * GDL_FLOATS(D, Dv);
        float* dst = gw_sh + (ch & 1) * GDW_BUF;
        if (D == DP) {                                     // Y and R, the faded keys and W in one run of memory
            for (int i = tid * 4; i < (3 * GDL + 1) * DP; i += 512) gd_copy<16>(dst + i, src + i);
        } else {
            for (int i = tid * 4; i < 2 * GDL * D; i += 512) gd_copy<16>(dst + i, src + i);
            for (int r = 2 * GDL + warp; r < 3 * GDL + 1; r += 4)
                if (lane * 4 < D) gd_copy<16>(dst + r * DP + lane * 4, src + (size_t)r * D + lane * 4);
        }
        const float* v = src + (size_t)(3 * GDL + 1) * D + col0;
        for (int i = tid; i < 2 * GDL * GDW_COLS / 4; i += 128) {
            const int t = i / (GDW_COLS / 4), e = (i % (GDW_COLS / 4)) * 4;
            if (col0 + e < Dv) gd_copy<16>(dst + (3 * GDL + 1) * DP + t * GDW_COLS + e, v + (size_t)t * Dv + e);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto share = [&]() {                                   // the state for the first product
#pragma unroll
        for (int c = 0; c < 4; c += 2) {
            const float a[4] = {gdw_lo(S[c].lo), gdw_hi(S[c].lo), gdw_lo(S[c].hi), gdw_hi(S[c].hi)};
            const float b[4] = {gdw_lo(S[c + 1].lo), gdw_hi(S[c + 1].lo), gdw_lo(S[c + 1].hi), gdw_hi(S[c + 1].hi)};
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *reinterpret_cast<float4*>(sS + (d0 + i) * GDW_SP + (cq + c) * 2) = make_float4(a[i], a[i], b[i], b[i]);
        }
    };
    fetch(0);
    share();
    for (int ch = 0; ch < n_chunks; ++ch) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                   // this chunk and the state are here, the other buffer is free
        if (ch + 1 < n_chunks) fetch(ch + 1);
        const float* m = gw_sh + (ch & 1) * GDW_BUF;
        const int nt = min(GDL, n - ch * GDL);
        // [column][rows r0, r0 + 1 | r0 + 2, r0 + 3], every fourth eight channels in sums of their own, added at the end: one chain of 128 would round
        // each of its sums at the size of the whole
        unsigned long long part[4][2][2], acc[2][2];
#pragma unroll
        for (int i = 0; i < 16; ++i) (&part[0][0][0])[i] = 0ull;
        {   // eight channels' operands in registers while the next eight are on their way
            const uint32_t ya = (uint32_t)__cvta_generic_to_shared(m + r0), xa = (uint32_t)__cvta_generic_to_shared(sS + cp * 2);
            SsmQuad y[2][8], x[2][8];
#pragma unroll
            for (int u = 0; u < 8; ++u) { y[0][u] = gdw_load(ya + u * 2 * GDL * 4); x[0][u] = gdw_load(xa + u * GDW_SP * 4); }
#pragma unroll
            for (int k = 0; k < DP; k += 8) {
                const int b = (k >> 3) & 1;
                if (k + 8 < DP) {
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        y[b ^ 1][u] = gdw_load(ya + (k + 8 + u) * 2 * GDL * 4);
                        x[b ^ 1][u] = gdw_load(xa + (k + 8 + u) * GDW_SP * 4);
                    }
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    unsigned long long (&a)[2][2] = part[(k >> 3) & 3];
                    ssm_fma2(a[0][0], y[b][u].lo, x[b][u].lo); ssm_fma2(a[0][1], y[b][u].hi, x[b][u].lo);
                    ssm_fma2(a[1][0], y[b][u].lo, x[b][u].hi); ssm_fma2(a[1][1], y[b][u].hi, x[b][u].hi);
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int r = 0; r < 2; ++r) acc[c][r] = gdw_add2(gdw_add2(part[0][c][r], part[1][c][r]), gdw_add2(part[2][c][r], part[3][c][r]));
        const float* add = m + (3 * GDL + 1) * DP + r0 * GDW_COLS + cp;        // U, then B U
        const float a[4] = {gdw_lo(acc[0][0]), gdw_hi(acc[0][0]), gdw_lo(acc[0][1]), gdw_hi(acc[0][1])};
        const float b[4] = {gdw_lo(acc[1][0]), gdw_hi(acc[1][0]), gdw_lo(acc[1][1]), gdw_hi(acc[1][1])};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 u = *reinterpret_cast<const float2*>(add + i * GDW_COLS);
            if (warp < 2) {
                *reinterpret_cast<float4*>(sZ + (r0 + i) * 2 * GDW_COLS + cp * 2) = make_float4(u.x - a[i], u.x - a[i], u.y - b[i], u.y - b[i]);
            } else if (r0 + i - GDL < nt) {
                float* o = p.out + ((size_t)(row0 + ch * GDL + r0 + i - GDL) * heads + hd) * Dv + col0 + cp;
                if (col0 + cp < Dv) o[0] = u.x + a[i];     // (Dv is a multiple of 4: two columns are there together)
                if (col0 + cp + 1 < Dv) o[1] = u.y + b[i];
            }
        }
        __syncthreads();                                   // Z is here, the state's copy has been read
        const SsmQuad w = ssm_quad(m + 3 * GDL * DP + d0);
#pragma unroll
        for (int c = 0; c < 4; ++c) { S[c].lo = gdw_mul2(S[c].lo, w.lo); S[c].hi = gdw_mul2(S[c].hi, w.hi); }
        {
            const uint32_t ka = (uint32_t)__cvta_generic_to_shared(m + 2 * GDL * DP + d0), za = (uint32_t)__cvta_generic_to_shared(sZ + cq * 2);
            SsmQuad k[2][4], z[2][4][2];
            auto ask = [&](int b, int j) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    k[b][u] = gdw_load(ka + (j + u) * DP * 4);
                    z[b][u][0] = gdw_load(za + (j + u) * 2 * GDW_COLS * 4);
                    z[b][u][1] = gdw_load(za + (j + u) * 2 * GDW_COLS * 4 + 16);
                }
            };
            ask(0, 0);
#pragma unroll
            for (int j = 0; j < GDL; j += 4) {
                const int b = (j >> 2) & 1;
                if (j + 4 < GDL) ask(b ^ 1, j + 4);
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const unsigned long long zz = (c & 1) ? z[b][u][c >> 1].hi : z[b][u][c >> 1].lo;
                        ssm_fma2(S[c].lo, k[b][u].lo, zz);
                        ssm_fma2(S[c].hi, k[b][u].hi, zz);
                    }
            }
        }
        share();
    }
    if (d0 >= D) return;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        if (col0 + cq + c < Dv) *reinterpret_cast<ulonglong2*>(st + (size_t)c * D) = make_ulonglong2(S[c].lo, S[c].hi);
}

// qkv, beta and the decays (ready) as for cml_delta_scan; chunks: scratch of GDL_FLOATS(D, Dv) floats per (tile of 32 rows, head).
extern "C" int cml_gated_chunks(const float* qkv, long ldq, const float* beta_in, long ldb, int beta_col, const float* decay, int decay_dim,
                                const int* tile_seq, const int* tile_q0, int n_tiles, const int* seq_row0, const int* seq_new,
                                const int* seq_start, const int* seq_slot, float* chunks, float* state, float* out, int n_seqs, int heads,
                                int qk_heads, int D, int Dv, int least, void* stream) {
    if (n_tiles <= 0 || n_seqs <= 0) return 0;
    if (heads < 1 || heads > 65535 || qk_heads < 1 || heads % qk_heads || (decay_dim != 1 && decay_dim != D)) return CML_ERR_BAD_SIZE;
    if (D < 4 || D > 128 || (D & 3) || Dv < 4 || (Dv & 3) || (Dv + GDW_COLS - 1) / GDW_COLS > 65535) return CML_ERR_BAD_SIZE;
    if ((((uintptr_t)chunks) | ((uintptr_t)state)) & 15) return CML_ERR_BAD_ALIGN;
    GatedChunks p = {qkv, ldq, beta_in, ldb, beta_col, decay, decay_dim, tile_seq, tile_q0, seq_row0, seq_new, seq_start, seq_slot, chunks,
                     state, out, heads, qk_heads, D, Dv, least};
    cudaStream_t s = (cudaStream_t)stream;
    constexpr size_t smem = (size_t)3 * GDL * 128 * sizeof(float), smem_walk = (size_t)(2 * GDW_BUF + 128 * GDW_SP + 2 * GDL * GDW_COLS) * sizeof(float);
    if (cml_allow_smem<gated_chunks_kernel>(smem) != cudaSuccess || cml_allow_smem<gated_walk_kernel>(smem_walk) != cudaSuccess) return CML_ERR_BAD_SIZE;
    launch_pdl(gated_chunks_kernel, dim3(n_tiles, heads), dim3(128), smem, s, p);
    launch_pdl(gated_walk_kernel, dim3(n_seqs, heads, (Dv + GDW_COLS - 1) / GDW_COLS), dim3(128), smem_walk, s, p);
    return cml_launch_status();
}

// ------------------------------------------------------------------------------------
// Rotation of heads inside float rows, in place: x [rows, ld] holds `heads` heads of D channels from column col0; the
// first rot_dim channels of every head are turned by angle = position * inv_freq[i] (pairing 1: channels (2i, 2i + 1);
// 0: channels (i, i + rot_dim / 2)), sines and cosines times `amp`; then heads from number `scaled_from` on are
// multiplied by `scale` (all their channels). A warp owns one (row, head); both members of a pair are read before
// either is written.
__global__ void rotate_rows_kernel(float* __restrict__ x, long ld, int col0, int rows, int heads, int D, int rot_dim,
                                   int pairing, const float* __restrict__ inv_freq, float amp, const int* __restrict__ row_pos,
                                   int scaled_from, float scale) {
    pdl_wait();
    pdl_launch_dependents();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= rows * heads) return;
    const int r = warp / heads, hd = warp % heads;
    float* h = x + (size_t)r * ld + col0 + (size_t)hd * D;
    const float pos = (float)row_pos[r];
    const float mul = hd >= scaled_from ? scale : 1.0f;
    const int half = rot_dim / 2;
    for (int i = lane; i < half; i += 32) {
        const int a = pairing ? 2 * i : i, b = pairing ? 2 * i + 1 : i + half;
        float sn, cs;
        sincosf(pos * inv_freq[i], &sn, &cs);
        sn *= amp; cs *= amp;
        const float u = h[a], v = h[b];
        h[a] = (u * cs - v * sn) * mul;
        h[b] = (v * cs + u * sn) * mul;
    }
    if (mul != 1.0f)
        for (int c = rot_dim + lane; c < D; c += 32) h[c] *= mul;
}

extern "C" int cml_rotate_rows(float* x, long ld, int col0, int rows, int heads, int D, int rot_dim, int pairing,
                               const float* inv_freq, float amp, const int* row_pos, int scaled_from, float scale, void* stream) {
    if (rows <= 0 || heads <= 0) return 0;
    if (rot_dim < 0 || rot_dim > D || (rot_dim & 1)) return CML_ERR_BAD_SIZE;
    const long warps = (long)rows * heads;
    launch_pdl(rotate_rows_kernel, dim3((unsigned)((warps + 3) / 4)), dim3(128), 0, (cudaStream_t)stream, x, ld, col0, rows, heads,
               D, rot_dim, pairing, inv_freq, amp, row_pos, scaled_from, scale);
    return cml_launch_status();
}

// ------------------------------------------------------------------------------------
// After a scan: per (row, head) o = raw / den (den = max(|n . q|, exp(-m)) + 1e-6 where the
// raw rows carry them, else 1), y = o / sqrt(mean(o^2) + eps) * w * sigmoid(gate) (or * silu(gate)), written in
// the compute type for the output projection. A warp owns one (row, head). raw [rows, heads, ldh]
// with ldh = Dv (+ 2 with a denominator); w [Dv] shared by the heads (w_head_stride 0) or
// [heads x Dv]; gate [rows, ldg] at column gate_col + head * Dv. Heads of up to 128 channels: everything a lane needs is
// asked for at once, into registers (row, then gate and weight behind the row's sum, were two trips to memory: 3.7 us -> 2.0 in a step's chain).
template <typename TO>
__global__ void head_norm_gate_kernel(const float* __restrict__ raw, int ldh, int with_den, const float* __restrict__ w,
                                      int w_head_stride, const float* __restrict__ gate, long ldg, int gate_col,
                                      TO* __restrict__ out, long ldo, int rows, int heads, int Dv, float eps, int gate_silu) {
    pdl_wait();
    pdl_launch_dependents();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= rows * heads) return;
    const int r = warp / heads, hd = warp % heads;
    const float* x = raw + ((size_t)r * heads + hd) * ldh;
    const float* wv = w ? w + (size_t)hd * w_head_stride : nullptr;      // null: a norm without weight
    const float* gt = gate + (size_t)r * ldg + gate_col + hd * Dv;
    TO* o = out + (size_t)r * ldo + (size_t)hd * Dv;
    float inv = 1.0f, den = 0.f, neg = 0.f;
    if (with_den) den = x[Dv], neg = x[Dv + 1];
    float ss = 0.f;
    if (Dv > 0 && Dv <= 128) {
        float v[4], g[4], m[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int c = min(lane + 32 * e, Dv - 1);
            v[e] = x[c];
            g[e] = gt[c];
            m[e] = wv ? wv[c] : 1.0f;
        }
        if (with_den) inv = 1.0f / (fmaxf(fabsf(den), expf(-neg)) + 1e-6f);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float q = v[e] * inv;
            if (lane + 32 * e < Dv) ss = fmaf(q, q, ss);
        }
        ss = warp_sum(ss);
        const float scale = inv / sqrtf(ss / (float)Dv + eps);
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (lane + 32 * e < Dv) o[lane + 32 * e] = from_f32<TO>(v[e] * scale * m[e] * (gate_silu ? silu_f(g[e]) : sigmoid_f(g[e])));
        return;
    }
    if (with_den) inv = 1.0f / (fmaxf(fabsf(den), expf(-neg)) + 1e-6f);
    for (int c = lane; c < Dv; c += 32) {
        const float o = x[c] * inv;
        ss = fmaf(o, o, ss);
    }
    ss = warp_sum(ss);
    const float scale = inv / sqrtf(ss / (float)Dv + eps);
    for (int c = lane; c < Dv; c += 32) o[c] = from_f32<TO>(x[c] * scale * (wv ? wv[c] : 1.0f) * (gate_silu ? silu_f(gt[c]) : sigmoid_f(gt[c])));
}

extern "C" int cml_head_norm_gate(const float* raw, int ldh, int with_den, const float* w, int w_head_stride, const float* gate,
                                  long ldg, int gate_col, void* out, long ldo, int out_dtype, int rows, int heads, int Dv, float eps,
                                  int gate_silu, void* stream) {
    if (rows <= 0) return 0;
    const long warps = (long)rows * heads;
    dim3 grid((unsigned)((warps + 3) / 4));
    cudaStream_t s = (cudaStream_t)stream;
    if (out_dtype == CML_DTYPE_F32)
        launch_pdl(head_norm_gate_kernel<float>, grid, dim3(128), 0, s, raw, ldh, with_den, w, w_head_stride, gate, ldg, gate_col,
                   (float*)out, ldo, rows, heads, Dv, eps, gate_silu);
    else if (out_dtype == CML_DTYPE_BF16)
        launch_pdl(head_norm_gate_kernel<bf16>, grid, dim3(128), 0, s, raw, ldh, with_den, w, w_head_stride, gate, ldg, gate_col,
                   (bf16*)out, ldo, rows, heads, Dv, eps, gate_silu);
    else
        return CML_ERR_BAD_DTYPE;
    return cml_launch_status();
}
