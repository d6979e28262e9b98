// Q8_0F x f32 GEMV, one activation vector: the reference's default quantisation pair (f32 block scales, f32
// activations) in a decode step.  Same role as the general GEMV of matmul_simt.cu (crates/ratchet-core/src/ops/gemv.rs:181-331),
// and the same products: every weight is (f32)code * scale rounded to f32 (quant.rs:114-120), multiplied into the sum by fma.
//
// HBM-bound: 36 bytes per 32 weights.  What the general kernel lost (11.5 us on [10240, 2560], 20.6 us on
// [2560, 10240], for 4.4 us of bytes):
//  * int8 -> f32 conversions run at a fraction of the FMA rate; here a code becomes a float by one byte permute into
//    2^23's mantissa and half of a packed add (exact), and product and sum are packed pairs (fma.rn.f32x2);
//  * a warp walked a whole row, up to twenty dependent steps; here the CTA's warps share the K range of four rows, one
//    or two steps of 512 values each, so nearly all bytes of a node are requested at once, and the x of a step is loaded
//    once for four rows;
//  * constant weights are requested before the kernel waits for its stream predecessor (programmatic dependent launch).
// The warps' sums meet in shared memory in warp order: deterministic.
#include <algorithm>

#include "common.cuh"
#include "f32x2.cuh"
#include "kernels.hpp"

namespace rt {

namespace {

constexpr int ROWS = 4;
constexpr int MAX_WARPS = 10;
constexpr int CHUNK = 512; // K values per warp and step: 16 codes per lane

__global__ void __launch_bounds__(MAX_WARPS * 32, 3) q8f_gemv_f32_kernel(MatmulParams p, int lhs_constant) {
    __shared__ float part[MAX_WARPS][ROWS];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!lhs_constant) asm volatile("griddepcontrol.wait;" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int row0 = blockIdx.x * ROWS, batch = blockIdx.z;
    const long long lb = batch % p.lhs_stack;
    const uint8_t *codes = (const uint8_t *)p.lhs + lb * p.lhs_batch_elems;
    const float *scales = (const float *)((const uint8_t *)p.lhs_scales + lb * p.lhs_batch_scale_bytes);
    const float *x = (const float *)p.rhs + (long long)(batch % p.rhs_stack) * p.K;

    uint4 q[ROWS];
    float d[ROWS];
    auto load = [&](int k) { // rows past the end repeat the last one and are not stored
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const long long at = (long long)min(row0 + r, p.M - 1) * p.K + k;
            q[r] = ldg_stream(codes + at);
            d[r] = __ldg(scales + (at >> 5));
        }
    };
    int k = warp * CHUNK + lane * 16;
    if (k < p.K) load(k);
    if (lhs_constant) asm volatile("griddepcontrol.wait;" ::: "memory");

    unsigned long long acc[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; r++) acc[r] = 0ull;
    const unsigned long long bias2 = pack2f(-8388736.f, -8388736.f); // 2^23 + 128
    while (k < p.K) {
        unsigned long long xv[8]; // written by the predecessor: plain loads, after the wait
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(x + k + 4 * j);
            xv[2 * j] = v.x;
            xv[2 * j + 1] = v.y;
        }
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const uint32_t w[4] = {q[r].x ^ 0x80808080u, q[r].y ^ 0x80808080u, q[r].z ^ 0x80808080u, q[r].w ^ 0x80808080u};
            const unsigned long long dd = pack2f(d[r], d[r]);
#pragma unroll
            for (int j = 0; j < 8; j++) acc[r] = fma2(mul2(add2(bytes2f(w[j >> 1], j & 1), bias2), dd), xv[j], acc[r]);
        }
        k += warps * CHUNK;
        if (k < p.K) load(k);
    }

    float sum[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
        sum[r] = sum2(acc[r]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], o);
    }
    if (lane == 0) {
#pragma unroll
        for (int r = 0; r < ROWS; r++) part[warp][r] = sum[r];
    }
    __syncthreads();
    const int row = row0 + (int)threadIdx.x;
    if (threadIdx.x < ROWS && row < p.M) {
        float s = part[0][threadIdx.x];
        for (int w = 1; w < warps; w++) s += part[w][threadIdx.x];
        const bool has_bias = p.bias_mode != BIAS_NONE;
        float bias = 0.f;
        if (has_bias) bias = load_bias(p.bias, p.bias_dt, p.bias_mode == BIAS_PER_M ? row : 0);
        ((float *)p.out)[(long long)batch * p.M + row] = epilogue_value<float>(s, has_bias, bias, p.epilogue);
    }
}

} // namespace

// Warps per CTA: the chunks of a row in as few equal steps as MAX_WARPS allows.
cudaError_t launch_q8f_gemv_f32(const MatmulParams &p, bool lhs_constant, cudaStream_t stream) {
    const int chunks = (p.K + CHUNK - 1) / CHUNK;
    const int steps = (chunks + MAX_WARPS - 1) / MAX_WARPS;
    const int warps = (chunks + steps - 1) / steps;
    return launch_pdl(q8f_gemv_f32_kernel, dim3((p.M + ROWS - 1) / ROWS, 1, p.stacks), dim3(warps * 32), 0, stream, p, lhs_constant ? 1 : 0);
}

} // namespace rt
