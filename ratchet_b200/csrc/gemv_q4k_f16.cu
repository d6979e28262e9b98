// Q4_K x f16 GEMV, one activation vector: a decode step against 4-bit weights.
//
// HBM-bound by size: 144 bytes per 256 weights.  The warp-MMA kernel (gemv_q4k_mma.cu), made for up to 16 vectors, spends a
// launch on latencies in a row: weights and activations staged in shared memory, a table of scales, the MMAs, two
// reductions and, for long rows, two cluster barriers.  With one vector nothing is reused but x, so here the nibbles go
// from global memory to registers to the sum:
//  * a warp takes 1024 values of four rows: a lane has 16 bytes of nibbles per row (16 values each of two neighbouring
//    sub-blocks) and that super-block's 16-byte header, all requested at once and, for constant weights, before the kernel
//    waits for its stream predecessor (programmatic dependent launch); x is loaded once for the four rows;
//  * the CTA's warps share the row's K range, so a node is thousands of independent warps of one or two steps each (CTAs that
//    stay and walk the row groups, the next group's loads in flight, were slower: 10.8 -> 15.2 us on [2560, 10240]);
//  * a nibble becomes a float by one byte permute into 2^23's mantissa and half of a packed add (exact); products and sums
//    are packed f32 pairs; scale and minimum enter once per sub-block: sc * sum(q x) - m * sum(x), all in f32;
//  * the warps' sums meet in shared memory in warp order (deterministic); with the gate/up fold a CTA has two gate rows and
//    their two up rows and writes the folded values itself.
// [3072, 8192]: 14.5 -> 10.3 us, [6144, 2048]: 11.0 -> 5.7, [3072, 1024]: 5.7 -> 3.1, [51865, 512]: 24.6 -> 17.3; about 3.6
// instructions a value and the latency of a warp's one or two steps bound it, not the bytes (2.1 us of them in the first).
#include <algorithm>

#include "common.cuh"
#include "f32x2.cuh"
#include "kernels.hpp"

namespace rt {

namespace {

constexpr int ROWS = 4; // per CTA; two of them (three CTAs per SM instead of two) were up to 8 % slower from [5120, 1280] on
constexpr int MAX_WARPS = 8;
constexpr int CHUNK_SB = 4; // super-blocks per warp and step

// 6-bit scale and minimum of sub-block 2 pair + h from a super-block's header (the packing of q4k_scale_min, decode.cuh)
__device__ __forceinline__ void header_scale_min(const uint4 &head, int pair, int h, uint32_t &sc, uint32_t &mn) {
    const int sh = 8 * ((pair & 1) * 2 + h);
    const uint32_t a = (head.y >> sh) & 0xFFu, b = (head.z >> sh) & 0xFFu, c = (head.w >> sh) & 0xFFu;
    sc = pair < 2 ? (a & 63u) : ((c & 0x0Fu) | ((a >> 6) << 4));
    mn = pair < 2 ? (b & 63u) : ((c >> 4) | ((b >> 6) << 4));
}

// The whole row again, element by element in f32: an infinity among the activations makes q * x or sum(x) a NaN that the
// product with the dequantised weight is not, so a NaN result is decided here by IEEE's rules for the plain sum.  One thread
// per row, 32 values per step from a 16-byte load of nibbles and one of the header: 221 us for [3072, 8192] and 112 for
// [512, 12288] (byte loads took 1603 and 799, the warp-MMA kernel takes 896 and 280).  A warp per row is faster (105, 41), but
// its vote at the end of every launch cost finite rows up to 10 % ([512, 1280] 2.32 -> 2.57 us).
__device__ __noinline__ float exact_row(const uint8_t *row, const __half *x, int nsb) {
    float acc = 0.f;
#pragma unroll 1
    for (int u = 0; u < nsb * 8; u++) {
        const int sb = u >> 3, pair = (u & 7) >> 1, half = u & 1;
        const uint8_t *blk = row + (long long)sb * 144;
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(blk + 16 + (u & 7) * 16)), head = __ldg(reinterpret_cast<const uint4 *>(blk));
        const float d = __half2float(__ushort_as_half((unsigned short)(head.x & 0xFFFFu)));
        const float dmin = __half2float(__ushort_as_half((unsigned short)(head.x >> 16)));
        const uint32_t ww[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t sc, mn;
            header_scale_min(head, pair, h, sc, mn);
            const float ds = __fmul_rn(d, (float)sc), dm = __fmul_rn(dmin, (float)mn);
            const __half *xp = x + sb * 256 + pair * 64 + h * 32 + half * 16;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const float code = (float)((ww[i >> 2] >> (8 * (i & 3) + 4 * h)) & 15u);
                acc += __fsub_rn(__fmul_rn(ds, code), dm) * __half2float(xp[i]);
            }
        }
    }
    return acc;
}

template <bool PAIR>
__global__ void __launch_bounds__(MAX_WARPS * 32, 2) q4k_gemv_f16_kernel(MatmulParams p, int lhs_constant) {
    __shared__ float part[MAX_WARPS][ROWS];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!lhs_constant) asm volatile("griddepcontrol.wait;" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int batch = blockIdx.z, nsb = p.K >> 8, ff = p.M >> 1;
    const uint8_t *w = (const uint8_t *)p.lhs + (long long)(batch % p.lhs_stack) * p.M * nsb * 144;
    const __half *x = (const __half *)p.rhs + (long long)(batch % p.rhs_stack) * p.K;
    constexpr int HALF = ROWS / 2; // with the fold: this many gate rows and their up rows
    // rows past the end repeat the last one and are not stored
    auto row_of = [&](int r) {
        return PAIR ? min((int)blockIdx.x * HALF + r % HALF, ff - 1) + (r / HALF) * ff : min((int)blockIdx.x * ROWS + r, p.M - 1);
    };
    const int pair = (lane & 7) >> 1, half = lane & 1; // this lane's pair of sub-blocks and which 16 of their 32 values

    uint4 q[ROWS], head[ROWS];
    auto load = [&](int sb) {
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const uint8_t *blk = w + ((long long)row_of(r) * nsb + sb) * 144;
            q[r] = __ldg(reinterpret_cast<const uint4 *>(blk + 16 + (lane & 7) * 16));
            head[r] = __ldg(reinterpret_cast<const uint4 *>(blk));
        }
    };
    int sb = warp * CHUNK_SB + (lane >> 3);
    if (sb < nsb) load(sb);
    if (lhs_constant) asm volatile("griddepcontrol.wait;" ::: "memory");

    float acc[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; r++) acc[r] = 0.f;
    const unsigned long long bias2 = pack2f(-8388608.f, -8388608.f);
    while (sb < nsb) {
        // the lane's 16 activations of each sub-block (written by the predecessor: plain loads, after the wait), and their sums
        unsigned long long xv[2][8];
        float xs[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const __half *xp = x + sb * 256 + pair * 64 + h * 32 + half * 16;
            unsigned long long s2 = 0ull;
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const uint4 raw = *reinterpret_cast<const uint4 *>(xp + j * 8);
                const uint32_t ww[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&ww[e]));
                    xv[h][j * 4 + e] = pack2f(f.x, f.y);
                    s2 = add2(s2, xv[h][j * 4 + e]);
                }
            }
            xs[h] = sum2(s2);
        }
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const uint32_t ww[4] = {q[r].x, q[r].y, q[r].z, q[r].w};
            unsigned long long s[2] = {0ull, 0ull};
#pragma unroll
            for (int e = 0; e < 4; e++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t nib = (h ? ww[e] >> 4 : ww[e]) & 0x0F0F0F0Fu;
#pragma unroll
                    for (int j = 0; j < 2; j++) s[h] = fma2(add2(bytes2f(nib, j), bias2), xv[h][e * 2 + j], s[h]);
                }
            const float d = __half2float(__ushort_as_half((unsigned short)(head[r].x & 0xFFFFu)));
            const float dmin = __half2float(__ushort_as_half((unsigned short)(head[r].x >> 16)));
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint32_t sc, mn;
                header_scale_min(head[r], pair, h, sc, mn);
                acc[r] = fmaf(d * (float)sc, sum2(s[h]), acc[r]);
                acc[r] = fmaf(-(dmin * (float)mn), xs[h], acc[r]);
            }
        }
        sb += warps * CHUNK_SB;
        if (sb < nsb) load(sb);
    }

#pragma unroll
    for (int r = 0; r < ROWS; r++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
    }
    if (lane == 0) {
#pragma unroll
        for (int r = 0; r < ROWS; r++) part[warp][r] = acc[r];
    }
    __syncthreads();
    if (threadIdx.x < ROWS) {
        const int r = threadIdx.x, row = row_of(r);
        float s = part[0][r];
        for (int k = 1; k < warps; k++) s += part[k][r];
        if (s != s) s = exact_row(w + (long long)row * nsb * 144, x, nsb);
        const bool has_bias = p.bias_mode != BIAS_NONE;
        float bias = 0.f;
        if (has_bias) bias = load_bias(p.bias, p.bias_dt, p.bias_mode == BIAS_PER_M ? row : 0);
        const __half o = epilogue_value<__half>(s, has_bias, bias, p.epilogue);
        __half *out = (__half *)p.out;
        if (PAIR) {
            const __half up = __ushort_as_half((unsigned short)__shfl_down_sync((1u << ROWS) - 1u, (unsigned)__half_as_ushort(o), HALF));
            const int col = (int)blockIdx.x * HALF + r;
            if (r < HALF && col < ff) out[(long long)batch * ff + col] = silu_mul_value<__half>(o, up);
        } else if ((int)blockIdx.x * ROWS + r < p.M) {
            out[(long long)batch * p.M + row] = o;
        }
    }
}

} // namespace

cudaError_t launch_q4k_gemv_f16(const MatmulParams &p, bool silu_pairs, bool lhs_constant, cudaStream_t stream) {
    const int chunks = (p.K / 256 + CHUNK_SB - 1) / CHUNK_SB;
    const int steps = (chunks + MAX_WARPS - 1) / MAX_WARPS;
    const int warps = (chunks + steps - 1) / steps; // the chunks of a row in as few equal steps as MAX_WARPS allows
    const int ctas = silu_pairs ? (p.M / 2 + ROWS / 2 - 1) / (ROWS / 2) : (p.M + ROWS - 1) / ROWS;
    return launch_pdl(silu_pairs ? q4k_gemv_f16_kernel<true> : q4k_gemv_f16_kernel<false>, dim3(ctas, 1, p.stacks), dim3(warps * 32), 0, stream, p,
                      lhs_constant ? 1 : 0);
}

} // namespace rt
