// The 16-bit tensor-core GEMM with K split over the CTAs of a cluster; part of gemm_umma.cu (included inside its
// anonymous namespace), whose helpers, parameter block and tensor maps it shares.
//
// For problems with fewer output tiles than SMs (prompts of 25 .. some hundred rows, the narrow second matrix of an MLP
// block): one CTA per tile left most SMs idle while each busy one pulled a whole K range through its L2 port.  Here a
// cluster of `ksplit` CTAs works on one tile, CTA i on K blocks [i*n/ksplit, (i+1)*n/ksplit), so the operands come in
// through ksplit ports.  The partial sums meet in distributed shared memory:
//   1. every CTA copies its f32 accumulators from tensor memory into its own (by then drained) operand ring, row-major,
//      16-byte chunks XOR the row, which makes both sides free of bank conflicts;
//   2. one cluster barrier; CTA i then owns an equal share of the tile's VALID rows and adds the ksplit partial rows in
//      rank order (deterministic): a warp reads 512 contiguous bytes of a peer's row per instruction, so a lane has four
//      neighbouring columns, applies the epilogue and stores them; nothing is staged again;
//   3. a second cluster barrier keeps every CTA's shared memory alive until its peers have read it.
// [2560, 10240] x 77 rows: 50.6 -> 15.7 us (20 tiles, clusters of six).  Through global memory (f32 slices, fences, a counter
// per tile) the same split gained nothing.

template <int BN> struct KsCfg {
    using C = Cfg<BN>;
    static constexpr int SMEM_BYTES = C::STAGES * C::STAGE_BYTES + 1024 /*alignment*/ + 256 /*barriers*/ + BN * 4 /*bias*/;
    static_assert(BM * BN * 4 <= C::STAGES * C::STAGE_BYTES, "the partial tile lives in the operand ring");
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// CMAX: largest cluster the instantiation serves (4 or 8): how many partial rows are in flight per lane
template <int BN, typename OutT, bool PAIR, int CMAX>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_umma_ksplit_kernel(const __grid_constant__ CUtensorMap map_p, const __grid_constant__ CUtensorMap map_q, const UmmaParams prm, const int ksplit) {
    using C = Cfg<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *tiles = smem;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + C::STAGES * C::STAGE_BYTES); // full [S], empty [S], accumulator
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * C::STAGES + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    float *bias_s = reinterpret_cast<float *>(smem + C::STAGES * C::STAGE_BYTES + 256);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t bar_full = smem_u32(bars), bar_empty = smem_u32(bars + C::STAGES), bar_acc = smem_u32(bars + 2 * C::STAGES);
    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; s++) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_acc, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    // this cluster's tile and this CTA's K blocks (ksplit <= K blocks: never empty)
    const int rank = (int)cluster_ctarank(), tile = (int)blockIdx.x / ksplit;
    const int tiles_per_batch = prm.tiles_r * prm.tiles_s;
    const int b = tile / tiles_per_batch;
    int tr, ts;
    tile_coords(tile % tiles_per_batch, prm.tiles_r, prm.tiles_s, prm.group_r, tr, ts);
    const int r0 = tr * BM, s0 = ts * (PAIR ? BN / 2 : BN);
    const int num_k = (prm.K + BK - 1) / BK;
    const int kb0 = num_k * rank / ksplit, kb1 = num_k * (rank + 1) / ksplit;
    const int rows = min(BM, prm.R - r0); // valid rows of the tile

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        if (lane == 0) {
            const int bp = b % prm.p_stack, bq = b % prm.q_stack;
            int stage = 0;
            uint32_t phase = 0;
            for (int kb = kb0; kb < kb1; kb++) {
                if (!mbar_wait(bar_empty + 8 * stage, phase ^ 1, abort_flag, 1)) break;
                const uint32_t a_dst = smem_u32(tiles + stage * C::STAGE_BYTES);
                mbar_expect_tx(bar_full + 8 * stage, C::STAGE_BYTES);
                tma_load_3d(a_dst, &map_p, kb * BK, r0, bp, bar_full + 8 * stage);
                if (PAIR) tma_load_4d(a_dst + C::A_BYTES, &map_q, kb * BK, s0, 0, bq, bar_full + 8 * stage);
                else tma_load_3d(a_dst + C::A_BYTES, &map_q, kb * BK, s0, bq, bar_full + 8 * stage);
                if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int kb = kb0; kb < kb1; kb++) {
                if (!mbar_wait(bar_full + 8 * stage, phase, abort_flag, 3)) { ok = false; break; }
                tc_fence_after();
                const uint32_t a_addr = smem_u32(tiles + stage * C::STAGE_BYTES);
                const uint32_t b_addr = a_addr + C::A_BYTES;
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; k++)
                    umma_f16(tmem_base, umma_desc_sw128(a_addr + k * UMMA_K * 2), umma_desc_sw128(b_addr + k * UMMA_K * 2), prm.idesc,
                             (kb != kb0 || k != 0) ? 1u : 0u);
                umma_commit(bar_empty + 8 * stage);
                if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
            }
            if (ok) umma_commit(bar_acc);
        }
    } else {
        // ---------------------------------------------------------------- accumulators into the drained ring
        const int q = warp & 3, half = (warp - 2) >> 2;
        if (prm.bias_mode == BIAS_PER_N) {
            for (int j = threadIdx.x - 64; j < BN; j += EPI_WARPS * 32) {
                const int jj = PAIR ? j % (BN / 2) : j;
                const int wrow = PAIR ? (j / (BN / 2)) * prm.s_out + s0 + jj : s0 + j;
                bias_s[j] = (s0 + jj < prm.s_out) ? load_bias(prm.bias, prm.bias_dt, wrow) : 0.f;
            }
        }
        // the accumulator is complete: every MMA of this CTA has read its operands and every copy has landed
        if (__all_sync(0xffffffffu, mbar_wait(bar_acc, 0, abort_flag, 4)) && q * 32 < rows) {
            tc_fence_after();
            const int row = q * 32 + lane;
            uint8_t *line = tiles + (size_t)row * (BN * 4);
#pragma unroll 1
            for (int c = half; c < BN / 32; c += 2) {
                uint32_t v[32];
                tmem_ld32(tmem_base + c * 32 + ((uint32_t)(q * 32) << 16), v);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    *reinterpret_cast<uint4 *>(line + (((c * 8 + j) ^ (row & 7)) << 4)) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    cluster_sync_all(); // every partial tile of the cluster is in shared memory (or its CTA gave up: the host hears of it)

    if (warp >= 2) {
        // ---------------------------------------------------------------- this CTA's rows: sum, epilogue, store
        constexpr int OCH = (PAIR ? BN / 2 : BN) / 4;                      // chunks of four output columns per row
        constexpr int UNITS = PAIR ? 2 : 1;                                // accumulators per output
        constexpr int U = CMAX == 4 && !PAIR ? 2 : 1;                      // rows in flight per lane
        const int per = (rows + ksplit - 1) / ksplit;
        const int first = rank * per, mine = max(0, min(rows, first + per) - first);
        uint32_t peer[CMAX];
#pragma unroll
        for (int j = 0; j < CMAX; j++) peer[j] = j < ksplit ? map_to_cta(smem_u32(tiles), (uint32_t)j) : 0u;
        bool vec_ok = prm.s_out % 4 == 0 && prm.out_ld % 4 == 0 && prm.out_col % 4 == 0 && prm.out_batch_stride % 4 == 0;
        for (int d = 0; d < prm.n_out; d++) vec_ok = vec_ok && reinterpret_cast<uintptr_t>(prm.outs[d]) % 8 == 0;
        const bool has_bias = prm.bias_mode != BIAS_NONE;
        const int items = mine * OCH;
#pragma unroll 1
        for (int i0 = (int)threadIdx.x - 64; i0 < items; i0 += EPI_WARPS * 32 * U) {
            float4 part[U][UNITS][CMAX];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int i = min(i0 + u * EPI_WARPS * 32, items - 1);
                const int row = first + i / OCH, ch = i % OCH;
#pragma unroll
                for (int n = 0; n < UNITS; n++) {
                    const uint32_t off = (uint32_t)row * (BN * 4) + (uint32_t)(((ch + n * OCH) ^ (row & 7)) << 4);
#pragma unroll
                    for (int j = 0; j < CMAX; j++)
                        if (j < ksplit) part[u][n][j] = ld_cluster_f4(peer[j] + off);
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int i = i0 + u * EPI_WARPS * 32;
                if (i >= items) break;
                const int row = first + i / OCH, ch = i % OCH, rg = r0 + row, col = s0 + ch * 4;
                if (col >= prm.s_out) continue;
                float acc[UNITS][4];
#pragma unroll
                for (int n = 0; n < UNITS; n++) {
                    float4 s = part[u][n][0];
#pragma unroll
                    for (int j = 1; j < CMAX; j++)
                        if (j < ksplit) {
                            s.x += part[u][n][j].x; s.y += part[u][n][j].y;
                            s.z += part[u][n][j].z; s.w += part[u][n][j].w;
                        }
                    acc[n][0] = s.x; acc[n][1] = s.y; acc[n][2] = s.z; acc[n][3] = s.w;
                }
                if (HAS_OPERAND_FACTORS<OutT>) {
                    if (prm.p_scale) {
                        const float f = __ldg(prm.p_scale + (long long)(b % prm.p_stack) * prm.R + rg);
#pragma unroll
                        for (int n = 0; n < UNITS; n++)
#pragma unroll
                            for (int e = 0; e < 4; e++) acc[n][e] *= f;
                    }
                    if (!PAIR && prm.q_scale) {
                        const float *qs = prm.q_scale + (long long)(b % prm.q_stack) * prm.S;
#pragma unroll
                        for (int e = 0; e < 4; e++) acc[0][e] *= __ldg(qs + min(col + e, prm.S - 1));
                    }
                }
                OutT o[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    if (PAIR) {
                        const OutT gv = epilogue_value<OutT>(acc[0][e], has_bias, has_bias ? bias_s[ch * 4 + e] : 0.f, RT_EPILOGUE_NONE);
                        const OutT uv = epilogue_value<OutT>(acc[UNITS - 1][e], has_bias, has_bias ? bias_s[BN / 2 + ch * 4 + e] : 0.f, RT_EPILOGUE_NONE);
                        o[e] = silu_mul_value<OutT>(gv, uv);
                    } else {
                        o[e] = epilogue_value<OutT>(acc[0][e], has_bias, has_bias ? bias_s[ch * 4 + e] : 0.f, prm.epilogue);
                    }
                }
                const long long at = (long long)b * prm.out_batch_stride + (long long)rg * prm.out_ld + prm.out_col + col;
                for (int d = 0; d < prm.n_out; d++) {
                    OutT *dst = reinterpret_cast<OutT *>(prm.outs[d]) + at;
                    if (vec_ok) {
                        uint2 w;
                        w.x = (uint32_t)reinterpret_cast<unsigned short &>(o[0]) | (uint32_t)reinterpret_cast<unsigned short &>(o[1]) << 16;
                        w.y = (uint32_t)reinterpret_cast<unsigned short &>(o[2]) | (uint32_t)reinterpret_cast<unsigned short &>(o[3]) << 16;
                        *reinterpret_cast<uint2 *>(dst) = w;
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            if (col + e < prm.s_out) dst[e] = o[e];
                    }
                }
            }
        }
    }

    // ---------------------------------------------------------------- teardown
    __syncthreads();
    cluster_sync_all(); // the peers have read this CTA's partial tile
    if (*abort_flag) {
        report_wait_error();
        // give copies that may still be in flight time to land before the CTA's memory is released
        const unsigned long long t0 = wait_clock();
        while (wait_clock() - t0 < 400000ull) __nanosleep(1000);
    }
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(BN) : "memory");
    }
}
