// The same operator for few rows (M <= 64): decoding, small batches.  The weights B are then nearly all of the bytes, so the
// kernel is built around streaming them.
//
// The MMA's roles are exchanged: 128 columns of C (rows of B) are the M side of tcgen05.mma and the T >= M rows of C are its
// N side.  A tile is 128 columns x all rows of C, a TMEM buffer is T columns wide instead of 256, a promotion thread owns 16
// or 32 rows of one column of C, and no 128-row tile is padded with zeros.  K is cut over the `splits` CTAs of a
// thread-block cluster so that the weights are read by as many SMs as there are; each CTA sends its partial sums straight into
// the shared memory of the CTA that finishes a row (every CTA finishes 1/splits of the rows), one cluster barrier, and the
// sums are added in split order.  What bounds it is the latency chain launch -> first weights -> last K block -> reduction;
// shared memory is kept below half an SM's so that the next call's CTAs are set up while this call's are finishing.
//
// Warps: promotion (TMEM lane = column of C; four warps per TW rows), then one each for TMA, MMA and scale products (as in
// gemm_kernel.cuh).
// All waits are bounded as there.
//
// Measured on a B200 (CUDA graph, cold weights), 128-row tiles -> this kernel: 16 x 7168 x 2304 14.9 -> 7.9 us, 32 x 4096 x 2048
// 8.7 -> 5.8, 64 x 7168 x 2304 10.7 -> 9.4, 16 x 1536 x 7168 10.8 -> 6.1, 16 x 7168 x 7168 20.9 -> 14.0 (the weights alone take 2.5,
// 1.3, 2.5, 1.7 and 7.7 us at 6.65 TB/s); the smallest call, 16 x 128 x 128, 3.1 -> 2.3.
#pragma once
#include "gemm_kernel.cuh"

namespace fp8bs {

template <int T>
struct SmallMCfg {
    static_assert(T == 16 || T == 32 || T == 64, "rows of C a tile has room for");
    static constexpr int X_WIDTH = T < 32 ? 32 : T;     // bytes per k of the box of A, and its swizzle span
    static constexpr int W_BYTES = 128 * 128;           // box of B: 128 columns of C x 128 k
    static constexpr int X_BYTES = 128 * X_WIDTH;
    static constexpr int STAGE_BYTES = W_BYTES + X_BYTES;
    static constexpr int STAGES = T == 64 ? 3 : 4;
    static constexpr int NBUF = 4;                      // TMEM buffers of T columns
    static constexpr int TMEM_COLS = NBUF * T;
    static constexpr int SSLOTS = 2 * NBUF;             // scale products: [column half][row of C]
    static constexpr int SSLOT_FLOATS = 2 * T;
    static constexpr int SLOT_BYTES = SSLOTS * SSLOT_FLOATS * 4;
    static constexpr int RED_BYTES = (T + 7) * 512;     // partial sums received: [split][row of C][128 columns]
    static constexpr int TW = T == 64 ? 32 : 16;        // rows of C of a promotion thread: with one warp per scheduler the
                                                        // instruction count per thread is what the last microsecond is spent on
    static constexpr int PROMO_WARPS = 4 * (T / TW);
    static constexpr int THREADS = 32 * (PROMO_WARPS + 3);
    static constexpr int SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + RED_BYTES + SLOT_BYTES + 256;
    static_assert(2 * (SMEM_BYTES + 1024) <= 228 * 1024, "two CTAs per SM");
    static_assert((2 * STAGES + 2 * NBUF) * 8 + 16 <= 256, "barrier area");
};

// 16 or 32 columns from TMEM, complete on return (load and wait in one statement).
__device__ __forceinline__ void tmem_ld_x16_sync(uint32_t taddr, uint32_t (&v)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_x32_sync(uint32_t taddr, uint32_t (&v)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, "
        "%18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
          "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
          "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}

// grid = n_tiles * splits CTAs, cluster size = splits.
template <int T>
__global__ void __launch_bounds__(SmallMCfg<T>::THREADS, 2)
gemm_small_m_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const GemmParams p)
{
    using Cfg = SmallMCfg<T>;
    constexpr int STAGES = Cfg::STAGES, NBUF = Cfg::NBUF;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = ptx::smem_u32(smem_raw);
    const uint32_t stage_base = (raw + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (stage_base - raw);
    // layout: [stages][received partial sums][scale products][barriers + control words]
    const uint32_t red_base = stage_base + STAGES * Cfg::STAGE_BYTES;
    const float* red_ptr = reinterpret_cast<const float*>(aligned + STAGES * Cfg::STAGE_BYTES);
    const uint32_t slot_base = red_base + Cfg::RED_BYTES;
    float* slots_ptr = reinterpret_cast<float*>(aligned + STAGES * Cfg::STAGE_BYTES + Cfg::RED_BYTES);
    const uint32_t bar_base = slot_base + Cfg::SLOT_BYTES;
    volatile uint32_t* ctrl = reinterpret_cast<volatile uint32_t*>(aligned + STAGES * Cfg::STAGE_BYTES + Cfg::RED_BYTES +
                                                                    Cfg::SLOT_BYTES + (2 * STAGES + 2 * NBUF) * 8);
    // ctrl[0] TMEM base address, ctrl[1] abort flag
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
    auto tfull_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + b); };
    auto tempty_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + NBUF + b); };

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const int S = p.splits;
    const int rank = S > 1 ? static_cast<int>(ptx::cluster_ctarank()) : 0;
    const int n0 = static_cast<int>(blockIdx.x) / S * 128;
    const int KB = p.K / 128;
    const int kb0 = rank * KB / S, kb1 = (rank + 1) * KB / S;

    if (threadIdx.x == 0) {
        ptx::prefetch_tensormap(&tmX);
        ptx::prefetch_tensormap(&tmW);
        for (int s = 0; s < STAGES; ++s) {
            ptx::mbar_init(full_bar(s), 1);
            ptx::mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < NBUF; ++b) {
            ptx::mbar_init(tfull_bar(b), 2);          // the MMA warp's commit and the scale warp
            ptx::mbar_init(tempty_bar(b), Cfg::PROMO_WARPS);
        }
        ctrl[1] = 0u;
        ptx::fence_mbar_init();
    }
    if (warp == Cfg::PROMO_WARPS + 1) {
        ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(&ctrl[0])), Cfg::TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (S > 1) ptx::cluster_arrive();                 // waited for before anything is written into a peer: it has started
    ptx::tc_fence_after_sync();
    const uint32_t tmem_base = ctrl[0];
    volatile uint32_t* abort_flag = &ctrl[1];
    ptx::grid_dependency_wait();
    ptx::grid_launch_dependents();

    constexpr int TW = Cfg::TW;
    const int row0 = (warp >> 2) * TW;                // promotion warps: first row of C of this thread
    unsigned long long acc[TW / 2];                   // ... and its rows row0 + 2 i, row0 + 2 i + 1, one column
#pragma unroll
    for (int i = 0; i < TW / 2; ++i) acc[i] = 0ull;
    bool ok = true;

    if (warp == Cfg::PROMO_WARPS) {
        if (ptx::elect_one()) {
            // ---------------------------------------------------- TMA producer ----
            int s = 0;
            uint32_t ph = 0;
            for (int kb = kb0; kb < kb1; ++kb) {
                ok = wait_bounded(empty_bar(s), ph ^ 1u, abort_flag, p.status, DS_TIMEOUT_STAGE_EMPTY);
                if (!ok) break;
                const uint32_t dst = stage_base + s * Cfg::STAGE_BYTES;
                // whole boxes are written and counted: columns >= N and rows >= M read as 0
                ptx::mbar_arrive_expect_tx(full_bar(s), Cfg::STAGE_BYTES);
                ptx::tma_load_2d(dst, &tmW, n0, kb * 128, full_bar(s));
                ptx::tma_load_2d(dst + Cfg::W_BYTES, &tmX, 0, kb * 128, full_bar(s));
                if (++s == STAGES) { s = 0; ph ^= 1u; }
            }
            if (!ok) {
                // aborting with loads possibly in flight: a bounded time to land
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000LL) __nanosleep(1000);
            }
        }
        __syncwarp();
    } else if (warp == Cfg::PROMO_WARPS + 1) {
        if (ptx::elect_one()) {
            // ---------------------------------------------------- MMA issuer ------
            constexpr uint32_t idesc = ptx::make_idesc_e4m3_mnmajor(128, T);
            constexpr uint32_t x_atom = 8 * Cfg::X_WIDTH;                 // 8 k-rows of the box of A
            constexpr uint32_t x_swizzle = Cfg::X_WIDTH == 64 ? 4u : 6u;  // 64- or 32-byte swizzle
            int s = 0;
            uint32_t ph = 0, item = 0;
            for (int kb = kb0; kb < kb1; ++kb, ++item) {
                const int b = item % NBUF;
                ok = wait_bounded(full_bar(s), ph, abort_flag, p.status, DS_TIMEOUT_STAGE_FULL);
                if (!ok) break;
                ok = wait_bounded(tempty_bar(b), ((item / NBUF) & 1u) ^ 1u, abort_flag, p.status, DS_TIMEOUT_TMEM_EMPTY);
                if (!ok) break;
                ptx::tc_fence_after_sync();
                const uint32_t w_addr = stage_base + s * Cfg::STAGE_BYTES;
                const uint64_t wdesc = ptx::make_smem_desc_sw128(w_addr, Cfg::W_BYTES, 1024);
                const uint64_t xdesc = ptx::make_smem_desc(w_addr + Cfg::W_BYTES, Cfg::X_BYTES, x_atom, x_swizzle);
                const uint32_t d = tmem_base + static_cast<uint32_t>(b * T);
#pragma unroll
                for (int j = 0; j < 4; ++j)           // K = 32 per instruction = 4 swizzle atoms of 8 k-rows
                    ptx::mma_f8f6f4(d, wdesc + static_cast<uint64_t>(j * (4096 >> 4)),
                                    xdesc + static_cast<uint64_t>(j * ((4 * x_atom) >> 4)), idesc, j > 0 ? 1u : 0u);
                ptx::mma_commit(tfull_bar(b));
                ptx::mma_commit(empty_bar(s));
                if (++s == STAGES) { s = 0; ph ^= 1u; }
            }
        }
        __syncwarp();
    } else if (warp == Cfg::PROMO_WARPS + 2) {
        // ---------------------------------------------------- scale products -------
        // a_scale[m, kb] * b_scale[n / 128, kb]: the tile's 128 columns touch at most two blocks of b_scale, one per 64
        // columns.  Same hand-over and order of waits as in gemm_kernel.cuh.
        constexpr int AHEAD = 4, NA = T < 32 ? 1 : T / 32;
        float av[AHEAD][NA], bv[AHEAD][2];
        int nb[2];
        for (int h = 0; h < 2; ++h) {
            const int n = (p.n_off + n0 + h * 64) >> 7;
            nb[h] = n < p.sn ? n : p.sn - 1;
        }
        int fkb = kb0;
        auto fetch = [&](float (&a)[NA], float (&b)[2]) {
            if (fkb < kb1) {
#pragma unroll
                for (int i = 0; i < NA; ++i) {
                    const int m = (T < 32 ? (lane & (T - 1)) : lane) + 32 * i;
                    a[i] = m < p.M ? __ldg(p.a_scale + static_cast<size_t>(fkb) * p.M + m) : 0.0f;
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) b[h] = __ldg(p.b_scale + static_cast<size_t>(fkb) * p.sn + nb[h]) * p.elem_scale;
            }
            ++fkb;
        };
#pragma unroll
        for (int d = 0; d < AHEAD; ++d) fetch(av[d], bv[d]);
        uint32_t item = 0;
        const uint32_t items = static_cast<uint32_t>(kb1 - kb0);
        while (ok && item < items) {
#pragma unroll
            for (int d = 0; d < AHEAD; ++d) {
                if (!ok || item >= items) break;
                if (item >= NBUF) {
                    ok = wait_bounded(tfull_bar(item % NBUF), ((item / NBUF) - 1u) & 1u, abort_flag, p.status, DS_TIMEOUT_SCALE_EMPTY);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                }
                float* dst = slots_ptr + (item % Cfg::SSLOTS) * Cfg::SSLOT_FLOATS;
                if constexpr (T == 16) {
                    dst[lane] = av[d][0] * (lane < 16 ? bv[d][0] : bv[d][1]);
                } else {
#pragma unroll
                    for (int i = 0; i < NA; ++i) {
                        dst[lane + 32 * i] = av[d][i] * bv[d][0];
                        dst[T + lane + 32 * i] = av[d][i] * bv[d][1];
                    }
                }
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(tfull_bar(item % NBUF));
                ++item;
                fetch(av[d], bv[d]);
            }
        }
    } else {
        // ---------------------------------------------------- promotion -------------
        const uint32_t my_slot = slot_base + static_cast<uint32_t>((((warp >> 1) & 1) * T + row0) * 4);   // [column half][row]
        const uint32_t my_tmem = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(row0);
        uint32_t item = 0;
        for (int kb = kb0; kb < kb1; ++kb, ++item) {
            const int b = item % NBUF;
            ok = wait_bounded(tfull_bar(b), (item / NBUF) & 1u, abort_flag, p.status, DS_TIMEOUT_TMEM_FULL);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            ptx::tc_fence_after_sync();
            const uint32_t sa = my_slot + (item % Cfg::SSLOTS) * (Cfg::SSLOT_FLOATS * 4);
            uint32_t v[TW];
            if constexpr (TW == 16) tmem_ld_x16_sync(my_tmem + static_cast<uint32_t>(b * T), v);
            else tmem_ld_x32_sync(my_tmem + static_cast<uint32_t>(b * T), v);
#pragma unroll
            for (int i = 0; i < TW / 4; ++i) {
                unsigned long long s0, s1;            // products of rows 4 i .. 4 i + 3
                ptx::ld_shared_v2_b64(sa + static_cast<uint32_t>(16 * i), s0, s1);
                acc[2 * i] = ptx::fma_f32x2((static_cast<unsigned long long>(v[4 * i + 1]) << 32) | v[4 * i], s0, acc[2 * i]);
                acc[2 * i + 1] = ptx::fma_f32x2((static_cast<unsigned long long>(v[4 * i + 3]) << 32) | v[4 * i + 2], s1, acc[2 * i + 1]);
            }
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(tempty_bar(b));
        }
    }

    // ---------------------------------------------------------------- result -------
    if (S == 1) {
        // straight from the registers (through shared memory, for wider stores, it took 0.6 us longer)
        const int n = n0 + (warp & 3) * 32 + lane;
        if (warp < Cfg::PROMO_WARPS && ok && n < p.N) {
#pragma unroll
            for (int t = 0; t < TW; ++t)
                if (row0 + t < p.M)
                    p.C[static_cast<size_t>(row0 + t) * p.N + n] = __float2bfloat16_rn(t & 1 ? f32x2_hi(acc[t / 2]) : f32x2_lo(acc[t / 2]));
        }
    } else {
        // partial sums to the CTA that finishes a row: [split][row of C][column] in its shared memory
        const int per = (p.M + S - 1) / S;            // rows of C each CTA finishes
        ptx::cluster_wait();                          // every CTA of the cluster runs
        if (warp < Cfg::PROMO_WARPS && ok) {
            const uint32_t mine = red_base + static_cast<uint32_t>((rank * per * 128 + (warp & 3) * 32 + lane) * 4);
            int owner = row0 / per, local = row0 - owner * per;
            uint32_t dst = ptx::mapa(mine, static_cast<uint32_t>(owner < S ? owner : 0));
#pragma unroll
            for (int t = 0; t < TW; ++t)
                if (row0 + t < p.M) {
                    ptx::st_shared_cluster_f32(dst + static_cast<uint32_t>(local * 512), t & 1 ? f32x2_hi(acc[t / 2]) : f32x2_lo(acc[t / 2]));
                    if (++local == per) {
                        local = 0;
                        ++owner;
                        dst = ptx::mapa(mine, static_cast<uint32_t>(owner < S ? owner : 0));
                    }
                }
        }
        ptx::cluster_sync();
        if (*abort_flag == 0u) {
            const int t0 = rank * per, rows = t0 + per < p.M ? per : p.M - t0;
            // four columns of one row per thread and round, all splits' loads in flight together
            for (int idx = static_cast<int>(threadIdx.x); idx < rows * 32; idx += Cfg::THREADS) {
                const int t = idx >> 5, c = (idx & 31) * 4;
                const float4* src = reinterpret_cast<const float4*>(red_ptr + t * 128 + c);
                float4 v[8];
#pragma unroll
                for (int s = 0; s < 8; ++s)
                    if (s < S) v[s] = src[static_cast<size_t>(s) * per * 32];
                float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                for (int s = 0; s < 8; ++s)           // split order
                    if (s < S) { sum.x += v[s].x; sum.y += v[s].y; sum.z += v[s].z; sum.w += v[s].w; }
                if (n0 + c < p.N) {
                    uint2 q;
                    q.x = pack_bf16x2(sum.x, sum.y);
                    q.y = pack_bf16x2(sum.z, sum.w);
                    *reinterpret_cast<uint2*>(p.C + static_cast<size_t>(t0 + t) * p.N + n0 + c) = q;
                }
            }
        }
    }

    ptx::tc_fence_before_sync();
    __syncthreads();
    if (warp == Cfg::PROMO_WARPS + 1) {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
    }
}

}  // namespace fp8bs
