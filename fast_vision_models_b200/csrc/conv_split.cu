// Dense convolution for small problems: one output tile per thread-block cluster, the reduction split over its CTAs.
//
// A layer with few output pixels (one image, or the 14x14 and 7x7 maps of a small batch) has a handful of 128-pixel
// tiles: the persistent kernels then leave most SMs idle and the busy ones stream the whole reduction through one SM's
// port (about 110 GB/s). Here a cluster of `split` CTAs shares a tile of 128 pixels x BN channels: CTA r multiplies its
// run of k-blocks (TMA -> tcgen05.mma -> fp32 accumulator in its own TMEM), then sends row slice o of its partial tile to
// CTA o's shared memory (distributed shared memory, 16-byte stores), and after one cluster barrier every CTA adds the
// `split` partial sums of its slice in rank order, applies bias / scale / residual / activation in fp32 and writes the
// result with 16-byte stores. (One bulk copy per slice instead of the remote stores was 0.5 to 2 us slower per launch.)
// No scratch in global memory, no flags, the same order of additions on every run. Graph of 20 launches, against the best
// CTA-pair tile, us: 3x3 512 -> 512 at 7x7, one image 6.5 / 18.8; 3x3 256 -> 256 at 14x14, one image 5.4 / 11.1; 1x1
// 2048 -> 512 at 7x7 4.9 / 9.4; classifier 2048 -> 1000 5.2 / 9.4; but 1x1 256 -> 1024 at 14x14 5.4 / 4.5 and the second of
// these at batch 64 38 / 17: the per-layer timing decides.
// The stages and the exchange buffer stay below half of an SM's shared memory where the pipeline allows it, so that the
// next layer's CTAs (programmatic dependent launch) can already fetch their weights beside this layer's last tiles.
#include <cuda.h>

#include <cstdint>
#include <cstring>

#include "fvm_internal.h"
#include "ptx_sm100.cuh"

namespace fvm {

static constexpr int CS_EPI_WARPS = 8;
static constexpr int CS_THREADS = 32 * (2 + CS_EPI_WARPS);     // producer, MMA issuer, epilogue warps
static constexpr int CS_MAX_STAGES = 8;
static constexpr int CS_UNITS = 4;                             // 8-channel output units per epilogue thread, at most
static constexpr uint32_t CS_A_BYTES = 128 * 64 * 2;
static constexpr int STATUS_WAIT_SPLIT = 0x107;

__device__ __forceinline__ void cs_cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cs_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void cs_push(uint32_t addr, const uint32_t* v) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}

// 8 fp32 sums + bias (* scale) (+ residual) -> activation -> 8 fp16: the arithmetic of the persistent kernels' epilogue
__device__ __forceinline__ uint4 cs_finish(const SplitParams& p, const float (&v)[8], const uint4& bias, const uint4& res, int n) {
    const uint32_t b4[4] = {bias.x, bias.y, bias.z, bias.w}, r4[4] = {res.x, res.y, res.z, res.w};
    uint32_t o[4];
    const bool fast = p.scale == nullptr && (p.act == 0 || p.act == 1 || p.act == 3 || p.act == 5);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        unsigned long long t = f2_add(f2_pack(__float_as_uint(v[2 * k]), __float_as_uint(v[2 * k + 1])), h2_to_f2(b4[k]));
        if (p.scale) t = f2_mul(t, f2_pack(__float_as_uint(__ldg(p.scale + n + 2 * k)), __float_as_uint(__ldg(p.scale + n + 2 * k + 1))));
        if (p.res) t = f2_add(t, h2_to_f2(r4[k]));
        if (fast) {
            if (p.act == 3) t = f2_silu(t);
            else if (p.act == 5) t = f2_gelu_erf(t);
            o[k] = f2_to_h2(t);
            if (p.act == 1) o[k] = h2_relu(o[k]);
        } else {
            float lo, hi;
            f2_unpack(t, lo, hi);
            lo = act_f(lo, p.act);
            hi = act_f(hi, p.act);
            o[k] = f2_to_h2(f2_pack(__float_as_uint(lo), __float_as_uint(hi)));
        }
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

// A CTA's part of the output: `units` runs of 8 channels, rows row0 .., columns n0 .., thread `et` of the epilogue warps takes
// units u0 + et, u0 + et + 256, .. (CS_UNITS of them). cs_residual requests the residual, cs_output adds the partial sums of
// the exchange (in CTA order) and writes.
__device__ __forceinline__ void cs_residual(const SplitParams& p, uint4 (&res)[CS_UNITS], int u0, int units, int lg8, int row0, int n0) {
#pragma unroll
    for (int k = 0; k < CS_UNITS; ++k) {
        const int u = u0 + k * 32 * CS_EPI_WARPS, n = n0 + ((u & ((1 << lg8) - 1)) << 3);
        res[k] = make_uint4(0u, 0u, 0u, 0u);
        if (p.res && u < units && n < p.K)
            res[k] = *reinterpret_cast<const uint4*>(p.res + static_cast<long long>(row0 + (u >> lg8)) * p.ldr + n);
    }
}
__device__ __forceinline__ void cs_output(const SplitParams& p, const uint4 (&res)[CS_UNITS], int u0, int units, int lg8, int row0,
                                          int n0, uint32_t red_base, int rsp) {
#pragma unroll
    for (int k = 0; k < CS_UNITS; ++k) {
        const int u = u0 + k * 32 * CS_EPI_WARPS;
        if (u >= units) break;
        const int rl = u >> lg8, c8 = u & ((1 << lg8) - 1), n = n0 + (c8 << 3);
        if (n >= p.K) continue;
        float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int q = 0; q < p.split; ++q) {
            const uint32_t a = red_base + static_cast<uint32_t>((q * (p.BN >> 2) + 2 * c8) * rsp + rl) * 16u;
            const uint4 x0 = lds128(a), x1 = lds128(a + static_cast<uint32_t>(rsp) * 16u);
            v[0] += __uint_as_float(x0.x); v[1] += __uint_as_float(x0.y); v[2] += __uint_as_float(x0.z); v[3] += __uint_as_float(x0.w);
            v[4] += __uint_as_float(x1.x); v[5] += __uint_as_float(x1.y); v[6] += __uint_as_float(x1.z); v[7] += __uint_as_float(x1.w);
        }
        const uint4 bias = p.bias ? __ldg(reinterpret_cast<const uint4*>(p.bias + n)) : make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4*>(p.y + static_cast<long long>(row0 + rl) * p.ldy + n) = cs_finish(p, v, bias, res[k], n);
    }
}
// This thread's row of the partial tile (16 columns at a time) into the exchange of the CTA that finishes the row.
__device__ __forceinline__ void cs_send(const SplitParams& p, uint32_t t_row, uint32_t dst, int c_begin, int c_end, int rsp, bool valid) {
    for (int c = c_begin; c < c_end; c += 16) {
        uint32_t v[16];
        tmem_ld_32x32b_x16(t_row + static_cast<uint32_t>(c), v);
        tmem_ld_wait();
        if (valid) {
#pragma unroll
            for (int k = 0; k < 4; ++k) cs_push(dst + static_cast<uint32_t>(((c >> 2) + k) * rsp) * 16u, v + 4 * k);
        }
        __syncwarp();
    }
}

// Shared memory: [stages x (A tile 16 KB | B tile BN x 128 B)] [exchange: split x BN/4 x rows, float4] [barriers] [tmem slot,
// abort flag]. The exchange is [source CTA][column / 4][row of the slice] with an odd row count: the sender's lanes (one
// row each) write 16-byte neighbours.
__global__ void __launch_bounds__(CS_THREADS)
conv_split_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const SplitParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t stage_bytes = CS_A_BYTES + static_cast<uint32_t>(p.BN) * 128u;
    const uint32_t red_base = smem_base + static_cast<uint32_t>(p.stages) * stage_bytes;
    const uint32_t bar_base = red_base + p.red_bytes;
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (CS_MAX_STAGES + s); };
    const uint32_t tfull_bar = bar_base + 8u * (2 * CS_MAX_STAGES);
    const uint32_t misc_off = (bar_base - smem_u32(smem_raw)) + 8u * (2 * CS_MAX_STAGES + 1);
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_raw + misc_off);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_raw + misc_off + 4);

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const int rank = static_cast<int>(cluster_ctarank());
    const int tile = static_cast<int>(fastdiv(blockIdx.x, p.div_split));
    const int m_tile = static_cast<int>(fastdiv(static_cast<uint32_t>(tile), p.div_ntiles));
    const int n0 = (tile - m_tile * p.n_tiles) * p.BN;
    const int m0 = m_tile * 128;
    const int kb0 = rank * p.kblocks / p.split, nkb = (rank + 1) * p.kblocks / p.split - kb0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(tfull_bar, 1);
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmap_a);
        tma_prefetch_desc(&tmap_b);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), static_cast<uint32_t>(p.tmem_cols));
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // after the TMEM of this CTA is secured: a dependent grid's CTA on this SM can then never hold what this one waits for
    if (threadIdx.x == 0) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    cs_cluster_arrive();          // (1) this CTA runs: its shared memory may be written by the others

    if (warp == 0) {
        if (elect_one()) {
            int tap = kb0 / p.cchunks, cc = kb0 - tap * p.cchunks;
            const int pre = nkb < p.stages ? nkb : p.stages;
            if (!p.wdyn) {        // weights are constants: requested before the wait for the preceding kernel
                int t2 = tap, c2 = cc;
                for (int i = 0; i < pre; ++i) {
                    mbar_expect_tx(full_bar(i), stage_bytes);
                    tma_load_3d(smem_base + static_cast<uint32_t>(i) * stage_bytes + CS_A_BYTES, &tmap_b, full_bar(i), c2 * 64, t2, n0);
                    if (++c2 == p.cchunks) { c2 = 0; ++t2; }
                }
            }
            int img = 0, h0 = 0, w0 = 0;
            if (p.im2col) {
                img = static_cast<int>(fastdiv(static_cast<uint32_t>(m0), p.div_pq));
                const int rem = m0 - img * p.P * p.Q;
                const int pp = static_cast<int>(fastdiv(static_cast<uint32_t>(rem), p.div_q));
                h0 = pp * p.sh - p.ph;
                w0 = (rem - pp * p.Q) * p.sw - p.pw;
            }
            int r = tap / p.S, s = tap - r * p.S;
            int stage = 0;
            uint32_t phase = 0;
            asm volatile("griddepcontrol.wait;" ::: "memory");
            for (int i = 0; i < nkb; ++i) {
                const uint32_t dst = smem_base + static_cast<uint32_t>(stage) * stage_bytes, bar = full_bar(stage);
                if (i >= pre && !mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag)) {
                    atomicExch(p.status, STATUS_WAIT_SPLIT);
                    break;
                }
                if (i >= pre || p.wdyn) {
                    mbar_expect_tx(bar, stage_bytes);
                    tma_load_3d(dst + CS_A_BYTES, &tmap_b, bar, cc * 64, tap, n0);
                }
                if (p.im2col) tma_load_im2col_4d(dst, &tmap_a, bar, cc * 64, w0, h0, img, static_cast<uint16_t>(s * p.dw), static_cast<uint16_t>(r * p.dh));
                else tma_load_2d(dst, &tmap_a, bar, cc * 64, m0);
                if (++cc == p.cchunks) {
                    cc = 0;
                    ++tap;
                    if (++s == p.S) { s = 0; ++r; }
                }
                if (++stage == p.stages) { stage = 0; phase ^= 1u; }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t idesc = umma_idesc_f16_f32(128, p.BN);
            const uint32_t hi128 = static_cast<uint32_t>(umma_desc_sw128(0) >> 32);
            const uint32_t lo0 = ((smem_base & 0x3ffffu) >> 4) | 0x10000u;
            int stage = 0;
            uint32_t phase = 0;
            bool failed = false;
            for (int i = 0; i < nkb; ++i) {      // every load is waited for, also after a wait that ran out
                failed |= !mbar_wait(full_bar(stage), phase, abort_flag);
                tc_fence_after();
                const uint32_t lo = lo0 + static_cast<uint32_t>(stage) * (stage_bytes >> 4);
                umma_f16_kblock(tmem_base, lo, hi128, lo + (CS_A_BYTES >> 4), hi128, idesc, static_cast<uint32_t>(i != 0));
                umma_commit(empty_bar(stage));
                if (++stage == p.stages) { stage = 0; phase ^= 1u; }
            }
            umma_commit(tfull_bar);
            if (failed) atomicExch(p.status, STATUS_WAIT_SPLIT);
        }
        __syncwarp();
    }

    if (warp < 2) {
        cs_cluster_wait();
        cs_cluster_arrive();
        cs_cluster_wait();
        if (warp == 1) {
            __syncwarp();
            tc_fence_after();
            tmem_dealloc(tmem_base, static_cast<uint32_t>(p.tmem_cols));
        }
        return;
    }

    // ------------------------------------------------------------------ epilogue
    const int et = static_cast<int>(threadIdx.x) - 64;
    const int valid = min(128, p.M - m0);
    const int rs = (valid + p.split - 1) / p.split, rsp = rs | 1;     // rows of a slice, padded to an odd count
    const int r0 = rank * rs;
    const int lg8 = p.lg_bn - 3;                                      // log2 of the 8-channel units per row
    const int units = max(0, min(rs, valid - r0)) << lg8;
    asm volatile("griddepcontrol.wait;" ::: "memory");                // the residual may be the preceding kernel's output
    uint4 res[CS_UNITS];
    cs_residual(p, res, et, units, lg8, m0 + r0, n0);
    if (!mbar_wait<32>(tfull_bar, 0u, abort_flag)) {
        if (lane == 0) atomicExch(p.status, STATUS_WAIT_SPLIT);
    }
    tc_fence_after();
    cs_cluster_wait();            // (1)
    {
        const int row = (warp & 3) * 32 + lane;
        const int owner = row < valid ? row / rs : 0;
        const uint32_t peer = mapa_shared(red_base, static_cast<uint32_t>(owner)) +
                              static_cast<uint32_t>((rank * (p.BN >> 2)) * rsp + (row - owner * rs)) * 16u;
        const int half = p.BN >> 1, c_begin = ((warp - 2) >> 2) * half;
        cs_send(p, tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16), peer, c_begin, c_begin + half, rsp, row < valid);
    }
    tc_fence_before();
    cs_cluster_arrive();          // (2) this CTA's partial sums are where they belong
    cs_cluster_wait();
    cs_output(p, res, et, units, lg8, m0 + r0, n0, red_base, rsp);
}

// The same with CTA pairs: a cluster of 2 x split CTAs shares a tile of 256 pixels x BN channels, pair q (ranks 2q, 2q + 1)
// multiplies its run of k-blocks with tcgen05.mma.cta_group::2 (each CTA holds 128 rows of A and half of the B tile, as in
// conv_pair_kernel) and row slice o of a CTA's 128 rows is finished by the CTA of the same half in pair o. For layers that have
// very many k-blocks and about half as many tiles as there are pairs: a 256-wide tile needs a third less L2 -> SM traffic per
// product than a single CTA's. 3x3 2048 -> 256 at 64x128, dilation 12 (288 k-blocks, 32 tiles): 59.4 us with two pairs per tile
// against 69.0 stream-K and 71.7 plain pairs; with 72 k-blocks or fewer the exchange of 128 KB per CTA (about 8 us) costs more.
// The exchange (fp32, 128 x BN per CTA) takes the place of the pipeline stages once every MMA of the cluster has finished.
__global__ void __launch_bounds__(CS_THREADS, 1)
conv_split_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const SplitParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t stage_bytes = CS_A_BYTES + static_cast<uint32_t>(p.BN) * 64u;
    const uint32_t red_base = smem_base;
    const uint32_t bar_base = smem_base + p.red_bytes;       // red_bytes covers the stages and the exchange
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (CS_MAX_STAGES + s); };
    const uint32_t tfull_bar = bar_base + 8u * (2 * CS_MAX_STAGES);
    const uint32_t misc_off = (bar_base - smem_u32(smem_raw)) + 8u * (2 * CS_MAX_STAGES + 1);
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_raw + misc_off);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_raw + misc_off + 4);

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const int rank = static_cast<int>(cluster_ctarank()), side = rank & 1, run = rank >> 1;
    const int tile = static_cast<int>(fastdiv(blockIdx.x >> 1, p.div_split));
    const int m_tile = static_cast<int>(fastdiv(static_cast<uint32_t>(tile), p.div_ntiles));
    const int n0 = (tile - m_tile * p.n_tiles) * p.BN;
    const int m0 = (2 * m_tile + side) * 128;
    const int kb0 = run * p.kblocks / p.split, nkb = (run + 1) * p.kblocks / p.split - kb0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(full_bar(s), 2);               // one arrive.expect_tx per CTA of the pair (used in the even CTA only)
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(tfull_bar, 1);
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmap_a);
        tma_prefetch_desc(&tmap_b);
    }
    if (warp == 1) {
        tmem_pair_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), static_cast<uint32_t>(p.tmem_cols));
        tmem_pair_relinquish();
    }
    // both CTAs' barriers exist before either signals one of the other's
    tc_fence_before();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (threadIdx.x == 0) pdl_trigger();      // after the TMEM of this CTA is secured

    if (warp == 0) {
        if (elect_one()) {
            int tap = kb0 / p.cchunks, cc = kb0 - tap * p.cchunks;
            const int pre = nkb < p.stages ? nkb : p.stages;
            const uint32_t lead_full0 = mapa_shared(full_bar(0), static_cast<uint32_t>(rank & ~1));
            const int b_row0 = n0 + side * (p.BN / 2);
            {
                int t2 = tap, c2 = cc;
                for (int i = 0; i < pre; ++i) {     // weights are constants: requested before the wait for the preceding kernel
                    const uint32_t bar = lead_full0 + 8u * static_cast<uint32_t>(i);
                    mbar_expect_tx_cluster(bar, stage_bytes);
                    tma_pair_load_3d(smem_base + static_cast<uint32_t>(i) * stage_bytes + CS_A_BYTES, &tmap_b, bar, c2 * 64, t2, b_row0);
                    if (++c2 == p.cchunks) { c2 = 0; ++t2; }
                }
            }
            const int ml = m0 < p.M ? m0 : m0 - 128;     // rows past the last pixel: the even CTA's once more, results dropped
            int img = 0, h0 = 0, w0 = 0;
            if (p.im2col) {
                img = static_cast<int>(fastdiv(static_cast<uint32_t>(ml), p.div_pq));
                const int rem = ml - img * p.P * p.Q;
                const int pp = static_cast<int>(fastdiv(static_cast<uint32_t>(rem), p.div_q));
                h0 = pp * p.sh - p.ph;
                w0 = (rem - pp * p.Q) * p.sw - p.pw;
            }
            int r = tap / p.S, s = tap - r * p.S;
            int stage = 0;
            uint32_t phase = 0;
            pdl_wait();
            for (int i = 0; i < nkb; ++i) {
                const uint32_t dst = smem_base + static_cast<uint32_t>(stage) * stage_bytes;
                const uint32_t bar = lead_full0 + 8u * static_cast<uint32_t>(stage);
                if (i >= pre) {
                    if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag)) {
                        atomicExch(p.status, STATUS_WAIT_SPLIT);
                        break;
                    }
                    mbar_expect_tx_cluster(bar, stage_bytes);
                    tma_pair_load_3d(dst + CS_A_BYTES, &tmap_b, bar, cc * 64, tap, b_row0);
                }
                if (p.im2col) tma_pair_load_im2col_4d(dst, &tmap_a, bar, cc * 64, w0, h0, img, static_cast<uint16_t>(s * p.dw), static_cast<uint16_t>(r * p.dh));
                else tma_pair_load_2d(dst, &tmap_a, bar, cc * 64, ml);
                if (++cc == p.cchunks) {
                    cc = 0;
                    ++tap;
                    if (++s == p.S) { s = 0; ++r; }
                }
                if (++stage == p.stages) { stage = 0; phase ^= 1u; }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (side == 0 && elect_one()) {
            const uint32_t idesc = umma_idesc_f16_f32(256, p.BN);
            const uint32_t hi128 = static_cast<uint32_t>(umma_desc_sw128(0) >> 32);
            const uint32_t lo0 = ((smem_base & 0x3ffffu) >> 4) | 0x10000u;
            const uint32_t peer_empty0 = mapa_shared(empty_bar(0), static_cast<uint32_t>(rank | 1));
            const uint32_t peer_tfull = mapa_shared(tfull_bar, static_cast<uint32_t>(rank | 1));
            int stage = 0;
            uint32_t phase = 0;
            bool failed = false;
            for (int i = 0; i < nkb; ++i) {      // every load is waited for, also after a wait that ran out
                failed |= !mbar_wait(full_bar(stage), phase, abort_flag);
                tc_fence_after();
                const uint32_t lo = lo0 + static_cast<uint32_t>(stage) * (stage_bytes >> 4);
                umma_pair_f16_kblock(tmem_base, lo, hi128, lo + (CS_A_BYTES >> 4), hi128, idesc, static_cast<uint32_t>(i != 0));
                umma_pair_commit(empty_bar(stage));
                umma_pair_commit(peer_empty0 + 8u * static_cast<uint32_t>(stage));
                if (++stage == p.stages) { stage = 0; phase ^= 1u; }
            }
            umma_pair_commit(tfull_bar);
            umma_pair_commit(peer_tfull);
            if (failed) atomicExch(p.status, STATUS_WAIT_SPLIT);
        }
        __syncwarp();
    }

    if (warp < 2) {
        cs_cluster_arrive();
        cs_cluster_wait();
        cs_cluster_arrive();
        cs_cluster_wait();
        if (warp == 1) {
            __syncwarp();
            tc_fence_after();
            tmem_pair_dealloc(tmem_base, static_cast<uint32_t>(p.tmem_cols));
        }
        return;
    }

    const int et = static_cast<int>(threadIdx.x) - 64;
    const int valid = max(0, min(128, p.M - m0));
    const int rs = max(1, (valid + p.split - 1) / p.split), rsp = rs | 1;
    const int r0 = run * rs;
    const int lg8 = p.lg_bn - 3;
    const int units = max(0, min(rs, valid - r0)) << lg8;
    pdl_wait();                   // the residual may be the preceding kernel's output
    uint4 res[CS_UNITS];
    cs_residual(p, res, et, units, lg8, m0 + r0, n0);
    if (!mbar_wait<32>(tfull_bar, 0u, abort_flag)) {
        if (lane == 0) atomicExch(p.status, STATUS_WAIT_SPLIT);
    }
    tc_fence_after();
    cs_cluster_arrive();          // (1) the MMAs that read this CTA's stages have finished: the exchange may be written there
    cs_cluster_wait();
    {
        const int row = (warp & 3) * 32 + lane;
        const int owner = row < valid ? row / rs : 0;
        const uint32_t peer = mapa_shared(red_base, static_cast<uint32_t>(2 * owner + side)) +
                              static_cast<uint32_t>((run * (p.BN >> 2)) * rsp + (row - owner * rs)) * 16u;
        const int half = p.BN >> 1, c_begin = ((warp - 2) >> 2) * half;
        cs_send(p, tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16), peer, c_begin, c_begin + half, rsp, row < valid);
    }
    tc_fence_before();
    cs_cluster_arrive();          // (2) this CTA's partial sums are where they belong
    cs_cluster_wait();
    for (int u0 = et; ; u0 += CS_UNITS * 32 * CS_EPI_WARPS) {
        cs_output(p, res, u0, units, lg8, m0 + r0, n0, red_base, rsp);
        if (u0 - et + CS_UNITS * 32 * CS_EPI_WARPS >= units) break;
        cs_residual(p, res, u0 + CS_UNITS * 32 * CS_EPI_WARPS, units, lg8, m0 + r0, n0);
    }
}

// Stages, exchange buffer and TMEM columns for `split` CTAs per tile of 128 x BN; false if the shape cannot run this way.
bool conv_split_plan(SplitParams* p, size_t* smem) {
    if (p->pair) {
        if ((p->BN != 64 && p->BN != 128 && p->BN != 256) || p->split < 2 || p->split > 4 || p->split > p->kblocks || p->wdyn) return false;
        const int rs = (128 + p->split - 1) / p->split;
        p->lg_bn = p->BN == 64 ? 6 : p->BN == 128 ? 7 : 8;
        p->tmem_cols = p->BN;
        const uint32_t stage = CS_A_BYTES + static_cast<uint32_t>(p->BN) * 64u;
        const uint32_t fixed = 1024 + 8 * (2 * CS_MAX_STAGES + 1) + 16;
        int stages = static_cast<int>((226u * 1024 - fixed) / stage);
        const int need = (p->kblocks + p->split - 1) / p->split;
        if (stages > need) stages = need;
        if (stages > CS_MAX_STAGES) stages = CS_MAX_STAGES;
        p->stages = stages;
        const uint32_t red = static_cast<uint32_t>(p->split * (p->BN >> 2) * (rs | 1) * 16);
        const uint32_t pipe = static_cast<uint32_t>(stages) * stage;
        p->red_bytes = ((red > pipe ? red : pipe) + 1023) & ~1023u;
        *smem = fixed + p->red_bytes;
        if (*smem < 120 * 1024) *smem = 120 * 1024;       // one CTA per SM
        return *smem <= 227 * 1024;
    }
    if (p->BN != 32 && p->BN != 64 && p->BN != 128) return false;
    if (p->split < 1 || p->split > 8 || p->split > p->kblocks) return false;
    const int rs = (128 + p->split - 1) / p->split;
    if ((rs * p->BN >> 3) > CS_UNITS * 32 * CS_EPI_WARPS) return false;
    p->lg_bn = p->BN == 32 ? 5 : p->BN == 64 ? 6 : 7;
    p->red_bytes = static_cast<uint32_t>(p->split * (p->BN >> 2) * ((rs | 1) + 1) * 16 + 1023) & ~1023u;
    p->tmem_cols = p->BN;
    const uint32_t stage = CS_A_BYTES + static_cast<uint32_t>(p->BN) * 128u;
    const uint32_t fixed = 1024 + p->red_bytes + 8 * (2 * CS_MAX_STAGES + 1) + 16;
    const int need = (p->kblocks + p->split - 1) / p->split;
    // below 104 KB two CTAs (also one of this kernel and one of the persistent kernels' 120 KB) share an SM; a pipeline that
    // would have fewer than three stages there takes what the SM has
    int stages = static_cast<int>((104u * 1024 - fixed) / stage);
    if (fixed > 104u * 1024 || (stages < 3 && stages < need)) stages = static_cast<int>((226u * 1024 - fixed) / stage);
    if (stages > need) stages = need;
    if (stages > CS_MAX_STAGES) stages = CS_MAX_STAGES;
    if (stages < 1) return false;
    p->stages = stages;
    *smem = fixed + static_cast<size_t>(stages) * stage;
    return true;
}

int conv_split_launch(const CUtensorMap& tmap_a, const CUtensorMap& tmap_b, const SplitParams& p, size_t smem, cudaStream_t stream) {
    auto kernel = p.pair ? conv_split_pair_kernel : conv_split_kernel;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) return FVM_ERR_SETUP;
    const int cluster = p.pair ? 2 * p.split : p.split;
    const int m_tiles = p.pair ? (p.M + 255) / 256 : (p.M + 127) / 128;
    return launch_pdl(kernel, dim3(static_cast<unsigned>(m_tiles * p.n_tiles * cluster)), dim3(CS_THREADS), smem, stream, cluster,
                      tmap_a, tmap_b, p);
}

}  // namespace fvm
