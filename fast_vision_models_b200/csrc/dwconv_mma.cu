// Depthwise 7x7 convolution (stride 1, no dilation) on the tensor cores, NHWC fp16, fp32 accumulation.
//
// One row of a depthwise filter applied to 16 consecutive input columns of ONE channel gives 8 output columns: a
// [16 columns] x [16 x 8 Toeplitz matrix of the row's taps] product. dw7_mma_kernel makes that the shape of an
// mma.sync.m16n8k16: the 16 rows of A are 16 "strips" (a strip = 8 output columns, marching down the rows of its part of
// the map; strips of a block are neighbours in x, row segments, or images), B is the Toeplitz matrix of one filter row, held
// in two registers per lane, and each loaded input row feeds the 7 output rows it belongs to: 7 fp32 accumulator
// fragments rotate through the registers. Per 128 outputs that is 7 matrix instructions and little more than one ldmatrix;
// 7 of 16 products are useful. The fp16x2 FMA kernel (dw_tile_kernel) is bound by the FMA pipe and by reading every input
// vector several times from shared memory; this one by the four barriers of a tile and its serial chains (with a predicate per matrix
// instruction, 39 us for 56x56x96, the hmma pipe was busy 39 % of the time, the schedulers 43 %; three blocks per SM instead of
// two need 80 registers a thread and gain nothing: 29.0 us).
// ConvNeXt-T layers, batch 64, us with the FMA kernel / this one (share of HBM bandwidth): 56x56x96 62.7 / 27.9 (0.43),
// 28x28x192 35.0 / 18.5 (0.32), 14x14x384 29.2 / 12.6, 7x7x768 14.0 / 9.3; batch 8 at 56x56x96 12.1 / 8.2.
// With 3 or 5 taps the useful share is too small: 95x95x192 3x3 191 us against 128, 48x48x336 5x5 125 against 86 (tile kernel).
//
// The matrix unit wants one channel's columns side by side, NHWC has the channels side by side, so a block's input patch is
// transposed once in shared memory (8x8 blocks, ldmatrix.trans -> stmatrix, about two shared-memory cycles per 64 elements)
// and the outputs are transposed back the same way on their way to a TMA store:
//   A: patch as TMA writes it  [image][row][column][8 channels]   -> B: planes [channel][image][row][column]
//   B: planes                  -> mma                             -> C: planes [channel][output row][strip][8]
//   C: output planes           -> B: [image][row][column][8 channels], stored by one TMA copy (clipped at the map's edges).
// Blocks are persistent: a block keeps its 8 channels (a warp its channel, with the Toeplitz matrices in registers) and walks
// tiles; the next patch is on its way to A while the present one is multiplied. Two blocks share an SM. Blocks of 8 channels
// were faster than 16 and 32 (56x56x96, batch 64, with predicates: 39 / 50 / 90 us): they allow the tallest segments, and a segment pays six
// rows of border.
//
// A column outside an output's window meets a zero of the Toeplitz matrix, which is harmless for finite values only. The
// transposition therefore looks at every staged value; a tile that holds an infinity or a NaN takes the direct sum
// (dw7_direct_part) over the same planes, so that exactly the outputs whose window holds the value are affected.
#include <cuda.h>

#include <cstdint>
#include <cstring>

#include "fvm_internal.h"
#include "ptx_sm100.cuh"

namespace fvm {

static constexpr int DM_S = 7;
static constexpr int DM_CB = 8;                    // channels per block, one per warp
static constexpr int DM_THREADS = 32 * DM_CB;
static constexpr int DM_STRIPS = 16;               // rows of the mma's A operand
static constexpr int DM_SMEM_LIMIT = 112 * 1024;   // two blocks per SM
static constexpr int STATUS_WAIT_DM = 0x106;

struct DmParams {
    int C, P, Q, N, ph, pw;
    int xb, segs, nimg;      // strips of a tile: xb 8-column blocks x segs row segments x nimg images, at most 16
    int rr;                  // output rows of a segment
    int tile_h, tile_w;      // staged patch: segs * rr + 6 rows, xb * 8 + 8 columns
    int tiles_x, tiles_y, vblocks;
    int tiles;               // tiles_x * tiles_y * ceil(N / nimg)
    int groups;              // 8-pixel groups of the staged patch
    int plane, oplane;       // bytes of one channel's input / output plane (odd multiples of 16: conflict-free 8x8 blocks)
    int buf_a, buf_b, buf_c; // bytes of the three buffers
    int act;
    int* status;
};

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void stsm_x4(uint32_t addr, const uint32_t (&r)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
__device__ __forceinline__ void stsm_x2(uint32_t addr, uint32_t r0, uint32_t r1) {
    asm volatile("stmatrix.sync.aligned.m8n8.x2.shared.b16 [%0], {%1, %2};" ::"r"(addr), "r"(r0), "r"(r1) : "memory");
}
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, float c0, float c1,
                                          float c2, float c3) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}

struct TrueTag { static constexpr bool value = true; };
struct FalseTag { static constexpr bool value = false; };

// fp32 pair -> rounded fp16 pair -> activation (evaluated on the rounded sum, rounded again: as dw_tile_kernel does)
template <int ACT>
__device__ __forceinline__ uint32_t dm_finish(float lo, float hi, int act) {
    uint32_t h;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(hi), "f"(lo));
    if (ACT != 0) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
        const __half2 o = __floats2half2_rn(act_f(f.x, act), act_f(f.y, act));
        return *reinterpret_cast<const uint32_t*>(&o);
    }
    return h;
}

// Direct sums over the planes of a tile whose patch holds a value that is not finite: same outputs, same places.
template <int ACT>
__device__ __noinline__ void dw7_direct_part(const DmParams& p, const uint8_t* planes, uint8_t* oplanes, const __half* w_s,
                                             const __half* __restrict__ bias, const int* strip_off, int c0) {
    const int ns = p.xb * p.segs * p.nimg;
    for (int i = threadIdx.x; i < DM_CB * p.rr * ns * 8; i += DM_THREADS) {
        const int px = i & 7;
        int k = i >> 3;
        const int strip = k % ns;
        k /= ns;
        const int row = k % p.rr, c = k / p.rr;
        const __half* src = reinterpret_cast<const __half*>(planes + c * p.plane + strip_off[strip]) + row * p.tile_w + px;
        float acc = bias ? __half2float(bias[c0 + c]) : 0.f;
        for (int r = 0; r < DM_S; ++r)
            for (int s = 0; s < DM_S; ++s)
                acc = fmaf(__half2float(src[r * p.tile_w + s]), __half2float(w_s[(r * DM_S + s) * DM_CB + c]), acc);
        const uint32_t h = dm_finish<ACT>(acc, 0.f, p.act);
        *reinterpret_cast<uint16_t*>(oplanes + c * p.oplane + row * 256 + strip * 16 + px * 2) = static_cast<uint16_t>(h & 0xffffu);
    }
}

// ANYROWS: segments of any height; false: a multiple of 7 rows, so that the first and the last 7 input rows of a strip know at
// compile time which products they have (no predicate per matrix instruction).
template <int ACT, bool ANYROWS>
__global__ void __launch_bounds__(DM_THREADS, 2)
dw7_mma_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_y,
              const __half* __restrict__ w, const __half* __restrict__ bias, float* __restrict__ pool_partial,
              const DmParams p) {
    constexpr int S = DM_S;
    extern __shared__ __align__(128) uint8_t dm_smem[];
    uint8_t* buf_a = dm_smem + ((128u - (smem_u32(dm_smem) & 127u)) & 127u);
    uint8_t* buf_b = buf_a + p.buf_a;
    uint8_t* buf_c = buf_b + p.buf_b;
    float* pool_s = reinterpret_cast<float*>(buf_c + p.buf_c);                    // [channel][strip]
    __half* w_s = reinterpret_cast<__half*>(pool_s + DM_CB * DM_STRIPS);          // [tap][channel]
    int* strip_off = reinterpret_cast<int*>(w_s + S * S * DM_CB);                 // byte offset of a strip inside a plane
    int* strip_px = strip_off + DM_STRIPS;                                        // first pixel of a strip in the output tile
    volatile int* abort_flag = strip_px + DM_STRIPS;
    const uint32_t a0 = smem_u32(buf_a), b0 = smem_u32(buf_b), o0 = smem_u32(buf_c), bar = smem_u32(strip_px + DM_STRIPS) + 8u;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // the channel blocks of one tile run side by side (they share cache lines); a block keeps its channels and walks tiles
    const int vb = blockIdx.x % p.vblocks, tile_step = gridDim.x / p.vblocks;
    const int c0 = vb * DM_CB;
    const int ns = p.xb * p.segs * p.nimg;
    const uint32_t tx_bytes = static_cast<uint32_t>(p.groups) * 128u;
    auto tile_pos = [&](int tile, int& q0, int& p0, int& n0) {
        const int ty = tile / p.tiles_x;
        q0 = (tile - ty * p.tiles_x) * p.xb * 8;
        const int im = ty / p.tiles_y;
        p0 = (ty - im * p.tiles_y) * p.segs * p.rr;
        n0 = im * p.nimg;
    };
    int tile = blockIdx.x / p.vblocks;
    int q0, p0, n0;

    if (tid == 0) {
        *abort_flag = 0;
        mbar_init(bar, 1);
        mbar_fence_init();
        tile_pos(tile, q0, p0, n0);
        pdl_wait();                // the copy is the block's first access to the input
        mbar_expect_tx(bar, tx_bytes);
        tma_load_4d(a0, &tmap_x, bar, c0, q0 - p.pw, p0 - p.ph, n0);
    }
    {
        if (tid < S * S)
            reinterpret_cast<uint4*>(w_s)[tid] = __ldg(reinterpret_cast<const uint4*>(w + static_cast<long long>(tid) * p.C + c0));
        if (tid < DM_STRIPS) {
            const int st = tid < ns ? tid : ns - 1;       // rows past the last strip repeat it; nothing of them is stored
            const int x = st % p.xb, sg = st / p.xb % p.segs, im = st / (p.xb * p.segs);
            strip_off[tid] = ((im * p.tile_h + sg * p.rr) * p.tile_w + x * 8) * 2;
            strip_px[tid] = (im * p.segs + sg) * p.rr * p.xb * 8 + x * 8;
        }
    }
    __syncthreads();

    // lane's part in a move of four 8x8 blocks: row lane % 8 of pixel group lane / 8
    const int pg = lane >> 3, li = lane & 7;
    const int g = lane >> 2, t = lane & 3;
    // taps this lane holds of the Toeplitz matrix: B[k][n] = w[k - n], k = 2t, 2t + 1, 2t + 8, 2t + 9, n = g
    const int i0 = 2 * t - g, i1 = i0 + 1, i2 = i0 + 8, i3 = i0 + 9;
    const uint32_t a_lane = b0 + static_cast<uint32_t>(strip_off[lane & 15] + (lane >> 4) * 16);
    const uint32_t row_bytes = static_cast<uint32_t>(p.tile_w) * 2u;
    const int rows = p.rr + S - 1;
    const int c = warp;                        // this warp's channel of the block
    uint32_t bw[S][2];
#pragma unroll
    for (int r = 0; r < S; ++r) {
        const unsigned short* wr = reinterpret_cast<const unsigned short*>(w_s) + r * S * DM_CB + c;
        const uint32_t v0 = (i0 >= 0 && i0 < S) ? wr[i0 * DM_CB] : 0u, v1 = (i1 >= 0 && i1 < S) ? wr[i1 * DM_CB] : 0u;
        const uint32_t v2 = (i2 >= 0 && i2 < S) ? wr[i2 * DM_CB] : 0u, v3 = (i3 >= 0 && i3 < S) ? wr[i3 * DM_CB] : 0u;
        bw[r][0] = v0 | (v1 << 16);
        bw[r][1] = v2 | (v3 << 16);
    }
    const float bc = bias ? __half2float(bias[c0 + c]) : 0.f;
    pdl_wait();                    // every thread, before the outputs and squeeze sums

    for (uint32_t phase = 0; tile < p.tiles; tile += tile_step, phase ^= 1u) {
        tile_pos(tile, q0, p0, n0);
        if (!mbar_wait<32>(bar, phase, abort_flag)) {
            if (tid == 0) atomicExch(p.status, STATUS_WAIT_DM);
            return;
        }
        if (tid == 0) tma_store_wait_read();       // the previous tile has left buffer B
        __syncthreads();
        __half2 seen = __float2half2_rn(0.f);
        for (int gr = warp * 4; gr < p.groups; gr += DM_CB * 4) {
            const int gi = min(gr + pg, p.groups - 1);
            uint32_t r[4];
            ldsm_x4_trans(r, a0 + static_cast<uint32_t>(gi * 8 + li) * 16u);
#pragma unroll
            for (int k = 0; k < 4; ++k) seen = __hfma2(*reinterpret_cast<const __half2*>(&r[k]), __float2half2_rn(0.f), seen);
            stsm_x4(b0 + static_cast<uint32_t>(li * p.plane + gi * 16), r);
        }
        const bool odd = (*reinterpret_cast<const uint32_t*>(&seen) & 0x7fff7fffu) != 0u;      // 0 * x is not 0
        const bool direct = __syncthreads_or(odd);
        if (tid == 0 && tile + tile_step < p.tiles) {        // the patch has been read: the next one may land in A
            int q1, p1, n1;
            tile_pos(tile + tile_step, q1, p1, n1);
            mbar_expect_tx(bar, tx_bytes);
            tma_load_4d(a0, &tmap_x, bar, c0, q1 - p.pw, p1 - p.ph, n1);
        }

        if (!direct) {
            int rows_ok[2] = {0, 0}, cols_ok[2] = {0, 0};              // squeeze: valid rows / columns of strips g, g + 8
            if (pool_partial) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int st = g + 8 * h;
                    if (st < ns) {
                        const int x = st % p.xb, sg = st / p.xb % p.segs, im = st / (p.xb * p.segs);
                        cols_ok[h] = p.Q - (q0 + x * 8 + 2 * t);
                        rows_ok[h] = n0 + im < p.N ? p.P - (p0 + sg * p.rr) : 0;
                    }
                }
            }
            {
                float acc[S][4];
                float sum0 = 0.f, sum1 = 0.f;
                uint32_t src = a_lane + static_cast<uint32_t>(c * p.plane);
                uint32_t dst = o0 + static_cast<uint32_t>(c * p.oplane + (lane & 15) * 16);
                uint32_t nxt[4];
                ldsm_x4(nxt, src);
                auto emit = [&](const float (&d)[4], int row) {
                    const uint32_t h0 = dm_finish<ACT>(d[0], d[1], p.act), h1 = dm_finish<ACT>(d[2], d[3], p.act);
                    stsm_x2(dst, h0, h1);
                    dst += 256;
                    if (pool_partial) {
                        const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&h0));
                        const float2 f1 = __half22float2(*reinterpret_cast<const __half2*>(&h1));
                        if (row < rows_ok[0]) sum0 += (cols_ok[0] > 0 ? f0.x : 0.f) + (cols_ok[0] > 1 ? f0.y : 0.f);
                        if (row < rows_ok[1]) sum1 += (cols_ok[1] > 0 ? f1.x : 0.f) + (cols_ok[1] > 1 ? f1.y : 0.f);
                    }
                };
                // rotating accumulators: input row y belongs to output rows y - r, r = 0 .. S - 1; row y - r sits in slot
                // (y - r) mod S; products for rows before the first or past the last are skipped.
                if constexpr (ANYROWS) {
                    for (int y0 = 0; y0 < rows; y0 += S) {
#pragma unroll
                        for (int j = 0; j < S; ++j) {
                            const int y = y0 + j;
                            if (y < rows) {
                                uint32_t a[4] = {nxt[0], nxt[1], nxt[2], nxt[3]};
                                if (y + 1 < rows) src += row_bytes;
                                ldsm_x4(nxt, src);                       // the next row under this row's products
#pragma unroll
                                for (int r = 0; r < S; ++r) {
                                    float (&d)[4] = acc[(j - r + S) % S];
                                    if (y - r < p.rr) {
                                        if (r == 0) mma_16816(d, a, bw[r][0], bw[r][1], bc, bc, bc, bc);
                                        else if (j >= r || y0 > 0) mma_16816(d, a, bw[r][0], bw[r][1], d[0], d[1], d[2], d[3]);
                                    }
                                }
                                if (y >= S - 1) emit(acc[(j + 1) % S], y - (S - 1));
                            }
                        }
                    }
                } else {
                    auto seven = [&](auto first_, auto last_, int y0) {
                        constexpr bool FIRST = decltype(first_)::value, LAST = decltype(last_)::value;
#pragma unroll
                        for (int j = 0; j < (LAST ? S - 1 : S); ++j) {
                            uint32_t a[4] = {nxt[0], nxt[1], nxt[2], nxt[3]};
                            if (!LAST || j < S - 2) {
                                src += row_bytes;
                                ldsm_x4(nxt, src);                       // the next row under this row's products
                            }
#pragma unroll
                            for (int r = 0; r < S; ++r) {
                                float (&d)[4] = acc[(j - r + S) % S];
                                if ((!FIRST || j >= r) && (!LAST || j < r)) {
                                    if (r == 0) mma_16816(d, a, bw[r][0], bw[r][1], bc, bc, bc, bc);
                                    else mma_16816(d, a, bw[r][0], bw[r][1], d[0], d[1], d[2], d[3]);
                                }
                            }
                            if (!FIRST || j == S - 1) emit(acc[(j + 1) % S], y0 + j - (S - 1));
                        }
                    };
                    seven(TrueTag{}, FalseTag{}, 0);
                    for (int y0 = S; y0 < p.rr; y0 += S) seven(FalseTag{}, FalseTag{}, y0);
                    seven(FalseTag{}, TrueTag{}, p.rr);
                }
                if (pool_partial) {
                    sum0 += __shfl_xor_sync(0xffffffffu, sum0, 1);
                    sum1 += __shfl_xor_sync(0xffffffffu, sum1, 1);
                    sum0 += __shfl_xor_sync(0xffffffffu, sum0, 2);
                    sum1 += __shfl_xor_sync(0xffffffffu, sum1, 2);
                    if (t == 0) {
                        pool_s[c * DM_STRIPS + g] = sum0;
                        pool_s[c * DM_STRIPS + g + 8] = sum1;
                    }
                }
            }
        } else {
            dw7_direct_part<ACT>(p, buf_b, buf_c, w_s, bias, strip_off, c0);
            if (pool_partial) {
                __syncthreads();
                for (int i = tid; i < DM_CB * ns; i += DM_THREADS) {
                    const int ch = i / ns, st = i % ns;
                    const int x = st % p.xb, sg = st / p.xb % p.segs, im = st / (p.xb * p.segs);
                    const int cols = min(8, p.Q - (q0 + x * 8)), nrow = n0 + im < p.N ? min(p.rr, p.P - (p0 + sg * p.rr)) : 0;
                    float s = 0.f;
                    for (int r = 0; r < nrow; ++r)
                        for (int k = 0; k < cols; ++k)
                            s += __half2float(*reinterpret_cast<const __half*>(buf_c + ch * p.oplane + r * 256 + st * 16 + k * 2));
                    pool_s[ch * DM_STRIPS + st] = s;
                }
            }
        }
        __syncthreads();

        // output planes -> [image][row][column][channel]
        const uint32_t out_row = static_cast<uint32_t>(p.xb * 8);
        for (int it = warp; it < p.rr * 4; it += DM_CB) {            // four strips of a row at a time
            const int row = it >> 2, s0 = (it & 3) * 4;
            if (s0 >= ns) continue;
            const int st = min(s0 + pg, ns - 1);
            uint32_t r[4];
            ldsm_x4_trans(r, o0 + static_cast<uint32_t>(li * p.oplane + row * 256 + st * 16));
            stsm_x4(b0 + (static_cast<uint32_t>(strip_px[st]) + row * out_row + li) * 16u, r);
        }
        fence_proxy_async_smem();
        __syncthreads();
        if (tid == 0) {
            tma_store_4d(&tmap_y, b0, c0, q0, p0, n0);
            tma_store_commit();
        }
        if (pool_partial) {
            const int per_img = p.xb * p.segs, slot = tile % (p.tiles_x * p.tiles_y);
            for (int i = tid; i < DM_CB * p.nimg; i += DM_THREADS) {
                const int ch = i % DM_CB, im = i / DM_CB;
                if (n0 + im < p.N) {
                    float s = 0.f;
                    for (int k = 0; k < per_img; ++k) s += pool_s[ch * DM_STRIPS + im * per_img + k];
                    pool_partial[(static_cast<long long>(n0 + im) * (p.tiles_x * p.tiles_y) + slot) * p.C + c0 + ch] = s;
                }
            }
        }
    }
    // only now: blocks of the next kernel that sit beside this one's tiles slowed both down (ConvNeXt-T, batch 64: 1648 us per
    // forward, 1674 with the trigger at the start)
    pdl_trigger();
    if (tid == 0) tma_store_wait_read();
}

struct DmPlan {
    DmParams p;
    size_t smem;
    unsigned grid;
    double cost;
};

// Tile geometry: the candidate with the least modelled time, per round of the persistent blocks: the matrix instructions
// (about 310 cycles per output row of a tile's 16 strips x 8 channels, 200 without predicates) and the copies in and out of the two blocks of an SM,
// or, for a block alone, its own plus the latency of its copies and barriers. Fitted to a sweep of all geometries for 18 maps
// (batch 1 to 64); a grid that puts a second block on each SM starts later (8x14x14x384: 5.9 us with 96 blocks, 6.5 with 192).
static bool dm_plan(int N, int H, int W, int C, int ph, int pw, int sms, DmPlan* out) {
    constexpr int S = DM_S;
    DmParams base;
    memset(&base, 0, sizeof(base));
    base.C = C; base.N = N; base.ph = ph; base.pw = pw;
    base.P = H + 2 * ph - S + 1;
    base.Q = W + 2 * pw - S + 1;
    if (base.P <= 0 || base.Q <= 0) return false;
    bool any = false;
    for (int xb = 1; xb <= DM_STRIPS && (xb == 1 || (xb - 1) * 8 < base.Q); ++xb)
        for (int segs = 1; segs * xb <= DM_STRIPS; ++segs)
            for (int rr = 2; rr <= 32; ++rr) {
                if (segs > 1 && (segs - 1) * rr >= base.P) break;
                const bool whole = xb * 8 >= base.Q && segs * rr >= base.P;
                for (int nimg = 1; nimg * segs * xb <= DM_STRIPS && nimg <= N && (nimg == 1 || whole); ++nimg) {
                    DmPlan d;
                    d.p = base;
                    DmParams& p = d.p;
                    p.xb = xb; p.segs = segs; p.nimg = nimg; p.rr = rr;
                    p.tile_h = segs * rr + S - 1;
                    p.tile_w = xb * 8 + 8;
                    if (p.tile_h > 256 || p.tile_w > 256) continue;
                    p.groups = nimg * p.tile_h * (xb + 1);
                    p.plane = p.groups * 16 + (p.groups & 1 ? 0 : 16);
                    p.oplane = rr * 256 + 16;
                    const int out_bytes = nimg * segs * rr * xb * 16 * DM_CB;
                    p.buf_a = p.groups * 16 * DM_CB;
                    p.buf_b = ((DM_CB * p.plane > out_bytes ? DM_CB * p.plane : out_bytes) + 127) / 128 * 128;
                    p.buf_c = DM_CB * p.oplane;
                    d.smem = 128 + static_cast<size_t>(p.buf_a) + p.buf_b + p.buf_c + DM_CB * DM_STRIPS * 4 + S * S * DM_CB * 2 + 2 * DM_STRIPS * 4 + 16;
                    if (d.smem > static_cast<size_t>(DM_SMEM_LIMIT)) break;
                    p.tiles_x = (base.Q + xb * 8 - 1) / (xb * 8);
                    p.tiles_y = (base.P + segs * rr - 1) / (segs * rr);
                    p.vblocks = C / DM_CB;
                    const long long tiles = static_cast<long long>(p.tiles_x) * p.tiles_y * ((N + nimg - 1) / nimg);
                    if (tiles > 0x3fffffff) break;
                    p.tiles = static_cast<int>(tiles);
                    const int slots = 2 * sms;
                    long long per_vb = slots / p.vblocks > 0 ? slots / p.vblocks : 1;
                    if (per_vb > tiles) per_vb = tiles;
                    d.grid = static_cast<unsigned>(per_vb * p.vblocks);
                    const double rounds = static_cast<double>((tiles + per_vb - 1) / per_vb) * ((d.grid + slots - 1) / slots);
                    const double on_sm = d.grid > static_cast<unsigned>(sms) ? 2.0 : 1.0;
                    if (on_sm > 1.0) {
                        const double busy = (rr % S ? 310.0 : 200.0) * rr + 3.0 * p.groups + 700.0;
                        d.cost = rounds * (2500.0 + busy > 2.0 * busy ? 2500.0 + busy : 2.0 * busy) + 4000.0;
                    } else {
                        d.cost = rounds * (2500.0 + (rr % S ? 230.0 : 160.0) * rr + 3.0 * p.groups);
                    }
                    if (!any || d.cost < out->cost) {
                        *out = d;
                        any = true;
                    }
                }
            }
    return any;
}

// The plan depends on sizes only; each thread keeps the last ones it made (a search of some thousand candidates).
static bool dm_plan_cached(int N, int H, int W, int C, int ph, int pw, DmPlan* out) {
    struct Entry { int key[7]; bool ok; DmPlan plan; };
    static thread_local Entry cache[64];
    const DeviceState* st = device_state();
    const int key[7] = {N, H, W, C, ph, pw, st ? st->sms : 148};
    uint32_t h = 2166136261u;
    for (int k : key) h = (h ^ static_cast<uint32_t>(k)) * 16777619u;
    Entry& e = cache[(h >> 16) & 63];
    if (memcmp(e.key, key, sizeof(key)) != 0) {
        e.ok = dm_plan(N, H, W, C, ph, pw, key[6], &e.plan);
        memcpy(e.key, key, sizeof(key));
    }
    *out = e.plan;
    return e.ok;
}

// Every stride-1 7x7 layer: also at the small end this one is faster (us, tile kernel / this one: one image 56x56x96 4.7 / 4.1,
// 14x14x384 5.1 / 3.9; 20 images 9x9x768 9.7 / 8.2).
bool dw_mma_runs(int N, int H, int W, int C, int ph, int pw) {
    DmPlan d;
    return dm_plan_cached(N, H, W, C, ph, pw, &d);
}

int dw_mma_slots(int N, int H, int W, int C, int ph, int pw) {
    DmPlan d;
    return dm_plan_cached(N, H, W, C, ph, pw, &d) ? d.p.tiles_x * d.p.tiles_y : -1;
}

int dw_mma_launch(const void* x, const void* w, const void* bias, void* y, float* pool_partial, int N, int H, int W, int C,
                  int ph, int pw, long long ldx, long long ldy, int act, cudaStream_t stream) {
    DeviceState* st = device_state();
    if (!st) return FVM_ERR_SETUP;
    DmPlan d;
    if (!dm_plan_cached(N, H, W, C, ph, pw, &d)) return FVM_ERR_ARG;
    DmParams& p = d.p;
    p.act = act;
    p.status = st->status_dev;
    CUtensorMap tx, ty;
    for (int o = 0; o < 2; ++o) {
        const unsigned long long w_ = o ? p.Q : W, h_ = o ? p.P : H, ld = o ? ldy : ldx;
        const unsigned long long dims[4] = {static_cast<unsigned long long>(C), w_, h_, static_cast<unsigned long long>(N)};
        const unsigned long long strides[3] = {ld * 2, w_ * ld * 2, h_ * w_ * ld * 2};
        const unsigned box[4] = {static_cast<unsigned>(DM_CB), static_cast<unsigned>(o ? p.xb * 8 : p.tile_w),
                                 static_cast<unsigned>(o ? p.segs * p.rr : p.tile_h), static_cast<unsigned>(p.nimg)};
        const int rc = encode_tiled_f16(o ? &ty : &tx, o ? y : x, 4, dims, strides, box, false);
        if (rc != FVM_OK) return rc;
    }
    const bool any = p.rr % DM_S != 0;
    auto kernel = act == 0 ? (any ? dw7_mma_kernel<0, true> : dw7_mma_kernel<0, false>)
                           : (any ? dw7_mma_kernel<-1, true> : dw7_mma_kernel<-1, false>);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DM_SMEM_LIMIT) != cudaSuccess) return FVM_ERR_SETUP;
    return launch_pdl(kernel, dim3(d.grid), dim3(DM_THREADS), d.smem, stream, 1, tx, ty, static_cast<const __half*>(w),
                      static_cast<const __half*>(bias), pool_partial, p);
}

}  // namespace fvm
