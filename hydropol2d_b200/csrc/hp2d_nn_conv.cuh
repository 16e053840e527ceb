// 3x3 convolutions of the screening network whose input tile is read once (sm_100a, TMA + tcgen05):
// the forward / backward-data convolution k_conv_halo, the convolution of inputs of a few channels
// k_conv_small, and the weight gradient k_wgrad.
//
// Output tiles are 8 x 16 pixels (kTX x kTY).  TMA brings the tile with its one-pixel halo, 10 x 18
// pixels of CB = 32 or 64 channels, into shared memory as consecutive rows of one pixel each (64 or
// 128 bytes, the TMA's 64- or 128-byte swizzle; outside the image reads zeros, the convolution's
// padding).  The operand of one tap is the same tile seen from another start address: the eight
// pixels of a tile row are eight consecutive rows, and the next tile row lies 10 rows further (the
// descriptor's stride), so a tap (ty, tx) only shifts the start by ty * 10 + tx rows.  The swizzle is
// a function of the shared-memory address itself, so shifted starts need no correction.  The
// implicit GEMM this replaces re-read the input from L2 once per tap, nine times, and was bound by
// that traffic (tensor pipe 8-16 % busy on the 32-channel layers).
#pragma once

#include "hp2d_nn_gemm.cuh"

namespace hp2d {
namespace nn {

constexpr int kHX = kTX + 2, kHY = kTY + 2;      // with the halo

template <int CB> __host__ __device__ constexpr uint32_t halo_bytes() { return uint32_t(kHX * kHY * CB * 2); }
template <int CB> __host__ __device__ constexpr uint32_t halo_stage() { return (halo_bytes<CB>() + CB * 2 + 1023u) & ~1023u; }

// descriptors of tiles of CB-channel rows (128-byte swizzle for 64 channels, 64-byte for 32)
template <int CB> __device__ __forceinline__ uint64_t row_desc(uint32_t addr, uint32_t lead, uint32_t stride) {
    uint64_t d = 0;
    d |= uint64_t((addr >> 4) & 0x3FFFu);
    d |= uint64_t((lead >> 4) & 0x3FFFu) << 16;
    d |= uint64_t((stride >> 4) & 0x3FFFu) << 32;
    d |= uint64_t(1u) << 46;                       // descriptor version
    d |= uint64_t(CB == 64 ? 2u : 4u) << 61;       // 128- or 64-byte swizzle
    return d;
}
// ---- BF16 output tiles through shared memory -----------------------------------------------------
// A thread holds a pixel's channels: stored straight to memory, a warp's 16-byte stores are 64 or more
// bytes apart, and the layers' time followed their output (16 x 256^2, 32 -> 32 channels 82 us,
// 32 -> 64 127 us).  Instead the tile is laid out in shared memory, rows of BN channels a pixel with
// their 16-byte pieces exchanged so that neither side meets bank conflicts, and written out along its
// rows, 512 contiguous bytes a warp (written by TMA, the two layers took 57 us each, now 45 and 55).
template <int BN> __host__ __device__ constexpr uint32_t out_bytes() { return uint32_t(kBM * BN * 2); }
template <int ID, int NTH> __device__ __forceinline__ void epi_sync() { asm volatile("barrier.sync %0, %1;" ::"n"(ID), "n"(NTH) : "memory"); }
template <int ID, int NTH> __device__ __forceinline__ bool epi_any(bool p) {
    int any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.red.or.pred q, %2, %3, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
                 : "=r"(any) : "r"(int(p)), "n"(ID), "n"(NTH) : "memory");
    return any != 0;
}
template <int BN> __device__ __forceinline__ uint32_t staged_at(uint32_t tile, int m, uint32_t piece) {
    const uint32_t flip = BN == 32 ? uint32_t((m >> 1) & 3) : uint32_t(m & 7);
    return tile + uint32_t(m) * (BN * 2) + 16u * (piece ^ flip);
}
// 32 accumulator columns (channels col0 ..) of pixel m through the epilogue into the staged tile, two
// channels an instruction; s_bias holds the columns' biases.  An epilogue warp has a scheduler almost
// to itself, so its instructions are the tile's time.
template <int BN>
__device__ __forceinline__ void stage_row32(const float (&v)[32], int col0, const float* s_bias, bool relu, uint32_t tile, int m) {
    const __nv_bfloat162 zero = __floats2bfloat162_rn(0.0f, 0.0f);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
            const int c = 8 * q + 2 * i;
            const float4 bb = *reinterpret_cast<const float4*>(s_bias + col0 + c);
            __nv_bfloat162 lo = __floats2bfloat162_rn(v[c] + bb.x, v[c + 1] + bb.y);
            __nv_bfloat162 hi = __floats2bfloat162_rn(v[c + 2] + bb.z, v[c + 3] + bb.w);
            if (relu) {   // rounding keeps the sign, so it may come first
                lo = __hmax2(lo, zero);
                hi = __hmax2(hi, zero);
            }
            w[i] = *reinterpret_cast<uint32_t*>(&lo);
            w[i + 1] = *reinterpret_cast<uint32_t*>(&hi);
        }
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(staged_at<BN>(tile, m, uint32_t(col0 / 8 + q))), "r"(w[0]),
                     "r"(w[1]), "r"(w[2]), "r"(w[3])
                     : "memory");
    }
}
// the staged tile to the output, by 128 threads (e: this thread's place among them): its pieces lie
// whole tile rows apart
template <int BN>
__device__ __forceinline__ void write_tile(uint32_t tile, const TileGeom& g, int b, int y0, int x0, int Co, uint16_t* out, int ldy,
                                           int e) {
    constexpr int PP = BN / 8;             // 16-byte pieces of a pixel
    constexpr int kStep = kBM / PP;        // pixels between a thread's pieces
    const int m = e / PP, piece = e % PP;
    const int x = x0 + m % kTX;
    int y = y0 + m / kTX;
    if (x >= g.W || 8 * piece >= Co) return;
    uint16_t* p = out + (size_t(b * g.H + y) * g.W + x) * ldy + 8 * piece;
    const size_t step = size_t(kStep / kTX) * g.W * ldy;
    uint32_t at = staged_at<BN>(tile, m, uint32_t(piece));   // kStep is a multiple of 8: the exchange stays
#pragma unroll
    for (int i = 0; i < PP; ++i) {
        uint32_t w0, w1, w2, w3;
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w0), "=r"(w1), "=r"(w2), "=r"(w3) : "r"(at));
        if (y < g.H) *reinterpret_cast<uint4*>(p) = make_uint4(w0, w1, w2, w3);
        at += uint32_t(kStep) * (BN * 2);
        p += step;
        y += kStep / kTX;
    }
}
// the biases of BN output columns (zero beyond Co) into shared memory
__device__ __forceinline__ void load_bias(float* s_bias, int bn, const float* __restrict__ bias, int Co, int tid, int nt) {
    for (int c = tid; c < bn; c += nt) s_bias[c] = bias && c < Co ? bias[c] : 0.0f;
}
// One 10 x 18 pixel halo tile of CB channels into shared memory by the kLoaders threads of the loading
// warps (e: this thread's place among them), 16 bytes a copy, in the layout TMA would give it: 64- or
// 128-byte swizzle, zeros outside the image.  A thread keeps its column and piece and steps down the
// tile.  The 32 -> 32 channel layer loads so: by TMA its tile of 180 rows of 64 bytes took as long as
// one of 128 (16 x 256^2: 57 us by TMA, 45 us so; the layers with 64 channels on either side are
// faster by TMA, 64 -> 32 68 against 72 us, 32 -> 64 55 against 63 us).
constexpr int kLoaders = 160;
template <int CB, int BN> __host__ __device__ constexpr int conv_loaders() { return CB == 32 && BN == 32 ? kLoaders : 32; }
template <int CB> __device__ __forceinline__ void load_halo(const uint16_t* __restrict__ x, const TileGeom& g, int b, int y0, int x0,
                                                            uint32_t stage, int e) {
    constexpr int PP = CB / 8, kLine = kHX * PP, kStep = kLoaders / kLine;   // pieces of a line of the tile; lines a pass
    static_assert(kLoaders % kLine == 0, "whole lines a pass");
    const int hy0 = e / kLine, hx = (e % kLine) / PP, piece = e % PP;
    const int xx = x0 - 1 + hx;
    const bool in_x = xx >= 0 && xx < g.W;
    const uint16_t* p = x + ((int64_t(b) * g.H + (y0 - 1 + hy0)) * g.W + xx) * CB + 8 * piece;
#pragma unroll
    for (int i = 0; i < (kHY + kStep - 1) / kStep; ++i) {
        const int hy = hy0 + i * kStep, yy = y0 - 1 + hy;
        if (kHY % kStep == 0 || hy < kHY) {
            const int r = hy * kHX + hx;
            const bool in = in_x && yy >= 0 && yy < g.H;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                             stage + uint32_t(r) * (CB * 2) + 16u * uint32_t(piece ^ (CB == 64 ? r & 7 : (r >> 1) & 3))),
                         "l"(in ? p + int64_t(i) * kStep * g.W * CB : x), "r"(in ? 16 : 0)
                         : "memory");
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// ---------------------------------------------------------------------------------------------
// y[P, Co] (epilogue) = conv3x3(x[B, H, W, C]) with w[Co, >= 9C], C = CB.  Persistent CTAs: the weights
// stay in shared memory, the loading warps stream halo tiles, one warp issues a tile's 9 * CB/16 MMAs
// into TMEM accumulator i % 2, groups of four warps store the accumulators through the epilogue.  K
// runs over taps, then channels, in steps of 16, as in the GEMMs: the results are the same bit for bit.
// What bounds it: the shared-memory pipe, which feeds the MMAs (a 128 x 32 x 16 MMA reads 5 KB) and
// carries the waits' polls, about 60 % each on the 64 -> 32 layer; DRAM is at 28 % there.
template <int CB, int BN> __host__ __device__ constexpr int conv_stages() {
    // halo tiles beside the weights and the staged output: 3, or the 2 that fit beside 128 x 64 channels' weights
    return CB == 64 && BN == 128 ? 2 : 3;
}
// groups of four epilogue warps, a tile each in turn, with a staged tile each (one where the weights
// leave no more room, or three CTAs share an SM)
template <int CB, int BN> __host__ __device__ constexpr int conv_groups() {
    return (CB == 64 && BN == 128) || conv_loaders<CB, BN>() > 32 ? 1 : 2;
}
template <int CB, int BN> __host__ __device__ constexpr int conv_threads() {
    return 32 + conv_loaders<CB, BN>() + 128 * conv_groups<CB, BN>();
}
template <int CB, int BN> __host__ __device__ constexpr size_t conv_smem() {
    return size_t(9) * CB * BN * 2 + size_t(conv_stages<CB, BN>()) * halo_stage<CB>() + conv_groups<CB, BN>() * out_bytes<BN>() + 1024;
}
// CTAs an SM holds
template <int CB, int BN> __host__ __device__ constexpr int conv_ctas() {
    return conv_smem<CB, BN>() * 3 <= 224 * 1024 ? 3 : conv_smem<CB, BN>() * 2 <= 224 * 1024 ? 2 : 1;
}
template <int CB, int BN>
__global__ void __launch_bounds__(conv_threads<CB, BN>(), conv_ctas<CB, BN>())
k_conv_halo(const uint16_t* __restrict__ x, const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
            int staged, int Co, void* y, int ldy, const float* __restrict__ bias, int epi, int* err, const TileGeom g) {
    constexpr int NS = conv_stages<CB, BN>(), NG = conv_groups<CB, BN>(), kLoadWarps = conv_loaders<CB, BN>() / 32;
    constexpr bool kCopy = kLoadWarps > 1;   // halo tiles by the warps' own copies, else by TMA
    __shared__ __align__(16) float s_bias[BN];
    static_assert(NS >= 2, "a halo tile must load while another is used");
    constexpr uint32_t kW = CB * BN * 2;   // one tap's weights
    constexpr uint32_t kRow = CB * 2;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) unsigned long long bar_full[NS], bar_empty[NS], acc_full[2], acc_empty[2], bar_w, bar_done;
    __shared__ uint32_t s_tmem;
    __shared__ int s_fail;
    volatile int* fail = &s_fail;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;
    const uint32_t sW = base, sX = base + 9 * kW;   // 9 * kW is a multiple of 1024 (BN >= 32)
    const uint32_t sY = sX + uint32_t(NS) * halo_stage<CB>();

    if (warp == 0) tmem_alloc(smem_addr(&s_tmem), uint32_t(2 * BN));
    load_bias(s_bias, BN, bias, Co, tid, conv_threads<CB, BN>());
    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(smem_addr(&bar_full[s]), kCopy ? uint32_t(kLoaders) : 1u);
            mbar_init(smem_addr(&bar_empty[s]), 1u);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_addr(&acc_full[b]), 1u);
            mbar_init(smem_addr(&acc_empty[b]), 128u);
        }
        mbar_init(smem_addr(&bar_w), 1u);
        mbar_init(smem_addr(&bar_done), 1u);
        mbar_fence_init();
        s_fail = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);

    uint32_t issued = 0;
    if (warp < kLoadWarps) {
        if constexpr (kCopy) {
            // NS - 1 tiles are on their way; a tile is handed over when its copies have landed
            uint32_t it = 0;
            const auto landed = [&](uint32_t i) {
                fence_proxy_async_smem();
                mbar_arrive(smem_addr(&bar_full[i % NS]));
            };
            for (int t = blockIdx.x; t < g.total && !pt_failed(fail); t += gridDim.x, ++it) {
                int b, y0, x0;
                g.at(t, b, y0, x0);
                const int s = int(it % NS);
                if (it >= uint32_t(NS - 1)) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(NS - 2) : "memory");
                    landed(it - uint32_t(NS - 1));
                }
                if (it >= uint32_t(NS) && !bar_wait(smem_addr(&bar_empty[s]), ((it / NS) - 1u) & 1u)) {
                    *fail = 1;
                    break;
                }
                load_halo<CB>(x, g, b, y0, x0, sX + uint32_t(s) * halo_stage<CB>(), tid);
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            for (uint32_t i = it >= uint32_t(NS - 1) ? it - uint32_t(NS - 1) : 0u; i < it; ++i) landed(i);
        } else if (lane == 0) {
            for (int t = blockIdx.x; t < g.total && !pt_failed(fail); t += gridDim.x) {
                int b, y0, x0;
                g.at(t, b, y0, x0);
                const int s = int(issued % NS);
                if (issued >= uint32_t(NS) && !bar_wait(smem_addr(&bar_empty[s]), ((issued / NS) - 1u) & 1u)) {
                    *fail = 1;
                    break;
                }
                mbar_expect_tx(smem_addr(&bar_full[s]), halo_bytes<CB>());
                tma_load_4d(sX + uint32_t(s) * halo_stage<CB>(), &tmX, 0, x0 - 1, y0 - 1, b, smem_addr(&bar_full[s]));
                ++issued;
            }
        }
    } else if (warp == kLoadWarps) {
        if (lane == 0) {
            mbar_expect_tx(smem_addr(&bar_w), 9 * kW);
            for (int tap = 0; tap < 9; ++tap) tma_load_2d(sW + tap * kW, &tmW, tap * CB, 0, smem_addr(&bar_w));
        }
        __syncwarp();
        constexpr uint32_t idesc = bf16_idesc<BN>();
        uint32_t it = 0;
        bool ok = bar_wait_warp(smem_addr(&bar_w), 0u);
        for (int t = blockIdx.x; ok && t < g.total && !pt_failed_warp(fail); t += gridDim.x, ++it) {
            const int s = int(it % NS), b = int(it & 1u);
            if (it >= 2 && !bar_wait_warp(smem_addr(&acc_empty[b]), ((it >> 1) - 1u) & 1u)) { ok = false; break; }
            if (!bar_wait_warp(smem_addr(&bar_full[s]), (it / NS) & 1u)) { ok = false; break; }
            tc_fence_after();
            const uint32_t acc = tmem + uint32_t(b * BN);
            const uint64_t da = row_desc<CB>(sX + uint32_t(s) * halo_stage<CB>(), 16u, uint32_t(kHX) * kRow);
            const uint64_t db = row_desc<CB>(sW, 16u, 8u * kRow);
#pragma unroll
            for (int tap = 0; tap < 9; ++tap) {   // offsets in the descriptors' 16-byte units
                const uint64_t oa = uint64_t(uint32_t((tap / 3) * kHX + tap % 3) * kRow / 16u), ob = uint64_t(uint32_t(tap) * kW / 16u);
#pragma unroll
                for (int kk = 0; kk < CB / 16; ++kk)
                    tc_mma_bf16(acc, da + (oa + uint64_t(2 * kk)), db + (ob + uint64_t(2 * kk)), idesc, (tap | kk) != 0 ? 1u : 0u);
            }
            tc_commit(smem_addr(&bar_empty[s]));
            tc_commit(smem_addr(&acc_full[b]));
        }
        if (!ok) *fail = 1;
        // every MMA this warp issued has completed before the TMEM can be released
        tc_commit(smem_addr(&bar_done));
        if (!bar_wait_warp(smem_addr(&bar_done), 0u)) *fail = 1;
    } else {
        const int q = warp & 3;   // TMEM lanes 32q .. 32q + 31 = pixels of the tile
        constexpr int kFirst = 1 + kLoadWarps;   // the first epilogue warp
        const int grp = NG == 2 ? (warp - kFirst) >> 2 : 0;   // its tiles: every NG-th of the CTA's
        const uint32_t tile = sY + uint32_t(grp) * out_bytes<BN>();
        const int e = (warp - kFirst - 4 * grp) * 32 + lane;
        uint32_t it = 0;
        for (int t = blockIdx.x; t < g.total; t += gridDim.x, ++it) {
            const int b = int(it & 1u);
            if (NG == 2 && b != grp) continue;
            const bool ready = !pt_failed(fail) && bar_wait(smem_addr(&acc_full[b]), (it >> 1) & 1u);
            if (grp == 0 ? epi_any<1, 128>(!ready) : epi_any<2, 128>(!ready)) {   // a group leaves together
                *fail = 1;
                break;
            }
            tc_fence_after();
            int img, y0, x0;
            g.at(t, img, y0, x0);
            const int m = q * 32 + lane;
            if (staged) {   // (the group has written its tile before out: the barrier above)
#pragma unroll 1
                for (int c0 = 0; c0 < BN; c0 += 32) {
                    float v[32];
                    tmem_ld32(tmem + (uint32_t(q * 32) << 16) + uint32_t(b * BN + c0), v);
                    stage_row32<BN>(v, c0, s_bias, epi == EPI_BF16_BIAS_RELU, tile, m);
                }
                tc_fence_before();
                mbar_arrive(smem_addr(&acc_empty[b]));
                if (grp == 0) epi_sync<3, 128>();
                else epi_sync<4, 128>();
                write_tile<BN>(tile, g, img, y0, x0, Co, static_cast<uint16_t*>(y), ldy, e);
            } else {
                const int row = g.row(img, y0, x0, m);
#pragma unroll 1
                for (int c0 = 0; c0 < BN; c0 += 32) {
                    float v[32];
                    tmem_ld32(tmem + (uint32_t(q * 32) << 16) + uint32_t(b * BN + c0), v);
                    if (row >= 0) store_row32(v, row, c0, row + 1, Co, y, ldy, bias, epi);
                }
                tc_fence_before();
                mbar_arrive(smem_addr(&acc_empty[b]));
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (s_fail) {
        if (tid == 0) {
            atomicExch(err, 1);
            // let the copies already issued land before the shared memory is released
            bar_wait(smem_addr(&bar_w), 0u);
            for (uint32_t i = issued > uint32_t(NS) ? issued - NS : 0u; i < issued; ++i)
                bar_wait(smem_addr(&bar_full[i % NS]), (i / NS) & 1u);
        }
        __syncthreads();
    }
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, uint32_t(2 * BN));
}

// ---------------------------------------------------------------------------------------------
// Rows of the im2col matrix of an input of C = 1, 2 or 4 channels (9C <= 36 of a row's 64 columns,
// the rest zero) written by the threads into shared memory, 128 bytes a pixel in the 128-byte
// swizzle: the operand of k_conv_small and of k_wgrad's first layer.
template <int C>
__device__ __forceinline__ void gather_row(const uint16_t* __restrict__ x, const TileGeom& g, int b, int y, int x0,
                                           uint32_t row_addr, int row) {
    static_assert(C == 1 || C == 2 || C == 4, "few channels");
    uint16_t v[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) v[i] = 0;
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
        const int yy = y + tap / 3 - 1, xx = x0 + tap % 3 - 1;
        if (yy >= 0 && yy < g.H && xx >= 0 && xx < g.W) {
            const uint16_t* p = x + ((size_t(b) * g.H + yy) * g.W + xx) * C;
            if constexpr (C == 4) {
                const uint2 u = *reinterpret_cast<const uint2*>(p);
                v[4 * tap] = uint16_t(u.x);
                v[4 * tap + 1] = uint16_t(u.x >> 16);
                v[4 * tap + 2] = uint16_t(u.y);
                v[4 * tap + 3] = uint16_t(u.y >> 16);
            } else if constexpr (C == 2) {
                const uint32_t u = *reinterpret_cast<const uint32_t*>(p);
                v[2 * tap] = uint16_t(u);
                v[2 * tap + 1] = uint16_t(u >> 16);
            } else {
                v[tap] = *p;
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = uint32_t(v[8 * c + 2 * q]) | (uint32_t(v[8 * c + 2 * q + 1]) << 16);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_addr + 16u * uint32_t(c ^ (row & 7))), "r"(w[0]),
                     "r"(w[1]), "r"(w[2]), "r"(w[3])
                     : "memory");
    }
}

// y[P, Co] (epilogue) = conv3x3 of an input of C channels, Co <= BN.  A CTA of 128 threads per tile
// (grid-stride): each thread writes its pixel's im2col row, one thread issues ceil(9C / 16) MMAs (the
// zero columns beyond add nothing), all store.  Two CTAs and more per SM overlap the phases.
// The im2col matrix this replaces was written to and read from HBM (128 bytes a pixel each way).
template <int C, int BN>
__global__ void __launch_bounds__(128)
k_conv_small(const uint16_t* __restrict__ x, const __grid_constant__ CUtensorMap tmW, int staged, int Co, void* y, int ldy, const float* __restrict__ bias, int epi, int* err, const TileGeom g) {
    constexpr uint32_t kA = kBM * 128u, kB = BN * 128u;
    __shared__ __align__(16) float s_bias[BN];
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) unsigned long long bar_w, bar_acc;
    __shared__ uint32_t s_tmem;
    __shared__ int s_fail;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;
    const uint32_t sA = base, sB = base + kA, sY = sB + kB;
    if (warp == 0) tmem_alloc(smem_addr(&s_tmem), uint32_t(BN));
    load_bias(s_bias, BN, bias, Co, tid, 128);
    if (tid == 0) {
        mbar_init(smem_addr(&bar_w), 1u);
        mbar_init(smem_addr(&bar_acc), 1u);
        mbar_fence_init();
        s_fail = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);
    if (tid == 0) {
        mbar_expect_tx(smem_addr(&bar_w), kB);
        tma_load_2d(sB, &tmW, 0, 0, smem_addr(&bar_w));
    }
    bool ok = bar_wait(smem_addr(&bar_w), 0u);
    uint32_t it = 0;
    for (int t = blockIdx.x; t < g.total; t += gridDim.x, ++it) {
        int b, y0, x0;
        g.at(t, b, y0, x0);
        gather_row<C>(x, g, b, y0 + (tid >> 3), x0 + (tid & 7), sA + uint32_t(tid) * 128u, tid);
        fence_proxy_async_smem();
        tc_fence_before();
        __syncthreads();
        if (warp == 0) {
            tc_fence_after();
            const uint64_t da = sw128_kmajor_desc(sA), db = sw128_kmajor_desc(sB);
#pragma unroll
            for (int kk = 0; kk < (9 * C + 15) / 16; ++kk)
                tc_mma_bf16(tmem, da + uint64_t(2 * kk), db + uint64_t(2 * kk), bf16_idesc<BN>(), kk != 0 ? 1u : 0u);
            tc_commit(smem_addr(&bar_acc));
        }
        ok = bar_wait(smem_addr(&bar_acc), it & 1u) && ok;
        if (!ok) atomicExch(&s_fail, 1);
        tc_fence_after();
        if (staged) {
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += 32) {
                float v[32];
                tmem_ld32(tmem + (uint32_t(warp * 32) << 16) + uint32_t(c0), v);
                stage_row32<BN>(v, c0, s_bias, epi == EPI_BF16_BIAS_RELU, sY, tid);
            }
            __syncthreads();   // (the next tile is staged after the barrier that follows its gather)
            if (ok) write_tile<BN>(sY, g, b, y0, x0, Co, static_cast<uint16_t*>(y), ldy, tid);
        } else {
            const int row = g.row(b, y0, x0, tid);
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += 32) {
                float v[32];
                tmem_ld32(tmem + (uint32_t(warp * 32) << 16) + uint32_t(c0), v);
                if (ok && row >= 0) store_row32(v, row, c0, row + 1, Co, y, ldy, bias, epi);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (s_fail && tid == 0) atomicExch(err, 1);
    if (warp == 0) tmem_dealloc(tmem, uint32_t(BN));
}

// ---------------------------------------------------------------------------------------------
// Weight gradient gW[co, tap*Ci + c] += sum over pixels dy[p, co] x[p + tap, c], read straight from the
// NHWC activations: D[m, n] with m over (tap, c) and n over co, K over the pixels, both operands
// MN-major (their channels are contiguous, their pixels rows of shared memory).  A unit is one block
// of CB input channels and BN output channels; its CTAs share the tiles, each accumulates all nine
// taps of its tiles in TMEM and adds them into gW at the end.
//   CB = 64: an MMA's 128 rows are two taps (the descriptor's leading offset is the distance of their
//            starts), five MMAs per 16 pixels, the tenth half thrown away;
//   CB = 32: 128 rows are the taps tx = -1, 0, 1 of one ty and one more shift thrown away (leading
//            offset one row), three MMAs.
// SMALL = C > 0: the input has C = 1, 2 or 4 channels: the operand is the gathered im2col row (64
// columns), one MMA.  BSMALL: dy has at most 4 channels, gathered into rows of 32.
// This replaces a transposed copy of dy and a transposed im2col of x in HBM (18 bytes moved per
// input byte, three quarters of a training step).
template <int CB, int SMALL> __host__ __device__ constexpr int wgrad_mmas() { return SMALL ? 1 : CB == 64 ? 5 : 3; }
template <int CB, int SMALL> __host__ __device__ constexpr uint32_t wgrad_a() { return SMALL ? kBM * 128u : halo_stage<CB>(); }
template <int CB, int BN, int SMALL> __host__ __device__ constexpr int wgrad_stages() {
    // (four stages leave room for a second CTA where the operands are small)
    return int((200u * 1024u) / (wgrad_a<CB, SMALL>() + kBM * BN * 2)) < 4 ? int((200u * 1024u) / (wgrad_a<CB, SMALL>() + kBM * BN * 2)) : 4;
}
template <int CB, int BN, int SMALL> __host__ __device__ constexpr size_t wgrad_smem() {
    return size_t(wgrad_stages<CB, BN, SMALL>()) * (wgrad_a<CB, SMALL>() + kBM * BN * 2) + 1024;
}
__host__ __device__ constexpr uint32_t tmem_cols(int n) { return n <= 32 ? 32u : n <= 64 ? 64u : n <= 128 ? 128u : n <= 256 ? 256u : 512u; }

// idesc of MN-major operands
template <int BN> __device__ __forceinline__ constexpr uint32_t bf16_idesc_mn() {
    return bf16_idesc<BN>() | (1u << 15) | (1u << 16);
}

template <int CB, int BN, int SMALL, bool BSMALL>
__global__ void __launch_bounds__(kPtThreads, 1)
k_wgrad(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmD, const uint16_t* __restrict__ x,
        const uint16_t* __restrict__ dy, int Ci, int Co, float* gW, int ldw, int* err, const TileGeom g, int ci_blocks, int halves) {
    constexpr int NS = wgrad_stages<CB, BN, SMALL>();
    constexpr int NM = wgrad_mmas<CB, SMALL>();
    constexpr uint32_t kA = wgrad_a<CB, SMALL>(), kB = kBM * BN * 2, kStage = kA + kB;
    constexpr uint32_t kRow = CB * 2;
    constexpr bool kGather = SMALL != 0 || BSMALL;
    constexpr uint32_t kTx = (SMALL ? 0u : halo_bytes<CB>()) + (BSMALL ? 0u : kB);
    constexpr uint32_t kCols = tmem_cols(NM * BN);
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) unsigned long long bar_full[NS], bar_empty[NS], bar_done;
    __shared__ uint32_t s_tmem;
    __shared__ int s_fail;
    volatile int* fail = &s_fail;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;
    const int cb = int(blockIdx.y) % ci_blocks, nb = int(blockIdx.y) / ci_blocks;
    // the CTA's work items: tiles, or half tiles (halves = 2: the product runs over half of the pixels)
    const int items = g.total * halves;
    const int n_tiles = int(blockIdx.x) < items ? (items - int(blockIdx.x) + int(gridDim.x) - 1) / int(gridDim.x) : 0;
    const auto item = [&](int i) { return int(blockIdx.x) + i * int(gridDim.x); };
    const auto tile_of = [&](int i) { return halves == 2 ? item(i) >> 1 : item(i); };

    if (warp == 0) tmem_alloc(smem_addr(&s_tmem), kCols);
    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(smem_addr(&bar_full[s]), 1u + (kGather ? 128u : 0u));
            mbar_init(smem_addr(&bar_empty[s]), 1u);
        }
        mbar_init(smem_addr(&bar_done), 1u);
        mbar_fence_init();
        s_fail = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);

    int issued = 0;
    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < n_tiles && !pt_failed(fail); ++i) {
                int b, y0, x0;
                g.at(tile_of(i), b, y0, x0);
                const int s = i % NS;
                const uint32_t fb = smem_addr(&bar_full[s]);
                if (i >= NS && !bar_wait(smem_addr(&bar_empty[s]), uint32_t((i / NS) - 1) & 1u)) {
                    *fail = 1;
                    break;
                }
                const uint32_t sa = base + uint32_t(s) * kStage;
                if (kTx) mbar_expect_tx(fb, kTx);
                else mbar_arrive(fb);
                if (!SMALL) tma_load_4d(sa, &tmX, cb * CB, x0 - 1, y0 - 1, b, fb);
                if (!BSMALL) tma_load_4d(sa + kA, &tmD, nb * BN, x0, y0, b, fb);
                issued = i + 1;
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = bf16_idesc_mn<BN>();
        bool ok = true;
        for (int i = 0; i < n_tiles && !pt_failed_warp(fail); ++i) {
            const int s = i % NS;
            if (!bar_wait_warp(smem_addr(&bar_full[s]), uint32_t(i / NS) & 1u)) { ok = false; break; }
            tc_fence_after();
            const uint32_t sa = base + uint32_t(s) * kStage, sb = sa + kA;
            const uint64_t db = row_desc<BN>(sb, 16u, 8u * (BN * 2));
            // the descriptor of each of the NM products; a 16-pixel step moves its start
            uint64_t da[NM];
#pragma unroll
            for (int q = 0; q < NM; ++q) {
                if (SMALL) {
                    da[q] = row_desc<64>(sa, 0u, 1024u);   // rows 64..127 repeat 0..63
                } else if (CB == 64) {
                    const int t0 = 2 * q, t1 = t0 + 1;
                    const uint32_t o0 = uint32_t((t0 / 3) * kHX + t0 % 3), o1 = uint32_t((t1 / 3) * kHX + t1 % 3);
                    da[q] = row_desc<CB>(sa + o0 * kRow, t1 < 9 ? (o1 - o0) * kRow : kRow, uint32_t(kHX) * kRow);
                } else {
                    da[q] = row_desc<CB>(sa + uint32_t(q * kHX) * kRow, kRow, uint32_t(kHX) * kRow);
                }
            }
            const int half = item(i) & 1;
            bool first = i == 0;
#pragma unroll
            for (int kk = 0; kk < kBM / 16; ++kk) {   // 16 pixels: two rows of the tile
                if (halves == 2 && kk / (kBM / 32) != half) continue;
                const uint64_t oa = uint64_t((SMALL ? uint32_t(16 * kk) * 128u : uint32_t(2 * kk * kHX) * kRow) / 16u);
                const uint64_t ob = uint64_t(uint32_t(16 * kk) * (BN * 2) / 16u);
#pragma unroll
                for (int q = 0; q < NM; ++q)
                    tc_mma_bf16(tmem + uint32_t(q * BN), da[q] + oa, db + ob, idesc, first ? 0u : 1u);
                first = false;
            }
            tc_commit(smem_addr(&bar_empty[s]));
        }
        if (!ok) *fail = 1;
        tc_commit(smem_addr(&bar_done));   // arrives once every MMA issued above has completed
    } else if (kGather) {
        const int m = tid - 64;   // pixel of the tile
        for (int i = 0; i < n_tiles && !pt_failed(fail); ++i) {
            int b, y0, x0;
            g.at(tile_of(i), b, y0, x0);
            const int s = i % NS;
            if (i >= NS && !bar_wait(smem_addr(&bar_empty[s]), uint32_t((i / NS) - 1) & 1u)) {
                *fail = 1;
                break;
            }
            const uint32_t sa = base + uint32_t(s) * kStage, sb = sa + kA;
            if constexpr (SMALL != 0)
                gather_row<SMALL>(x, g, b, y0 + (m >> 3), x0 + (m & 7), sa + uint32_t(m) * 128u, m);
            if constexpr (BSMALL) {   // dy's Co <= 4 channels and zeros, rows of 32 in the 64-byte swizzle
                static_assert(!BSMALL || BN == 32, "rows of 32 channels");
                const int yy = y0 + (m >> 3), xx = x0 + (m & 7);
                uint32_t w0 = 0u, w1 = 0u;
                if (yy < g.H && xx < g.W) {
                    const uint16_t* p = dy + ((size_t(b) * g.H + yy) * g.W + xx) * Co;
                    w0 = uint32_t(p[0]) | (Co > 1 ? uint32_t(p[1]) << 16 : 0u);
                    if (Co > 2) w1 = uint32_t(p[2]) | (Co > 3 ? uint32_t(p[3]) << 16 : 0u);
                }
                const uint32_t row = sb + uint32_t(m) * 64u;
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row + 16u * uint32_t(c ^ ((m >> 1) & 3))),
                                 "r"(c == 0 ? w0 : 0u), "r"(c == 0 ? w1 : 0u), "r"(0u), "r"(0u)
                                 : "memory");
            }
            fence_proxy_async_smem();
            mbar_arrive(smem_addr(&bar_full[s]));
        }
    }
    __syncwarp();
    const bool landed = bar_wait(smem_addr(&bar_done), 0u);
    if (!landed) atomicExch(&s_fail, 1);
    tc_fence_after();
    __syncthreads();
    if (warp >= 2 && !s_fail && n_tiles > 0) {
        const int q = warp & 3;
        const int r = q * 32 + lane;   // row of an MMA's 128
#pragma unroll 1
        for (int p = 0; p < NM; ++p) {
            int k = -1;   // column of gW, without the channel block
            if (SMALL) k = r < 9 * SMALL ? r : -1;
            else if (CB == 64) { const int tap = 2 * p + (r >> 6); k = tap < 9 ? tap * Ci + cb * CB + (r & 63) : -1; }
            else { const int tx = r >> 5; k = tx < 3 ? (3 * p + tx) * Ci + cb * CB + (r & 31) : -1; }
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += 32) {
                float v[32];
                tmem_ld32(tmem + (uint32_t(q * 32) << 16) + uint32_t(p * BN + c0), v);
                if (k >= 0) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int n = nb * BN + c0 + i;
                        if (n < Co) atomicAdd(gW + size_t(n) * ldw + k, v[i]);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (s_fail) {
        if (tid == 0) {
            atomicExch(err, 1);
            // let the copies already issued land before the shared memory is released
            for (int i = max(0, issued - NS); kTx != 0u && i < issued; ++i)
                bar_wait(smem_addr(&bar_full[i % NS]), uint32_t(i / NS) & 1u);
        }
        __syncthreads();
    }
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, kCols);
}

}  // namespace nn
}  // namespace hp2d
