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
// bytes apart and each writes half a sector, and the layers' time followed their output (16 x 256^2,
// 32 -> 32 channels 82 us, 32 -> 64 127 us).  Instead the tile is laid out in shared memory as TMA
// stores it, rows of OB = 32 or 64 channels a pixel in the 64- or 128-byte swizzle, and one TMA copy
// writes it; rows and columns outside the image are left out by the copy.
template <int BN> __host__ __device__ constexpr int out_box() { return BN >= 64 ? 64 : 32; }   // channels of a box
template <int BN> __host__ __device__ constexpr uint32_t out_bytes() { return uint32_t(kBM * BN * 2); }
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
                 : "memory");
}
__device__ __forceinline__ void store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// at most N of this thread's latest stores still read shared memory / are not complete
template <int N> __device__ __forceinline__ void store_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
template <int N> __device__ __forceinline__ void store_wait() { asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory"); }
template <int ID, int NTH> __device__ __forceinline__ void epi_sync() { asm volatile("barrier.sync %0, %1;" ::"n"(ID), "n"(NTH) : "memory"); }
template <int ID, int NTH> __device__ __forceinline__ bool epi_any(bool p) {
    int any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.red.or.pred q, %2, %3, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
                 : "=r"(any) : "r"(int(p)), "n"(ID), "n"(NTH) : "memory");
    return any != 0;
}
// 32 accumulator columns (channels col0 ..) of pixel m through the epilogue into the staged tile
template <int BN>
__device__ __forceinline__ void stage_row32(const float (&v)[32], int col0, int Co, const float* __restrict__ bias, bool relu,
                                            uint32_t tile, int m) {
    constexpr int OB = out_box<BN>();
    const uint32_t row = tile + uint32_t(col0 / OB) * uint32_t(kBM * OB * 2) + uint32_t(m) * (OB * 2);
    const uint32_t chunk0 = uint32_t(col0 % OB) / 8u, flip = OB == 64 ? uint32_t(m & 7) : uint32_t((m >> 1) & 3);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int c = 8 * q + 2 * i;
            float a = v[c] + (col0 + c < Co ? bias[col0 + c] : 0.0f);
            float b = v[c + 1] + (col0 + c + 1 < Co ? bias[col0 + c + 1] : 0.0f);
            if (relu) { a = fmaxf(a, 0.0f); b = fmaxf(b, 0.0f); }
            w[i] = uint32_t(f2bf(a)) | (uint32_t(f2bf(b)) << 16);
        }
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row + 16u * ((chunk0 + uint32_t(q)) ^ flip)), "r"(w[0]),
                     "r"(w[1]), "r"(w[2]), "r"(w[3])
                     : "memory");
    }
}

// ---------------------------------------------------------------------------------------------
// y[P, Co] (epilogue) = conv3x3(x[B, H, W, C]) with w[Co, >= 9C], C = CB.  One persistent CTA: the
// weights stay in shared memory, warp 0 streams halo tiles, warp 1 issues a tile's 9 * CB/16 MMAs
// into TMEM accumulator i % 2, warps 2-5 store accumulator i % 2 through the epilogue.  K runs over
// taps, then channels, in steps of 16, as in the GEMMs: the results are the same bit for bit.
// output tiles staged: two, one where the weights leave no more room
template <int CB, int BN> __host__ __device__ constexpr int conv_outs() { return CB == 64 && BN == 128 ? 1 : 2; }
template <int CB, int BN> __host__ __device__ constexpr int conv_stages() {
    // halo tiles beside the weights and the staged outputs: 2 beside 128 x 64 channels' weights, 3 where
    // several CTAs then share an SM, else 4
    return CB == 64 && BN == 128 ? 2 : CB == 64 && BN == 64 ? 4 : 3;
}
template <int CB, int BN> __host__ __device__ constexpr size_t conv_smem() {
    return size_t(9) * CB * BN * 2 + size_t(conv_stages<CB, BN>()) * halo_stage<CB>() + conv_outs<CB, BN>() * out_bytes<BN>() + 1024;
}

template <int CB, int BN>
__global__ void __launch_bounds__(kPtThreads, 1)
k_conv_halo(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
            const __grid_constant__ CUtensorMap tmY, int staged, int Co, void* y, int ldy, const float* __restrict__ bias,
            int epi, int* err, const TileGeom g) {
    constexpr int NS = conv_stages<CB, BN>(), NO = conv_outs<CB, BN>();
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
    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(smem_addr(&bar_full[s]), 1u);
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
    if (warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(smem_addr(&bar_w), 9 * kW);
            for (int tap = 0; tap < 9; ++tap) tma_load_2d(sW + tap * kW, &tmW, tap * CB, 0, smem_addr(&bar_w));
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
    } else if (warp == 1) {
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
        uint32_t it = 0;
        for (int t = blockIdx.x; t < g.total; t += gridDim.x, ++it) {
            const int b = int(it & 1u);
            const bool ready = !pt_failed(fail) && bar_wait(smem_addr(&acc_full[b]), (it >> 1) & 1u);
            if (epi_any<2, 128>(!ready)) {   // the four warps leave together (they meet at barriers below)
                *fail = 1;
                break;
            }
            tc_fence_after();
            int img, y0, x0;
            g.at(t, img, y0, x0);
            const int m = q * 32 + lane;
            if (staged) {
                const uint32_t tile = sY + (NO == 2 ? (it & 1u) : 0u) * out_bytes<BN>();
                // the store that used this tile has read it (thread 64 issues the stores)
                if (tid == 64) store_wait_read<NO - 1>();
                epi_sync<1, 128>();
#pragma unroll 1
                for (int c0 = 0; c0 < BN; c0 += 32) {
                    float v[32];
                    tmem_ld32(tmem + (uint32_t(q * 32) << 16) + uint32_t(b * BN + c0), v);
                    stage_row32<BN>(v, c0, Co, bias, epi == EPI_BF16_BIAS_RELU, tile, m);
                }
                tc_fence_before();
                mbar_arrive(smem_addr(&acc_empty[b]));
                fence_proxy_async_smem();
                epi_sync<1, 128>();
                if (tid == 64) {
                    constexpr int OB = out_box<BN>();
                    for (int c0 = 0; c0 < BN && c0 < Co; c0 += OB)
                        tma_store_4d(&tmY, tile + uint32_t(c0 / OB) * uint32_t(kBM * OB * 2), c0, x0, y0, img);
                    store_commit();
                }
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
        if (staged && tid == 64) store_wait<0>();
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
k_conv_small(const uint16_t* __restrict__ x, const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmY,
             int staged, int Co, void* y, int ldy, const float* __restrict__ bias, int epi, int* err, const TileGeom g) {
    constexpr uint32_t kA = kBM * 128u, kB = BN * 128u;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) unsigned long long bar_w, bar_acc;
    __shared__ uint32_t s_tmem;
    __shared__ int s_fail;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;
    const uint32_t sA = base, sB = base + kA, sY = sB + kB;
    if (warp == 0) tmem_alloc(smem_addr(&s_tmem), uint32_t(BN));
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
            if (tid == 0) store_wait_read<0>();
            __syncthreads();
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += 32) {
                float v[32];
                tmem_ld32(tmem + (uint32_t(warp * 32) << 16) + uint32_t(c0), v);
                stage_row32<BN>(v, c0, Co, bias, epi == EPI_BF16_BIAS_RELU, sY, tid);
            }
            fence_proxy_async_smem();
            __syncthreads();
            if (tid == 0 && ok) {
                constexpr int OB = out_box<BN>();
                for (int c0 = 0; c0 < BN && c0 < Co; c0 += OB)
                    tma_store_4d(&tmY, sY + uint32_t(c0 / OB) * uint32_t(kBM * OB * 2), c0, x0, y0, b);
                store_commit();
            }
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
    if (staged && tid == 0) store_wait<0>();
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
        const uint16_t* __restrict__ dy, int Ci, int Co, float* gW, int ldw, int* err, const TileGeom g, int ci_blocks) {
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
    const int n_tiles = int(blockIdx.x) < g.total ? (g.total - int(blockIdx.x) + int(gridDim.x) - 1) / int(gridDim.x) : 0;

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
                g.at(int(blockIdx.x) + i * int(gridDim.x), b, y0, x0);
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
#pragma unroll
            for (int kk = 0; kk < kBM / 16; ++kk) {   // 16 pixels: two rows of the tile
                const uint64_t oa = uint64_t((SMALL ? uint32_t(16 * kk) * 128u : uint32_t(2 * kk * kHX) * kRow) / 16u);
                const uint64_t ob = uint64_t(uint32_t(16 * kk) * (BN * 2) / 16u);
#pragma unroll
                for (int q = 0; q < NM; ++q)
                    tc_mma_bf16(tmem + uint32_t(q * BN), da[q] + oa, db + ob, idesc, (i | kk) != 0 ? 1u : 0u);
            }
            tc_commit(smem_addr(&bar_empty[s]));
        }
        if (!ok) *fail = 1;
        tc_commit(smem_addr(&bar_done));   // arrives once every MMA issued above has completed
    } else if (kGather) {
        const int m = tid - 64;   // pixel of the tile
        for (int i = 0; i < n_tiles && !pt_failed(fail); ++i) {
            int b, y0, x0;
            g.at(int(blockIdx.x) + i * int(gridDim.x), b, y0, x0);
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
