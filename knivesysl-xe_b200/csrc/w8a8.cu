// w8a8.cu — the W8A8 tier (int8 weights with one plain FP16 scale per (row, K32), no zero
// point): the reference's high-fidelity fallback for the few matrices that need more than four
// weight bits, lm_head first (xpu/src/kernels_dpas.cpp:345-395 repack, 768-843 GEMV,
// 1578-1629 GEMM). Weights: codes[Mt][Kt][16 rows][32 B] (a row's 32 codes are contiguous),
// scales[Mt][Kt][16]. Activations are the W4A8 staging unchanged.
//
// Both kernels are HBM-bound streams of 512-byte tiles. The GEMV keeps the W4A8 GEMV's
// mapping (a half-warp per tile, the two halves of a warp = the reference's two accumulators,
// a team of S warps per row-group, partial sums added in split order through shared memory)
// with plain batched loads: the one weight this tier serves in practice is hundreds of
// megabytes, so ramp and tail do not matter. The general GEMM gives a warp one (row-group, eight
// tokens) task, as the reference does, on mma.sync m16n8k32: its A fragment is word c and
// word 4 + c of rows r and r + 8 of the tile, read straight from global memory. It is left for
// activations that do not fit in shared memory (K above 25,800), for unaligned buffers and where its plan costs
// less (head_plan).
#include "stream.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace tq {

namespace {

constexpr int kW = 16;     // warps per GEMV CTA
constexpr int kU = 4;      // tiles a half-warp loads per batch

__global__ void __launch_bounds__(kW * 32)
gemv_w8a8_kernel(const uint8_t *__restrict__ codes, const uint16_t *__restrict__ scales,
                 const int8_t *__restrict__ q, const float *__restrict__ as,
                 const float *__restrict__ residual, float *__restrict__ y, int groups, int Kt,
                 int S) {
    __shared__ float part[kW * 16];
    pdl_trigger();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = lane >> 4, n = lane & 15;
    const int tpc = kW / S, team = warp / S, split = warp - team * S;
    const int kt_begin = Kt * split / S;
    const int cnt = Kt * (split + 1) / S - kt_begin;
    for (int g0 = blockIdx.x * tpc; g0 < groups; g0 += gridDim.x * tpc) {
        const int g = g0 + team;
        float acc = 0.0f;
        if (g < groups) {
            const uint8_t *bbase = codes + ((size_t)g * Kt + kt_begin) * 512u + (size_t)n * 32u;
            const uint16_t *sbase = scales + ((size_t)g * Kt + kt_begin) * 16u + n;
            // this half-warp's tiles: offsets h, h + 2, ... (even offsets = accumulator 0)
            for (int i0 = h; i0 < cnt; i0 += 2 * kU) {
                uint4 wa[kU], wb[kU];
                uint32_t sc[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const int i = i0 + 2 * u;
                    if (i < cnt) {
                        wa[u] = ldg_stream_v4(bbase + (size_t)i * 512u);
                        wb[u] = ldg_stream_v4(bbase + (size_t)i * 512u + 16);
                        sc[u] = __ldg(sbase + (size_t)i * 16u);
                    }
                }
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const int i = i0 + 2 * u;
                    if (i >= cnt) break;
                    const int kt = kt_begin + i;
                    const uint4 a0 = __ldg(reinterpret_cast<const uint4 *>(q + (size_t)kt * 32));
                    const uint4 a1 = __ldg(reinterpret_cast<const uint4 *>(q + (size_t)kt * 32) + 1);
                    int d = __dp4a((int)wa[u].x, (int)a0.x, 0);
                    d = __dp4a((int)wa[u].y, (int)a0.y, d);
                    d = __dp4a((int)wa[u].z, (int)a0.z, d);
                    d = __dp4a((int)wa[u].w, (int)a0.w, d);
                    d = __dp4a((int)wb[u].x, (int)a1.x, d);
                    d = __dp4a((int)wb[u].y, (int)a1.y, d);
                    d = __dp4a((int)wb[u].z, (int)a1.z, d);
                    d = __dp4a((int)wb[u].w, (int)a1.w, d);
                    const float ws = __half2float(__ushort_as_half((unsigned short)sc[u]));
                    acc = fmaf(__fmul_rn((float)d, ws), __ldg(as + kt), acc);
                }
            }
        }
        acc = __fadd_rn(acc, __shfl_down_sync(0xffffffffu, acc, 16));    // acc0 + acc1
        const int row = g * 16 + n;
        if (S == 1) {
            // unsplit: the accumulator is stored as is; a residual is a separate add
            if (g < groups && h == 0) y[row] = residual ? __fadd_rn(acc, residual[row]) : acc;
            continue;
        }
        if (h == 0) part[warp * 16 + n] = acc;
        __syncthreads();
        if (g < groups && split == 0 && h == 0) {
            float sum = 0.0f;
            for (int i = 0; i < S; ++i) sum = __fadd_rn(sum, part[(warp + i) * 16 + n]);
            y[row] = __fadd_rn(sum, residual ? residual[row] : 0.0f);
        }
        __syncthreads();      // part is rewritten by the next round
    }
}

constexpr int kGW = 8;     // warps per GEMM CTA

__global__ void __launch_bounds__(kGW * 32)
gemm_w8a8_kernel(const uint8_t *__restrict__ codes, const uint16_t *__restrict__ scales,
                 const int8_t *__restrict__ aq, const float *__restrict__ as,
                 float *__restrict__ y, int M, int Kt, int T) {
    pdl_trigger();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = lane >> 2, c = lane & 3;
    const int tgroups = T / 8;
    const long tasks = (long)(M / 16) * tgroups;
    int czero[4];
    make_const_quad(czero, 0);
    for (long task = (long)blockIdx.x * kGW + warp; task < tasks; task += (long)gridDim.x * kGW) {
        const int rg = (int)(task / tgroups), tg = (int)(task - (long)rg * tgroups);
        const uint8_t *bbase = codes + (size_t)rg * Kt * 512u + (size_t)r * 32u + c * 4;
        const uint16_t *sbase = scales + (size_t)rg * Kt * 16u + r;
        const int8_t *abase = aq + ((size_t)tg * 8 + r) * 32 + c * 4;
        const float *asb = as + (size_t)tg * 8 + 2 * c;
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int kt = 0; kt < Kt; ++kt) {
            const uint8_t *t = bbase + (size_t)kt * 512u;
            const uint32_t a0 = ldg_stream_u32(t), a2 = ldg_stream_u32(t + 16);
            const uint32_t a1 = ldg_stream_u32(t + 256), a3 = ldg_stream_u32(t + 272);
            const int8_t *ab = abase + (size_t)kt * T * 32;
            const uint32_t b0 = __ldg(reinterpret_cast<const uint32_t *>(ab));
            const uint32_t b1 = __ldg(reinterpret_cast<const uint32_t *>(ab + 16));
            int d[4];
            mma_s8_c(d, a0, a1, a2, a3, b0, b1, czero);
            const float ws0 = __half2float(__ushort_as_half(__ldg(sbase + (size_t)kt * 16u)));
            const float ws1 = __half2float(__ushort_as_half(__ldg(sbase + (size_t)kt * 16u + 8)));
            const float2 as2 = __ldg(reinterpret_cast<const float2 *>(asb + (size_t)kt * T));
            acc[0] = fmaf((float)d[0], __fmul_rn(ws0, as2.x), acc[0]);
            acc[1] = fmaf((float)d[1], __fmul_rn(ws0, as2.y), acc[1]);
            acc[2] = fmaf((float)d[2], __fmul_rn(ws1, as2.x), acc[2]);
            acc[3] = fmaf((float)d[3], __fmul_rn(ws1, as2.y), acc[3]);
        }
        const size_t row = (size_t)rg * 16 + r, tok = (size_t)tg * 8 + 2 * c;
        y[tok * M + row] = acc[0];
        y[(tok + 1) * M + row] = acc[1];
        y[tok * M + row + 8] = acc[2];
        y[(tok + 1) * M + row + 8] = acc[3];
    }
}

// The same with the activations of a token window in shared memory: a warp takes a row-group and 8 NTG tokens.
// What bounded the kernel above at 8 tokens was not the weight stream but its reads of the activations: every
// warp of an SM comes to a k-tile's 256 bytes at about the same time and waits out an L2 latency for them. Here
// one CTA per SM and window stages them once; a warp walks row-groups and keeps two register batches of U k-tiles
// of its weight stream, the first one requested before the wait for the staging kernel. The last window of a
// call may hold fewer than NTG groups of tokens (RAGGED, a form of its own: the test costs two groups a warp 7 %): its
// warps multiply what lies in shared memory for the others and do not store it. head_plan() chooses NTG and the warps.
// W = 28 warps (72 registers) carry the 27.7 row-groups per SM of a 65536-row head in one round; 16 warps have
// registers for twice the tiles (20000 x 2048, 8 tokens: 18.5 against 22.2 us with 28). us of the launch alone, weights from
// HBM, kernel above / this one: 65536 x 5120 at 8 / 16 / 24 / 32 / 48 / 64 tokens 66 / 108 / 160 / 218 / 318 / 422 -> 58 / 63 / 95 /
// 92 / 169 / 170; 20000 x 5120 at 8 / 24 / 48 tokens 53 / 57 / 110 -> 38 / 45 / 56.
constexpr int kSActTile = 256 + 32;        // staged codes and scales of a k-tile and eight tokens
constexpr size_t kSSmem = 227 * 1024;
constexpr int kWide = 28, kNarrow = 16;    // warps per CTA

template <int NTG, int U, int W, bool RAGGED = false>
__global__ void __launch_bounds__(W * 32, 1)
gemm_w8a8_staged_kernel(const uint8_t *__restrict__ codes, const uint16_t *__restrict__ scales,
                        const int8_t *__restrict__ aq, const float *__restrict__ as,
                        float *__restrict__ y, int M, int Kt, int T) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int r = lane >> 2, c = lane & 3;
    const int groups = M / 16, tok0 = blockIdx.y * (8 * NTG);
    const int real = RAGGED ? min(NTG, T / 8 - (int)blockIdx.y * NTG) : NTG;
    const int first = blockIdx.x + gridDim.x * warp, stride = gridDim.x * nw;
    // Lane (r, c) holds k = 8c..8c+7 of rows r and r + 8 as the fragment's two k positions, and takes the
    // same bytes of token r: a 32-byte row is one 8-byte load of four lanes.
    const uint32_t lane_c = r * 32 + c * 8;
    // one batch: the codes of U tiles, and their scales, two a lane
    auto load = [&](uint2 (&w)[U][2], uint32_t &sc, int g, int kt0) {
        const uint8_t *cp = codes + ((size_t)g * Kt + kt0) * 512u + lane_c;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (kt0 + u < Kt) {
                w[u][0] = ldg_stream_v2(cp + u * 512);
                w[u][1] = ldg_stream_v2(cp + u * 512 + 256);
            }
        if ((lane >> 3) < U && kt0 + (lane >> 3) < Kt) sc = ldg_stream_u32(scales + ((size_t)g * Kt + kt0) * 16u + lane * 2);
    };
    uint2 w0[U][2], w1[U][2];
    uint32_t s0 = 0, s1 = 0;
    pdl_trigger();
    if (first < groups) load(w0, s0, first, 0);
    pdl_wait();      // so far only weights were read
    const uint32_t act = smem_u32(smem);
    for (int i = threadIdx.x; i < Kt * NTG * 16; i += blockDim.x) {       // 16 bytes of codes each
        const int kt = i / (NTG * 16), rem = i - kt * (NTG * 16);
        if (!RAGGED || (rem >> 4) < real)
            cp_async16_plain(act + (uint32_t)(kt * NTG + (rem >> 4)) * kSActTile + (rem & 15) * 16,
                             aq + ((size_t)kt * T + tok0) * 32 + rem * 16);
    }
    for (int i = threadIdx.x; i < Kt * NTG * 8; i += blockDim.x) {        // one scale each
        const int kt = i / (NTG * 8), rem = i - kt * (NTG * 8);
        if (!RAGGED || (rem >> 3) < real)
            cp_async4(act + (uint32_t)(kt * NTG + (rem >> 3)) * kSActTile + 256 + (rem & 7) * 4,
                      as + (size_t)kt * T + tok0 + rem);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const f32x2 neg_magic = pack2(-kMagicF, -kMagicF);
    int cmagic[4];
    make_const_quad(cmagic, kMagicBits);
    f32x2 acc01[NTG], acc23[NTG];
    auto batch = [&](uint2 (&w)[U][2], uint32_t sc, int kt0) {
        const uint32_t at = act + (uint32_t)(kt0 * NTG) * kSActTile;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (kt0 + u >= Kt) break;
            const uint32_t sa = __shfl_sync(0xffffffffu, sc, u * 8 + (r >> 1));
            const uint32_t sb = __shfl_sync(0xffffffffu, sc, u * 8 + 4 + (r >> 1));
            const int sh = (r & 1) * 16;
            const float ws0 = __half2float(__ushort_as_half((unsigned short)(sa >> sh)));
            const float ws1 = __half2float(__ushort_as_half((unsigned short)(sb >> sh)));
            const f32x2 ws0p = pack2(ws0, ws0), ws1p = pack2(ws1, ws1);
#pragma unroll
            for (int t = 0; t < NTG; ++t) {
                uint2 b;
                f32x2 as2;
                const uint32_t tile = at + (u * NTG + t) * kSActTile;
                asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(b.x), "=r"(b.y) : "r"(tile + lane_c));
                asm volatile("ld.shared.u64 %0, [%1];" : "=l"(as2) : "r"(tile + 256 + c * 8));
                int d[4];      // the dot + kMagicBits: as fp32, 12582912 + dot
                mma_s8_c(d, w[u][0].x, w[u][1].x, w[u][0].y, w[u][1].y, b.x, b.y, cmagic);
                fma2_acc(acc01[t], add2(pack2i(d[0], d[1]), neg_magic), mul2(ws0p, as2));
                fma2_acc(acc23[t], add2(pack2i(d[2], d[3]), neg_magic), mul2(ws1p, as2));
            }
        }
    };
#pragma unroll 1
    for (int g = first; g < groups; g += stride) {
#pragma unroll
        for (int t = 0; t < NTG; ++t) acc01[t] = acc23[t] = 0ull;
#pragma unroll 1
        for (int kt = 0;; kt += 2 * U) {
            // the batch after w0's: of this row-group or the first one of the next
            if (kt + U < Kt) load(w1, s1, g, kt + U);
            else if (g + stride < groups) load(w1, s1, g + stride, 0);
            batch(w0, s0, kt);
            if (kt + U >= Kt) {
#pragma unroll
                for (int u = 0; u < U; ++u) { w0[u][0] = w1[u][0]; w0[u][1] = w1[u][1]; }
                s0 = s1;
                break;
            }
            if (kt + 2 * U < Kt) load(w0, s0, g, kt + 2 * U);
            else if (g + stride < groups) load(w0, s0, g + stride, 0);
            batch(w1, s1, kt + U);
            if (kt + 2 * U >= Kt) break;
        }
        const size_t row = (size_t)g * 16 + r;
#pragma unroll
        for (int t = 0; t < NTG; ++t) {
            if (RAGGED && t >= real) break;
            float o[4];
            unpack2(acc01[t], o[0], o[1]);
            unpack2(acc23[t], o[2], o[3]);
            const size_t tok = (size_t)tok0 + t * 8 + 2 * c;
            y[tok * M + row] = o[0];
            y[(tok + 1) * M + row] = o[1];
            y[tok * M + row + 8] = o[2];
            y[(tok + 1) * M + row + 8] = o[3];
        }
    }
}

int g_sms = 0;
int sms() {
    if (!g_sms) {
        int dev = 0;
        TQ_CHECK(cudaGetDevice(&dev));
        TQ_CHECK(cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev));
        if (g_sms <= 0) g_sms = 148;
    }
    return g_sms;
}

}  // namespace

void launch_gemv_w8a8(const uint8_t *codes, const uint16_t *scales, const int8_t *q,
                      const float *as, const float *residual, float *y, int M, int K, int splits) {
    const int groups = M / 16, Kt = K / 32;
    if (groups <= 0 || splits <= 0 || splits > kW || (kW % splits)) return;
    const int tpc = kW / splits;
    const int grid = std::min(8 * sms(), (groups + tpc - 1) / tpc);
    launch_pdl(gemv_w8a8_kernel, dim3(grid), dim3(kW * 32), 0, codes, scales, q, as, residual, y,
               groups, Kt, splits);
    TQ_LAUNCH_CHECK("gemv_w8a8_kernel");
}

// How a call of `groups` row-groups, `tgroups` groups of 8 tokens and Kt k-tiles runs: the plan whose busiest SM
// needs the fewest clocks for a k-tile of all its rounds of row-groups. A round of the staged kernel is bound by latency,
// so it costs much the same with few row-groups as with many. Measured on 65536 x 5120 and 57 other weights of 1040 to
// 262144 rows, 8 to 2400 tokens: 475 to 505 clocks with one group of tokens a warp, 580 to 630 with two, 760 to 990 with
// four on 17 to 28 warps; 370 to 470, 400 to 490 and 550 to 600 on up to 16; with one or two windows at least the weight
// stream, 25 or 20 clocks a warp. The general kernel holds 32 tasks an SM: about 500 clocks a round of them and 8 a task,
// 27.5 a task where the weights serve 8 tokens only. It is left the heads that are one round of its own and two
// of the staged kernel (66,320 to 75,776 rows, 8 tokens: 66320 x 5120 67 us against 78), and long K, where few groups
// fit and many windows leave SMs idle. An odd number of token groups is no reason for windows of one: 65536 x 5120, 24
// tokens 150 us so and 95 in a window of four, 600 tokens 5810 (75 windows, one CTA each; 4110 in the general kernel) and
// 1740. Over those calls no choice was more than 2 % behind the general kernel.
HeadPlan head_plan(int groups, int tgroups, int Kt, int sms) {
    HeadPlan best{};
    if (groups <= 0 || tgroups <= 0) return best;
    const double tasks = (double)groups * tgroups / sms;      // of an SM
    for (int ntg = 4; ntg >= 1; ntg >>= 1) {
        const int windows = (tgroups + ntg - 1) / ntg;
        if ((size_t)Kt * ntg * kSActTile > kSSmem || windows > sms || (ntg > 1 && 2 * tgroups <= ntg)) continue;
        HeadPlan p{ntg, windows, std::min(groups, sms / windows), 0, 0, 0.0};
        const int per = (groups + p.ctas - 1) / p.ctas;
        p.rounds = (per + kWide - 1) / kWide;
        p.warps = std::max(8, (per + p.rounds - 1) / p.rounds);
        double round;
        if (p.warps > kNarrow)
            round = ntg == 4 ? 400 + 21 * p.warps
                  : ntg == 2 ? (windows <= 2 ? 565 : 545) + 2.5 * p.warps : windows <= 2 ? 505 : 475;
        else
            round = ntg == 4 ? 590 : (ntg == 2 ? 410 : 375) + (windows == 1 ? 80 : windows == 2 ? 20 : 0);
        if (windows <= 2) round = std::max(round, (windows == 1 ? 25.0 : 20.0) * p.warps);
        p.clocks = p.rounds * round * (tgroups % ntg ? 1.04 : 1.0);
        if (!best.ntg || p.clocks < best.clocks) best = p;
    }
    const double general = std::max(500 * std::ceil(tasks / 32) + 8 * tasks, tgroups == 1 ? 27.5 * tasks : 0.0);
    if (best.ntg && best.clocks > general) best = HeadPlan{};
    return best;
}

void launch_gemm_w8a8(const uint8_t *codes, const uint16_t *scales, const int8_t *aq,
                      const float *as, float *y, int M, int K, int T) {
    const int Kt = K / 32;
    const HeadPlan p = head_plan(M / 16, T / 8, Kt, sms());
    if (p.ntg && !((uintptr_t)aq & 15) && !((uintptr_t)codes & 7) && !(((uintptr_t)scales | (uintptr_t)as) & 3)) {
        auto go = [&](auto kernel) {
            static const void *done[10];      // kernels of one type: by address
            for (const void *&d : done) {
                if (d == (const void *)kernel) break;
                if (d) continue;
                TQ_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSSmem));
                d = (const void *)kernel;
                break;
            }
            launch_pdl(kernel, dim3(p.ctas, p.windows), dim3(p.warps * 32), (size_t)Kt * p.ntg * kSActTile, codes,
                       scales, aq, as, y, M, Kt, T);
        };
        auto pick = [&](auto ragged) {
            constexpr bool R = decltype(ragged)::value;
            if (p.warps <= kNarrow) {
                if (p.ntg == 4) go(gemm_w8a8_staged_kernel<4, 4, kNarrow, R>);
                else if (p.ntg == 2) go(gemm_w8a8_staged_kernel<2, 4, kNarrow, R>);
                else go(gemm_w8a8_staged_kernel<1, 4, kNarrow>);
            } else {
                if (p.ntg == 4) go(gemm_w8a8_staged_kernel<4, 2, kWide, R>);
                else if (p.ntg == 2) go(gemm_w8a8_staged_kernel<2, 2, kWide, R>);
                else go(gemm_w8a8_staged_kernel<1, 4, kWide>);
            }
        };
        if (T / 8 % p.ntg) pick(std::true_type{});
        else pick(std::false_type{});
        TQ_LAUNCH_CHECK("gemm_w8a8_staged_kernel");
        return;
    }
    const long tasks = (long)(M / 16) * (T / 8);
    if (tasks <= 0) return;
    const int grid = (int)std::min<long>((tasks + kGW - 1) / kGW, 16L * sms());
    launch_pdl(gemm_w8a8_kernel, dim3(grid), dim3(kGW * 32), 0, codes, scales, aq, as, y, M, K / 32, T);
    TQ_LAUNCH_CHECK("gemm_w8a8_kernel");
}

}  // namespace tq
