// gemm_batch.cu — batched W4A8 GEMM for decode batches of 16 to 64 tokens in the reference's
// arithmetic (a scale per (token, K32) block; x_gemm_w4a8, xpu/src/kernels_dpas.cpp:1379-1489).
//
// The reference's split rule leaves such a call few and long (row-group, split) tasks: 64 tokens on 5120 x 17408
// are 320 chains of 544 k-tiles. The kernels of gemm_stream.cu cut the tokens into windows of 8 on CTA
// columns then, because the activations of a split do not fit beside their weight rings, and every
// window loads, unpacks and scales all weights again; what is left on an SM is a few warps that
// each wait on their own dependency chains. Here
//  * a CTA keeps the activations of ALL tokens in shared memory, of a whole split if they fit, else one
//    phase of the K range at a time in two buffers (cp.async into the other one while a phase is
//    computed). They are copied as the staging kernel left them; a lane's 8 bytes of a token are
//    its B fragment if the nibbles of a weight word are put into the same order (two byte permutes a word),
//    and the code sums become floats where they arrive;
//  * a warp carries NTG groups of 8 tokens of one row-group: the weight words, which it loads a chunk of
//    eight k-tiles ahead into registers, their unpacking and scales are paid once for them. CTAs
//    take contiguous ranges of (row-group, window) tasks of one split, so that the SMs share a call evenly;
//  * at most 12 (168 registers) or 16 warps (128), so that the chains of a warp's units can overlap.
// Arithmetic, order of the sums and the split reduction are those of gemm_stream.cu.
//
// What bounds it: the latency between a warp's instructions (32 a unit of 16 x 8 x 32 at NTG 2, 24 at 4). At 64 tokens on
// 5120 x 17408 an SM has nine warps, 2.25 a scheduler, each 4.7 clocks from one instruction to the next: 47 % of the issue
// slots. us of the launch alone, weights from HBM, the kernels before / this one: 5120 x 17408 K32 at 64 / 24 / 16 tokens
// 104.5 / 34.0 / 25.3 -> 92.0 / 30.7 / 23.6; 17408 x 17408 at 64 252 -> 172; 4096 x 4096 at 64 23.7 -> 18.6; 2048 x 8192
// K64 at 64 / 16 26.5 / 11.2 -> 20.9 / 8.5; 17408 x 5120 K64 at 48 52.9 -> 41.9; three of 6000 x 6016 at 24 43.9 -> 31.2;
// 704 x 8992 at 64 26.6 -> 11.1. (The first of them is not what the kernel is for: windows of 8 tokens on 18 warps, a form
// of the ring kernel that was not built in, came to the same time there.)
// Tried without gain: {ws, ws, z, z} in the scale buffer instead of pairs built from two words (105 against 99 us
// at 64 tokens: the reads' latency), 20 warps of 96 registers (126).
#include "stream.cuh"

#include <algorithm>
#include <type_traits>

namespace tq {

namespace {

constexpr int kCT = 8;                          // k-tiles per chunk: one register buffer of weights
constexpr int kExpBytes = kCT * 16 * 8;         // expanded scales of one chunk, per warp
constexpr size_t kSmemLimit = 227 * 1024;

struct BatchArgs {
    int P;            // k-tiles of one phase (a multiple of kCT)
    int phases;       // of a task: 1 = the split's activations stay for the whole kernel
    int buf_bytes;    // one phase's activations
};

__device__ __forceinline__ f32x2 lds_f32x2(uint32_t addr) {
    f32x2 v;
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint2 lds_u2(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t ldg_u16(const uint16_t *p) {
    uint16_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}

template <int NTG, int W>
__global__ void __launch_bounds__(W * 32, 1)
gemm_w4a8_batch_kernel(const GemmArgs a, const BatchArgs b, float *__restrict__ part, int *__restrict__ count) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, nthr = blockDim.x;
    const int r = lane >> 2, c = lane & 3, row16 = lane & 15, th = lane >> 4;
    const int T = a.T, windows = T / (8 * NTG);
    const int S = a.max_splits, split = blockIdx.x % S, ci = blockIdx.x / S;
    const int nctas = (gridDim.x - split + S - 1) / S;
    const int Kt = a.K >> 5, ksh = a.ksh, Ktg = Kt >> ksh;
    const int kt_begin = Kt * split / S, cnt = Kt * (split + 1) / S - kt_begin;
    const int nch = (cnt + kCT - 1) / kCT;
    const int groups_all = a.goff[a.count];
    const long tasks = (long)groups_all * windows;
    const int t_begin = (int)(tasks * ci / nctas), t_end = (int)(tasks * (ci + 1) / nctas);
    const int rounds = (t_end - t_begin + nw - 1) / nw;

    float2 *expw = reinterpret_cast<float2 *>(smem) + warp * 128;
    const uint32_t buf0 = smem_u32(smem) + (uint32_t)nw * kExpBytes;

    // ---- weights: the next chunk to load ---------------------------------------------------
    int p_ci = 0, p_task = t_begin + warp;
    const uint8_t *t_c = nullptr, *nx_c = nullptr;
    const uint16_t *t_s = nullptr;
    int nx_nt = 0, nx_kt0 = 0;
    auto advance = [&]() {
        if (p_task >= t_end) {
            nx_nt = 0;
            return;
        }
        if (p_ci == 0) {
            const int g = p_task / windows;
            int wi = 0;
            while (wi + 1 < a.count && g >= a.goff[wi + 1]) ++wi;
            const int lg = g - a.goff[wi];
            t_c = a.codes[wi] + ((size_t)lg * Kt + kt_begin) * 256u + r * 16 + c * 4;
            t_s = a.scales[wi] + (size_t)lg * Ktg * 16u + row16;
        }
        nx_c = t_c + (size_t)p_ci * (kCT * 256);
        nx_nt = min(kCT, cnt - p_ci * kCT);
        nx_kt0 = kt_begin + p_ci * kCT;
        if (++p_ci == nch) {
            p_ci = 0;
            p_task += nw;
        }
    };
    uint32_t w0[kCT][2], w1[kCT][2], sr[4];
    auto load_chunk = [&](uint32_t (&w)[kCT][2]) {
#pragma unroll
        for (int u = 0; u < kCT; ++u)
            if (u < nx_nt) {
                w[u][0] = ldg_stream_u32(nx_c + u * 256);
                w[u][1] = ldg_stream_u32(nx_c + u * 256 + 128);
            }
    };
    auto load_scales = [&]() {
#pragma unroll
        for (int m = 0; m < 4; ++m)
            if (2 * m + th < nx_nt) sr[m] = ldg_u16(t_s + (size_t)((nx_kt0 + 2 * m + th) >> ksh) * 16);
    };
    pdl_trigger();
    advance();
    load_chunk(w0);
    load_scales();
    int cur_nt = nx_nt;
    // the task whose scales are in sr has its pointers in t_s until the next advance()
    advance();
    pdl_wait();      // everything above reads only packed weights

    // ---- activations: one phase, copied as it lies ([k-tile][token]) ---------------------------
    auto stage = [&](int ph, uint32_t buf) {
        const int kt0 = kt_begin + ph * b.P, n = min(b.P, cnt - ph * b.P);
        const int8_t *sc = a.aq + (size_t)kt0 * T * 32;
        for (int i = threadIdx.x; i < n * T * 2; i += nthr) cp_async16_plain(buf + i * 16, sc + (size_t)i * 16);
        const uint32_t fa = buf + (uint32_t)(b.P * T) * 32, fs = fa + (uint32_t)(b.P * T) * 4;
        const float *sa = a.as + (size_t)kt0 * T;
        const int32_t *ss = a.asum + (size_t)kt0 * T;
        for (int i = threadIdx.x; i < n * T / 4; i += nthr) {
            cp_async16_plain(fa + i * 16, sa + (size_t)i * 4);
            cp_async16_plain(fs + i * 16, ss + (size_t)i * 4);
        }
        cp_async_commit();
    };
    // its code sums as negated floats (every thread converts what it copied)
    auto finish = [&](int ph, uint32_t buf) {
        cp_async_wait<0>();
        const int n = min(b.P, cnt - ph * b.P);
        unsigned char *fs = smem + (buf - smem_u32(smem)) + (size_t)(b.P * T) * 36;
        for (int i = threadIdx.x; i < n * T / 4; i += nthr) {
            const int4 v = reinterpret_cast<const int4 *>(fs)[i];
            reinterpret_cast<float4 *>(fs)[i] = make_float4(-(float)v.x, -(float)v.y, -(float)v.z, -(float)v.w);
        }
        __syncthreads();
    };
    stage(0, buf0);

    const f32x2 neg_magic2 = pack2(-kMagicF, -kMagicF);
    int cmagic[4];
    make_const_quad(cmagic, kMagicBits);
    uint32_t buf = buf0;
    int qpar = 0;
    for (int j = 0; j < rounds; ++j) {
        const int task = t_begin + j * nw + warp;
        const bool have = task < t_end;
        const int g = task / windows, win = task - g * windows, tok0 = win * 8 * NTG;
        f32x2 acc01[NTG], acc23[NTG];
#pragma unroll
        for (int t = 0; t < NTG; ++t) acc01[t] = acc23[t] = 0ull;
        for (int ph = 0; ph < b.phases; ++ph) {
            if (b.phases > 1 || j == 0) {
                finish(ph, buf);
                // the other buffer was read last before this barrier
                if (b.phases > 1 && (ph + 1 < b.phases || j + 1 < rounds))
                    stage(ph + 1 < b.phases ? ph + 1 : 0, buf == buf0 ? buf0 + b.buf_bytes : buf0);
            }
            if (have) {
                const int left_ph = min(b.P, cnt - ph * b.P);
                uint32_t bl = buf + (uint32_t)(tok0 + r) * 32 + c * 8;
                uint32_t al = buf + (uint32_t)(b.P * T) * 32 + (tok0 + 2 * c) * 4;
                const uint32_t sums = (uint32_t)(b.P * T) * 4, bstep = T * 32, astep = T * 4;
                for (int k0 = 0; k0 < left_ph; k0 += kCT, qpar ^= 1) {
                    auto chunk = [&](uint32_t (&w)[kCT][2], uint32_t (&wn)[kCT][2]) {
                        // expand this chunk's scale words: {ws, z + 8} of tile 2m + th, row row16
#pragma unroll
                        for (int m = 0; m < 4; ++m) {
                            const float ws = __half2float(__ushort_as_half((unsigned short)(sr[m] & 0xFFF0u)));
                            expw[(m * 16 + row16) * 2 + th] = make_float2(ws, (float)(int)((sr[m] ^ 8u) & 15u));
                        }
                        __syncwarp();
                        load_scales();
                        load_chunk(wn);
                        auto tile_pair = [&](auto full_tag, const int jp) {
                            constexpr bool FULL = decltype(full_tag)::value;
                            const float4 ea = *reinterpret_cast<const float4 *>(expw + (jp * 16 + r) * 2);
                            const float4 eb = *reinterpret_cast<const float4 *>(expw + (jp * 16 + r + 8) * 2);
#pragma unroll
                            for (int uu = 0; uu < 2; ++uu) {
                                const int u = 2 * jp + uu;
                                if (!FULL && u >= cur_nt) continue;
                                // natural k order: the even and the odd codes of a word interleaved
                                const uint32_t l0 = nib_plus8(w[u][0]), h0 = nib_plus8(w[u][0] >> 4);
                                const uint32_t l1 = nib_plus8(w[u][1]), h1 = nib_plus8(w[u][1] >> 4);
                                const uint32_t A0 = __byte_perm(l0, h0, 0x5140), A2 = __byte_perm(l0, h0, 0x7362);
                                const uint32_t A1 = __byte_perm(l1, h1, 0x5140), A3 = __byte_perm(l1, h1, 0x7362);
                                const float ws0 = uu ? ea.z : ea.x, nz0 = uu ? ea.w : ea.y;
                                const float ws1 = uu ? eb.z : eb.x, nz1 = uu ? eb.w : eb.y;
                                const f32x2 ws0p = pack2(ws0, ws0), ws1p = pack2(ws1, ws1);
                                const f32x2 nz0p = pack2(nz0, nz0), nz1p = pack2(nz1, nz1);
#pragma unroll
                                for (int t = 0; t < NTG; ++t) {
                                    const uint2 bb = lds_u2(bl + t * 256);
                                    const f32x2 as2 = lds_f32x2(al + t * 32);
                                    const f32x2 sm2 = lds_f32x2(al + sums + t * 32);
                                    int d[4];
                                    mma_s8_c(d, A0, A1, A2, A3, bb.x, bb.y, cmagic);
                                    const f32x2 f01 = fma2(nz0p, sm2, add2(pack2i(d[0], d[1]), neg_magic2));
                                    const f32x2 f23 = fma2(nz1p, sm2, add2(pack2i(d[2], d[3]), neg_magic2));
                                    fma2_acc(acc01[t], f01, mul2(ws0p, as2));
                                    fma2_acc(acc23[t], f23, mul2(ws1p, as2));
                                }
                                bl += bstep;
                                al += astep;
                            }
                        };
                        if (cur_nt == kCT) {
#pragma unroll
                            for (int jp = 0; jp < kCT / 2; ++jp) tile_pair(std::true_type{}, jp);
                        } else {
#pragma unroll
                            for (int jp = 0; jp < kCT / 2; ++jp) tile_pair(std::false_type{}, jp);
                        }
                        __syncwarp();      // expw is rewritten by the next chunk
                        cur_nt = nx_nt;
                        advance();
                    };
                    if (qpar) chunk(w1, w0);
                    else chunk(w0, w1);
                }
            }
            if (b.phases > 1) buf = buf == buf0 ? buf0 + b.buf_bytes : buf0;
        }
        if (!have) continue;
        int wi = 0;
        while (wi + 1 < a.count && g >= a.goff[wi + 1]) ++wi;
        const int lg = g - a.goff[wi];
        float out[NTG][4];
#pragma unroll
        for (int t = 0; t < NTG; ++t) {
            unpack2(acc01[t], out[t][0], out[t][1]);
            unpack2(acc23[t], out[t][2], out[t][3]);
        }
        if (S > 1) {
            // partial of this split -> scratch; the last split to arrive sums 0..S-1
            const size_t slot = (size_t)win * groups_all + g;
            float *pp = part + (slot * S + split) * (NTG * 128) + lane;
#pragma unroll
            for (int t = 0; t < NTG; ++t)
#pragma unroll
                for (int k = 0; k < 4; ++k) pp[(t * 4 + k) * 32] = out[t][k];
            __threadfence();
            __syncwarp();
            int old = 0;
            if (lane == 0) old = atomicAdd(count + slot, 1);
            old = __shfl_sync(0xffffffffu, old, 0);
            if (old != S - 1) continue;
            __threadfence();
            const float *base = part + slot * S * (NTG * 128) + lane;
#pragma unroll
            for (int t = 0; t < NTG; ++t) {
                float v[4][16];
#pragma unroll
                for (int s2 = 0; s2 < 16; ++s2)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        v[k][s2] = s2 < S ? __ldcg(base + (size_t)s2 * (NTG * 128) + (t * 4 + k) * 32) : 0.0f;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float sum = 0.0f;
#pragma unroll
                    for (int s2 = 0; s2 < 16; ++s2)
                        if (s2 < S) sum = __fadd_rn(sum, v[k][s2]);
                    out[t][k] = sum;
                }
            }
            if (lane == 0) count[slot] = 0;      // ready for the next launch
        }
        const size_t row = (size_t)lg * 16 + r;
        const int M = a.M[wi];
        float *y = a.y[wi];
#pragma unroll
        for (int t = 0; t < NTG; ++t) {
            const size_t tok = (size_t)tok0 + t * 8 + 2 * c;
            y[tok * M + row] = out[t][0];
            y[(tok + 1) * M + row] = out[t][1];
            y[tok * M + row + 8] = out[t][2];
            y[(tok + 1) * M + row + 8] = out[t][3];
        }
    }
}

}  // namespace

// Which kernel: both plans are turned into clocks of the busiest SM for the call, and the smaller one is taken, the
// other kernel's unless this kernel's is 4.5 % below it. (The other kernel is the ring kernel, or the streaming kernel where the
// activations of 8 tokens do not fit beside the rings: a split of more than 266 k-tiles.) The terms are what the
// kernels are made of: per k-tile, what a unit of one (row-group, token groups) costs by the warps that share an SM; the
// rounds of a warp's tasks, the last one with the warps that it has; launch and staging; the phases; with splits, the
// partials and their ordered sum, again for each further round.
// The constants are on one scale with each other rather than clocks: they minimise the time of the kernels chosen, with
// a penalty where that is this one and it loses against the other, over 3500 calls drawn from 128 to 17408 rows,
// one to four weights, K 512 to 17408, both scale groups and 16 to 64 tokens, every plan measured. There the calls run
// in 0.80 of the other kernel's time, 0.2 % above the best plan of each; 15 are more than 3 % behind the other kernel, two more
// than 8 %, and of 440 calls that the constants had not seen nine, the worst by 9 % (960 x 2528, 24 tokens: 6.9 us
// against 6.3). Counting a warp's instructions alone, without the sums of the splits and the rounds, left 243 of the
// 3500 more than 3 % behind, one by 46 % (912 x 6464 K64, 40 tokens: 13.3 us against 9.2).
namespace {

constexpr double kLead = 1.045;

// rounds of `per` tasks on `warps` warps: the clocks of a k-tile in all of them
template <typename F>
double all_rounds(int per, int warps, F clocks) {
    return per / warps * clocks(warps) + (per % warps ? clocks(per % warps) : 0.0);
}

double other_clocks(const RingShape &r, int splits) {
    const double unit = all_rounds(r.per, r.warps, [&](int w) {
        switch (r.kernel) {
            case RingShape::kStream: return std::max(180.0, (r.ntg == 1 ? 18.6 : 30.0) * w);
            case RingShape::kSmall: return 18.6 * w + 8;
            case RingShape::kLarge: return 12.4 * w + 116;
            default: return (16 + 19 * r.ntg) * std::max(4.6, 0.38 * w);
        }
    });
    static const double lead_in[4] = {2800, 4200, 4000, 8200};
    const bool one = r.ntg == 1, wide = r.kernel == RingShape::kSeveral;
    const double sums = splits == 1 ? 0.0 : !one ? 2800.0 * r.ntg : r.kernel == RingShape::kLarge ? 9600.0 : 4200.0;
    const int rounds = (r.per + r.warps - 1) / r.warps;
    return lead_in[r.kernel] + r.span * (unit + (wide ? 19 * r.ntg : 0)) + sums + (splits > 1 ? 19000.0 * (rounds - 1) : 0);
}

double batch_clocks(const BatchPlan &p, int splits) {
    static const double shared[4] = {4.0, 5.8, 7.9, 10.0};      // 1 to 4 warps on a scheduler
    const double unit = all_rounds(p.per, p.warps, [&](int w) { return (19 + 10 * p.ntg) * shared[(w - 1) / 4]; });
    // many splits on four or five warps: measured, the longer a split, without a cause that is known
    const double few = splits >= 8 && p.warps <= 5 ? 38.0 * p.ntg * p.span : 0.0;
    const int passes = p.phases > 1 ? p.phases * p.rounds : 1;
    return 6000 + p.span * unit + few + 4000.0 * (passes - 1) +
           (splits > 1 ? 1200 * p.ntg + 20500 * (p.rounds - 1) + (p.wide ? 4700 * p.rounds : 0) : 0);
}

}  // namespace

bool batch_plan(const GemmArgs &a, int sms, const RingShape &other, BatchPlan &best) {
    if (a.mode || a.x || a.dump || a.npeer || a.T < 16 || a.T > 64 || a.T % 8) return false;
    for (int i = 0; i < a.count; ++i)
        if (a.ld[i] && a.ld[i] != a.M[i]) return false;
    const int S = a.max_splits, Kt = a.K / 32, groups = a.goff[a.count], tg = a.T / 8;
    if (S > 16 || S > sms || groups <= 0) return false;
    best = BatchPlan{};
    for (int ntg = 8; ntg >= 2; --ntg) {
        if (tg % ntg) continue;
        const long tasks = (long)groups * (tg / ntg);
        for (int wide = 0; wide <= (ntg == 3 || ntg == 4 ? 1 : 0); ++wide) {
            BatchPlan p{};
            p.ntg = ntg;
            p.wide = wide;
            p.ctas = (int)std::max(1L, std::min<long>(sms / S, tasks));
            p.per = (int)((tasks + p.ctas - 1) / p.ctas);
            if (wide && p.per <= 12) continue;
            const int most = wide ? 16 : 12;
            p.rounds = (p.per + most - 1) / most;
            p.warps = std::max(4, (p.per + p.rounds - 1) / p.rounds);
            p.span = (Kt + S - 1) / S;
            const size_t room = kSmemLimit - (size_t)p.warps * kExpBytes, tile = (size_t)a.T * 40;
            p.P = (p.span + kCT - 1) / kCT * kCT;
            p.phases = 1;
            if (p.P * tile > room) {
                p.P = (int)(room / 2 / tile) / kCT * kCT;
                p.phases = (p.span + p.P - 1) / p.P;
            }
            p.clocks = batch_clocks(p, S);
            if (!best.ntg || p.clocks < best.clocks) best = p;
        }
    }
    return best.ntg && kLead * best.clocks < other_clocks(other, S);
}

bool launch_gemm_batch(const GemmArgs &a, int sms, const RingShape &other) {
    BatchPlan plan;
    if (((uintptr_t)a.aq | (uintptr_t)a.as | (uintptr_t)a.asum) & 15) return false;      // 16-byte copies
    if (!batch_plan(a, sms, other, plan)) return false;
    const int S = a.max_splits, groups = a.goff[a.count];
    const int ntg = plan.ntg, nw = plan.warps, ctas = plan.ctas;
    const long tasks = (long)groups * (a.T / 8 / ntg);
    const BatchArgs b = {plan.P, plan.phases, (int)(plan.P * (size_t)a.T * 40)};
    const size_t smem = (size_t)nw * kExpBytes + (size_t)b.buf_bytes * (b.phases > 1 ? 2 : 1);
    float *part = nullptr;
    int *count = nullptr;
    if (S > 1) split_scratch((size_t)tasks * S * ntg * 128, (int)tasks, part, count);
    auto go = [&](auto kernel) {
        static const void *done[12];      // kernels of one type: by address
        for (const void *&d : done) {
            if (d == (const void *)kernel) break;
            if (d) continue;
            TQ_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));
            d = (const void *)kernel;
            break;
        }
        launch_pdl(kernel, dim3(ctas * S), dim3(nw * 32), smem, a, b, part, count);
    };
    switch (ntg * 2 + plan.wide) {
        case 4: go(gemm_w4a8_batch_kernel<2, 12>); break;
        case 6: go(gemm_w4a8_batch_kernel<3, 12>); break;
        case 7: go(gemm_w4a8_batch_kernel<3, 16>); break;
        case 8: go(gemm_w4a8_batch_kernel<4, 12>); break;
        case 9: go(gemm_w4a8_batch_kernel<4, 16>); break;
        case 10: go(gemm_w4a8_batch_kernel<5, 12>); break;
        case 12: go(gemm_w4a8_batch_kernel<6, 12>); break;
        case 14: go(gemm_w4a8_batch_kernel<7, 12>); break;
        case 16: go(gemm_w4a8_batch_kernel<8, 12>); break;
        default: return false;
    }
    TQ_LAUNCH_CHECK("gemm_w4a8_batch_kernel");
    return true;
}

}  // namespace tq
