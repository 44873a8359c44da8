// gemm_tc.cu — prefill W4A8 GEMM on the sm_100a tensor cores: tcgen05.mma kind::f16 on
// integer-valued fp16 operands, fp32 accumulators in tensor memory (TMEM).
//
// Replaces gemm_rc16 / the unsplit path of x_gemm_w4a8 (xpu/src/kernels_dpas.cpp:1255-1332,
// 1371-1378): Y[tok][n] = sum over k-tiles, ascending, of (float)(d - z*asum) * (ws*as) with
// d the exact int32 dot of one 16-row x K32 tile, accumulated with fma into one fp32
// accumulator per output - the arithmetic and the order of the reference.
//
// Why the f16 pipe for an integer dot. The 4-bit codes less their zero point (-15..15) and the int8
// activations are exact in fp16, their products (< 2^11) and a k-tile's sum of them (< 2^16; a
// K64 group: < 2^17) are exact in the tensor core's fp32 accumulation, so the accumulator IS
// (float)(d - z*asum), bit for bit, and the promote is one fma per output. With kind::i8 the
// accumulator is int32 and every output costs an integer add and a float add more per k-tile
// on the CUDA cores (the exact conversion), which is what bounded that version of the
// kernel: the tensor pipe, at half the int8 rate, is still far from being the wall.
//
// Mapping. Weights are the M side of the MMA (128 output rows = 128 TMEM lanes), tokens the
// N side (128, 192 or 256 per CTA tile: choose_tile_tokens), a k-tile (K = 32) is two K = 16
// instructions, so one accumulator read-out yields exactly the per-k-tile dots the reference
// promotes. The K loop advances in steps of two k-tiles. Both operands come from images that one
// pre-pass writes in the operand layout (canonical no-swizzle K-major core matrices): the
// activation image and the weight image, every 4-bit code expanded to fp16 q - z once per call.
// Tiles are walked token block fastest, so the CTAs that run together share a few row blocks of
// the weight image while the whole activation image stays in L2.
//
// A CTA (20 warps, one per SM, persistent over tiles) runs three roles connected by
// mbarriers (step slots in shared memory, accumulator buffers in the 512 columns of TMEM):
//  * one thread starts the bulk (TMA) copies of a step: 16 KiB of weights and the activations of
//    the tile's tokens, each contiguous in its image;
//  * two MMA threads (in two warps): two tcgen05.mma (M=128, N=tokens, K=16) per k-tile into the
//    promote group's accumulator buffer (the first one overwrites it), then tcgen05.commit;
//  * workers (16 warps): thread = weight row x a quarter of the tile's tokens. Per promote group:
//    wait for the group's accumulator, then 16 columns at a time tcgen05.ld and
//    acc = fma(d, ws*as, acc); the accumulators stay in registers for the whole K loop and are
//    stored at the end (coalesced over rows).
//
// What bounds it: the workers' latencies and the hand-offs. At 256 tokens a tile a worker issues
// 184 instructions a K32 group for its 64 outputs (64 fma, 32 packed ws*as, 16 shared loads) and
// 135 a K64 group in per-token mode; ncu shows 65 / 58 % of the issue slots used, the FMA pipe
// 50 / 41 % busy and the tensor pipe 23 / 55 %. With two 256-column buffers a group's cycle is MMA,
// hand-off, promote, hand-off, overlapped with one other group. Measured, staging included, against
// 128-token tiles with the zero point applied in the promote: 17408 x 5120 K64, 4096 tokens in the
// reference's arithmetic 1.59 against 1.77 ms; 2048 tokens with per-token scales 0.43 against
// 0.49 ms; 1024 tokens W4A4 with zero points 0.32 against 0.57 ms; 5120 x 17408, 1000 tokens, zero
// points 0.60 against 0.88 ms; 10240 x 5120 K32, 136 tokens, zero points 114 against 216 us.
// Wider tiles pay a group's fixed work (barrier, scale word, counters: about 70 instructions) once
// for 64 outputs instead of 32. Tried and slower (4096 tokens, reference arithmetic, 1.60 ms): the
// 16x256b TMEM load with four rows x 16 tokens per thread, which reads a quarter of the activation
// scales from shared memory (1.74 to 1.83 ms); 8 workers x 128 tokens and 12 x 64 or 80 with the
// next load under the promote (1.74 to 1.81, 1.63 to 1.74); the activation scales loaded ahead of
// the TMEM wait (1.72, spills); the two groups of a step in a rolled loop (1.85).
//
// Every mbarrier wait is bounded; on expiry the kernel records a status word, stops
// issuing work, still frees its TMEM and returns.
#include "tc.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

namespace tq {

namespace {

constexpr int kTM = 128;                 // weight rows per tile (TMEM lanes)
constexpr int kABytes = kTM * 64;        // expanded fp16 weights of one k-tile
constexpr int kWorkWarps = 16;
constexpr int kMmaWarps = 2;
// Workers, the warp that starts the copies, the MMA warps, and one idle warp that completes the
// last group of four (setmaxnreg moves registers between groups of four warps).
constexpr int kThreads = (kWorkWarps + 4) * 32;
// A launch with 20 warps gives every thread 96 registers (61440 of the SM's); the workers of the
// widest tile, whose 64 accumulators and loaded columns do not fit in that, take 104 and the other
// four warps keep 64: 512 * 104 + 128 * 64 = 61440, exactly what the launch holds. A few words still
// spill at that split: 8 bytes a thread in block mode and 12 (40 loaded) in W4A4 at 256 tokens, none
// with per-token scales, up to 88 in the SUMS variants. (112 and 32: the MMA and copy threads spill
// too, and per-token prefill of 4096 tokens took 0.80 instead of 0.69 ms.)
constexpr int kLaunchRegs = 96, kWorkRegs = 104, kRoleRegs = 64;
static_assert(kWorkWarps * 32 * kWorkRegs + 4 * 32 * kRoleRegs <= kThreads * kLaunchRegs,
              "the register split must not exceed what the launch holds");
// Suspend-time hint of the waits: a thread that polls back to back takes issue slots from the warps
// beside it, one that waits with the hint stays off the scheduler until the phase completes.
constexpr uint32_t kNapNs = 2000;

// Geometry of a tile of TN = 4 * WT tokens (a worker thread promotes WT of them).
template <int WT>
struct TcTile {
    static constexpr int TN = kWorkWarps / 4 * WT;                        // tokens per tile (accumulator columns)
    static constexpr int NB = 512 / TN < 8 ? 512 / TN : 8;   // accumulator buffers in TMEM
    static constexpr int NBP = NB >= 8 ? 8 : NB >= 4 ? 4 : 2;// ... as a power of two
    static constexpr int kBStep = TN * 128;                  // fp16 activations of a step (two k-tiles)
    static constexpr int kScales = TN * 8;                   // as of both k-tiles; as many bytes of sum differences
    static constexpr int kImgStep = kBStep + 2 * kScales;    // activation image of one step
    static constexpr int kSlot = 2 * kABytes + kImgStep;     // step slot: weights, then the image
    static constexpr int kSlots = 230000 / kSlot < 8 ? 230000 / kSlot : 8;
    static constexpr int kSmem = kSlots * kSlot;             // > half an SM's shared memory: one CTA per SM,
                                                             // which the 512-column TMEM allocation requires
    static_assert(kSmem > 116 * 1024 && kSlots >= 3 && kSlot % 128 == 0, "slots");
};

// fp16 operands: four 16-byte K-chunks per row of a k-tile, 128 bytes apart; row groups of 8
// are 512 bytes apart; the second K = 16 instruction of a k-tile starts two chunks further
constexpr uint32_t kLboH = 128, kSboH = 512;

// Device words that say which variant of the GEMM does a call. The pre-pass stamps `diff` with the
// generation if some asum of the call is not the sum of its codes, and `zp` if some zero point of the
// weight is not 0; only where both are stamped does z * (sum of codes - asum) enter the result. The SUMS
// kernel, last of the call, moves the generation on, so that nothing has to be cleared and a captured
// call decides by the data of each replay.
struct SumsState {
    unsigned gen, diff, zp;      // read together, with `arrived`, as one 16-byte word
    unsigned arrived;            // CTAs of the SUMS kernel that have read the words
    unsigned last;               // the call before: did its SUMS kernel do the work?
};
// Stamps *word unless it is stamped already: a store by every CTA costs far more than the look (136
// tokens on 10240 x 5120 with zero points: 167 us instead of 113, 258 with a store by every warp).
__device__ __forceinline__ void stamp(unsigned *word, unsigned gen) {
    if (__ldcg(word) != gen) *word = gen;
}
// Never 0, what the stamps start from.
__device__ __forceinline__ unsigned next_generation(unsigned g) { return g + 1 ? g + 1 : 1; }

struct TcParams {
    const uint8_t *wimg;     // per (128-row block, k-tile): kABytes of fp16 weights in operand layout
    const uint16_t *scales;
    const uint8_t *img;      // per (TN-token block, step): kImgStep bytes (see the pre-pass)
    void *y;
    const float *as_tok;     // per-token scales (PERTOK kernels)
    SumsState *sums;
    int *status;
    unsigned long long wait_ns;   // limit of every mbarrier wait
    int M, Kt, ksh, T, tok_blocks, out_bf16;
};

// Four int8 codes (one word) -> fp16: flipping the sign bit makes a byte code + 128, which put
// under fp16's exponent of 1024 reads 1152 + code; subtracting 1152 is exact. Returns the
// halves of bytes sel (two selector nibbles pairs) as one word.
__device__ __forceinline__ uint32_t bytes_to_h2(uint32_t flipped_lo, uint32_t flipped_hi, uint32_t sel) {
    uint32_t t, r;
    // bytes a (of lo) and b (of hi) into the low bytes of two halves, then the exponent
    t = __byte_perm(flipped_lo, flipped_hi, sel) & 0x00FF00FFu;
    t |= 0x64006400u;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(t), "r"(0x64806480u));
    return r;
}

// Eight int8 codes (k = 0..3 in lo, 4..7 in hi) -> one 16-byte fp16 K-chunk in the order
// 0,4,1,5,2,6,3,7 (the order the weight expansion produces).
__device__ __forceinline__ uint4 codes_to_chunk(uint32_t lo, uint32_t hi) {
    lo ^= 0x80808080u;
    hi ^= 0x80808080u;
    return make_uint4(bytes_to_h2(lo, hi, 0x4400u), bytes_to_h2(lo, hi, 0x5511u),
                      bytes_to_h2(lo, hi, 0x6622u), bytes_to_h2(lo, hi, 0x7733u));
}

// Eight two's-complement nibbles of w (nibble i = code k = i) -> eight fp16 values, as four
// words holding the codes (0,4), (1,5), (2,6), (3,7). Per word: the two nibbles land in the
// low bits of the two halves; xor with 0x6408 sets fp16's exponent of 1024 and flips the
// code's sign bit, so the half reads 1024 + (q + 8); subtracting `base` = 1032 + z leaves q - z.
__device__ __forceinline__ uint4 nib8_to_h8(uint32_t w, uint32_t mask, uint32_t bias, uint32_t base) {
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t t;                                        // ((w >> 4i) & mask) ^ bias in one logic op
        asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(t) : "r"(w >> (4 * i)), "r"(mask), "r"(bias));
        asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r[i]) : "r"(t), "r"(base));
    }
    return make_uint4(r[0], r[1], r[2], r[3]);
}

struct PrepassArgs {
    const uint8_t *codes;
    const uint16_t *scales;
    const int8_t *aq;        // int8 codes [kt][tok][32], or for S4 the int4 codes [kt64][tok][32]
    const float *as;
    const int32_t *asum;
    uint8_t *wimg, *img;
    SumsState *sums;
    int M, Kt, ksh, T, TN, Tpad;
    int wblocks;             // CTAs that expand weights; the others convert activations
};

// Pre-pass: both operands of the GEMM into the layout its tiles copy, in one launch.
//  * Weights (the first wblocks CTAs): packed codes [row group][k-tile][16 rows][16 B] -> per
//    (128-row block, k-tile) the kABytes of fp16 values q - z in the operand layout (row groups
//    of 8 are kSboH apart, a row's four 16-byte K-chunks kLboH apart). With the zero point taken
//    off here the tensor core's dot is d - z * sum(codes) itself (integers below 2^18, exact), so
//    the GEMM promotes asymmetric weights like symmetric ones. A thread expands one row of one
//    k-tile; 8 consecutive lanes write 128 contiguous bytes per chunk. 4 bytes out per packed
//    byte: 178 MB for 17408 x 5120, written and read once per call.
//  * Activations: the caller's staging -> per (TN-token block, step of two k-tiles) the fp16
//    codes of k-tile 0 then 1 as [TN / 8][4 K-chunks][8 tokens][16 B], as[2][TN], and
//    (sum of the codes - asum)[2][TN], 0 unless the caller's asum is something else than the sum
//    of its codes (SumsState).
//    Tokens >= T are padded with zeros. S4: int4 codes; a K64 block's scale and sum go with its
//    first k-tile.
template <bool S4>
__global__ void __launch_bounds__(256) gemm_tc_prepass_kernel(const PrepassArgs a) {
    pdl_trigger();
    pdl_wait();      // the images may still be read by the previous call's kernel
    const unsigned gen = __ldcg(&a.sums->gen);
    if ((int)blockIdx.x < a.wblocks) {
        const uint32_t mask = 0x000F000Fu, bias = 0x64086408u;
        const size_t n = (size_t)a.M * a.Kt;
        const int Ktg = a.Kt >> a.ksh;
        uint32_t any = 0;
        for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)a.wblocks * 256) {
            const int kt = (int)(i / a.M), m = (int)(i % a.M);
            const uint4 c4 = ldg_stream_v4(a.codes + ((size_t)(m >> 4) * a.Kt + kt) * 256 + (m & 15) * 16);
            const uint32_t sw = __ldg(a.scales + ((size_t)(m >> 4) * Ktg + (kt >> a.ksh)) * 16 + (m & 15));
            any |= sw & 15u;
            const uint32_t base = (0x6400u + ((sw ^ 8u) & 15u)) * 0x00010001u;      // 1032 + z
            const int r = m & (kTM - 1);
            uint8_t *dst = a.wimg + ((size_t)(m / kTM) * a.Kt + kt) * kABytes + (r >> 3) * kSboH + (r & 7) * 16;
            *reinterpret_cast<uint4 *>(dst) = nib8_to_h8(c4.x, mask, bias, base);                 // k 0..7
            *reinterpret_cast<uint4 *>(dst + kLboH) = nib8_to_h8(c4.y, mask, bias, base);         // k 8..15
            *reinterpret_cast<uint4 *>(dst + 2 * kLboH) = nib8_to_h8(c4.z, mask, bias, base);     // k 16..23
            *reinterpret_cast<uint4 *>(dst + 3 * kLboH) = nib8_to_h8(c4.w, mask, bias, base);     // k 24..31
        }
        if (__syncthreads_or((int)any) && threadIdx.x == 0) stamp(&a.sums->zp, gen);
        return;
    }
    const int T = a.T, TN = a.TN, nsteps = a.Kt >> 1;
    const size_t nrow = (size_t)nsteps * a.Tpad;
    const size_t img_step = (size_t)TN * 144;
    int diff = 0;
    for (size_t i = (size_t)(blockIdx.x - a.wblocks) * 256 + threadIdx.x; i < nrow;
         i += (size_t)(gridDim.x - a.wblocks) * 256) {
        const int st = (int)(i / a.Tpad), tok = (int)(i % a.Tpad);
        const int tb = tok / TN, tl = tok - tb * TN;
        uint8_t *blk = a.img + ((size_t)tb * nsteps + st) * img_step;
        float *sv = reinterpret_cast<float *>(blk + (size_t)TN * 128);
        int sum[2] = {0, 0};
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            uint32_t w[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
            if (tok < T) {
                if (S4) {
                    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(a.aq + ((size_t)st * T + tok) * 32) + g);
                    const uint32_t p[4] = {v.x, v.y, v.z, v.w};
                    // byte b of the half = k 2b (low nibble), 2b + 1 (high nibble), two's complement:
                    // to bytes in k order, sign extended
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint32_t lo = p[j] & 0x0F0F0F0Fu, hi = (p[j] >> 4) & 0x0F0F0F0Fu;
                        lo = __vsub4(lo ^ 0x08080808u, 0x08080808u);
                        hi = __vsub4(hi ^ 0x08080808u, 0x08080808u);
                        w[2 * j] = __byte_perm(lo, hi, 0x5140);
                        w[2 * j + 1] = __byte_perm(lo, hi, 0x7362);
                    }
                } else {
                    const uint4 *src = reinterpret_cast<const uint4 *>(a.aq + ((size_t)(2 * st + g) * T + tok) * 32);
                    const uint4 x = __ldg(src), y = __ldg(src + 1);    // k = 0..15, 16..31
                    w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w;
                    w[4] = y.x; w[5] = y.y; w[6] = y.z; w[7] = y.w;
                }
            }
            uint8_t *dst = blk + (size_t)g * TN * 64 + (tl >> 3) * kSboH + (tl & 7) * 16;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                *reinterpret_cast<uint4 *>(dst + j * kLboH) = codes_to_chunk(w[2 * j], w[2 * j + 1]);
                sum[g] = __dp4a((int)w[2 * j], 0x01010101, sum[g]);
                sum[g] = __dp4a((int)w[2 * j + 1], 0x01010101, sum[g]);
            }
        }
        float s0 = 0.0f, s1 = 0.0f;
        int d0 = 0, d1 = 0;
        if (tok < T) {
            if (S4) {
                s0 = a.as[(size_t)st * T + tok];
                d0 = sum[0] + sum[1] - a.asum[(size_t)st * T + tok];
            } else {
                const size_t j0 = (size_t)(2 * st) * T + tok, j1 = j0 + T;
                if (a.as) {
                    s0 = a.as[j0];
                    s1 = a.as[j1];
                }
                d0 = sum[0] - a.asum[j0];
                d1 = sum[1] - a.asum[j1];
            }
        }
        sv[tl] = s0;
        sv[TN + tl] = s1;
        sv[2 * TN + tl] = (float)d0;
        sv[3 * TN + tl] = (float)d1;
        diff |= d0 | d1;
    }
    if (__syncthreads_or(diff) && threadIdx.x == 0) stamp(&a.sums->diff, gen);
}

constexpr int kWaitMma = 21, kWaitEpi = 22, kWaitProd = 23;   // status codes of failed waits

template <int REGS>
__device__ __forceinline__ void reg_alloc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS));
}
template <int REGS>
__device__ __forceinline__ void reg_dealloc() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS));
}

__device__ __forceinline__ void tmem_ldn(uint32_t taddr, uint32_t (&v)[16]) { tmem_ld16(taddr, v); }
__device__ __forceinline__ void tmem_ldn(uint32_t taddr, uint32_t (&v)[32]) { tmem_ld32(taddr, v); }
__device__ __forceinline__ void tmem_wait_ldn(uint32_t (&v)[16]) { tmem_wait_ld16(v); }
__device__ __forceinline__ void tmem_wait_ldn(uint32_t (&v)[32]) { tmem_wait_ld32(v); }

// GW = k-tiles accumulated in TMEM before one fp32 promote (1: the reference's arithmetic with
// a scale per (token, K32); 2: K64 weight groups with per-token activation scales, or - not
// PERTOK - with one activation scale per (token, K64): the W4A4 arithmetic). PERTOK:
// the activation scale is applied once at the end (y = acc * as_tok).
//
// The K loop advances in steps of two k-tiles (K is a multiple of 64); step n of the CTA
// (counted across its tiles) uses step slot n % kSlots, promote group n uses accumulator buffer
// n % NBP. A worker warp owns 32 TMEM lanes (rows) and WT of the tile's tokens.
//
// SUMS: the kernel applies z * (sum of codes - asum), for callers whose asum is not the sum of
// their codes, on weights with zero points. Both variants are launched; the one that SumsState does
// not select returns at once.
template <int GW, bool PERTOK, bool SUMS, int WT>
__global__ void __maxnreg__(kLaunchRegs) gemm_w4a8_tc_kernel(const TcParams p) {
    using G = TcTile<WT>;
    constexpr int TN = G::TN, NB = G::NBP, kSS = G::kSlots;
    constexpr int kCols = WT == 32 ? 32 : 16;            // columns of one TMEM load
    constexpr uint32_t kIdesc = idesc_f16(kTM, TN);
    // what a step copies of the image: the codes, the activation scales, the sum differences
    constexpr uint32_t kImgCopy = SUMS ? G::kImgStep : (PERTOK ? G::kBStep : G::kBStep + G::kScales);
    // per-token scales: the promote reads nothing from the slot, so its MMAs free it
    constexpr bool kReadsSlot = !PERTOK || SUMS, kSlotFreedByMma = !kReadsSlot;
    // How the two MMA threads share the work: whole steps in turn, or - two groups per step and only
    // two accumulator buffers - the first k-tile of every step for one thread and the second for the
    // other. Either way a buffer belongs to one thread for good, so a thread that waits for a
    // buffer's phase has seen the phase before it (a parity wait cannot tell phases two apart).
    constexpr bool kByTile = GW == 1 && NB == 2;
    static_assert(kByTile || (NB / (GW == 1 ? 2 : 1)) % kMmaWarps == 0, "a buffer belongs to one MMA thread");
    constexpr int kStepStride = kByTile ? 1 : kMmaWarps;
    // The same for the slots: each is always filled for the same thread, or the accumulator that the
    // thread's previous step needed was free only after the slot's previous use had been promoted.
    static_assert(kByTile || kSS % kMmaWarps == 0 || kSS >= NB / (GW == 1 ? 2 : 1) + kMmaWarps, "slot phases");
    // One K64 group per step, per-token scales: the promote is a bare fma per output, as packed
    // fma on token pairs (5 % faster there; in every other mode the packed form measured slower).
    constexpr bool kPacked = PERTOK && !SUMS && GW == 2;
    pdl_trigger();
    pdl_wait();      // everything below reads what earlier kernels wrote (words, images)
    const uint4 sw = __ldcg(reinterpret_cast<const uint4 *>(p.sums));      // gen, diff, zp, arrived
    if ((sw.y == sw.x && sw.z == sw.x) != SUMS) {
        // A CTA that reads the words after this store finds old stamps: not selected either.
        if (SUMS && blockIdx.x == 0 && threadIdx.x == 0) {
            p.sums->last = 0;
            p.sums->gen = next_generation(sw.x);
        }
        return;
    }
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t bars[2 * kSS + 2 * NB];   // full[kSS], empty[kSS], accfull[NB], accempty[NB]
    __shared__ uint32_t tmem_base_s;
    __shared__ int dead_s;                      // a wait gave up somewhere in the CTA
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t smem_u = smem_u32(smem);
    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[kSS]),
                   acc0 = smem_u32(&bars[2 * kSS]), accempty0 = smem_u32(&bars[2 * kSS + NB]);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kSS; ++s) {
            mbar_init(full0 + s * 8, 1);                 // the copy thread's arrive with the step's byte count
            // a slot is free when every worker warp has read its activation scales - or, in
            // the variant whose workers read nothing from the slot, when its MMAs are complete
            mbar_init(empty0 + s * 8, kSlotFreedByMma ? (kByTile ? kMmaWarps : 1) : kWorkWarps);
        }
        for (int b = 0; b < NB; ++b) {
            mbar_init(acc0 + b * 8, kReadsSlot ? 2 : 1); // tcgen05.commit; the committing thread (below)
            mbar_init(accempty0 + b * 8, kWorkWarps);    // one arrive per worker warp
        }
        dead_s = 0;
        mbar_init_fence();
    }
    if (warp == 0) {                                     // one warp allocates all 512 columns
        tmem_alloc(smem_u32(&tmem_base_s), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;
    // all threads of this CTA have read the words; the last CTA to say so moves the generation on
    if (SUMS && threadIdx.x == 0 && atomicInc(&p.sums->arrived, gridDim.x - 1) == gridDim.x - 1) {
        p.sums->last = 1;
        p.sums->gen = next_generation(sw.x);
    }

    const int spt = p.Kt >> 1;                           // steps per tile
    const int ntiles = (p.M / kTM) * p.tok_blocks;
    const int my_tiles = (ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;

    // Bounded wait that also gives up when another role already has. Inlined: a call would have to
    // fit the register shares that setmaxnreg hands out.
    auto wait_on = [&](uint32_t bar, uint32_t parity, int code) -> bool {
        if (mbar_test_wait(bar, parity)) return true;
        uint64_t t0 = 0;
        for (uint32_t polls = 1;; ++polls) {
            if (mbar_try_wait_hint(bar, parity, kNapNs)) return true;
            if (*(volatile int *)&dead_s) return false;
            if ((polls & 1023u) == 0) {
                const uint64_t now = global_timer_ns();
                if (t0 == 0) t0 = now;
                else if (now - t0 > p.wait_ns) break;
            }
        }
        atomicCAS(p.status, 0, code);
        *(volatile int *)&dead_s = 1;
        return false;
    };

    if (warp < kWorkWarps) {
        // ====================== workers: promote the accumulators ==========================
        reg_alloc<kWorkRegs>();
        const int q4 = warp & 3, chalf = (warp >> 2) * WT;   // lane quarter, first token
        const int rloc = q4 * 32 + lane;                  // row inside the tile = TMEM lane
        const uint32_t lane_base = tmem_base + ((uint32_t)(q4 * 32) << 16) + chalf;
        const int Ktg = p.Kt >> p.ksh;
        // activation scales of this thread's tokens inside a step slot
        const unsigned char *sv_base = smem + 2 * kABytes + G::kBStep + chalf * 4;
        int ss = 0;                                       // step slot, kept as a counter
        int b = 0;                                        // accumulator buffer and its parity
        uint32_t par = 0;

        for (int ti = 0; ti < my_tiles; ++ti) {
            const int tile = (int)blockIdx.x + ti * (int)gridDim.x;
            const int tb = tile % p.tok_blocks, rb = tile / p.tok_blocks;
            const int row = rb * kTM + rloc;
            // the scale word of the group being promoted
            const uint16_t *scn = p.scales + ((size_t)(row >> 4) * Ktg) * 16 + (row & 15);
            float acc[WT];
            f32x2 accp[WT / 2];                           // the same as pairs (kPacked)
            if constexpr (kPacked) {
#pragma unroll
                for (int i = 0; i < WT / 2; ++i) accp[i] = 0ull;
            } else {
#pragma unroll
                for (int i = 0; i < WT; ++i) acc[i] = 0.0f;
            }
            uint32_t scw = __ldg(scn);
#pragma unroll 1
            for (int s = 0; s < spt; ++s)
#pragma unroll
            for (int g = 0; g < (GW == 2 ? 1 : 2); ++g) {     // k-tile of the step
                int zp = 0;
                float ws;
                if (SUMS) unpack_scale(scw, zp, ws);
                else ws = __half2float(__ushort_as_half((unsigned short)(scw & 0xFFF0u)));
                // the next group's word: the next one in the row's run, except inside a K64
                // pair promoted per k-tile, whose second tile shares the first one's
                if (GW == 2 || g == 1 || p.ksh == 0) scn += 16;
                if (GW == 2 ? s + 1 < spt : (g == 0 || s + 1 < spt)) scw = __ldg(scn);
                const f32x2 ws2 = pack2(ws, ws);
                const float zf = (float)zp;
                if (!__all_sync(0xffffffffu, wait_on(acc0 + b * 8, par, kWaitEpi))) goto gave_up;
                tc_fence_after();
                const ulonglong2 *sv = reinterpret_cast<const ulonglong2 *>(
                    sv_base + (size_t)ss * G::kSlot + g * (TN * 4));
                // the accumulator holds (float)(d - z * sum of codes) of the group (the group's
                // first MMA overwrites it): nothing has to be converted
                uint32_t d[kCols];
#pragma unroll
                for (int c = 0; c < WT / kCols; ++c) {
                    tmem_ldn(lane_base + b * TN + c * kCols, d);
                    tmem_wait_ldn(d);
                    if constexpr (kPacked) {
#pragma unroll
                        for (int j = 0; j < kCols / 2; ++j)
                            fma2_acc(accp[c * (kCols / 2) + j],
                                     pack2(__uint_as_float(d[2 * j]), __uint_as_float(d[2 * j + 1])), ws2);
                    } else {
#pragma unroll
                        for (int j = 0; j < kCols / 4; ++j) {     // four tokens at a time
                            const int jj = c * (kCols / 4) + j;
                            float f[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) f[i] = __uint_as_float(d[4 * j + i]);
                            if constexpr (SUMS) {
                                ulonglong2 sm = sv[2 * TN / 4 + jj];
                                if (GW == 2) {                                     // exact: small integers
                                    const ulonglong2 sm1 = sv[3 * TN / 4 + jj];
                                    sm.x = add2(sm.x, sm1.x);
                                    sm.y = add2(sm.y, sm1.y);
                                }
                                float m[4];
                                unpack2(sm.x, m[0], m[1]);
                                unpack2(sm.y, m[2], m[3]);
#pragma unroll
                                for (int i = 0; i < 4; ++i) f[i] = fmaf(zf, m[i], f[i]);
                            }
                            float w[4] = {ws, ws, ws, ws};
                            if constexpr (!PERTOK) {
                                const ulonglong2 a4 = sv[jj];                      // four activation scales
                                unpack2(mul2(ws2, a4.x), w[0], w[1]);              // ws * as, rounded once
                                unpack2(mul2(ws2, a4.y), w[2], w[3]);
                            }
#pragma unroll
                            for (int i = 0; i < 4; ++i) acc[4 * jj + i] = fmaf(f[i], w[i], acc[4 * jj + i]);
                        }
                    }
                }
                // Tell the MMA that it may overwrite the buffer and, behind the step's last group, the copy
                // thread that the slot's images may be replaced. The copies write through the
                // async proxy, which an arrive does not order behind this warp's shared-memory reads: in
                // a kernel of 64-token tiles, whose workers take eight slots in a row at the start of a tile,
                // reads still under way got the scales of the slot's next use (step n + 8; W4A4, a third of
                // the calls). So the proxy fence comes first. With one group per step both arrives follow it
                // as one instruction; with two, the accumulator is given back before it (4096 tokens:
                // 1585 us against 1618 with the fence first and 1607 without; W4A4, 1024 tokens: 324
                // against 318 and 318).
                constexpr bool kOneArrive = kReadsSlot && GW == 2;
                if (kOneArrive) fence_proxy_async_smem();
                tc_fence_before();
                __syncwarp();
                if (kOneArrive) {
                    mbar_arrive_if(lane == 0 ? accempty0 + b * 8 : empty0 + ss * 8, lane < 2);
                } else {
                    mbar_arrive_if(accempty0 + b * 8, lane == 0);
                    if (kReadsSlot && g == 1) {
                        fence_proxy_async_smem();
                        __syncwarp();
                        mbar_arrive_if(empty0 + ss * 8, lane == 0);
                    }
                }
                if (++b == NB) {
                    b = 0;
                    par ^= 1u;
                }
                if ((GW == 2 || g == 1) && ++ss == kSS) ss = 0;
            }
            // store: thread = row, its tokens; rows are contiguous in y, so a warp writes 128 B
#pragma unroll
            for (int i = 0; i < WT / 2; ++i) {
                float v0, v1;
                if constexpr (kPacked) unpack2(accp[i], v0, v1);
                else { v0 = acc[2 * i]; v1 = acc[2 * i + 1]; }
                const int tok = tb * TN + chalf + 2 * i;
                if (PERTOK) {
                    if (tok < p.T) v0 = __fmul_rn(v0, __ldg(p.as_tok + tok));
                    if (tok + 1 < p.T) v1 = __fmul_rn(v1, __ldg(p.as_tok + tok + 1));
                }
                if (p.out_bf16) {
                    __nv_bfloat16 *y = static_cast<__nv_bfloat16 *>(p.y);
                    if (tok < p.T) __stcs(reinterpret_cast<unsigned short *>(y + (size_t)tok * p.M + row), __bfloat16_as_ushort(__float2bfloat16_rn(v0)));
                    if (tok + 1 < p.T) __stcs(reinterpret_cast<unsigned short *>(y + (size_t)(tok + 1) * p.M + row), __bfloat16_as_ushort(__float2bfloat16_rn(v1)));
                } else {
                    float *y = static_cast<float *>(p.y);
                    if (tok < p.T) __stcs(y + (size_t)tok * p.M + row, v0);
                    if (tok + 1 < p.T) __stcs(y + (size_t)(tok + 1) * p.M + row, v1);
                }
            }
        }
    gave_up:
        // ---- teardown, also after a failed wait: all roles have stopped issuing work when the
        // others have arrived at barrier 1; then the TMEM goes back
        tmem_wait_ld_all();
        tc_fence_before();
        asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
        tc_fence_after();
        if (warp == 0) tmem_dealloc(tmem_base, 512);
        return;
    }
    reg_dealloc<kRoleRegs>();
    if (warp == kWorkWarps) {
        // ====================== copies (one thread) =======================================
        // Two bulk copies per step: the fp16 weights of the tile's row block (both k-tiles) and
        // the activation image of its token block; the slot's previous contents must have been
        // consumed (by the MMAs, or by every worker warp whose MMAs are then complete).
        if (elect_one()) {
            int ss = 0;                    // step slot and the parity of its use, kept as counters
            uint32_t ph = 0;
            for (int ti = 0; ti < my_tiles; ++ti) {
                const int tile = (int)blockIdx.x + ti * (int)gridDim.x;
                const int tb = tile % p.tok_blocks, rb = tile / p.tok_blocks;
                const uint8_t *src = p.img + (size_t)tb * spt * G::kImgStep;
                const uint8_t *wsrc = p.wimg + (size_t)rb * p.Kt * kABytes;
                bool ok = true;
                for (int s = 0; s < spt; ++s, src += G::kImgStep, wsrc += 2 * kABytes) {
                    ok = wait_on(empty0 + ss * 8, ph ^ 1u, kWaitProd);
                    if (!ok) break;
                    const uint32_t fb = full0 + ss * 8;
                    const uint32_t dst = smem_u + ss * G::kSlot;
                    mbar_expect_tx(fb, 2 * kABytes + kImgCopy);
                    bulk_g2s_plain(dst, wsrc, 2 * kABytes, fb);
                    bulk_g2s_plain(dst + 2 * kABytes, src, kImgCopy, fb);
                    if (++ss == kSS) {
                        ss = 0;
                        ph ^= 1u;
                    }
                }
                if (!ok) break;
            }
            // No copy may still be in flight when the CTA gives its shared memory back: wait
            // (bounded) until the last armed use of every slot has all its bytes. On the normal
            // path every one of them was consumed long ago and these tests return at once; after
            // a wait that gave up somewhere, this is where the copies already started drain.
            for (int s2 = 0; s2 < kSS; ++s2) {
                const uint32_t last = (s2 < ss) ? ph : (ph ^ 1u);     // this round's use, or the one before
                const uint64_t t0 = global_timer_ns();
                while (!mbar_try_wait_hint(full0 + s2 * 8, last, kNapNs))
                    if (global_timer_ns() - t0 > p.wait_ns) {
                        atomicCAS(p.status, 0, kWaitProd);
                        break;
                    }
                // nor may a commit still have to arrive on a slot's barrier
                if (kSlotFreedByMma) wait_on(empty0 + s2 * 8, last, kWaitProd);
            }
        }
        __syncwarp();
    } else if (warp <= kWorkWarps + kMmaWarps) {
        // ====================== MMA issuers (one thread per warp, steps in turn) ===========
        const int mw = warp - (kWorkWarps + 1);
        if (elect_one()) {
            const uint64_t desc0 = smem_desc_at(smem_u, kLboH, kSboH);
            const int n_total = my_tiles * spt;            // steps of this CTA
            int ss = kByTile ? 0 : mw;     // step slot and the parity of its use, kept as counters
            uint32_t ph = 0;
            static_assert(kMmaWarps < kSS, "the first step of every MMA thread is in the first round of slots");
            for (int n = ss; n < n_total; n += kStepStride) {
                if (!wait_on(full0 + ss * 8, ph, kWaitMma)) break;
                bool ok = true;
#pragma unroll
                for (int hh = 0; hh < (kByTile ? 1 : 2); ++hh) {   // the step's two k-tiles, or this thread's
                    const uint32_t h = kByTile ? (uint32_t)mw : (uint32_t)hh;
                    const uint32_t gi = (GW == 2) ? (uint32_t)n : 2u * n + h;      // promote group
                    const uint32_t b = gi % NB, par = (gi / NB) & 1u;
                    const bool last = kByTile || hh == 1;
                    // the group's accumulator buffer has been read out
                    if (GW == 1 || hh == 0) {
                        ok = wait_on(accempty0 + b * 8, par ^ 1u, kWaitMma);
                        if (!ok) break;
                        tc_fence_after();
                    }
                    const uint64_t da = desc0 + (uint64_t)((ss * G::kSlot + h * kABytes) >> 4);
                    const uint64_t db = desc0 + (uint64_t)((ss * G::kSlot + 2 * kABytes + h * (TN * 64)) >> 4);
                    // the first MMA of a promote group overwrites the accumulator
                    tc_mma_f16(tmem_base + b * TN, da, db, kIdesc, (GW == 2 && hh == 1) ? 1u : 0u);
                    tc_mma_f16(tmem_base + b * TN, da + (2 * kLboH >> 4), db + (2 * kLboH >> 4), kIdesc, 1u);
                    if (GW == 1 || hh == 1) {
                        tc_commit(acc0 + b * 8);
                        // A commit tracks MMAs only. This thread has seen the slot's copies complete, and
                        // its own arrival passes that on to the workers, who read scales and sums from the
                        // slot behind this barrier. (Every worker thread testing the slot's barrier itself
                        // instead: 4096 tokens in block mode 1655 against 1607 us, W4A4 1024 336 against 316.)
                        if (kReadsSlot) mbar_arrive(acc0 + b * 8);
                    }
                    // the step's operands have been read when its MMAs are complete
                    if (kSlotFreedByMma && last) tc_commit(empty0 + ss * 8);
                }
                if (!ok) break;
                ss += kStepStride;
                if (ss >= kSS) {
                    ss -= kSS;
                    ph ^= 1u;
                }
            }
        }
        __syncwarp();
    }
    asm volatile("bar.arrive 1, %0;" ::"n"(kThreads) : "memory");
}

struct TcScratch {
    uint8_t *img = nullptr;
    size_t img_bytes = 0;
    uint8_t *wimg = nullptr;      // fp16 image of the call's weight (4 bytes per packed byte)
    size_t wimg_bytes = 0;
    SumsState *sums = nullptr;
} g_tc;

int g_tc_sms = 0;

template <int GW, bool PERTOK, int WT>
void launch_both(const TcParams &p, int grid) {
    static bool once = false;
    if (!once) {
        for (auto k : {gemm_w4a8_tc_kernel<GW, PERTOK, false, WT>, gemm_w4a8_tc_kernel<GW, PERTOK, true, WT>})
            TQ_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, TcTile<WT>::kSmem));
        once = true;
    }
    launch_pdl(gemm_w4a8_tc_kernel<GW, PERTOK, false, WT>, dim3(grid), dim3(kThreads), (size_t)TcTile<WT>::kSmem, p);
    launch_pdl(gemm_w4a8_tc_kernel<GW, PERTOK, true, WT>, dim3(grid), dim3(kThreads), (size_t)TcTile<WT>::kSmem, p);
}

template <int WT>
void launch_mode(const GemmTcArgs &a, const TcParams &p, int grid) {
    if (a.aq4) launch_both<2, false, WT>(p, grid);
    else if (!a.as_tok) launch_both<1, false, WT>(p, grid);
    else if (a.ksh) launch_both<2, true, WT>(p, grid);
    else launch_both<1, true, WT>(p, grid);
}

// Tokens per tile: the width whose rounds of tiles over the SMs cost least, a round counted as
// (tokens + 96) units. One constant for five modes whose own ones differ: a round of 148 tiles takes,
// at 128 / 192 / 256 tokens and K 5120, 63 / 78 / 102 us in block mode on K32 weights (constant 83),
// 58 / 78 / 102 on K64 (45), 48 / 56 / 69 with per-token scales on K32 (172; 89 at K 2048),
// 25 / 35 / 42 on K64 (57), 39 / 51 / 66 in W4A4 (56). The rest is how many rounds the tiles of a width
// need (136 tokens on 10240 rows: 2 / 1 / 1 rounds, so 192). Over 128 to 2048 tokens on 10240 x 5120,
// 5120 x 17408, 17408 x 5120 and 2048 x 5120 in these modes the choice is at most 3.5 % behind the
// fastest width (17408 x 5120, K64 blocks, 776 tokens: 453 us at 256, 438 at 192).
int choose_tile_tokens(int M, int T, int sms) {
    int best = 0;
    long best_cost = 0;
    for (int tn : {256, 192, 128}) {
        const long tiles = (long)(M / kTM) * ((T + tn - 1) / tn);
        const long cost = (tiles + sms - 1) / sms * (tn + 96);
        if (!best || cost < best_cost) {
            best = tn;
            best_cost = cost;
        }
    }
    return best;
}

}  // namespace

int launch_gemm_tc(const GemmTcArgs &a) {
    // covered: per-block activation scales (the reference's x_gemm_w4a8 arithmetic) or
    // per-token scales, rows a multiple of 128, K a multiple of 64
    if (!a.as == !a.as_tok) return -1;          // exactly one kind of activation scale
    if (a.aq4 && (!a.as || !a.ksh)) return -1;  // W4A4: K64 weights, scale per (token, K64)
    if (a.M % kTM || a.K % 64 || a.T < 128) return -1;     // steps of two k-tiles
    const int Kt = a.K / 32;
    if (!g_tc_sms) {
        int dev = 0;
        TQ_CHECK(cudaGetDevice(&dev));
        TQ_CHECK(cudaDeviceGetAttribute(&g_tc_sms, cudaDevAttrMultiProcessorCount, dev));
        if (g_tc_sms <= 0) g_tc_sms = 148;
        g_tc.sums = static_cast<SumsState *>(tq_dev_alloc(sizeof(SumsState), "gemm.tc.sums.state"));
        const SumsState first = {1, 0, 0, 0, 0};
        TQ_CHECK(cudaMemcpyAsync(g_tc.sums, &first, sizeof first, cudaMemcpyHostToDevice, stream()));
    }
    ProfScope prof(a.M, a.K, a.T, a.aq4 ? 44 : (a.ksh ? 64 : 4));
    const int TN = choose_tile_tokens(a.M, a.T, g_tc_sms);
    const int tok_blocks = (a.T + TN - 1) / TN, Tpad = tok_blocks * TN;
    const size_t ibytes = (size_t)(Kt / 2) * Tpad * 144;
    if (ibytes > g_tc.img_bytes) {
        if (g_tc.img) tq_dev_free(g_tc.img);
        g_tc.img = static_cast<uint8_t *>(tq_dev_alloc(ibytes, "gemm.tc.activation.image"));
        g_tc.img_bytes = ibytes;
    }
    const size_t wbytes = (size_t)a.M * a.K * 2;
    if (wbytes > g_tc.wimg_bytes) {
        if (g_tc.wimg) tq_dev_free(g_tc.wimg);
        g_tc.wimg = static_cast<uint8_t *>(tq_dev_alloc(wbytes, "gemm.tc.weight.image"));
        g_tc.wimg_bytes = wbytes;
    }
    PrepassArgs q{};
    q.codes = a.codes; q.scales = a.scales; q.as = a.as; q.asum = a.asum;
    q.aq = a.aq4 ? reinterpret_cast<const int8_t *>(a.aq4) : a.aq;
    q.wimg = g_tc.wimg; q.img = g_tc.img; q.sums = g_tc.sums;
    q.M = a.M; q.Kt = Kt; q.ksh = a.ksh; q.T = a.T; q.TN = TN; q.Tpad = Tpad;
    // one round of CTAs (8 per SM), shared between the two jobs by their items
    const size_t witems = (size_t)a.M * Kt, aitems = (size_t)(Kt / 2) * Tpad * 3;
    const int room = g_tc_sms * 8;
    const int ablocks = (int)std::min<size_t>((aitems / 3 + 255) / 256,
                                              std::max<size_t>(1, room * aitems / (aitems + witems)));
    q.wblocks = (int)std::min<size_t>((witems + 255) / 256, (size_t)std::max(1, room - ablocks));
    if (a.aq4) launch_pdl(gemm_tc_prepass_kernel<true>, dim3(q.wblocks + ablocks), dim3(256), 0, q);
    else launch_pdl(gemm_tc_prepass_kernel<false>, dim3(q.wblocks + ablocks), dim3(256), 0, q);
    TQ_LAUNCH_CHECK("gemm_tc_prepass_kernel");
    TcParams p{};
    p.wimg = g_tc.wimg; p.scales = a.scales; p.img = g_tc.img; p.y = a.y;
    p.as_tok = a.as_tok;
    p.sums = g_tc.sums;
    p.status = device_status_word();
    p.wait_ns = wait_limit_ns();
    p.M = a.M; p.Kt = Kt; p.ksh = a.ksh; p.T = a.T; p.tok_blocks = tok_blocks; p.out_bf16 = a.out_bf16;
    const int grid = std::min(g_tc_sms, (a.M / kTM) * tok_blocks);
    switch (TN) {
        case 256: launch_mode<64>(a, p, grid); break;
        case 192: launch_mode<48>(a, p, grid); break;
        default: launch_mode<32>(a, p, grid); break;
    }
    TQ_LAUNCH_CHECK("gemm_w4a8_tc_kernel");
    return 0;
}

int prefill_sums_variant() {
    if (!g_tc.sums) return -1;
    unsigned last = 0;
    if (cudaMemcpyAsync(&last, &g_tc.sums->last, sizeof last, cudaMemcpyDeviceToHost, stream()) != cudaSuccess ||
        cudaStreamSynchronize(stream()) != cudaSuccess)
        return -1;
    return (int)last;
}

}  // namespace tq
