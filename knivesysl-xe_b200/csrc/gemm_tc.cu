// gemm_tc.cu — prefill W4A8 GEMM on the sm_100a tensor cores: tcgen05.mma kind::f8f6f4 on
// integer-valued e4m3 operands, fp32 accumulators in tensor memory (TMEM).
//
// Replaces gemm_rc16 / the unsplit path of x_gemm_w4a8 (xpu/src/kernels_dpas.cpp:1255-1332,
// 1371-1378): Y[tok][n] = sum over k-tiles, ascending, of (float)(d - z*asum) * (ws*as) with
// d the exact int32 dot of one 16-row x K32 tile, accumulated with fma into one fp32
// accumulator per output - the arithmetic and the order of the reference.
//
// Why a floating-point pipe for an integer dot. The accumulator is a float already: with kind::i8 it is
// int32, and every output costs an integer add and a float add more per k-tile on the CUDA cores
// (the exact conversion). And why e4m3 rather than fp16: the 4-bit codes less their zero point (-15..15)
// are exact in its four significant bits, and an int8 activation is the sum of two numbers that are, its low
// nibble (0..15) and the multiple of 16 that is left (-128..112). So a k-tile is two MMAs of K = 32,
// W x high and W x low, as many tensor cycles as two of K = 16 in fp16, on weights of half the bytes;
// 4-bit activations need one. The products (< 2^11) and the sums of a k-tile (< 2^16) or a K64 group
// (< 2^17) are exact in the fp32 accumulation (checked on random and extreme operands against integers), so
// the accumulator IS (float)(d - z*asum), bit for bit, and the promote is one fma per output.
//
// Mapping. Weights are the M side of the MMA (128 output rows = 128 TMEM lanes), tokens the
// N side, and one accumulator read-out yields exactly the per-k-tile dots the reference
// promotes. A CTA's tile is two row blocks x 32 to 128 tokens, or one x 256, where the promote reads an activation
// scale per token and group (block and 4-bit modes), one row block x 128, 192 or 256 tokens with per-token
// scales (choose_tile_tokens). The K loop advances in steps of two k-tiles. Both operands come from images
// that one pre-pass writes in the operand layout (canonical no-swizzle K-major core matrices): the
// activation image and the weight image, every 4-bit code expanded to e4m3 q - z once per call.
// Tiles are walked token block fastest, so the CTAs that run together share a few row blocks of
// the weight image while the whole activation image stays in L2.
//
// A CTA (20 warps, one per SM, persistent over tiles) runs three roles connected by
// mbarriers (step slots in shared memory, accumulator buffers in the 512 columns of TMEM):
//  * one thread starts the bulk (TMA) copies of a step: 8 KiB of weights a row block, with 1 KiB of their scales unless
//    the activation scales are per token, and the activations of the tile's tokens, each contiguous in its image;
//  * two MMA threads (in two warps): the tcgen05.mma of a k-tile into the
//    promote group's accumulator buffer (the first one overwrites it), then tcgen05.commit;
//  * workers (16 warps): thread = a row of every row block x a quarter of the tile's tokens. Per promote group:
//    wait for the group's accumulator, then a few columns at a time tcgen05.ld and
//    acc = fma(d, ws*as, acc); the accumulators stay in registers for the whole K loop and are
//    stored at the end (coalesced over rows).
//
// What bounds it: the workers, in block mode 1060 clocks a group of 256 x 128 outputs (900 of them at work).
// Their multiplies and fmas alone take 640: a packed multiply and two fmas of a token pair measure 5 clocks per
// scheduler, not 4. The loop without MMAs measures 740, with MMAs running a quarter of the time 940:
// an activation scale is a broadcast read of shared memory (two cycles for 16 bytes), which the MMAs' operand
// reads hold up. Hence two rows per thread: a scale that is read serves both, half the reads (one row of 256
// tokens: 183 instructions a group of 64 outputs, 1210 clocks). With per-token scales nothing is read there, one
// row block and wide tokens move fewer operand bytes, and the wait for hand-offs is a quarter of the time.
//
// Measured, staging included, against fp16 operands and 128-row tiles of 128 to 256 tokens: 17408 x 5120
// K64, 4096 tokens in the reference's arithmetic 1.44 against 1.59 ms; 2048 tokens with per-token scales
// 378 against 428 us; 1024 tokens W4A4 254 against 321 us; 5120 x 17408, 1000 tokens 479 against 598 us;
// 10240 x 5120 K32, 136 tokens 70 against 114 us (with per-token scales, minutes on end, the power limit takes
// most of the gain: 420 against 430 us). Where that came from, block mode at 4096 tokens: row pairs
// alone 1.74 ms (they spill); weight scales as fp32 from the step slot instead of a load, a conversion and a
// pointer per row, walking addresses instead of products of counters, a barrier test by the whole warp: 1.44.
// Tried and slower: TMEM loads issued a chunk ahead (1.47), in chunks of four (1.59), packed fma (1.55: a
// register move per value), scales read a group ahead (by 5 % in a copy of the loop), the 16x256b TMEM
// load (910 against 740 clocks in such a copy).
//
// Every mbarrier wait is bounded; on expiry the kernel records a status word, stops
// issuing work, still frees its TMEM and returns.
#include "tc.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

namespace tq {

namespace {

constexpr int kTM = 128;                 // weight rows of one MMA (TMEM lanes)
constexpr int kABytes = kTM * 32;        // expanded e4m3 weights of 128 rows of one k-tile
constexpr int kWScales = kTM * 4;        // their fp32 scales
constexpr int kWImgStep = 2 * kABytes + 2 * kWScales;    // weight image of a row block and step (two k-tiles)
constexpr int kWorkWarps = 16;
constexpr int kMmaWarps = 2;
// Workers, the warp that starts the copies, the MMA warps, and one idle warp that completes the
// last group of four (setmaxnreg moves registers between groups of four warps).
constexpr int kThreads = (kWorkWarps + 4) * 32;
// A launch with 20 warps gives every thread 96 registers (61440 of the SM's); the workers of the
// widest tiles, whose 64 accumulators and loaded columns do not fit in that, take 104 and the other
// four warps keep 64: 512 * 104 + 128 * 64 = 61440, exactly what the launch holds. (112 and 32: the
// MMA and copy threads spill, and per-token prefill of 4096 tokens took 0.80 instead of 0.69 ms.) No form
// without sums spills but the 80-token tile in W4A4 (24 bytes, both forms in one kernel); with sums the widest ones do (up to
// 148).
constexpr int kLaunchRegs = 96, kWorkRegs = 104, kRoleRegs = 64;
static_assert(kWorkWarps * 32 * kWorkRegs + 4 * 32 * kRoleRegs <= kThreads * kLaunchRegs,
              "the register split must not exceed what the launch holds");
// Suspend-time hint of the waits: a thread that polls back to back takes issue slots from the warps
// beside it, one that waits with the hint stays off the scheduler until the phase completes.
constexpr uint32_t kNapNs = 2000;

// What one accumulator read-out is promoted with.
enum Mode {
    kBlock,      // a scale per (token, K32): the reference's arithmetic
    kInt4,       // 4-bit activations, a scale per (token, K64)
    kToken,      // per-token scales, K32 weight groups
    kToken64     // per-token scales, K64 weight groups
};

// Geometry of a tile of R * 128 rows x TN = 4 * WT tokens (a worker thread promotes R rows x WT tokens).
template <int MODE, int WT>
struct TcTile {
    static constexpr bool kPerTok = MODE == kToken || MODE == kToken64;
    static constexpr int GW = MODE == kInt4 || MODE == kToken64 ? 2 : 1;  // k-tiles per promote
    static constexpr int R = kPerTok || WT > 32 ? 1 : 2;     // row blocks of 128
    static constexpr int TN = kWorkWarps / 4 * WT;           // tokens per tile
    static constexpr int kChunk = kPerTok ? 16 : 8;          // tokens of one TMEM load of a worker
    static constexpr int kRest = WT % kChunk, kMain = WT - kRest;
    static constexpr int kRowCols = (TN + 31) / 32 * 32;     // accumulator columns of a row block
    static constexpr int kAccCols = R * kRowCols;            // ... of a promote group
    static constexpr int NB = 512 / kAccCols >= 8 ? 8 : 512 / kAccCols >= 4 ? 4 : 2;     // accumulator buffers in TMEM
    static constexpr int kParts = MODE == kInt4 ? 1 : 2;     // e4m3 operands that an activation code makes
    static constexpr int kBPart = TN * 32;                   // one of them, one k-tile
    static constexpr int kBTile = kParts * kBPart;
    static constexpr int kBStep = 2 * kBTile;                // a step is two k-tiles
    static constexpr int kScales = TN * 8;                   // as of both k-tiles; as many bytes of sum differences
    static constexpr int kImgStep = kBStep + 2 * kScales;    // activation image of one step
    // weights of a row block and step: the e4m3 codes of both k-tiles, then (not per token) their scales
    static constexpr int kABlock = kPerTok ? 2 * kABytes : kWImgStep;
    static constexpr int kAStep = R * kABlock;
    static constexpr int kSlot = kAStep + kImgStep;          // step slot: weights, then the image
    static constexpr int kSlots = 230000 / kSlot < 8 ? 230000 / kSlot : 8;
    static constexpr int kSmem = kSlots * kSlot;             // > half an SM's shared memory: one CTA per SM,
                                                             // which the 512-column TMEM allocation requires
    static_assert(kSmem > 116 * 1024 && kSlots >= 3 && kSlot % 128 == 0, "slots");
    static_assert(kMain % kChunk == 0 && (kRest == 0 || R == 2), "chunks");
    static_assert(TN % 16 == 0 && NB * kAccCols <= 512, "tile");
};
// bytes of the activation image per token and step: the codes, two scales, two sum differences
__host__ __device__ constexpr int image_step_bytes(bool int4) { return (int4 ? 64 : 128) + 16; }

// Device words that say which variant of the GEMM does a call. The pre-pass stamps `diff` with the
// generation if some asum of the call is not the sum of its codes, and `zp` if some zero point of the
// weight is not 0; only where both are stamped does z * (sum of codes - asum) enter the result. The call's
// last kernel moves the generation on, so that nothing has to be cleared and a captured
// call decides by the data of each replay.
struct SumsState {
    unsigned gen, diff, zp;      // read together, with `arrived`, as one 16-byte word
    unsigned arrived;            // CTAs of the last kernel that have read the words
    unsigned last;               // the call before: did it apply the sums?
};
// Stamps *word unless it is stamped already: a store by every CTA costs far more than the look (54 us of a call with
// 1184 CTAs of the pre-pass, 145 with a store by every warp; 10240 x 5120, 136 tokens, in the version with fp16 operands).
__device__ __forceinline__ void stamp(unsigned *word, unsigned gen) {
    if (__ldcg(word) != gen) *word = gen;
}
// Never 0, what the stamps start from.
__device__ __forceinline__ unsigned next_generation(unsigned g) { return g + 1 ? g + 1 : 1; }

struct TcParams {
    const uint8_t *wimg;     // per (128-row block, step): kWImgStep bytes, the e4m3 weights of both k-tiles, then their scales
    const uint16_t *scales;
    const uint8_t *img;      // per (TN-token block, step): kImgStep bytes (see the pre-pass)
    void *y;
    const float *as_tok;     // per-token scales (PERTOK kernels)
    SumsState *sums;
    int *status;
    unsigned long long wait_ns;   // limit of every mbarrier wait
    int M, Kt, ksh, T, tok_blocks, out_bf16;
};

// e4m3 of the integers that the operands are made of. Its four significant bits hold 0..16 and their
// multiples by a power of two; a word is four table entries.
constexpr uint32_t kE0 = 0x44403800u, kE4 = 0x4E4C4A48u, kE8 = 0x53525150u, kE12 = 0x57565554u;   // 0..15
constexpr uint32_t kN8 = 0x4A4C4E50u, kN4 = 0x38404448u;                                          // 8..5, 4..1
constexpr uint32_t kTimes16 = 0x20202020u, kH0 = 0x64605800u;       // times 16: four more in the exponent; 0 stays 0

// Four lookups in a table of 16 bytes (a0 the first four): per nibble of the low half of s its low three
// bits select one of the first and one of the last eight, and its top bit (mask: 0xFF or 0) chooses.
__device__ __forceinline__ uint32_t lut16(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t s,
                                          uint32_t mask) {
    const uint32_t i = s & 0x7777u, lo = __byte_perm(a0, a1, i), hi = __byte_perm(a2, a3, i);
    return (hi & mask) | (lo & ~mask);
}
// Per nibble of the low half of s: 0xFF if its top bit is set, else 0. (The permute replicates the
// sign bit of the selected byte, 0x80, where a selector's top bit is set, and copies the byte where not.)
__device__ __forceinline__ uint32_t top_bits(uint32_t s) {
    uint32_t m;
    asm("prmt.b32 %0, %1, %1, %2;" : "=r"(m) : "r"(0x80808080u), "r"(s));
    return (m & 0x7F7F7F7Fu) | ((m << 1) & 0x80808080u);
}
// Four nibbles (the low half of s), two's complement, as e4m3.
__device__ __forceinline__ uint32_t nib4_to_e4m3(uint32_t s) {
    const uint32_t m = top_bits(s);
    return lut16(kE0, kE4, kN8, kN4, s, m) | (m & 0x80808080u);
}
// Four int8 codes -> e4m3 of their low nibbles (0..15) and of what is left (a multiple of 16, -128..112),
// whose sum a code is. A half word's four nibbles are low, high, low, high: each half is looked up in
// both tables, and the bytes that belong to either are picked.
__device__ __forceinline__ void codes_to_e4m3(uint32_t w, uint32_t &high, uint32_t &low) {
    const uint32_t w1 = w >> 16, m0 = top_bits(w), m1 = top_bits(w1);
    low = __byte_perm(lut16(kE0, kE4, kE8, kE12, w, m0), lut16(kE0, kE4, kE8, kE12, w1, m1), 0x6420);
    constexpr uint32_t h4 = kE4 + kTimes16, h8 = kN8 + kTimes16, h12 = kN4 + kTimes16;
    high = __byte_perm(lut16(kH0, h4, h8, h12, w, m0) | (m0 & 0x80808080u),
                       lut16(kH0, h4, h8, h12, w1, m1) | (m1 & 0x80808080u), 0x7531);
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
//    (128-row block, step) twice the kABytes of e4m3 values q - z of a k-tile in the operand layout (row groups
//    of 8 are kSbo apart, a row's two 16-byte K-chunks kLbo apart), then twice the rows' scales as fp32. With the zero point taken
//    off here the tensor core's dot is d - z * sum(codes) itself (integers below 2^17, exact), so
//    the GEMM promotes asymmetric weights like symmetric ones. A thread expands one row of one
//    k-tile, by a table of the 16 codes for the row's zero point; 8 consecutive lanes write 128
//    contiguous bytes per chunk. 2.25 bytes out per packed byte: 100 MB for 17408 x 5120, written once per call
//    and read by every token block's tiles, from L2 where they run together.
//  * Activations: the caller's staging -> per (TN-token block, step of two k-tiles) the e4m3
//    codes of k-tile 0 then 1 as [TN / 8][2 K-chunks][8 tokens][16 B], of an int8 code first the part that is
//    a multiple of 16, then the low nibbles; as[2][TN], and (sum of the codes - asum)[2][TN], 0
//    unless the caller's asum is something else than the sum of its codes (SumsState).
//    Tokens >= T are padded with zeros. S4: int4 codes; a K64 block's scale and sum go with its
//    first k-tile.
// CTAs per SM: 48 registers a thread, and the grid is one round of them (60 registers and the second round that
// they bring: 2048 x 2048, 512 tokens, 29 us for the call instead of 25).
constexpr int kPreCtas = 5;
template <bool S4>
__global__ void __launch_bounds__(256, kPreCtas) gemm_tc_prepass_kernel(const PrepassArgs a) {
    __shared__ uint4 table[16];      // per zero point (z + 8): e4m3 of q - z, by nibble
    pdl_trigger();
    {
        const int z8 = threadIdx.x >> 4, v = (int)((threadIdx.x & 15) ^ 8) - z8, mag = v < 0 ? -v : v;
        const int e = 31 - __clz(mag);
        reinterpret_cast<uint8_t *>(table)[threadIdx.x] =
            (uint8_t)(mag == 0 ? 0 : (v < 0 ? 0x80 : 0) | ((e + 7) << 3) | (((mag << 3) >> e) & 7));
    }
    __syncthreads();
    pdl_wait();      // the images may still be read by the previous call's kernel
    const unsigned gen = __ldcg(&a.sums->gen);
    if ((int)blockIdx.x < a.wblocks) {
        const uint32_t n = (uint32_t)a.M * a.Kt;
        const int Ktg = a.Kt >> a.ksh;
        uint32_t any = 0;
        for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < n; i += a.wblocks * 256) {
            const int kt = (int)(i / (uint32_t)a.M), m = (int)(i - (uint32_t)kt * a.M);
            const uint4 c4 = ldg_stream_v4(a.codes + ((size_t)(m >> 4) * a.Kt + kt) * 256 + (m & 15) * 16);
            const uint32_t sw = __ldg(a.scales + ((size_t)(m >> 4) * Ktg + (kt >> a.ksh)) * 16 + (m & 15));
            any |= sw & 15u;
            const uint4 t = table[(sw ^ 8u) & 15u];
            const uint32_t w[4] = {c4.x, c4.y, c4.z, c4.w};      // k = 8 j..8 j + 7, nibble i = k 8 j + i
            uint32_t o[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                o[2 * j] = lut16(t.x, t.y, t.z, t.w, w[j], top_bits(w[j]));
                o[2 * j + 1] = lut16(t.x, t.y, t.z, t.w, w[j] >> 16, top_bits(w[j] >> 16));
            }
            const int r = m & (kTM - 1);
            uint8_t *blk = a.wimg + ((size_t)(m / kTM) * (a.Kt >> 1) + (kt >> 1)) * kWImgStep;
            uint8_t *dst = blk + (kt & 1) * kABytes + (r >> 3) * kSbo + (r & 7) * 16;
            reinterpret_cast<float *>(blk + 2 * kABytes + (kt & 1) * kWScales)[r] =
                __half2float(__ushort_as_half((unsigned short)(sw & 0xFFF0u)));
            *reinterpret_cast<uint4 *>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
            *reinterpret_cast<uint4 *>(dst + kLbo) = make_uint4(o[4], o[5], o[6], o[7]);
        }
        if (__syncthreads_or((int)any) && threadIdx.x == 0) stamp(&a.sums->zp, gen);
        return;
    }
    const int T = a.T, TN = a.TN, nsteps = a.Kt >> 1;
    const uint32_t n = (uint32_t)(S4 ? nsteps : a.Kt) * a.Tpad;
    const size_t img_step = (size_t)TN * image_step_bytes(S4);
    const int part = TN * 32;                    // one e4m3 operand of one k-tile
    int diff = 0;
    for (uint32_t i = (blockIdx.x - a.wblocks) * 256 + threadIdx.x; i < n; i += (gridDim.x - a.wblocks) * 256) {
        const int kk = (int)(i / (uint32_t)a.Tpad), tok = (int)(i - (uint32_t)kk * a.Tpad);   // k-tile, S4: step
        const int st = S4 ? kk : kk >> 1, tb = tok / TN, tl = tok - tb * TN;
        const bool real = tok < T;
        const size_t at = (size_t)kk * T + tok;
        uint8_t *blk = a.img + ((size_t)tb * nsteps + st) * img_step;
        uint8_t *dst = blk + (tl >> 3) * kSbo + (tl & 7) * 16;
        float *sv = reinterpret_cast<float *>(blk + (size_t)part * (S4 ? 2 : 4)) + tl;
        int sum = 0;
        uint4 v[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
        float sc = 0.0f;
        int asum = 0;
        if (real) {
            v[0] = __ldg(reinterpret_cast<const uint4 *>(a.aq + at * 32));
            v[1] = __ldg(reinterpret_cast<const uint4 *>(a.aq + at * 32) + 1);
            if (a.as) sc = __ldg(a.as + at);
            asum = __ldg(a.asum + at);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {            // k = 0..15, 16..31 of the k-tile; S4: k-tile 0, 1 of the step
            const uint32_t p[4] = {v[h].x, v[h].y, v[h].z, v[h].w};
            if (S4) {                            // byte b = k 2b (low nibble), 2b + 1 (high nibble)
                uint32_t o[8];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    o[2 * j] = nib4_to_e4m3(p[j]);
                    o[2 * j + 1] = nib4_to_e4m3(p[j] >> 16);
                    // codes + 8 as bytes; 8 of them to a word
                    sum = __dp4a((int)((p[j] & 0x0F0F0F0Fu) ^ 0x08080808u), 0x01010101, sum);
                    sum = __dp4a((int)(((p[j] >> 4) & 0x0F0F0F0Fu) ^ 0x08080808u), 0x01010101, sum) - 64;
                }
                *reinterpret_cast<uint4 *>(dst + h * part) = make_uint4(o[0], o[1], o[2], o[3]);
                *reinterpret_cast<uint4 *>(dst + h * part + kLbo) = make_uint4(o[4], o[5], o[6], o[7]);
            } else {
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    codes_to_e4m3(p[j], hi[j], lo[j]);
                    sum = __dp4a((int)p[j], 0x01010101, sum);
                }
                uint8_t *d = dst + (kk & 1) * 2 * part + h * kLbo;
                *reinterpret_cast<uint4 *>(d) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4 *>(d + part) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
        }
        const int d = sum - asum;
        sv[S4 ? 0 : (kk & 1) * TN] = sc;
        sv[(S4 ? 2 : 2 + (kk & 1)) * TN] = (float)d;
        if (S4) sv[TN] = sv[3 * TN] = 0.0f;
        diff |= d;
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

__device__ __forceinline__ void tmem_ldn(uint32_t taddr, uint32_t (&v)[4]) { tmem_ld4(taddr, v); }
__device__ __forceinline__ void tmem_ldn(uint32_t taddr, uint32_t (&v)[8]) { tmem_ld8(taddr, v); }
__device__ __forceinline__ void tmem_ldn(uint32_t taddr, uint32_t (&v)[16]) { tmem_ld16(taddr, v); }
__device__ __forceinline__ void tmem_wait_ldn(uint32_t (&v)[8]) { tmem_wait_ld8(v); }
__device__ __forceinline__ void tmem_wait_ldn(uint32_t (&v)[16]) { tmem_wait_ld16(v); }
// one wait for two loads
__device__ __forceinline__ void tmem_wait_ldn2(uint32_t (&v)[4], uint32_t (&w)[4]) { tmem_wait_ld4x2(v, w); }
__device__ __forceinline__ void tmem_wait_ldn2(uint32_t (&v)[8], uint32_t (&w)[8]) { tmem_wait_ld8x2(v, w); }
__device__ __forceinline__ float lds_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
// four fp32 values of shared memory as two pairs; volatile, so that it stays where it is written, ahead of
// the wait for the TMEM loads whose latency it shares
__device__ __forceinline__ ulonglong2 lds_pairs(uint32_t addr) {
    ulonglong2 v;
    asm volatile("ld.shared.v2.u64 {%0,%1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(addr) : "memory");
    return v;
}

// GW = k-tiles accumulated in TMEM before one fp32 promote (1: the reference's arithmetic with
// a scale per (token, K32); 2: K64 weight groups with per-token activation scales, or
// one activation scale per (token, K64): the W4A4 arithmetic). With per-token scales
// the activation scale is applied once at the end (y = acc * as_tok).
//
// The K loop advances in steps of two k-tiles (K is a multiple of 64); step n of the CTA
// (counted across its tiles) uses step slot n % kSlots, promote group n uses accumulator buffer
// n % NB. A worker warp owns 32 TMEM lanes (a row of each row block) and WT of the tile's tokens.
//
// SUMS: z * (sum of codes - asum) is applied, for callers whose asum is not the sum of
// their codes, on weights with zero points. ADVANCE: this is the call's last kernel.
template <int MODE, bool SUMS, bool ADVANCE, int WT>
__device__ __forceinline__ void tc_gemm(const TcParams &p, const unsigned gen) {
    using G = TcTile<MODE, WT>;
    constexpr int TN = G::TN, NB = G::NB, kSS = G::kSlots, R = G::R, GW = G::GW;
    constexpr bool PERTOK = G::kPerTok;
    constexpr uint32_t kIdesc = idesc_f8(kTM, TN);
    // what a step copies of the image: the codes, the activation scales, the sum differences
    constexpr uint32_t kImgCopy = SUMS ? G::kImgStep : (PERTOK ? G::kBStep : G::kBStep + G::kScales);
    // per-token scales: the promote reads nothing from the slot, so its MMAs free it
    constexpr bool kReadsSlot = !PERTOK || SUMS, kSlotFreedByMma = !kReadsSlot;
    // the weight scales come with the step's weights (as fp32; SUMS needs the zero points beside them)
    constexpr bool kScalesFromSlot = !PERTOK && !SUMS;
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
    if (ADVANCE && threadIdx.x == 0 && atomicInc(&p.sums->arrived, gridDim.x - 1) == gridDim.x - 1) {
        p.sums->last = SUMS;
        p.sums->gen = next_generation(gen);
    }

    const int spt = p.Kt >> 1;                           // steps per tile
    const int ntiles = (p.M / kTM + R - 1) / R * p.tok_blocks;
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
        const int q4 = warp & 3, cq = warp >> 2;          // lane quarter, token quarter
        // Its tokens: kMain from c_main, taken kChunk at a time, and kRest from c_rest. (All chunks start on a
        // multiple of their width.) With 64 accumulators a thread c0 goes into the addresses, which saves the
        // registers that spill otherwise; the narrower tiles are up to 3 to 8 % faster without it.
        constexpr bool kFold = R * WT == 64;
        const int c_main = cq * G::kMain, c_rest = 4 * G::kMain + cq * G::kRest, c0 = kFold ? c_main : 0;
        const int rloc = q4 * 32 + lane;                  // row inside the row block = TMEM lane
        const uint32_t lane_base = tmem_base + ((uint32_t)(q4 * 32) << 16) + c0;
        const int Ktg = p.Kt >> p.ksh, nrb = p.M / kTM;
        // inside a step slot: the activation scales, the scales of this thread's rows
        const uint32_t sv_base = smem_u + G::kAStep + G::kBStep;
        const uint32_t ws_off = 2 * kABytes + rloc * 4 - (G::kAStep + G::kBStep + c0 * 4);
        uint32_t sv = sv_base + c0 * 4, ebar = empty0;    // slot ss: its scales, its barrier
        uint32_t tcol = lane_base, abar = acc0, par = 0;  // the accumulator buffer, its barrier and parity

        for (int ti = 0; ti < my_tiles; ++ti) {
            const int tile = (int)blockIdx.x + ti * (int)gridDim.x;
            const int tb = tile % p.tok_blocks, rb = tile / p.tok_blocks * R;
            // The scale words of the group being promoted, where they do not come with the step (kScalesFromSlot).
            const uint16_t *scn[R];
            uint32_t scw[R];
            if constexpr (!kScalesFromSlot) {
#pragma unroll
                for (int h = 0; h < R; ++h) {
                    const int row = min(rb + h, nrb - 1) * kTM + rloc;
                    scn[h] = p.scales + ((size_t)(row >> 4) * Ktg) * 16 + (row & 15);
                    scw[h] = __ldg(scn[h]);
                }
            }
            float acc[R][WT];
#pragma unroll
            for (int h = 0; h < R; ++h)
#pragma unroll
                for (int i = 0; i < WT; ++i) acc[h][i] = 0.0f;
#pragma unroll 1
            for (int s = 0; s < spt; ++s)
#pragma unroll
            for (int g = 0; g < (GW == 2 ? 1 : 2); ++g) {     // k-tile of the step
                float ws[R], zf[R];
                if constexpr (!kScalesFromSlot) {
#pragma unroll
                    for (int h = 0; h < R; ++h) {
                        int zp = 0;
                        if (SUMS) unpack_scale(scw[h], zp, ws[h]);
                        else ws[h] = __half2float(__ushort_as_half((unsigned short)(scw[h] & 0xFFF0u)));
                        // the next group's word: the next one in the row's run, except inside a K64
                        // pair promoted per k-tile, whose second tile shares the first one's
                        if (GW == 2 || g == 1 || p.ksh == 0) scn[h] += 16;
                        if (GW == 2 ? s + 1 < spt : (g == 0 || s + 1 < spt)) scw[h] = __ldg(scn[h]);
                        zf[h] = (float)zp;
                    }
                }
                // usually complete: one test by the whole warp; else every lane waits for itself
                if (!mbar_test_wait_warp(abar, par)) {
                    if (!__all_sync(0xffffffffu, wait_on(abar, par, kWaitEpi))) goto gave_up;
                }
                tc_fence_after();
                if constexpr (kScalesFromSlot) {
#pragma unroll
                    for (int h = 0; h < R; ++h)
                        ws[h] = lds_f32(sv + ws_off + h * G::kABlock + g * kWScales);
                }
                f32x2 ws2[R];
#pragma unroll
                for (int h = 0; h < R; ++h) ws2[h] = pack2(ws[h], ws[h]);
                // The accumulators hold (float)(d - z * sum of codes) of the group (the group's
                // first MMA overwrites them): nothing has to be converted.
                const uint32_t svg = sv + g * (TN * 4);           // activation scales of the k-tile
                // N accumulators of row block h from number i0, loaded to d, their scales (at `at`) in as
                auto promote = [&](auto &d, const ulonglong2 *as, const uint32_t at, const int h, const int i0) {
                    constexpr int N = sizeof(d) / 4;
#pragma unroll
                    for (int j = 0; j < N / 4; ++j) {             // four tokens
                        float f[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) f[i] = __uint_as_float(d[4 * j + i]);
                        if constexpr (SUMS) {
                            ulonglong2 sm = lds_pairs(at + 2 * TN * 4 + 16 * j);
                            if (GW == 2) {                                     // exact: small integers
                                const ulonglong2 sm1 = lds_pairs(at + 3 * TN * 4 + 16 * j);
                                sm.x = add2(sm.x, sm1.x);
                                sm.y = add2(sm.y, sm1.y);
                            }
                            float m[4];
                            unpack2(sm.x, m[0], m[1]);
                            unpack2(sm.y, m[2], m[3]);
#pragma unroll
                            for (int i = 0; i < 4; ++i) f[i] = fmaf(zf[h], m[i], f[i]);
                        }
                        float w[4] = {ws[h], ws[h], ws[h], ws[h]};
                        if constexpr (!PERTOK) {
                            // one row block: read here, not ahead of the TMEM wait, where they spill (119 against 114 us)
                            const ulonglong2 a4 = R == 1 ? lds_pairs(at + 16 * j) : as[j];
                            unpack2(mul2(ws2[h], a4.x), w[0], w[1]);           // ws * as, rounded once
                            unpack2(mul2(ws2[h], a4.y), w[2], w[3]);
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            acc[h][i0 + 4 * j + i] = fmaf(f[i], w[i], acc[h][i0 + 4 * j + i]);
                    }
                };
                // N tokens of every row, from token (and column) c0 + col
                auto chunk = [&](auto n_tag, const int col, const int i0) {
                    constexpr int N = decltype(n_tag)::value;
                    const uint32_t at = svg + col * 4;
                    if constexpr (R == 1) {
                        uint32_t d[N];
                        tmem_ldn(tcol + col, d);
                        tmem_wait_ldn(d);
                        promote(d, nullptr, at, 0, i0);
                    } else {
                        uint32_t d0[N], d1[N];
                        ulonglong2 as[N / 4];
                        tmem_ldn(tcol + col, d0);
                        tmem_ldn(tcol + G::kRowCols + col, d1);
#pragma unroll
                        for (int j = 0; j < N / 4; ++j) as[j] = lds_pairs(at + 16 * j);
                        tmem_wait_ldn2(d0, d1);
                        promote(d0, as, at, 0, i0);
                        promote(d1, as, at, 1, i0);
                    }
                };
#pragma unroll
                for (int i = 0; i < G::kMain; i += G::kChunk)
                    chunk(std::integral_constant<int, G::kChunk>{}, (kFold ? 0 : c_main) + i, i);
                if constexpr (G::kRest != 0) chunk(std::integral_constant<int, G::kRest>{}, c_rest, G::kMain);
                // Tell the MMA that it may overwrite the buffer and, behind the step's last group, the copy
                // thread that the slot's images may be replaced. The copies write through the
                // async proxy, which an arrive does not order behind this warp's shared-memory reads: in
                // a kernel of 64-token tiles, whose workers take eight slots in a row at the start of a tile,
                // reads still under way got the scales of the slot's next use (step n + 8; W4A4, a third of
                // the calls). So the proxy fence comes first. With one group per step both arrives follow it
                // as one instruction; with two, the accumulator is given back before it.
                constexpr bool kOneArrive = kReadsSlot && GW == 2;
                if (kOneArrive) fence_proxy_async_smem();
                tc_fence_before();
                __syncwarp();
                if (kOneArrive) {
                    mbar_arrive_if(lane == 0 ? abar + NB * 8 : ebar, lane < 2);
                } else {
                    mbar_arrive_if(abar + NB * 8, lane == 0);
                    if (kReadsSlot && g == 1) {
                        fence_proxy_async_smem();
                        __syncwarp();
                        mbar_arrive_if(ebar, lane == 0);
                    }
                }
                tcol += G::kAccCols;
                abar += 8;
                if (kByTile ? g == 1 : abar == acc0 + NB * 8) {
                    tcol -= NB * G::kAccCols;
                    abar -= NB * 8;
                    par ^= 1u;
                }
                if (GW == 2 || g == 1) {
                    sv += G::kSlot;
                    ebar += 8;
                    if (ebar == empty0 + kSS * 8) {
                        sv -= kSS * G::kSlot;
                        ebar -= kSS * 8;
                    }
                }
            }
            // store: thread = row, its tokens; rows are contiguous in y, so a warp writes 128 B
#pragma unroll
            for (int h = 0; h < R; ++h) {
                if (rb + h >= nrb) break;
                const int row = (rb + h) * kTM + rloc;
#pragma unroll
                for (int i = 0; i < WT / 2; ++i) {
                    float v0 = acc[h][2 * i], v1 = acc[h][2 * i + 1];
                    const int tok = tb * TN + (2 * i < G::kMain ? c_main + 2 * i : c_rest + 2 * i - G::kMain);
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
        // A bulk copy per row block for the step's weights (both k-tiles) and one for
        // the activation image of its token block; the slot's previous contents must have been
        // consumed (by the MMAs, or by every worker warp whose MMAs are then complete).
        if (elect_one()) {
            int ss = 0;                    // step slot and the parity of its use, kept as counters
            uint32_t ph = 0;
            for (int ti = 0; ti < my_tiles; ++ti) {
                const int tile = (int)blockIdx.x + ti * (int)gridDim.x;
                const int tb = tile % p.tok_blocks, rb = tile / p.tok_blocks * R;
                const uint8_t *src = p.img + (size_t)tb * spt * G::kImgStep;
                const uint8_t *wsrc = p.wimg + (size_t)rb * spt * kWImgStep;
                // the next row block's image; a last tile with one row block copies that one twice
                const size_t wnext = rb + 1 < p.M / kTM ? (size_t)spt * kWImgStep : 0;
                bool ok = true;
                for (int s = 0; s < spt; ++s, src += G::kImgStep, wsrc += kWImgStep) {
                    ok = wait_on(empty0 + ss * 8, ph ^ 1u, kWaitProd);
                    if (!ok) break;
                    const uint32_t fb = full0 + ss * 8;
                    const uint32_t dst = smem_u + ss * G::kSlot;
                    mbar_expect_tx(fb, G::kAStep + kImgCopy);
                    bulk_g2s_plain(dst, wsrc, G::kABlock, fb);
                    if (R == 2) bulk_g2s_plain(dst + G::kABlock, wsrc + wnext, G::kABlock, fb);
                    bulk_g2s_plain(dst + G::kAStep, src, kImgCopy, fb);
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
            const uint64_t desc0 = smem_desc(smem_u);
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
                    // the first MMA of a promote group overwrites the accumulator
#pragma unroll
                    for (int rr = 0; rr < R; ++rr) {
                        const uint32_t acc_t = tmem_base + b * G::kAccCols + rr * G::kRowCols;
                        const uint64_t da = desc0 + (uint64_t)((ss * G::kSlot + rr * G::kABlock + h * kABytes) >> 4);
                        const uint64_t db = desc0 + (uint64_t)((ss * G::kSlot + G::kAStep + h * G::kBTile) >> 4);
                        tc_mma_f8(acc_t, da, db, kIdesc, (GW == 2 && hh == 1) ? 1u : 0u);
                        if (G::kParts == 2) tc_mma_f8(acc_t, da, db + (G::kBPart >> 4), kIdesc, 1u);
                    }
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

// The call's data decide between the two forms (SumsState). A kernel of a narrow tile holds both behind one
// branch: the second launch, which returns at once, takes about 2 us of every call (10240 x 5120, 136 tokens: 69.9 us
// with it, 67.8 without; 1024 x 1024: 17.6 and 15.5). With more than kOneKernel accumulators a thread the
// registers of one form spill for the other's sake (17408 x 5120, 4096 tokens, 64 accumulators: 1687 against
// 1450 us), so there each is a kernel, both are launched and the one not selected returns.
constexpr int kOneKernel = 40;
enum Form { kPlain, kSums, kBothForms };
template <int MODE, int WT, int FORM>
__global__ void __maxnreg__(kLaunchRegs) gemm_w4a8_tc_kernel(const TcParams p) {
    pdl_trigger();
    pdl_wait();      // everything below reads what earlier kernels wrote (words, images)
    const uint4 sw = __ldcg(reinterpret_cast<const uint4 *>(p.sums));      // gen, diff, zp, arrived
    const bool sums = sw.y == sw.x && sw.z == sw.x;
    if (FORM == kBothForms ? sums : FORM == kSums) {
        if (FORM == kSums && !sums) {
            // A CTA that reads the words after this store finds old stamps: not selected either.
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                p.sums->last = 0;
                p.sums->gen = next_generation(sw.x);
            }
            return;
        }
        if constexpr (FORM != kPlain) tc_gemm<MODE, true, FORM != kPlain, WT>(p, sw.x);
    } else {
        if (FORM == kPlain && sums) return;
        if constexpr (FORM != kSums) tc_gemm<MODE, false, FORM == kBothForms, WT>(p, sw.x);
    }
}

struct TcScratch {
    uint8_t *img = nullptr;
    size_t img_bytes = 0;
    uint8_t *wimg = nullptr;      // e4m3 image of the call's weight, with its scales (2.25 bytes per packed byte)
    size_t wimg_bytes = 0;
    SumsState *sums = nullptr;
} g_tc;

int g_tc_sms = 0;

template <int MODE, int WT>
void launch_tile(const TcParams &p, int sms) {
    using G = TcTile<MODE, WT>;
    const int grid = std::min(sms, (p.M / kTM + G::R - 1) / G::R * p.tok_blocks);
    auto go = [&](auto form) {
        constexpr auto kernel = gemm_w4a8_tc_kernel<MODE, WT, decltype(form)::value>;
        static bool once = false;
        if (!once) {
            TQ_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, G::kSmem));
            once = true;
        }
        launch_pdl(kernel, dim3(grid), dim3(kThreads), (size_t)G::kSmem, p);
    };
    if constexpr (G::R * WT <= kOneKernel) {
        go(std::integral_constant<int, kBothForms>{});
    } else {
        go(std::integral_constant<int, kPlain>{});
        go(std::integral_constant<int, kSums>{});
    }
}

template <int MODE>
void launch_width(const TcParams &p, int TN, int sms) {
    if constexpr (TcTile<MODE, 32>::R == 2) {
        switch (TN) {
            case 256: launch_tile<MODE, 64>(p, sms); break;
            case 128: launch_tile<MODE, 32>(p, sms); break;
            case 112: launch_tile<MODE, 28>(p, sms); break;
            case 96: launch_tile<MODE, 24>(p, sms); break;
            case 80: launch_tile<MODE, 20>(p, sms); break;
            case 64: launch_tile<MODE, 16>(p, sms); break;
            case 48: launch_tile<MODE, 12>(p, sms); break;
            default: launch_tile<MODE, 8>(p, sms); break;
        }
    } else {
        switch (TN) {
            case 256: launch_tile<MODE, 64>(p, sms); break;
            case 192: launch_tile<MODE, 48>(p, sms); break;
            default: launch_tile<MODE, 32>(p, sms); break;
        }
    }
}

// Tokens per tile: the width whose rounds of tiles over the SMs cost least, a round counted as
// (tokens + a constant) units. In block mode a round of 148 tiles of 256 rows takes 34 / 44 / 51 / 62 / 69 / 80
// / 92 us at 32 / 48 / 64 / 80 / 96 / 112 / 128 tokens and K 5120 (0.6 us a token and 25 tokens' worth of fixed
// cost; W4A4 0.34 and 30); with per-token scales a round of 128 rows takes 24 / 33 / 40 us at 128 / 192 / 256
// tokens on K64 weights (57) and 44 / 56 / 67 on K32 (108). The rest is how many rounds the tiles of a
// width need: 136 tokens on 10240 rows are one round of 48 (us of the whole call: 67; 64 tokens: 81, 128: 122), 1000 on
// 5120 rows two of 80 (485; 96: 535, 128: 680). With one constant for both scale groups, and one for block mode and W4A4,
// the choice is within 1 % of the fastest width over twelve shapes in all modes. In block and 4-bit mode there is one tile of a single row block too, 256 tokens wide, for calls that it takes
// in one round and pairs do not, an odd number of row blocks most of all (4736 x 5120, 37 of them, 1024 tokens: 114
// against 138 us in two rounds of 80, W4A4 68 against 86). Where both are one round it is the slower one (9472 x 5120, 512
// tokens, 112 us in pairs), hence 256 - 82 units.
int choose_tile_tokens(int M, int T, int sms, bool per_token) {
    const int rows = (per_token ? 1 : 2) * kTM, widest = per_token ? 256 : 128, step = per_token ? 64 : 16;
    int best = 0;
    long best_cost = 0;
    for (int tn = widest; tn >= widest / (per_token ? 2 : 4); tn -= step) {
        const long tiles = (long)((M + rows - 1) / rows) * ((T + tn - 1) / tn);
        const long cost = (tiles + sms - 1) / sms * (tn + (per_token ? 96 : 26));
        if (!best || cost < best_cost) {
            best = tn;
            best_cost = cost;
        }
    }
    if (!per_token) {
        const long tiles = (long)(M / kTM) * ((T + 255) / 256);
        if ((tiles + sms - 1) / sms * (256 - 82) < best_cost) best = 256;
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
    const int TN = choose_tile_tokens(a.M, a.T, g_tc_sms, a.as_tok != nullptr);
    const int tok_blocks = (a.T + TN - 1) / TN, Tpad = tok_blocks * TN;
    const size_t ibytes = (size_t)(Kt / 2) * Tpad * image_step_bytes(a.aq4 != nullptr);
    if (ibytes > g_tc.img_bytes) {
        if (g_tc.img) tq_dev_free(g_tc.img);
        g_tc.img = static_cast<uint8_t *>(tq_dev_alloc(ibytes, "gemm.tc.activation.image"));
        g_tc.img_bytes = ibytes;
    }
    const size_t wbytes = (size_t)(a.M / kTM) * (Kt / 2) * kWImgStep;
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
    // one round of CTAs, shared between the two jobs by their items (an activation item is worth two)
    const size_t witems = (size_t)a.M * Kt, aitems = (size_t)(a.aq4 ? Kt / 2 : Kt) * Tpad;
    const size_t room = (size_t)g_tc_sms * kPreCtas;
    const int ablocks = (int)std::min<size_t>((aitems + 255) / 256,
                                              std::max<size_t>(1, room * 2 * aitems / (2 * aitems + witems)));
    q.wblocks = (int)std::min<size_t>((witems + 255) / 256, std::max<size_t>(1, room - ablocks));
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
    if (a.aq4) launch_width<kInt4>(p, TN, g_tc_sms);
    else if (!a.as_tok) launch_width<kBlock>(p, TN, g_tc_sms);
    else if (a.ksh) launch_width<kToken64>(p, TN, g_tc_sms);
    else launch_width<kToken>(p, TN, g_tc_sms);
    TQ_LAUNCH_CHECK("gemm_w4a8_tc_kernel");
    return 0;
}

int prefill_tile_tokens(int M, int T, int sms, bool per_token) { return choose_tile_tokens(M, T, sms, per_token); }

int prefill_sums_variant() {
    if (!g_tc.sums) return -1;
    unsigned last = 0;
    if (cudaMemcpyAsync(&last, &g_tc.sums->last, sizeof last, cudaMemcpyDeviceToHost, stream()) != cudaSuccess ||
        cudaStreamSynchronize(stream()) != cudaSuccess)
        return -1;
    return (int)last;
}

}  // namespace tq
