// net_u8_tc.cu -- a whole uint8 keyword-spotting network as ONE kernel: a one-channel first layer, depthwise-separable
// blocks (3x3 stride-1 'same' depthwise, then 1x1, 64 channels), global average pool, dense layer.  The layer list of the
// reference's include/small/models/DSCNNTiny.hpp; every requantisation's clamp is its ReLU.
//
// An image's activations (64 channels of at most 128 pixels) never leave shared memory, and all filters of the network stay
// there for the life of a CTA: 85 KB for four blocks, laid out once per set of weights (prepare_kernel) so that a CTA fetches
// them with one bulk copy.  16 warps work in groups of 4 or 8; a group takes one image through all layers, its lanes are
// the tensor memory's lanes and the image's pixels.  A layer is
//     operands in shared memory -> MMAs -> int32 sums in tensor memory -> requantised in registers -> the next layer's operand,
// a chain that a group cannot shorten; the other groups' images fill it.  Two more warps issue the MMAs, each for two groups in
// turn.  What bounds it: of the 9400 cycles an image takes with four groups, the tensor pipe is busy for some 4000
// (20 MMAs of 39 cycles a depthwise layer) and the integer ALU for 4600; the rest is the chain (hand-over 150 cycles,
// 320 from the last MMA to its sums) and groups that meet in the same phase.  With one issuing warp it takes 13100 (21 MMAs take a warp
// 2100 cycles from hand-over to hand-over), with one for every group 11500 (they share the pipe, finish together and then
// requantise together).
// 4096 images of the 49x10 network 223 -> 137 us against five launches of block_u8_tc.cu, one image 38.9 -> 14.4.
//
// The intermediate.  [copy][16-channel block][entry][16 B], three copies displaced by (1 - kw) pixels with the wrapping
// column zeroed, W + 1 zero entries above and below, as in block_u8_tc.cu: tap (kh, kw) of pixel p is entry p + kh * W of
// copy kw.  The middle copy is also the operand of the 1x1 layers (pixel p is entry p + W) and takes the first layer's
// im2col rows: nobody else needs it at the time, and zero entries stay zero.
// Depthwise layers on the tensor core: one MMA covers TWO taps of 16 channels (a tap is a 16-byte chunk of the operand, and the
// distance between the chunks is a field of the descriptor); the filter is two diagonals of 16.  20 MMAs of 16 columns for
// 64 channels, 10 KB of filter; one tap of 32 channels each takes 18 MMAs of 32 columns but 18 KB, and four layers of
// that leave room for two groups instead of four.  An MMA takes as long as its 128 rows of operand take to read (33 cycles).
// Per-channel constants enter as one more MMA: a tile of 127s and 1s times signed digits (block_u8_tc.cu).
#include "tc_common.cuh"

namespace
{
using namespace sb;

constexpr int BM = 128, K = 64, KB = K / CB, TAPS = 9, PAIRS = 5;
constexpr int MAX_BLOCKS = 6, MAX_STAGES = 1 + 2 * MAX_BLOCKS;
constexpr int STEM_BYTES = 4 * K * CB, PW_BYTES = K * K, DW_BYTES = PAIRS * KB * 512, DIGIT_BYTES = 2 * K * CB;
constexpr int WARPS = 16, ISSUERS = 2;
constexpr int IMAGE_BYTES = 8;            // raw image bytes a thread fetches ahead, at most
constexpr int DPITCH = K + 4;             // bytes per row of the dense filter in shared memory
constexpr int SMEM_LIMIT = 224 * 1024;    // beside some 2 KB of static arrays

struct Requant
{
    int lshift, rshift, mult, k_zero;
};
enum { STEM = 0, DW = 1, PW = 2 };
struct NetArgs
{
    int N, H, W, HW, E, stages, groups;
    int H0, W0, Fh, Fw, stride, pad_t, pad_l, pitch, img_bytes; // first layer: raw image, window, padded copy
    Requant q[MAX_STAGES], qp, qd;                               // stages, pool, dense
    int zero_in[MAX_STAGES], zero_pool, Kd, zero_in_d;
    uint32_t signed_in;  // bit s: stage s takes its operand as signed bytes (a zero point of 128), first layer and depthwise only
    // Byte offsets of the filters, the same in the prepared buffer and in shared memory: first layer, depthwise and 1x1 filters, digits of
    // the constants, the constant tile, the dense filter, tables ([stages][K] constants, [Kd] constants of the dense layer, a word
    // with a bit for every stage whose constants the digits do not hold).  The groups' own memory follows.
    uint32_t o_stem, o_dw, o_pw, o_digits, o_ones, o_dense, o_corr, o_dense_c, o_big, o_group, group_bytes;
};
struct Weights
{
    const uint8_t *filt[MAX_STAGES + 1]; // stages, dense
    const int32_t *bias[MAX_STAGES + 1];
};

__device__ __forceinline__ int dp4a_u8_s8(unsigned a, unsigned b, int c)
{
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ int kind_of(int s) { return s == 0 ? STEM : ((s & 1) ? DW : PW); }

// Everything a CTA keeps in shared memory, once per set of weights (one CTA).
__global__ void __launch_bounds__(512) prepare_kernel(const __grid_constant__ NetArgs a, const __grid_constant__ Weights wt, uint8_t *__restrict__ o)
{
    const int tid = threadIdx.x, threads = blockDim.x, blocks = a.stages / 2;
    int *corr = reinterpret_cast<int *>(o + a.o_corr), *big = reinterpret_cast<int *>(o + a.o_big);
    uint8_t *dense = o + a.o_dense;
    for (int i = tid; i < (int)a.o_group / 16; i += threads)
        reinterpret_cast<uint4 *>(o)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    for (int i = tid; i < 2 * BM; i += threads)
        reinterpret_cast<uint4 *>(o + a.o_ones)[i] = make_uint4(0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu, i < BM ? 0x7f7f7f7fu : 0x017f7f7fu);
    // first layer [K/16][1][Fh][Fw][1][16] -> K-major [chunk][n][16 B]: byte kh * 4 + kw of output channel n, signed
    for (int i = tid; i < STEM_BYTES; i += threads)
    {
        const int n = i / CB % K, k = i / (CB * K) * CB + i % CB, kh = k >> 2, kw = k & 3;
        if (kh < a.Fh && kw < a.Fw)
            o[a.o_stem + i] = wt.filt[0][((n / CB * a.Fh + kh) * a.Fw + kw) * CB + n % CB] ^ 0x80;
    }
    for (int b = 0; b < blocks; ++b)
    {
        // depthwise [K/16][3][3][16] -> [pair][16-channel block][chunk][16 n][16 B], diagonal; taps in the order kw * 3 + kh
        for (int i = tid; i < TAPS * K; i += threads)
        {
            const int ch = i % K, t = i / K;
            o[a.o_dw + b * DW_BYTES + ((t >> 1) * KB + ch / CB) * 512 + (t & 1) * 256 + (ch % CB) * 17] =
                wt.filt[2 * b + 1][(ch / CB * TAPS + t % 3 * 3 + t / 3) * CB + ch % CB] ^ 0x80;
        }
        for (int i = tid; i < PW_BYTES; i += threads) // 1x1 [K/16][C/16][16 c][16 k] as they lie in memory, signed
            o[a.o_pw + b * PW_BYTES + i] = wt.filt[2 * b + 2][i] ^ 0x80;
    }
    for (int i = tid; i < a.Kd * K; i += threads) // dense [Kd/16][K/16][16 c][16 k] -> rows [k][c] of signed bytes
        dense[(i / (CB * K) * CB + i % CB) * DPITCH + i / CB % K] = wt.filt[a.stages][i] ^ 0x80;
    __syncthreads();
    for (int i = tid; i < a.stages * K; i += threads)
    {
        const int n = i % K, s = i / K;
        int c = a.q[s].k_zero + (wt.bias[s] ? wt.bias[s][n] : 0);
        if (kind_of(s) == PW && a.zero_in[s] != 0)
        {
            int wsum = 0; // sum over input channels of (w + zero_filt)
            const int8_t *col = reinterpret_cast<const int8_t *>(o + a.o_pw + (s / 2 - 1) * PW_BYTES) + (n / CB) * KB * CB * CB + n % CB;
            for (int j = 0; j < K; ++j)
                wsum += col[j * CB];
            c += a.zero_in[s] * wsum;
        }
        corr[i] = c;
        int rest = c / 127;
        const int last = c - 127 * rest;
        if (rest > 31 * 127 || rest < -31 * 127)
            atomicOr(big, 1 << s);
        for (int e = 0; e < 32; ++e) // 31 digits worth 127 each, one worth 1: K-major [chunk][n][16 B]
        {
            const int d = e == 31 ? last : max(-127, min(127, rest));
            rest -= d;
            o[a.o_digits + s * DIGIT_BYTES + (e >> 4) * K * CB + n * CB + (e & 15)] = (uint8_t)d;
        }
    }
    for (int i = tid; i < a.Kd; i += threads)
    {
        int wsum = 0;
        for (int c = 0; c < K; ++c)
            wsum += (int)(int8_t)dense[i * DPITCH + c];
        reinterpret_cast<int *>(o + a.o_dense_c)[i] = a.qd.k_zero + (wt.bias[a.stages] ? wt.bias[a.stages][i] : 0) + a.zero_in_d * wsum;
    }
}

// 16 sums (constants included) -> 16 bytes, by the common quantiser
__device__ __forceinline__ uint4 requant16(const uint32_t *r, int mult, int bit, int sh1)
{
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
        w[e] = pack4_sat(requant_seeded_raw((int)r[4 * e], mult, 1ll << 30, bit, sh1),
                         requant_seeded_raw((int)r[4 * e + 1], mult, 1ll << 30, bit, sh1),
                         requant_seeded_raw((int)r[4 * e + 2], mult, 1ll << 30, bit, sh1),
                         requant_seeded_raw((int)r[4 * e + 3], mult, 1ll << 30, bit, sh1));
    return make_uint4(w[0], w[1], w[2], w[3]);
}
// The same for any quantiser, and for constants that the digits do not hold.  Out of line, and chosen once per stage: with the
// choice inside the loop over channel blocks, the common path executed 816 instructions per warp and stage, now 585.
__device__ __noinline__ uint4 requant16_any(uint32_t d, const int *corr, const Requant &q)
{
    uint32_t r[16], w[4];
    tmem_ld16(d, r);
    tmem_ld_wait();
#pragma unroll
    for (int e = 0; e < 4; ++e)
    {
        int v[4];
        for (int j = 0; j < 4; ++j)
            v[j] = (int)r[4 * e + j] + (corr ? corr[4 * e + j] : 0);
        w[e] = requant_pack4_general(v[0], v[1], v[2], v[3], q.lshift, q.rshift, q.mult);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// PARTS warps share a lane quarter, each with KB / PARTS of the channel blocks: a group is 4 * PARTS warps.
template <int PARTS>
__global__ void __launch_bounds__((WARPS + ISSUERS) * 32, 1)
net_u8_tc_kernel(const __grid_constant__ NetArgs a, const uint8_t *__restrict__ prepared, const uint8_t *__restrict__ in,
                 uint8_t *__restrict__ out, int *status)
{
    constexpr int GW = 4 * PARTS, GT = GW * 32, CBW = KB / PARTS, MAX_GROUPS = WARPS / GW;
    constexpr int PPARTS = GW / KB; // warps that share the pixels of a channel block in the pool
    extern __shared__ __align__(1024) uint8_t smem[];
    // A group's operand is complete; its sums are: of a depthwise layer the first half of the channels and the second, of another
    // layer all.  A wait by parity cannot tell a phase from the one two further on, so whoever waits on a barrier has to see
    // each of its phases; warps that need the first half alone wait for `half_done` in every depthwise layer and for `rest_done` in none.
    __shared__ __align__(8) uint64_t loaded, ready[MAX_GROUPS], half_done[MAX_GROUPS], rest_done[MAX_GROUPS], done[MAX_GROUPS];
    __shared__ uint32_t tmem_base_s;
    __shared__ int failed[MAX_GROUPS];
    __shared__ int4 quant[MAX_STAGES]; // multiplier, bit, shift, 0: not the common quantiser
    __shared__ int pool_part[MAX_GROUPS][PPARTS][K];
    __shared__ __align__(16) uint8_t pooled[MAX_GROUPS][K];

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31; // (uniform to the compiler too)
    const int workers = a.groups * GT;
    const uint32_t copy_bytes = (uint32_t)(KB * a.E * CB), copy16 = copy_bytes >> 4;
    const uint32_t tmem_cols = a.groups == 1 ? 64 : (a.groups == 2 ? 128 : 256);
    const bool worker = tid < workers;
    const int group = warp / GW, gw = warp % GW, gt = tid % GT;
    const int image = a.H0 * a.W0, step = gridDim.x * a.groups, first = blockIdx.x + gridDim.x * group;

    uint8_t ahead[IMAGE_BYTES]; // the next image
    auto fetch = [&](int n) {
        const uint8_t *src = in + (size_t)n * image;
#pragma unroll
        for (int u = 0; u < IMAGE_BYTES; ++u)
            ahead[u] = (n < a.N && gt + u * GT < image) ? __ldg(src + gt + u * GT) : 0;
    };
    if (warp == a.groups * GW)
    {
        if (lane == 0)
        {
            mbar_init(&loaded, 1);
            for (int g = 0; g < MAX_GROUPS; ++g)
            {
                mbar_init(&ready[g], GW); mbar_init(&half_done[g], 1); mbar_init(&rest_done[g], 1); mbar_init(&done[g], 1);
                failed[g] = 0;
            }
            fence_barrier_init();
            mbar_expect_tx(&loaded, a.o_group);
            tma_load_1d(smem, prepared, a.o_group, &loaded);
        }
        __syncwarp();
        if (lane < a.stages)
        {
            const Requant q = a.q[lane];
            const bool fast = requant_is_fast(q.lshift, q.rshift, q.mult);
            quant[lane] = fast ? make_int4(q.mult, 1 << (q.rshift - 2), q.rshift - 1, 1) : make_int4(0, 0, 0, 0);
        }
        tmem_alloc(&tmem_base_s, tmem_cols);
        tmem_relinquish();
    }
    else if (worker)
    {
        fetch(first);
        for (int i = tid; i < (int)(a.groups * a.group_bytes) / 16; i += workers)
            reinterpret_cast<uint4 *>(smem + a.o_group)[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    fence_proxy_async();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();

    if (!worker)
    {
        // ---------------- issuers: each the MMAs of every other group ----------------
        bool ok = __all_sync(0xffffffffu, mbar_wait(&loaded, 0, status, 71));
        const uint32_t big = __shfl_sync(0xffffffffu, *reinterpret_cast<const uint32_t *>(smem + a.o_big), 0), mem = smem_u32(smem + a.o_group);
        const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_s, 0);
        const uint64_t d_ones = make_smem_desc(smem_u32(smem + a.o_ones), BM * CB, 8 * CB, 0);
        const uint64_t d_digits = make_smem_desc(smem_u32(smem + a.o_digits), K * CB, 8 * CB, 0);
        const uint64_t d_dw = make_smem_desc(smem_u32(smem + a.o_dw), 256, 8 * CB, 0);
        const uint64_t d_pw = make_smem_desc(smem_u32(smem + a.o_pw), 8 * CB, KB * CB * CB, 0);
        const uint64_t d_stem = make_smem_desc(smem_u32(smem + a.o_stem), K * CB, 8 * CB, 0);
        const uint64_t d_mid = make_smem_desc(mem + copy_bytes + (uint32_t)(a.W * CB), (uint32_t)(a.E * CB), 8 * CB, 0);
        uint64_t d_pair[PAIRS]; // block 0 of the operand of a pair of taps
#pragma unroll
        for (int p = 0; p < PAIRS; ++p)
        {
            const int t0 = 2 * p, t1 = 2 * p + 1;
            const uint32_t e0 = (uint32_t)(t0 / 3) * copy16 + (uint32_t)(t0 % 3 * a.W);
            const uint32_t e1 = t1 < TAPS ? (uint32_t)(t1 / 3) * copy16 + (uint32_t)(t1 % 3 * a.W) : e0 + 1; // zero weights
            d_pair[p] = make_smem_desc(mem + e0 * CB, (e1 - e0) * CB, 8 * CB, 0);
        }
        // Its groups in turn; all of them come through the same stages, the last ones with an image less at most.
        const int me = warp - a.groups * GW;
        auto stages_of = [&](int g) { return (a.N - (int)(blockIdx.x + gridDim.x * g) + step - 1) / step * a.stages; };
        const int rounds = stages_of(me);
        uint32_t phase = 0;
        int s = 0;
#pragma unroll 1
        for (int round = 0; round < rounds && ok; ++round, phase ^= 1, s = s + 1 == a.stages ? 0 : s + 1)
#pragma unroll 1
            for (int g = me; g < a.groups; g += ISSUERS)
            {
                if (g != me && round >= stages_of(g))
                    continue;
                const int block = s >> 1;
                const uint32_t seeded = ((big >> s) & 1u) ^ 1u, sgn = (a.signed_in >> s) & 1u, d0 = tmem + (uint32_t)(g * K);
                const uint64_t at = (uint64_t)((uint32_t)g * (a.group_bytes >> 4));
                ok = __all_sync(0xffffffffu, mbar_wait(&ready[g], phase, status, 74));
                if (!ok)
                    break;
                tc_fence_after_sync();
                if (elect_one())
                {
                    if (seeded)
                        tc_mma_i8(d0, d_ones, d_digits + (uint64_t)(s * (DIGIT_BYTES >> 4)), make_idesc(2, 0, 1, 0, 0, BM, K), 0u);
                    if (s & 1)
                    {
                        const uint32_t idesc = make_idesc(2, 0, 1, 0, 0, BM, CB) | (sgn << 7);
                        const uint64_t b = d_dw + (uint64_t)(block * (DW_BYTES >> 4));
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                        {
#pragma unroll
                            for (int p = 0; p < PAIRS; ++p)
#pragma unroll
                                for (int cb = h * KB / 2; cb < (h + 1) * KB / 2; ++cb)
                                    tc_mma_i8(d0 + (uint32_t)(cb * CB), d_pair[p] + at + (uint64_t)(cb * a.E), b + (uint64_t)((p * KB + cb) * 32),
                                              idesc, p == 0 ? seeded : 1u);
                            // the epilogue of the first half runs under the MMAs of the second
                            tc_commit(h == 0 ? &half_done[g] : &rest_done[g]);
                        }
                    }
                    else
                    {
                        const bool stem = s == 0;
                        const uint32_t idesc = make_idesc(2, 0, 1, 0, stem ? 0u : 1u, BM, K) | (sgn << 7);
                        const uint64_t b = stem ? d_stem : d_pw + (uint64_t)((block - 1) * (PW_BYTES >> 4));
                        const uint32_t b_step = stem ? (uint32_t)(2 * K) : (uint32_t)(2 * CB);
                        tc_mma_i8(d0, d_mid + at, b, idesc, seeded); // 32 bytes of the reduction each
                        if (!stem || a.Fh > 8)
                            tc_mma_i8(d0, d_mid + at + (uint64_t)(2 * a.E), b + (uint64_t)b_step, idesc, 1u);
                        tc_commit(&done[g]);
                    }
                }
                __syncwarp();
            }
    }
    else
    {
        const int quarter = gw & 3, part = gw >> 2, cb0 = part * CBW;
        const int q = quarter * 32 + lane, oh = q / a.W, ow = q - oh * a.W; // this thread's pixel = tensor-memory lane
        const bool live = q < a.HW, to_left = live && ow != a.W - 1, to_right = live && ow != 0;
        const uint32_t d = tmem_base_s + (uint32_t)(group * K) + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(cb0 * CB);
        uint8_t *sP = smem + a.o_group + group * a.group_bytes, *sI = sP + 3 * copy_bytes;
        uint8_t *mid = sP + copy_bytes + (size_t)(q + a.W) * CB; // this pixel in block 0 of the middle copy
        const uint8_t *sDense = smem + a.o_dense;
        auto sync_group = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(GT) : "memory"); };
        const uint8_t in_xor = (a.signed_in & 1u) ? 0x80 : 0;
        auto store_image = [&]() {
#pragma unroll
            for (int u = 0; u < IMAGE_BYTES; ++u)
            {
                const int i = gt + u * GT;
                if (i < image)
                {
                    const int h = i / a.W0, w = i - h * a.W0;
                    sI[(h + a.pad_t) * a.pitch + (w + a.pad_l)] = ahead[u] ^ in_xor;
                }
            }
        };
        uint32_t phase = 0, dw_phase = 0; // of `done`; of `half_done` and `rest_done`
        bool ok = mbar_wait(&loaded, 0, status, 71);
        const uint32_t big = *reinterpret_cast<const uint32_t *>(smem + a.o_big);
        if (first < a.N)
        {
            store_image();
            sync_group();
        }
        for (int n = first; n < a.N; n += step)
        {
            // im2col of the first layer: row q, chunk j of 4 window rows
            if (live)
                for (int j = part; j * 4 < a.Fh; j += PARTS)
                {
                    const uint8_t *row = sI + (oh * a.stride + j * 4) * a.pitch + ow * a.stride;
                    unsigned wv[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if (j * 4 + t < a.Fh)
                        {
                            const uint8_t *pw = row + t * a.pitch;
                            const unsigned *al = reinterpret_cast<const unsigned *>(pw - ((size_t)pw & 3));
                            wv[t] = __funnelshift_r(al[0], al[1], 8 * (unsigned)((size_t)pw & 3));
                        }
                    *reinterpret_cast<uint4 *>(mid + (size_t)j * a.E * CB) = make_uint4(wv[0], wv[1], wv[2], wv[3]);
                }
#pragma unroll 1
            for (int s = 0; s < a.stages && ok; ++s)
            {
                fence_proxy_async();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(&ready[group]);
                if (s == 0)
                    fetch(n + step);
                const int4 rq = quant[s];
                const bool dw = s & 1, three = !dw && s + 1 < a.stages;
                const uint32_t sx = ((a.signed_in >> 1) >> s) & 1u ? 0x80808080u : 0u; // the next stage's operand
                auto put = [&](int cb, uint4 o) {
                    if (sx)
                    {
                        o.x ^= sx; o.y ^= sx; o.z ^= sx; o.w ^= sx;
                    }
                    uint8_t *p1 = mid + (size_t)cb * a.E * CB;
                    if (live)
                        *reinterpret_cast<uint4 *>(p1) = o;
                    // The depthwise layers' operand has three copies; the 1x1 layers and the pool read the middle one.  A
                    // copy's entry for a pixel that would wrap is zero from the start.
                    if (three && to_left)
                        *reinterpret_cast<uint4 *>(p1 - copy_bytes + CB) = o; // copy kw = 0, entry q + W + 1
                    if (three && to_right)
                        *reinterpret_cast<uint4 *>(p1 + copy_bytes - CB) = o; // copy kw = 2, entry q + W - 1
                };
                // its channels' sums: a depthwise layer's first half, second half or (a group of four warps) both in turn.  (One wait on
                // a barrier chosen beforehand: 4096 images 139.5 us.)
                const bool late = PARTS > 1 && cb0 * 2 >= KB;
                ok = !dw ? mbar_wait(&done[group], phase, status, 73)
                         : late ? mbar_wait(&rest_done[group], dw_phase, status, 75) : mbar_wait(&half_done[group], dw_phase, status, 72);
                tc_fence_after_sync();
                if (rq.w && !((big >> s) & 1u))
                {
                    uint32_t r[2][16];
                    tmem_ld16(d, r[0]);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < CBW; ++i)
                    {
                        if (i + 1 < CBW)
                        {
                            if (PARTS == 1 && i + 1 == KB / 2 && dw)
                            {
                                ok = mbar_wait(&rest_done[group], dw_phase, status, 75) && ok;
                                tc_fence_after_sync();
                            }
                            tmem_ld16(d + (uint32_t)((i + 1) * CB), r[(i + 1) & 1]);
                        }
                        put(cb0 + i, requant16(r[i & 1], rq.x, rq.y, rq.z));
                        if (i + 1 < CBW)
                            tmem_ld_wait();
                    }
                }
                else
                {
                    if (PARTS == 1 && dw)
                    {
                        ok = mbar_wait(&rest_done[group], dw_phase, status, 75) && ok;
                        tc_fence_after_sync();
                    }
#pragma unroll 1
                    for (int i = 0; i < CBW; ++i)
                        put(cb0 + i, requant16_any(d + (uint32_t)(i * CB),
                                                   ((big >> s) & 1u) ? reinterpret_cast<const int *>(smem + a.o_corr) + s * K + (cb0 + i) * CB : nullptr, a.q[s]));
                }
                phase ^= !dw;
                dw_phase ^= dw;
                if (s == 0)
                    store_image(); // everybody's im2col of this image is done
            }
            // a warp that gave up says so; the others' waits run out too (it did not arrive), and the group leaves together
            if (!ok)
                *reinterpret_cast<volatile int *>(&failed[group]) = 1;
            sync_group();
            if (*reinterpret_cast<volatile int *>(&failed[group]))
                break;
            {
                // A warp sums a channel block over every PPARTS-th group of eight pixels; a lane owns four channels of every
                // eighth of those.
                const int cbp = gw % KB, ppart = gw / KB, quad = lane & 3, pg = lane >> 2;
                unsigned s4[4] = {0u, 0u, 0u, 0u};
                const uint8_t *col = sP + copy_bytes + ((size_t)cbp * a.E + a.W) * CB + quad * 4;
                for (int px = ppart * 8 + pg; px < a.HW; px += PPARTS * 8)
                {
                    const unsigned wv = *reinterpret_cast<const unsigned *>(col + (size_t)px * CB);
                    s4[0] = __dp4a(wv, 0x00000001u, s4[0]);
                    s4[1] = __dp4a(wv, 0x00000100u, s4[1]);
                    s4[2] = __dp4a(wv, 0x00010000u, s4[2]);
                    s4[3] = __dp4a(wv, 0x01000000u, s4[3]);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int m = 16; m >= 4; m >>= 1)
                        s4[e] += __shfl_xor_sync(0xffffffffu, s4[e], m);
                if (lane < 4)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        pool_part[group][ppart][cbp * CB + quad * 4 + e] = (int)s4[e];
            }
            sync_group();
            if (gt < K)
            {
                int v = a.qp.k_zero + a.HW * a.zero_pool;
#pragma unroll
                for (int pp = 0; pp < PPARTS; ++pp)
                    v += pool_part[group][pp][gt];
                pooled[group][gt] = (uint8_t)requant_dev(v, a.qp.lshift, a.qp.rshift, a.qp.mult);
            }
            sync_group();
            if (gt < a.Kd)
            {
                int acc = reinterpret_cast<const int *>(smem + a.o_dense_c)[gt];
                const unsigned *wrow = reinterpret_cast<const unsigned *>(sDense + gt * DPITCH);
                const unsigned *pv = reinterpret_cast<const unsigned *>(pooled[group]);
#pragma unroll
                for (int c4 = 0; c4 < K / 4; ++c4)
                    acc = dp4a_u8_s8(pv[c4], wrow[c4], acc);
                out[(size_t)n * a.Kd + gt] = (uint8_t)requant_dev(acc, a.qd.lshift, a.qd.rshift, a.qd.mult);
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == a.groups * GW)
        tmem_dealloc(tmem_base_s, tmem_cols);
}

bool quant_ok(const small_b200_layer &L)
{
    return L.lshift >= 0 && L.lshift < 32 && L.rshift >= 0 && L.rshift < 32 && row_stride(&L) == L.stride && !L.accumulate;
}
bool no_pads(const small_b200_layer &L) { return !L.pad_t && !L.pad_b && !L.pad_l && !L.pad_r; }
Requant quant(const small_b200_layer &L) { return Requant{L.lshift, L.rshift, L.multiplier, L.k_zero}; }

// The layer list [first, (depthwise, 1x1) * b, average pool, dense]; false when it is not covered.
bool plan(const small_b200_layer *L, int n, NetArgs &a)
{
    if (!L || n < 5 || n % 2 == 0 || (n - 3) / 2 > MAX_BLOCKS)
        return false;
    a = NetArgs{};
    const small_b200_layer &c = L[0];
    // (images are counted in 32 bits, with a round of the CTAs' groups on top)
    if (c.N < 0 || c.N > 0x7fff0000 || c.H < 1 || c.W < 1 || c.C != 1 || c.K != K || c.zero_filt != -128 || (c.zero_in != 0 && c.zero_in != -128) || !quant_ok(c) || c.Fh < 1 ||
        c.Fh > 16 || c.Fw < 1 || c.Fw > 4 || c.stride < 1 || c.pad_t < 0 || c.pad_b < 0 || c.pad_l < 0 || c.pad_r < 0)
        return false;
    const long long tall = (long long)c.H + c.pad_t + c.pad_b, wide = (long long)c.W + c.pad_l + c.pad_r; // the padded image
    if ((long long)c.H * c.W > IMAGE_BYTES * 128 || tall > SMEM_LIMIT || wide > SMEM_LIMIT || tall * wide > SMEM_LIMIT)
        return false;
    a.N = c.N;
    a.H = out_dim(c.H, c.pad_t, c.pad_b, c.Fh, c.stride);
    a.W = out_dim(c.W, c.pad_l, c.pad_r, c.Fw, c.stride);
    a.HW = a.H * a.W;
    if (a.H <= 0 || a.W <= 0 || a.HW > BM)
        return false;
    a.H0 = c.H; a.W0 = c.W; a.Fh = c.Fh; a.Fw = c.Fw; a.stride = c.stride; a.pad_t = c.pad_t; a.pad_l = c.pad_l;
    a.pitch = (((int)wide + 12) + 3) & ~3; // room for the unaligned window read
    a.img_bytes = (((int)tall + 1) * a.pitch + 127) & ~127;
    a.E = (BM + 2 * a.W + 7) & ~7;
    a.q[0] = quant(c); a.zero_in[0] = c.zero_in;
    a.signed_in = c.zero_in != 0;
    const int blocks = (n - 3) / 2;
    a.stages = 1 + 2 * blocks;
    for (int s = 1; s < a.stages; ++s)
    {
        const small_b200_layer &l = L[s];
        const bool dw = s & 1;
        const int f = dw ? 3 : 1, p = dw ? 1 : 0;
        if (l.N != a.N || l.C != K || l.K != K || l.H != a.H || l.W != a.W || l.Fh != f || l.Fw != f || l.stride != 1 || l.pad_t != p ||
            l.pad_b != p || l.pad_l != p || l.pad_r != p || l.zero_filt != -128 || !quant_ok(l) ||
            (dw && l.zero_in != 0 && l.zero_in != -128))
            return false;
        a.q[s] = quant(l); a.zero_in[s] = l.zero_in;
        if (dw && l.zero_in != 0)
            a.signed_in |= 1u << s;
    }
    const small_b200_layer &pl = L[n - 2], &dn = L[n - 1];
    if (pl.N != a.N || pl.C != K || pl.H != a.H || pl.W != a.W || pl.Fh != a.H || pl.Fw != a.W || pl.stride < 1 || pl.stride > 3 ||
        !no_pads(pl) || !quant_ok(pl))
        return false;
    if (dn.N != a.N || dn.C != K || dn.H != 1 || dn.W != 1 || dn.Fh != 1 || dn.Fw != 1 || dn.stride != 1 || !no_pads(dn) ||
        dn.K <= 0 || dn.K % CB != 0 || dn.K > 128 || !quant_ok(dn) || dn.zero_filt != -128)
        return false;
    a.qp = quant(pl); a.zero_pool = pl.zero_in;
    a.qd = quant(dn); a.Kd = dn.K; a.zero_in_d = dn.zero_in;
    uint32_t o = 0;
    auto take = [&](uint32_t bytes) { const uint32_t at = o; o += (bytes + 127) & ~127u; return at; };
    a.o_stem = take(STEM_BYTES);
    a.o_dw = take(blocks * DW_BYTES);
    a.o_pw = take(blocks * PW_BYTES);
    a.o_digits = take(a.stages * DIGIT_BYTES);
    a.o_ones = take(2 * BM * CB);
    a.o_dense = take(a.Kd * DPITCH);
    a.o_corr = take(a.stages * K * 4);
    a.o_dense_c = take(a.Kd * 4);
    a.o_big = take(4);
    a.o_group = o;
    a.group_bytes = 3 * KB * a.E * CB + a.img_bytes;
    return a.o_group + a.group_bytes <= SMEM_LIMIT;
}

template <int PARTS>
int launch(NetArgs a, const uint8_t *prepared, const uint8_t *in, uint8_t *out, cudaStream_t st)
{
    auto kern = net_u8_tc_kernel<PARTS>;
    static PerDeviceOnce configured;
    int dev;
    if (configured.needed(&dev))
    {
        SB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT));
        configured.mark(dev);
    }
    int *status = device_status_ptr();
    if (!status)
        return fail(SMALL_B200_CUDA_ERROR, "device status word not available");
    a.groups = WARPS / (4 * PARTS);
    const int room = (int)((SMEM_LIMIT - a.o_group) / a.group_bytes);
    if (a.groups > room)
        a.groups = room;
    const int grid = a.N < num_sms() ? a.N : num_sms();
    kern<<<grid, a.groups * PARTS * 128 + ISSUERS * 32, a.o_group + a.groups * a.group_bytes, st>>>(a, prepared, in, out, status);
    return launched("net_u8_tc_kernel");
}
const char *NOT_COVERED = "separable network<quint8> ERROR: this list of layers is not covered by the one-kernel form; call the "
                          "layers separately.";
} // namespace

extern "C"
{
int small_b200_separable_network_u8_supported(const small_b200_layer *layers, int32_t n)
{
    NetArgs a;
    return plan(layers, n, a) ? 1 : 0;
}

size_t small_b200_separable_network_u8_prepared_bytes(const small_b200_layer *layers, int32_t n)
{
    NetArgs a;
    return plan(layers, n, a) ? a.o_group : 0;
}

int small_b200_separable_network_u8_prepare(const small_b200_layer *layers, int32_t n, const uint8_t *const *filts,
                                            const int32_t *const *biases, void *prepared, void *stream)
{
    NetArgs a;
    if (!plan(layers, n, a))
        return fail(SMALL_B200_INVALID_ARGUMENT, NOT_COVERED);
    if (reinterpret_cast<uintptr_t>(prepared) & 15)
        return fail(SMALL_B200_INVALID_ARGUMENT, "separable network<quint8> ERROR: the prepared buffer must be 16-byte aligned.");
    Weights w{};
    for (int s = 0; s <= a.stages; ++s)
    {
        const int i = s < a.stages ? s : n - 1;
        w.filt[s] = filts[i];
        w.bias[s] = biases ? biases[i] : nullptr;
    }
    prepare_kernel<<<1, 512, 0, as_stream(stream)>>>(a, w, static_cast<uint8_t *>(prepared));
    return launched("prepare_kernel");
}

int small_b200_separable_network_u8(const small_b200_layer *layers, int32_t n, const void *prepared, const uint8_t *in, uint8_t *out,
                                    void *stream)
{
    NetArgs a;
    if (!plan(layers, n, a))
        return fail(SMALL_B200_INVALID_ARGUMENT, NOT_COVERED);
    if (a.N == 0)
        return SMALL_B200_OK;
    if (reinterpret_cast<uintptr_t>(prepared) & 15)
        return fail(SMALL_B200_INVALID_ARGUMENT, "separable network<quint8> ERROR: the prepared buffer must be 16-byte aligned.");
    const uint8_t *p = static_cast<const uint8_t *>(prepared);
    // Groups of eight warps up to two images per SM, of four beyond: 148 images 14.4 and 16.5 us, 200 19.7 and 20.5,
    // 400 28.8 and 22.6 (groups of sixteen 14.4, 24.6, 32.8).
    if (a.N <= 2 * num_sms())
        return launch<2>(a, p, in, out, as_stream(stream));
    return launch<1>(a, p, in, out, as_stream(stream));
}
} // extern "C"
