// conv_u8_rgb.cu -- small::Conv2D<QUInt8Buffer> (include/small/interface_abstract.hpp:229-404, loop nest
// include/small/q_abstract_layer.hpp:894-1571) of the first layer on THREE-channel images, as an implicit GEMM on tcgen05.mma.kind::i8.
//
// Implicit GEMM.  A GEMM row is G = 4 / stride outputs side by side: their windows begin within four pixels and end within eight.
// Shared memory holds the input as chunks of four pixels of four bytes (the fourth meets rows of zeros of the filter), [row % stride][row / stride][chunk], so
// chunk m and the next one are the 32 bytes of a reduction step for GEMM row m = r * PW + c, and a kernel row only moves the start:
// one MMA per kernel row, G * 16 columns per 16 output channels.  The operand's 16-byte columns overlap, the distance between them is one row.
// Zero points as in conv_u8_patch.cu: sixteen more columns, the first G of which have ones at their output's window, give the sums of the
// bytes; a pixel outside the image holds the byte -zi.
//
// Roles: 16 epilogue warps (sets of four, an accumulator each), 12 producer warps (a tile each, from global memory through registers and a
// table of the patch's chunks), 2 issuing warps (tiles in turn: what one spends on a tile's MMAs and waits is 600 cycles and more).
//
// What bounds it: instructions.  A tile of 256 outputs of 16 channels takes 2000 warp instructions (five and a half per 32
// results, half of them on the half-rate integer pipe, some 35 a chunk of four pixels), at 57 % of the issue slots and 39 % of the ALU (512
// images of 96x96); its three MMAs take 132 cycles.  The CUDA cores' form
// has seven dp4a and the gather of the window beside the same requantisation.  us, that form -> this: 3 -> 16
// channels at 96x96 with a stride of two, 2048 images 98.8 -> 53.4 (19 at the rate of a copy of its bytes), 3 -> 32 149.7 -> 82;
// at 32x32, stride 1, 4096 images 84 -> 48; at 416x416, 16 images 53 -> 25.7.  On the way: one issuing warp in a rolled loop 76 (1150
// cycles a tile whatever its work), rows and columns from divisions instead of the table 66.
#include "tc_common.cuh"

#include <algorithm>
#include <type_traits>

namespace
{
using namespace sb;

constexpr int BM = 128, C3 = 3, SETS = 4, EPI_WARPS = 4 * SETS, PROD_WARPS = 12, STAGES = PROD_WARPS, ISSUERS = 2;
constexpr int THREADS = (EPI_WARPS + PROD_WARPS + ISSUERS) * 32;
static_assert(SETS % ISSUERS == 0 && STAGES % ISSUERS == 0, "who waits on a stage or an accumulator sees all of its phases");
constexpr int MAX_ROWS = 10; // of a window
constexpr int SMEM_LIMIT = 200 * 1024;
// Outputs from which on this kernel is the faster one.  us, the CUDA cores' form -> this, 96x96 images, a stride of two, 16 channels: 64 images
// (147 456 outputs) 6.1 -> 6.9, 256 images 15.5 -> 10.8; 16 images of 224x224 (200 704) 7.3 -> 7.2.
constexpr long long RGB_MIN = 200000;

struct RgbArgs
{
    int N, H, W, K, Ho, Wo, Fh, Fw, stride, pad_t, pad_l;
    int TH, TW, PW;           // output rows and chunks of a tile, chunks a row of its patch
    int rows_in, units;       // input rows of a patch, its chunks
    int tiles_x, tiles_y, tiles;
    int E;                    // entries of a plane of rows
    uint32_t stage_bytes, o_filter, o_table, smem;
    uint32_t outside;         // the byte of a tap outside the image, four times
    long long in_bytes;
    int zero_in, zero_filt, lshift, rshift, mult, k_zero;
    FastDiv by_tiles_x, by_tiles_y, by_PW;
};

// four outputs' bytes by any quantiser
__device__ __forceinline__ uint32_t quantise4(bool fast, int a, int b, int c, int d, const RgbArgs &p, int bit, int sh1)
{
    if (!fast)
        return requant_pack4_general(a, b, c, d, p.lshift, p.rshift, p.mult);
    return pack4_sat(requant_seeded_raw(a, p.mult, 1ll << 30, bit, sh1), requant_seeded_raw(b, p.mult, 1ll << 30, bit, sh1),
                     requant_seeded_raw(c, p.mult, 1ll << 30, bit, sh1), requant_seeded_raw(d, p.mult, 1ll << 30, bit, sh1));
}

__device__ __forceinline__ uint64_t desc_of(uint32_t low, uint32_t high)
{
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(low), "r"(high));
    return d;
}

// G outputs a GEMM row, KB blocks of 16 output channels a CTA; THREE: windows of three rows.
template <int G, int KB, bool THREE>
__global__ void __launch_bounds__(THREADS, 1)
conv_u8_rgb_kernel(const __grid_constant__ RgbArgs a, const uint8_t *__restrict__ in, const uint8_t *__restrict__ filt,
                   const int32_t *__restrict__ bias, uint8_t *__restrict__ out, int *status)
{
    constexpr int UNITS = G * KB, NCOLS = UNITS * 16 + 16;
    constexpr uint32_t TMEM_COLS = SETS * NCOLS <= 256 ? 256 : 512;
    static_assert(SETS * NCOLS <= 512, "");
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], acc_full[SETS], acc_empty[SETS];
    __shared__ uint32_t tmem_base_s;
    __shared__ __align__(16) int seed[KB * CB];

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int kb0 = blockIdx.y * KB, kbs = a.K / CB, R = a.Fh * a.Fw * C3;
    const int my_tiles = (a.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;

    // The filter: [kernel row][16-byte half][column][16 B], and the channels' constants.
    for (int i = tid; i < a.Fh * 2 * NCOLS * 4; i += THREADS)
    {
        const int px4 = i & 3, col = (i >> 2) % NCOLS, hk = (i >> 2) / NCOLS, kh = hk >> 1;
        const int unit = col / CB, g = unit < UNITS ? unit % G : col - UNITS * CB, kw = (hk & 1) * 4 + px4 - g * a.stride;
        uint32_t v = 0;
        if (g < G && kw >= 0 && kw < a.Fw)
        {
            v = 0x00010101u;
            if (unit < UNITS)
            {
                const uint8_t *w = filt + ((size_t)(kb0 + unit / G) * R + (size_t)(kh * a.Fw + kw) * C3) * CB + col % CB;
                v = (uint32_t)w[0] | (uint32_t)w[CB] << 8 | (uint32_t)w[2 * CB] << 16;
            }
        }
        reinterpret_cast<uint32_t *>(smem + a.o_filter)[i] = v;
    }
    if (tid < KB * CB)
    {
        const int k = kb0 * CB + tid;
        const uint8_t *w = filt + (size_t)(k / CB) * R * CB + k % CB;
        int sum = 0;
        for (int i = 0; i < R; ++i)
            sum += w[i * CB];
        seed[tid] = a.k_zero + (bias ? bias[k] : 0) + a.zero_in * sum + R * a.zero_in * a.zero_filt;
    }
    // A patch's chunks: where they go, how far from the first one they lie, row, column.
    uint4 *table = reinterpret_cast<uint4 *>(smem + a.o_table);
    for (int i = tid; i < a.units; i += THREADS)
    {
        const int r = a.by_PW.div(i), c = i - r * a.PW, sh = a.stride - 1; // (a stride of one or two)
        table[i] = make_uint4((uint32_t)(((r & sh) * a.E + (r >> sh) * a.PW + c) * 16), (uint32_t)((r * a.W + 4 * c) * C3), (uint32_t)r, (uint32_t)(4 * c));
    }
    fence_proxy_async();
    if (warp == EPI_WARPS + PROD_WARPS)
    {
        if (lane == 0)
        {
            for (int i = 0; i < STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
            for (int i = 0; i < SETS; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 4); }
            fence_barrier_init();
        }
        __syncwarp();
        tmem_alloc(&tmem_base_s, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_s, 0);

    // image, first output row and chunk of a tile
    auto decode = [&](int tile, int &n, int &r0, int &c0) {
        const int t1 = a.by_tiles_x.div(tile);
        n = a.by_tiles_y.div(t1); r0 = (t1 - n * a.tiles_y) * a.TH; c0 = (tile - t1 * a.tiles_x) * a.TW;
    };
    if (warp < EPI_WARPS)
    {
        // ---------------- epilogue: thread = GEMM row; set s takes tiles s, s + SETS, ...
        const int set = warp >> 2, quarter = warp & 3, m = quarter * 32 + lane;
        const int rl = a.by_PW.div(m), cl = m - rl * a.PW;
        const bool fast = requant_is_fast(a.lshift, a.rshift, a.mult), mine = cl < a.TW && rl < a.TH;
        const int bit = 1 << ((a.rshift - 2) & 31), sh1 = a.rshift - 1;
        const size_t plane = (size_t)a.Ho * a.Wo * CB;
        // two outputs side by side are one 32-byte store where every row begins at one
        const bool pairs = (a.Wo & 1) == 0 && (reinterpret_cast<uintptr_t>(out) & 31) == 0;
        const uint32_t d = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(set * NCOLS);
        bool ok = true;
        uint32_t turn = 0;
        auto tiles = [&](auto is_fast) {
#pragma unroll 1
            for (int i = set; i < my_tiles; i += SETS, turn ^= 1)
            {
                int n, r0, c0;
                decode(blockIdx.x + i * gridDim.x, n, r0, c0);
                const int oh = r0 + rl, ow = (c0 + cl) * G;
                const int live = mine && oh < a.Ho ? a.Wo - ow : 0; // outputs of this thread
                uint8_t *o = out + ((size_t)n * kbs + kb0) * plane + ((size_t)oh * a.Wo + ow) * CB;
                ok = mbar_wait(&acc_full[set], turn, status, 81);
                if (!ok)
                    break;
                tc_fence_after_sync();
                uint32_t sums[16];
                tmem_ld16(d + UNITS * 16, sums);
#pragma unroll
                for (int kb = 0; kb < KB; ++kb)
#pragma unroll
                    for (int g = 0; g < G; g += 2)
                    {
                        uint32_t x[2][16], w[8];
                        tmem_ld16(d + (uint32_t)((kb * G + g) * 16), x[0]);
                        tmem_ld16(d + (uint32_t)((kb * G + g + 1) * 16), x[1]);
                        tmem_ld_wait();
                        if (kb == KB - 1 && g == G - 2) // read
                        {
                            tc_fence_before_sync();
                            __syncwarp();
                            if (lane == 0)
                                mbar_arrive(&acc_empty[set]);
                        }
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                        {
                            const int4 s = reinterpret_cast<const int4 *>(seed + kb * CB)[e];
#pragma unroll
                            for (int h = 0; h < 2; ++h)
                            {
                                const int base = a.zero_filt * (int)sums[g + h];
                                w[4 * h + e] = quantise4(decltype(is_fast)::value, (int)x[h][4 * e] + s.x + base, (int)x[h][4 * e + 1] + s.y + base,
                                                         (int)x[h][4 * e + 2] + s.z + base, (int)x[h][4 * e + 3] + s.w + base, a, bit, sh1);
                            }
                        }
                        uint8_t *og = o + (size_t)kb * plane + g * CB;
                        if (pairs)
                        {
                            if (live > g)
                                asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(og), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                                             "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                                             : "memory");
                        }
                        else
                        {
                            if (live > g)
                                *reinterpret_cast<uint4 *>(og) = make_uint4(w[0], w[1], w[2], w[3]);
                            if (live > g + 1)
                                *reinterpret_cast<uint4 *>(og + CB) = make_uint4(w[4], w[5], w[6], w[7]);
                        }
                    }
            }
        };
        if (fast)
            tiles(std::true_type{});
        else
            tiles(std::false_type{});
    }
    else if (warp < EPI_WARPS + PROD_WARPS)
    {
        // ---------------- producers: a warp a tile, which has a stage of its own
        const int w = warp - EPI_WARPS;
        uint8_t *stage = smem + w * a.stage_bytes;
        const uintptr_t first = reinterpret_cast<uintptr_t>(in), last = first + (uintptr_t)a.in_bytes;
        const uint4 outside = make_uint4(a.outside, a.outside, a.outside, a.outside);
        bool ok = true;
        uint32_t used = 1; // parity of the stage's last release; the first round finds it free
        for (int i = w; i < my_tiles; i += PROD_WARPS, used ^= 1)
        {
            int n, r0, c0;
            decode(blockIdx.x + i * gridDim.x, n, r0, c0);
            const int ih0 = r0 * a.stride - a.pad_t, iw0 = c0 * 4 - a.pad_l;
            // (the address may lie before the buffer: it is only used where it does not)
            const uintptr_t image = first + (uintptr_t)((long long)n * a.H * a.W * C3);
            const uintptr_t src = image + (uintptr_t)(((long long)ih0 * a.W + iw0) * C3);
            // all words that hold bytes of the patch's chunks lie in the buffer
            const bool words = image + (uintptr_t)(((long long)max(ih0, 0) * a.W + iw0 - 1) * C3) >= first &&
                               image + (uintptr_t)(((long long)min(ih0 + a.rows_in, a.H) * a.W + 4 + 1) * C3) <= last;
            if (i >= PROD_WARPS)
                ok = __all_sync(0xffffffffu, mbar_wait(&empty[w], used, status, 82));
            if (!ok)
                break;
            if (words)
            {
                constexpr int U = 3; // chunks of a lane under way at once
                for (int u0 = lane; u0 < a.units; u0 += 32 * U)
                {
                    uint32_t p[U][4];
                    uint4 t[U];
                    int shift[U];
#pragma unroll
                    for (int v = 0; v < U; ++v)
                    {
                        t[v] = table[min(u0 + v * 32, a.units - 1)];
                        const int ih = ih0 + (int)t[v].z, iw = iw0 + (int)t[v].w;
                        const uintptr_t at = src + t[v].y;
                        const uint32_t *q = reinterpret_cast<const uint32_t *>(at & ~(uintptr_t)3);
                        shift[v] = (int)(at & 3) * 8;
                        t[v].z = (unsigned)ih < (unsigned)a.H && iw > -4 && iw < a.W;
                        t[v].w = (uint32_t)iw;
                        if (t[v].z)
                        {
                            p[v][0] = __ldg(q); p[v][1] = __ldg(q + 1); p[v][2] = __ldg(q + 2);
                            p[v][3] = shift[v] ? __ldg(q + 3) : 0u;
                        }
                    }
#pragma unroll
                    for (int v = 0; v < U; ++v)
                    {
                        uint4 x = outside;
                        if (t[v].z) // three words, of which pixels: their fourth bytes are the next one's first
                        {
                            const uint32_t w0 = __funnelshift_r(p[v][0], p[v][1], shift[v]), w1 = __funnelshift_r(p[v][1], p[v][2], shift[v]),
                                           w2 = __funnelshift_r(p[v][2], p[v][3], shift[v]);
                            x = make_uint4(w0, __funnelshift_r(w0, w1, 24), __funnelshift_r(w1, w2, 16), w2 >> 8);
                            const int iw = (int)t[v].w;
                            if (iw < 0 || iw + 4 > a.W)
                            {
                                x.x = (unsigned)iw < (unsigned)a.W ? x.x : a.outside;
                                x.y = (unsigned)(iw + 1) < (unsigned)a.W ? x.y : a.outside;
                                x.z = (unsigned)(iw + 2) < (unsigned)a.W ? x.z : a.outside;
                                x.w = (unsigned)(iw + 3) < (unsigned)a.W ? x.w : a.outside;
                            }
                        }
                        *reinterpret_cast<uint4 *>(stage + t[v].x) = x; // (the last chunk's by several lanes: the same bytes)
                    }
                }
            }
            else // at an end of the buffer: bytes
                for (int u = lane; u < a.units; u += 32)
                {
                    const uint4 t = table[u];
                    const int ih = ih0 + (int)t.z, iw = iw0 + (int)t.w;
                    uint32_t x[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                    {
                        x[j] = a.outside;
                        if ((unsigned)ih < (unsigned)a.H && (unsigned)(iw + j) < (unsigned)a.W)
                        {
                            const uint8_t *q = reinterpret_cast<const uint8_t *>(src + t.y) + j * C3;
                            x[j] = (uint32_t)q[0] | (uint32_t)q[1] << 8 | (uint32_t)q[2] << 16;
                        }
                    }
                    *reinterpret_cast<uint4 *>(stage + t.x) = make_uint4(x[0], x[1], x[2], x[3]);
                }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&full[w]);
        }
    }
    else
    {
        // ---------------- issuers: tiles in turn
        const int me = warp - EPI_WARPS - PROD_WARPS;
        const uint32_t idesc = make_idesc(2 /*s32*/, 0, 0, 0 /*A K-major*/, 0 /*B K-major*/, BM, NCOLS);
        const uint64_t da = make_smem_desc(smem_u32(smem), 16, 8 * 16, 0), db = make_smem_desc(smem_u32(smem) + a.o_filter, NCOLS * 16, 8 * 16, 0);
        auto row = [&](int kh) { return (uint32_t)((kh & (a.stride - 1)) * a.E + (kh >> (a.stride - 1)) * a.PW); }; // its entries' first
        const uint32_t row1 = row(1), row2 = row(2), da_high = (uint32_t)(da >> 32);
        bool ok = true;
        int st = me, buf = me;
        uint32_t turn = 0, acc_turn = 1;
        for (int i = me; i < my_tiles && ok; i += ISSUERS)
        {
            if (i >= SETS)
                ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], acc_turn, status, 83));
            ok = ok && __all_sync(0xffffffffu, mbar_wait(&full[st], turn, status, 84));
            if (!ok)
                break;
            tc_fence_after_sync();
            if (elect_one())
            {
                const uint32_t at = (uint32_t)da + (uint32_t)st * (a.stage_bytes >> 4), d = tmem + (uint32_t)(buf * NCOLS);
                if (THREE) // (the rolled loop takes 150 cycles an MMA)
                {
                    tc_mma_i8(d, desc_of(at, da_high), db, idesc, 0u);
                    tc_mma_i8(d, desc_of(at + row1, da_high), db + 2 * NCOLS, idesc, 1u);
                    tc_mma_i8(d, desc_of(at + row2, da_high), db + 4 * NCOLS, idesc, 1u);
                }
                else
                    for (int kh = 0; kh < a.Fh; ++kh)
                        tc_mma_i8(d, desc_of(at + row(kh), da_high), db + (uint64_t)(kh * 2 * NCOLS), idesc, kh > 0 ? 1u : 0u);
                tc_commit(&empty[st]);
                tc_commit(&acc_full[buf]);
            }
            __syncwarp();
            st += ISSUERS;
            if (st >= STAGES) { st -= STAGES; turn ^= 1; }
            buf += ISSUERS;
            if (buf >= SETS) { buf -= SETS; acc_turn ^= 1; }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == EPI_WARPS + PROD_WARPS)
        tmem_dealloc(tmem, TMEM_COLS);
}

template <int G, int KB, bool THREE>
int launch_rgb(const RgbArgs &a, const uint8_t *in, const uint8_t *filt, const int32_t *bias, uint8_t *out, cudaStream_t st)
{
    auto kern = conv_u8_rgb_kernel<G, KB, THREE>;
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
    const int parts = a.K / (KB * CB);
    kern<<<dim3((unsigned)std::min(a.tiles, std::max(1, num_sms() / parts)), (unsigned)parts), THREADS, a.smem, st>>>(a, in, filt, bias, out, status);
    return launched("conv_u8_rgb_kernel");
}
} // namespace

namespace sb
{
// Returns -1 when the layer is not covered by this kernel (or too small for it), otherwise a SMALL_B200_* code.
int conv2d_u8_rgb(const small_b200_layer *L, const uint8_t *in, const uint8_t *filt, const int32_t *bias, uint8_t *out, cudaStream_t st)
{
    RgbArgs a{};
    a.N = L->N; a.H = L->H; a.W = L->W; a.K = L->K; a.Fh = L->Fh; a.Fw = L->Fw; a.stride = L->stride; a.pad_t = L->pad_t; a.pad_l = L->pad_l;
    if (L->C != C3 || a.stride < 1 || a.stride > 2 || row_stride(L) != a.stride)
        return -1;
    const int G = 4 / a.stride;
    if (L->accumulate || a.K % CB != 0 || a.K <= 0 || a.Fh < 1 || a.Fh > MAX_ROWS || a.Fw < 1 || (G - 1) * a.stride + a.Fw > 8 || a.pad_t < 0 ||
        a.pad_l < 0 || L->zero_in > 0 || L->zero_in < -255 || (reinterpret_cast<uintptr_t>(out) & 15) != 0)
        return -1;
    a.Ho = out_dim(a.H, L->pad_t, L->pad_b, a.Fh, a.stride);
    a.Wo = out_dim(a.W, L->pad_l, L->pad_r, a.Fw, a.stride);
    if (a.N <= 0 || a.Ho <= 0 || a.Wo <= 0)
        return SMALL_B200_OK;
    if ((long long)a.H * a.W * C3 >= 1 << 30 || (long long)a.N * a.Ho * a.Wo < RGB_MIN)
        return -1;
    a.zero_in = L->zero_in; a.zero_filt = L->zero_filt;
    a.lshift = L->lshift; a.rshift = L->rshift; a.mult = L->multiplier; a.k_zero = L->k_zero;
    a.outside = (uint32_t)(-L->zero_in) * 0x01010101u;
    a.in_bytes = (long long)a.N * a.H * a.W * C3;
    // Chunks of a tile: the split of a row into parts, and the rows that fit 128 GEMM rows, which leave the fewest tiles.
    const int chunks = (a.Wo + G - 1) / G, more_r = (a.Fh - 1) / a.stride;
    long long best = -1;
    for (int parts = 1; parts <= chunks; ++parts)
    {
        const int TW = (chunks + parts - 1) / parts, PW = TW + 1;
        if (TW > BM)
            continue;
        const int TH = std::min((BM - TW) / PW + 1, a.Ho), tx = (chunks + TW - 1) / TW, ty = (a.Ho + TH - 1) / TH;
        const long long tiles = (long long)tx * ty * a.N;
        if (best < 0 || tiles < best)
        {
            best = tiles;
            a.TW = TW; a.PW = PW; a.TH = TH; a.tiles_x = tx; a.tiles_y = ty;
        }
        else if (TW <= 8)
            break;
    }
    if (best < 0 || best > 0x3fffffff)
        return -1;
    a.tiles = (int)best;
    // Tiles with few outputs, of images a little too large for one: from half of one on where a tile's pixels are fetched for several parts of the
    // channels, a third where for one.  us, the CUDA cores' form and this: 3 -> 32 at 11x11, 2048 images (0.24 of a tile, two parts)
    // 12.1 and 18.5, 3 -> 64 at 38x9, 2048 images (0.33, four) 43.6 and 61.6, at 30x30 / 2, 1024 images (0.44, two) 18.9 and 21.4; but at
    // 18x18, 1024 images (0.63, four) 23.6 and 19.5, 3 -> 16 at 15x15, 2048 images (0.44) 13.6 and 11.9.
    const double filled = (double)a.N * a.Ho * a.Wo / ((double)a.tiles * BM * G);
    if (filled < (a.K > (a.stride == 2 && a.K % (2 * CB) == 0 ? 2 * CB : CB) && a.Fh > 2 ? 0.5 : 0.35))
        return -1;
    a.rows_in = (a.TH - 1) * a.stride + a.Fh;
    a.units = a.rows_in * a.PW;
    a.E = std::max(BM + more_r * a.PW + 1, (a.rows_in + a.stride - 1) / a.stride * a.PW);
    a.by_tiles_x.set(a.tiles_x); a.by_tiles_y.set(a.tiles_y); a.by_PW.set(a.PW);
    a.stage_bytes = ((uint32_t)(a.stride * a.E * 16) + 127) & ~127u;
    a.o_filter = a.stage_bytes * STAGES;
    const bool two = a.stride == 2 && a.K % (2 * CB) == 0;
    a.o_table = a.o_filter + (uint32_t)(a.Fh * 2 * ((two ? 4 : G) * 16 + 16) * 16);
    a.smem = a.o_table + (uint32_t)a.units * 16;
    if (a.smem > (uint32_t)SMEM_LIMIT)
        return -1;
#define SB_RGB(G_, KB_) return a.Fh == 3 ? launch_rgb<G_, KB_, true>(a, in, filt, bias, out, st) : launch_rgb<G_, KB_, false>(a, in, filt, bias, out, st)
    if (a.stride == 1)
        SB_RGB(4, 1);
    if (two)
        SB_RGB(2, 2);
    SB_RGB(2, 1);
#undef SB_RGB
}
} // namespace sb
