// conv_u8_thin.cu -- small::Conv2D<QUInt8Buffer> (include/small/interface_abstract.hpp:229-404, loop nest
// include/small/q_abstract_layer.hpp:894-1571) of pointwise layers on 16, 32 and 64 channels, as one or two tcgen05.mma.kind::i8 a tile.
//
// A reduction step is 32 bytes: 32 channels of a pixel, or TWO pixels of 16.  The operand is memory as it is: runs of 128 pixels of 16
// bytes, which bulk copies put one behind the other: with 32 and 64 channels those of a tile's planes, with 16 the two halves of 256 pixels, and
// then a GEMM row is pixels m and m + 128 and the filter two diagonal blocks, 32 columns per 16 output channels.  A tile runs
// across images.  Zero points as in conv_u8_patch.cu: sixteen more columns, the first of which are ones, give the sums of the bytes.
//
// Roles: 24 epilogue warps (six sets of four, an accumulator each), two producing and two issuing warps (tiles in turn; with one producer, which
// computes a run for every plane and image, 32 -> 32 at 24x24 takes 28.9 us instead of 19.2).
//
// What bounds it: the epilogue's instructions, five and a half per 32 results, half of them on the half-rate integer pipe: a tile of 256
// pixels and 16 channels takes 1450 warp instructions and 580 cycles, its MMA 44 of them.  us, 2048 images, before (see the rule below) -> this:
// 16 -> 16 at 48x48 55.9 -> 38.0 (23 at the rate of a copy of its bytes), 16 -> 32 at 24x24 26.3 -> 17.0, 16 -> 128 88.9 -> 58.8, 32 -> 32
// 32.2 -> 19.2; 32 -> 64 at 12x12 15.9 -> 10.9, 64 -> 64 16.6 -> 11.7, 64 -> 16 12.1 -> 7.6; 64 -> 64 at 45x45, 48 images 8.6 -> 6.7.
#include "tc_common.cuh"

#include <algorithm>
#include <type_traits>

namespace
{
using namespace sb;

constexpr int BM = 128, SETS = 6, EPI_WARPS = 4 * SETS, ISSUERS = 2, PRODUCERS = 2, STAGES = 12;
constexpr int THREADS = (EPI_WARPS + PRODUCERS + ISSUERS) * 32;
constexpr uint32_t HALF = BM * CB; // 128 pixels of a plane
// Where this kernel is the faster one.  us, before (16 channels: the CUDA cores' kernel of quint8.cu, else conv_u8_tc.cu) -> this: 16 -> 16 at
// 48x48, 64 images (2.4 million results) 3.8 -> 4.2, 256 images 9.4 -> 7.4; 16 -> 32 at 24x24, 64 images 3.3 -> 3.9, 256 images (4.7
// million) 5.3 -> 5.1; 16 -> 64 at 24x24, 1 image 3.9 -> 3.7, 64 images 4.3 -> 4.2, but up to 128 pixels (a CTA there) 3.0 to 3.3 -> 3.7; 32 -> 64 at 12x12, 128 images (18 432 pixels) 4.1 -> 4.5,
// 256 images 5.2 -> 4.6; 64 -> 64 at 12x12, 64 images 4.2 -> 4.6, 256 images 5.6 -> 5.3.  128 channels stay where they were: 128 -> 128 at
// 14x14, 64 images 5.6 -> 6.8, at 8x8, 2048 images 14.4 -> 17.6.
constexpr long long MIN_RESULTS = 4 << 20, MIN_PIXELS = 30000;
bool large_enough(int C, int K, long long pixels)
{
    return C > CB ? pixels >= MIN_PIXELS : (K >= 64 && pixels > BM) || pixels * K >= MIN_RESULTS;
}
constexpr int MAX_STEPS = 2;             // reduction steps: up to 64 channels
constexpr int SMEM_LIMIT = 2 * MAX_STEPS * (STAGES * (int)HALF + 80 * 16);
static_assert(SETS % ISSUERS == 0 && STAGES % ISSUERS == 0 && STAGES % PRODUCERS == 0, "who waits on a stage or an accumulator sees all of its phases");

struct ThinArgs
{
    int N, P, C, K;       // P: pixels of an image
    int tiles, total;     // tiles, pixels
    int chunks;           // runs of 16 bytes a reduction takes: two pixels' or a pixel's blocks of channels
    int zero_in, zero_filt, lshift, rshift, mult, k_zero;
    FastDiv by_P;
};

__device__ __forceinline__ uint64_t desc_of(uint32_t low, uint32_t high)
{
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(low), "r"(high));
    return d;
}
// four outputs' bytes by any quantiser
__device__ __forceinline__ uint32_t quantise4(bool fast, int a, int b, int c, int d, const ThinArgs &p, int bit, int sh1)
{
    if (!fast)
        return requant_pack4_general(a, b, c, d, p.lshift, p.rshift, p.mult);
    return pack4_sat(requant_seeded_raw(a, p.mult, 1ll << 30, bit, sh1), requant_seeded_raw(b, p.mult, 1ll << 30, bit, sh1),
                     requant_seeded_raw(c, p.mult, 1ll << 30, bit, sh1), requant_seeded_raw(d, p.mult, 1ll << 30, bit, sh1));
}

// G pixels a GEMM row (2: 16 channels, 1: more), KB blocks of 16 output channels a CTA.
template <int G, int KB>
__global__ void __launch_bounds__(THREADS, 1)
conv_u8_thin_kernel(const __grid_constant__ ThinArgs a, const uint8_t *__restrict__ in, const uint8_t *__restrict__ filt,
                    const int32_t *__restrict__ bias, uint8_t *__restrict__ out, int *status)
{
    constexpr int UNITS = G * KB, NCOLS = UNITS * 16 + 16;
    constexpr uint32_t TMEM_COLS = SETS * NCOLS <= 256 ? 256 : 512;
    static_assert(SETS * NCOLS <= 512, "");
    extern __shared__ __align__(1024) uint8_t smem[]; // [stage][chunk][128][16 B], filter [chunk][column][16 B]
    __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], acc_full[SETS], acc_empty[SETS];
    __shared__ uint32_t tmem_base_s;
    __shared__ __align__(16) int seed[KB * CB];

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int kb0 = blockIdx.y * KB, kbs = a.K / CB;
    const int my_tiles = (a.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    const uint32_t stage_bytes = (uint32_t)a.chunks * HALF;
    uint8_t *sB = smem + STAGES * stage_bytes;

    for (int i = tid; i < a.chunks * NCOLS * 4; i += THREADS) // a word: four channels of a column
    {
        const int c4 = (i & 3) * 4, col = (i >> 2) % NCOLS, half = (i >> 2) / NCOLS, unit = col / CB;
        const int g = unit < UNITS ? unit % G : col - UNITS * CB; // the pixel this column is for
        uint32_t v = 0;
        if (G == 2 ? g == half : g == 0)
        {
            v = 0x01010101u;
            if (unit < UNITS)
            {
                const uint8_t *w = filt + ((size_t)(kb0 + unit / G) * a.C + (G == 1 ? half * CB : 0) + c4) * CB + col % CB;
                v = (uint32_t)w[0] | (uint32_t)w[CB] << 8 | (uint32_t)w[2 * CB] << 16 | (uint32_t)w[3 * CB] << 24;
            }
        }
        reinterpret_cast<uint32_t *>(sB)[i] = v;
    }
    if (tid < KB * CB)
    {
        const int k = kb0 * CB + tid;
        const uint8_t *w = filt + (size_t)(k / CB) * a.C * CB + k % CB;
        int sum = 0;
        for (int i = 0; i < a.C; ++i)
            sum += w[i * CB];
        seed[tid] = a.k_zero + (bias ? bias[k] : 0) + a.zero_in * sum + a.C * a.zero_in * a.zero_filt;
    }
    fence_proxy_async();
    if (warp == EPI_WARPS)
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

    if (warp < EPI_WARPS)
    {
        // ---------------- epilogue: thread = GEMM row; set s takes tiles s, s + SETS, ...
        const int set = warp >> 2, quarter = warp & 3, m = quarter * 32 + lane;
        const bool fast = requant_is_fast(a.lshift, a.rshift, a.mult);
        const int bit = 1 << ((a.rshift - 2) & 31), sh1 = a.rshift - 1;
        const size_t plane = (size_t)a.P * CB;
        const uint32_t d = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(set * NCOLS);
        bool ok = true;
        uint32_t turn = 0;
        auto tiles = [&](auto is_fast) {
#pragma unroll 1
            for (int i = set; i < my_tiles; i += SETS, turn ^= 1)
            {
                const int tile = blockIdx.x + i * gridDim.x;
                uint8_t *o[G];
                bool live[G];
#pragma unroll
                for (int g = 0; g < G; ++g)
                {
                    const int px = tile * G * BM + g * BM + m;
                    live[g] = px < a.total;
                    const int n = a.by_P.div(live[g] ? px : 0), p = px - n * a.P;
                    o[g] = out + ((size_t)n * kbs + kb0) * plane + (long long)p * CB;
                }
                ok = mbar_wait(&acc_full[set], turn, status, 91);
                if (!ok)
                    break;
                tc_fence_after_sync();
                uint32_t sums[16];
                tmem_ld16(d + UNITS * 16, sums);
#pragma unroll
                for (int u = 0; u < UNITS; ++u)
                {
                    const int kb = u / G, g = u % G;
                    uint32_t x[16], w[4];
                    tmem_ld16(d + (uint32_t)(u * 16), x);
                    tmem_ld_wait();
                    if (u == UNITS - 1) // read
                    {
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0)
                            mbar_arrive(&acc_empty[set]);
                    }
                    const int base = a.zero_filt * (int)sums[g];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                    {
                        const int4 s = reinterpret_cast<const int4 *>(seed + kb * CB)[e];
                        w[e] = quantise4(decltype(is_fast)::value, (int)x[4 * e] + s.x + base, (int)x[4 * e + 1] + s.y + base,
                                         (int)x[4 * e + 2] + s.z + base, (int)x[4 * e + 3] + s.w + base, a, bit, sh1);
                    }
                    if (live[g])
                        *reinterpret_cast<uint4 *>(o[g] + (size_t)kb * plane) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
        };
        if (fast)
            tiles(std::true_type{});
        else
            tiles(std::false_type{});
    }
    else if (warp < EPI_WARPS + PRODUCERS)
    {
        // ---------------- producers: tiles in turn (rows of a last tile behind its pixels keep stale bytes: their results are not stored)
        bool ok = true;
        int st = warp - EPI_WARPS;
        uint32_t used = 1;
        const int seg = G == 1 ? lane / a.chunks : 0, cb = lane - seg * a.chunks;
        for (int i = st; i < my_tiles; i += PRODUCERS)
        {
            if (i >= STAGES)
                ok = __all_sync(0xffffffffu, mbar_wait(&empty[st], used, status, 92));
            if (!ok)
                break;
            const int px0 = (blockIdx.x + i * gridDim.x) * G * BM, left = min(G * BM, a.total - px0);
            uint8_t *dst = smem + st * stage_bytes;
            if (lane == 0)
                mbar_expect_tx(&full[st], (uint32_t)(left * a.C));
            __syncwarp();
            if (G == 2)
            {
                if (lane == 0)
                    tma_load_1d(dst, in + (size_t)px0 * CB, (uint32_t)left * CB, &full[st]);
            }
            else
            {
                // a lane a plane and image: the pixels of at most three images (a.P >= 64); seg * a.P fits in 31 bits
                const int n = a.by_P.div(px0), p = px0 - n * a.P;
                const int row0 = seg ? min(seg, 2) * a.P - p : 0, rows = min(seg ? a.P : a.P - p, left - row0);
                if (seg < 3 && rows > 0)
                    tma_load_1d(dst + cb * HALF + row0 * CB, in + (((size_t)(n + seg) * a.chunks + cb) * a.P + (seg ? 0 : p)) * CB, (uint32_t)rows * CB,
                                &full[st]);
            }
            __syncwarp();
            st += PRODUCERS;
            if (st >= STAGES) { st -= STAGES; used ^= 1; }
        }
    }
    else
    {
        // ---------------- issuers: tiles in turn
        const int me = warp - EPI_WARPS - PRODUCERS;
        const uint32_t idesc = make_idesc(2 /*s32*/, 0, 0, 0 /*A K-major*/, 0 /*B K-major*/, BM, NCOLS);
        const uint64_t da = make_smem_desc(smem_u32(smem), HALF, 8 * CB, 0), db = make_smem_desc(smem_u32(sB), NCOLS * 16, 8 * CB, 0);
        const uint32_t da_high = (uint32_t)(da >> 32);
        bool ok = true;
        int st = me, buf = me;
        uint32_t turn = 0, acc_turn = 1;
        for (int i = me; i < my_tiles && ok; i += ISSUERS)
        {
            if (i >= SETS)
                ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], acc_turn, status, 93));
            ok = ok && __all_sync(0xffffffffu, mbar_wait(&full[st], turn, status, 94));
            if (!ok)
                break;
            tc_fence_after_sync();
            if (elect_one())
            {
                const uint32_t d = tmem + (uint32_t)(buf * NCOLS), at = (uint32_t)da + (uint32_t)st * (stage_bytes >> 4);
                tc_mma_i8(d, desc_of(at, da_high), db, idesc, 0u);
                if (G == 1)
#pragma unroll
                    for (int j = 1; j < MAX_STEPS; ++j)
                        if (2 * j < a.chunks)
                            tc_mma_i8(d, desc_of(at + (uint32_t)(j * 2 * (HALF >> 4)), da_high), db + (uint64_t)(j * 2 * NCOLS), idesc, 1u);
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
    if (warp == EPI_WARPS)
        tmem_dealloc(tmem, TMEM_COLS);
}

template <int G, int KB>
int launch_thin(const ThinArgs &a, const uint8_t *in, const uint8_t *filt, const int32_t *bias, uint8_t *out, cudaStream_t st)
{
    const uint32_t smem = (uint32_t)a.chunks * (STAGES * HALF + (G * KB * 16 + 16) * 16);
    auto kern = conv_u8_thin_kernel<G, KB>;
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
    kern<<<dim3((unsigned)std::min(a.tiles, std::max(1, num_sms() / parts)), (unsigned)parts), THREADS, smem, st>>>(a, in, filt, bias, out, status);
    return launched("conv_u8_thin_kernel");
}
} // namespace

namespace sb
{
// Returns -1 when the layer is not covered by this kernel (or too small for it), otherwise a SMALL_B200_* code.
int conv2d_u8_thin(const small_b200_layer *L, const uint8_t *in, const uint8_t *filt, const int32_t *bias, uint8_t *out, cudaStream_t st)
{
    if (L->accumulate || (L->C != CB && L->C % (2 * CB) != 0) || L->C <= 0 || L->C > MAX_STEPS * 2 * CB || L->K <= 0 || L->K % CB || L->K > 128 || L->Fh != 1 || L->Fw != 1 || L->stride != 1 ||
        row_stride(L) != 1 || L->pad_t || L->pad_b || L->pad_l || L->pad_r ||
        ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) != 0)
        return -1;
    const long long P = (long long)L->H * L->W, total = P * L->N;
    if (P <= 0 || L->N <= 0 || total > 0x3fffffff || !large_enough(L->C, L->K, total))
        return -1;
    ThinArgs a{};
    a.N = L->N; a.P = (int)P; a.C = L->C; a.K = L->K; a.total = (int)total;
    a.zero_in = L->zero_in; a.zero_filt = L->zero_filt;
    a.lshift = L->lshift; a.rshift = L->rshift; a.mult = L->multiplier; a.k_zero = L->k_zero;
    if (a.C > CB && P < BM / 2)
        return -1; // a tile would have many images' runs to fetch
    a.chunks = std::max(2, a.C / CB);
    a.tiles = (int)((total + (a.C == CB ? 2 * BM : BM) - 1) / (a.C == CB ? 2 * BM : BM));
    a.by_P.set(a.P);
    if (a.C == CB)
        return a.K % 32 == 0 ? launch_thin<2, 2>(a, in, filt, bias, out, st) : launch_thin<2, 1>(a, in, filt, bias, out, st);
    return a.K % 64 == 0   ? launch_thin<1, 4>(a, in, filt, bias, out, st)
           : a.K % 32 == 0 ? launch_thin<1, 2>(a, in, filt, bias, out, st)
                           : launch_thin<1, 1>(a, in, filt, bias, out, st);
}
} // namespace sb
