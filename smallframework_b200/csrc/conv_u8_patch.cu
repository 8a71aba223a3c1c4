// conv_u8_patch.cu -- small::Conv2D<QUInt8Buffer> (include/small/interface_abstract.hpp:229-404, loop nest
// include/small/q_abstract_layer.hpp:894-1571) for windows of more than one tap and strides 1 and 2, as an implicit GEMM on
// tcgen05.mma.kind::i8 whose pixels are fetched ONCE: conv_u8_ring.cu gathers every pixel once per tap.
//
// Implicit GEMM by linear shift.  A tile is TH x TW outputs of an image, or several whole small images; its input patch lies
// in shared memory as [16-channel block][phase][entry][16 B], phase = (row % stride, column % stride), entries of PW = TW + (Fw - 1) / stride a
// row.  Output (r, c) is GEMM row m = r * PW + c, and tap (kh, kw) of it is entry m + (kh / stride) * PW + kw / stride of phase
// (kh % stride, kw % stride): a tap only moves the start of the operand (a multiple of 16 bytes, any of which read at the same
// speed).  Rows with c >= TW are junk and are not stored.
// A reduction step of 32 bytes is two (block, tap) slabs of 16 channels.  The slabs of the filter, 256 bytes each, are put in the order of
// their operands' addresses, so that two neighbours are one step: the distance between their operands is a field of the
// descriptor.  An odd slab is paired with a region of zeros.
// Zero points.  Both operands are the unsigned bytes as they are.  sum (a + zi)(b + zf) = sum ab + zf sum a + zi sum b + n zi zf: the MMA
// gives the first, sixteen more columns with a filter column of ones the second, the others are constants of a channel.  A tap
// outside the image holds the byte -zi; where that is no byte, conv_u8_ring.cu takes the layer.
//
// Roles: 8 producer warps (16-byte cp.async through a table of the patch's pixels), 2 issuing warps (tiles in turn, an accumulator each:
// what a warp spends on issuing a tile's MMAs is hidden by the other's), 8 epilogue warps.  The filter stays in shared memory where it fits
// beside the stages of pixels, else its slabs travel with the pixels' channels.
//
// What bounds it: a tile of 64 channels takes 18 MMAs of 52 cycles and an epilogue of 900; a launch of a few tiles an SM
// begins with 9000 cycles until its first sums, most of them the first patches and the filter, which all SMs ask for at once.  (64 -> 64
// 3x3 at 45x37, 1024 images: 161 us; tensor core unit 35 %, issue slots 37 %, shared memory 33 %, DRAM 13 %: no unit's limit.)
// us, conv_u8_ring.cu -> this: 3x3 64 -> 64 channels at 45x37, 48 images 34.9 -> 12.4, 64 -> 128 with a stride of two 35.2 -> 11.9;
// 256 -> 256 at 20x20, 48 images 142 -> 39; 96 -> 96 at 30x11, 64 images 43.5 -> 11.3; 16 -> 32 at 112x112 with a stride of two, 24
// images 16.9 -> 14.9.
#include "tc_common.cuh"

#include <algorithm>

namespace
{
using namespace sb;

constexpr int BM = 128, EPI_WARPS = 8, PROD_WARPS = 8, ISSUERS = 2;
constexpr int THREADS = (EPI_WARPS + PROD_WARPS + ISSUERS) * 32, PROD_THREADS = PROD_WARPS * 32, EPI_THREADS = EPI_WARPS * 32;
constexpr int MAX_TAPS = 49, MAX_STAGES = 4, SLAB = CB * CB;
constexpr int SMEM_LIMIT = 216 * 1024;

struct PatchArgs
{
    int N, H, W, C, K, Ho, Wo, Fh, Fw, sh, sw, pad_t, pad_l;
    int cbs, taps;
    int TH, TW, PW, RI, ni;          // outputs of a tile, entries a row, rows an image takes, images a tile
    int rows_in, cols_in, units;     // input pixels of a patch: per image, together
    int tiles_x, tiles_y, tiles;
    int E, planes;                   // entries of a phase's plane (what the last GEMM row's last tap reads included), phases
    int cc, chunks, stages;          // channel blocks of a stage of pixels, such stages a tile, stages in shared memory
    int resident;                    // the filter stays; else a stage also holds its slabs
    int in_order;                    // ranks are the taps themselves
    uint32_t run;                    // bytes from 16 output channels' slabs to the next 16's
    uint32_t patch_bytes, stage_bytes, o_filter, o_table, o_zero, smem;
    uint32_t outside;                // the byte of a tap outside the image, four times
    int zero_in, zero_filt, lshift, rshift, mult, k_zero;
    FastDiv by_tiles_x, by_tiles_y, by_PW, by_RI, by_taps;
    uint16_t operand[MAX_TAPS];      // of the tap with this rank: entries from its block's first
    uint8_t rank[MAX_TAPS];
};

__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

__device__ __forceinline__ uint64_t desc_of(uint32_t low, uint32_t high)
{
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(low), "r"(high));
    return d;
}

// 16 sums by any quantiser; out of line and chosen once per tile
__device__ __noinline__ uint4 requant16_any(uint32_t d, const int *seed, int base, int lshift, int rshift, int mult)
{
    uint32_t r[16], w[4];
    tmem_ld16(d, r);
    tmem_ld_wait();
#pragma unroll
    for (int e = 0; e < 4; ++e)
    {
        int v[4];
        for (int j = 0; j < 4; ++j)
            v[j] = (int)r[4 * e + j] + seed[4 * e + j] + base;
        w[e] = requant_pack4_general(v[0], v[1], v[2], v[3], lshift, rshift, mult);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// NINE: windows of nine taps, whose steps are unrolled.
template <int NT, bool NINE>
__global__ void __launch_bounds__(THREADS, 1)
conv_u8_patch_kernel(const __grid_constant__ PatchArgs a, const uint8_t *__restrict__ in, const uint8_t *__restrict__ filt,
                     const int32_t *__restrict__ bias, uint8_t *__restrict__ out, int *status)
{
    constexpr int NCOLS = NT + 16, GROUPS = NT / CB;
    constexpr uint32_t TMEM_COLS = 2 * NCOLS <= 64 ? 64 : 2 * NCOLS <= 128 ? 128 : 2 * NCOLS <= 256 ? 256 : 512;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[MAX_STAGES], empty[MAX_STAGES], acc_full[2], acc_empty[2], filter_full;
    __shared__ uint32_t tmem_base_s;
    __shared__ __align__(16) int seed[NT];
    __shared__ uint8_t rank[MAX_TAPS];

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int nb = blockIdx.y, groups = min(GROUPS, a.K / CB - nb * GROUPS); // groups of 16 output channels this CTA really has
    const int my_tiles = (a.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    uint4 *table = reinterpret_cast<uint4 *>(smem + a.o_table);

    // Slabs of `blocks` channel blocks from cb0 on to `dst`.  In order they are one run per 16 output channels: bulk copies by a
    // warp, `bar` is told the bytes.  Else 16-byte copies by `count` threads (a bulk copy a slab: 24000 cycles for 64 -> 128 channels).
    const uint8_t *filt_nb = filt + (size_t)nb * GROUPS * a.cbs * a.taps * SLAB;
    const size_t filt_run = (size_t)a.cbs * a.taps * SLAB;
    auto fetch_runs = [&](uint8_t *dst, int cb0, int blocks, uint64_t *bar) {
        if (lane == 0)
            mbar_expect_tx(bar, (uint32_t)(groups * blocks * a.taps * SLAB));
        __syncwarp();
        for (int g = lane; g < groups; g += 32)
            tma_load_1d(dst + g * a.run, filt_nb + g * filt_run + (size_t)cb0 * a.taps * SLAB, (uint32_t)(blocks * a.taps * SLAB), bar);
    };
    auto fetch_slabs = [&](uint8_t *dst, int cb0, int blocks, int thread, int count) {
        const int slabs = blocks * a.taps;
        int g = 0, i = thread / CB;
        const uint8_t *src = filt_nb + (size_t)cb0 * a.taps * SLAB + (thread % CB) * CB;
        dst += (thread % CB) * CB;
        for (;; i += count / CB)
        {
            for (; i >= slabs; i -= slabs, ++g)
                ;
            if (g >= groups)
                break;
            const int b = a.by_taps.div(i), t = i - b * a.taps;
            cp_async16(dst + g * a.run + (b * a.taps + rank[t]) * SLAB, src + g * filt_run + (size_t)i * SLAB);
        }
    };
    if (warp == EPI_WARPS + PROD_WARPS)
    {
        if (lane == 0)
        {
            for (int i = 0; i < MAX_STAGES; ++i) { mbar_init(&full[i], PROD_WARPS + (!a.resident && a.in_order)); mbar_init(&empty[i], 1); }
            for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], EPI_WARPS); }
            mbar_init(&filter_full, 1 + EPI_WARPS);
            fence_barrier_init();
        }
        __syncwarp();
        if (a.resident && a.in_order)
            fetch_runs(smem + a.o_filter, 0, a.cbs, &filter_full);
        else if (lane == 0)
            mbar_arrive(&filter_full);
        tmem_alloc(&tmem_base_s, TMEM_COLS);
        tmem_relinquish();
    }
    else if (warp >= EPI_WARPS && warp < EPI_WARPS + PROD_WARPS)
    {
        // a patch's pixels in the order they lie in the image: where they go, how far from the first one they lie, row and column, image
        for (int i = tid - EPI_WARPS * 32; i < a.units; i += PROD_THREADS)
        {
            const int per = a.rows_in * a.cols_in, j = i / per, p = i - j * per, r = p / a.cols_in, c = p - r * a.cols_in;
            const int phase = (r & (a.sh - 1)) * a.sw + (c & (a.sw - 1)), entry = (j * a.RI + (r >> (a.sh - 1))) * a.PW + (c >> (a.sw - 1));
            table[i] = make_uint4((uint32_t)(phase * a.E + entry) * CB, ((uint32_t)j * a.cbs * a.H * a.W + (uint32_t)r * a.W + (uint32_t)c) * CB,
                                  (uint32_t)r << 16 | (uint32_t)c, (uint32_t)j);
        }
        for (int i = tid - EPI_WARPS * 32; i < BM; i += PROD_THREADS)
            reinterpret_cast<uint4 *>(smem + a.o_zero)[i] = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async();
    }
    else if (warp < EPI_WARPS)
    {
        if (tid < a.taps)
            rank[tid] = a.rank[tid];
        if (tid < NT)
            seed[tid] = a.k_zero + (bias && nb * NT + tid < a.K ? bias[nb * NT + tid] : 0) + a.taps * a.C * a.zero_in * a.zero_filt;
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_s, 0);

    // image, first output row and column of a tile
    auto decode = [&](int tile, int &n, int &r0, int &c0) {
        const int t1 = a.by_tiles_x.div(tile), t2 = a.by_tiles_y.div(t1);
        n = t2 * a.ni; r0 = (t1 - t2 * a.tiles_y) * a.TH; c0 = (tile - t1 * a.tiles_x) * a.TW;
    };
    if (warp < EPI_WARPS)
    {
        // ---------------- epilogue: thread = GEMM row, the channels split between the two warps of a lane quarter
        // First, while the first pixels are on their way: the filter column of ones, behind the last 16 output channels of the slabs
        // (never rewritten), and the part of the channels' constants that is zero_in * (sum of the filter bytes).
        if (a.resident && !a.in_order)
            fetch_slabs(smem + a.o_filter, 0, a.cbs, tid, EPI_THREADS);
        cp_async_commit();
        for (int i = tid; i < (int)(a.run / CB) * (a.resident ? 1 : a.stages); i += EPI_THREADS)
        {
            const int st = i / (int)(a.run / CB), r = i - st * (int)(a.run / CB);
            uint8_t *base = a.resident ? smem + a.o_filter : smem + st * a.stage_bytes + a.patch_bytes;
            reinterpret_cast<uint4 *>(base + GROUPS * a.run)[r] = make_uint4(1u, 0u, 0u, 0u);
        }
        cp_async_wait<0>();
        fence_proxy_async();
        __syncwarp();
        if (lane == 0)
            mbar_arrive(&filter_full);
        bool ok = mbar_wait(&filter_full, 0, status, 66);
        if (a.zero_in != 0) // a warp adds rows of 16 channels (from shared memory where they are: read from memory twice, the filter kept the pixels waiting)
        {
            constexpr int PARTS = EPI_WARPS >= GROUPS ? EPI_WARPS / GROUPS : 1;
            const int g = warp / PARTS, rows = a.cbs * a.taps * CB, stride = PARTS * 32;
            if (g < groups)
            {
                const uint4 *w = reinterpret_cast<const uint4 *>(a.resident ? smem + a.o_filter + g * a.run : filt_nb + g * filt_run);
                int sum[CB] = {};
                for (int r0 = tid - g * stride; r0 < rows; r0 += stride * 8)
                {
                    uint4 v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        v[u] = r0 + u * stride < rows ? w[r0 + u * stride] : make_uint4(0u, 0u, 0u, 0u);
                    unsigned even[4] = {0u, 0u, 0u, 0u}, odd[4] = {0u, 0u, 0u, 0u}; // pairs of sums of 8 bytes
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                    {
                        const unsigned x[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                        {
                            even[k] += x[k] & 0x00ff00ffu;
                            odd[k] += (x[k] >> 8) & 0x00ff00ffu;
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                    {
                        sum[4 * k] += (int)(even[k] & 0xffffu); sum[4 * k + 1] += (int)(odd[k] & 0xffffu);
                        sum[4 * k + 2] += (int)(even[k] >> 16); sum[4 * k + 3] += (int)(odd[k] >> 16);
                    }
                }
#pragma unroll
                for (int k = 0; k < CB; ++k)
                {
                    sum[k] = __reduce_add_sync(0xffffffffu, sum[k]);
                    if (lane == 0)
                        atomicAdd(&seed[g * CB + k], a.zero_in * sum[k]);
                }
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
        const int quarter = warp & 3, part = warp >> 2, m = quarter * 32 + lane;
        const int row = a.by_PW.div(m), cl = m - row * a.PW, j = a.by_RI.div(row), rl = row - j * a.RI;
        const bool fast = requant_is_fast(a.lshift, a.rshift, a.mult);
        const int bit = 1 << ((a.rshift - 2) & 31), sh1 = a.rshift - 1;
        const size_t plane = (size_t)a.Ho * a.Wo * CB;
        for (int i = 0; i < my_tiles && ok; ++i)
        {
            const int buf = i & 1;
            int n, r0, c0;
            decode(blockIdx.x + i * gridDim.x, n, r0, c0);
            n += j;
            const int oh = r0 + rl, ow = c0 + cl;
            const bool live = cl < a.TW && rl < a.TH && j < a.ni && n < a.N && oh < a.Ho && ow < a.Wo;
            uint8_t *o = out + ((size_t)n * (a.K / CB) + (size_t)nb * GROUPS) * plane + ((size_t)oh * a.Wo + ow) * CB;
            ok = mbar_wait(&acc_full[buf], (i >> 1) & 1, status, 61);
            if (!ok)
                break;
            tc_fence_after_sync();
            const uint32_t d = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * NCOLS);
            uint32_t r[2][16];
            tmem_ld16(d + NT, r[1]);
            tmem_ld16(d + (uint32_t)(part * CB), r[0]); // the load of the next 16 channels is in flight while 16 are requantised
            tmem_ld_wait();
            const int base = a.zero_filt * (int)r[1][0];
            if (fast)
            {
                constexpr int EACH = GROUPS > 1 ? GROUPS / (EPI_WARPS / 4) : 1;
#pragma unroll
                for (int u = 0; u < EACH; ++u)
                {
                    const int g = part + u * (EPI_WARPS / 4);
                    if (g >= groups)
                        break;
                    if (u + 1 < EACH)
                        tmem_ld16(d + (uint32_t)((g + EPI_WARPS / 4) * CB), r[(u + 1) & 1]);
                    const uint32_t *x = r[u & 1];
                    const int4 *s4 = reinterpret_cast<const int4 *>(seed + g * CB);
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                    {
                        const int4 s = s4[e];
                        w[e] = pack4_sat(requant_seeded_raw((int)x[4 * e] + s.x + base, a.mult, 1ll << 30, bit, sh1),
                                         requant_seeded_raw((int)x[4 * e + 1] + s.y + base, a.mult, 1ll << 30, bit, sh1),
                                         requant_seeded_raw((int)x[4 * e + 2] + s.z + base, a.mult, 1ll << 30, bit, sh1),
                                         requant_seeded_raw((int)x[4 * e + 3] + s.w + base, a.mult, 1ll << 30, bit, sh1));
                    }
                    if (live)
                        *reinterpret_cast<uint4 *>(o + (size_t)g * plane) = make_uint4(w[0], w[1], w[2], w[3]);
                    if (u + 1 < EACH)
                        tmem_ld_wait();
                }
            }
            else
#pragma unroll 1
                for (int g = part; g < groups; g += EPI_WARPS / 4)
                {
                    const uint4 v = requant16_any(d + (uint32_t)(g * CB), seed + g * CB, base, a.lshift, a.rshift, a.mult);
                    if (live)
                        *reinterpret_cast<uint4 *>(o + (size_t)g * plane) = v;
                }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&acc_empty[buf]);
        }
    }
    else if (warp < EPI_WARPS + PROD_WARPS)
    {
        // ---------------- producers ----------------
        const int pt = tid - EPI_WARPS * 32;
        const size_t plane = (size_t)a.H * a.W * CB;
        const uint32_t block = (uint32_t)(a.planes * a.E * CB);
        const uint4 outside = make_uint4(a.outside, a.outside, a.outside, a.outside);
        const int total = my_tiles * a.chunks, ahead = a.stages - 1; // stages whose copies are under way
        bool ok = true;
        int st = 0, done_st = 0;
        uint32_t used = 1; // parity of the stage's last release; the first round finds all free
        auto finish = [&]() { // the oldest outstanding stage is complete
            fence_proxy_async();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&full[done_st]);
            if (++done_st == a.stages)
                done_st = 0;
        };
        int i = 0;
        for (int tile = blockIdx.x, chunk = 0; i < total; ++i)
        {
            if (i >= a.stages)
                ok = __all_sync(0xffffffffu, mbar_wait(&empty[st], used, status, 62));
            if (!ok)
                break;
            int n, r0, c0;
            decode(tile, n, r0, c0);
            const int ih0 = r0 * a.sh - a.pad_t, iw0 = c0 * a.sw - a.pad_l, cb0 = chunk * a.cc, blocks = min(a.cc, a.cbs - cb0);
            uint8_t *stage = smem + st * a.stage_bytes;
            // (the first pixel may lie outside the image: only addresses inside are used)
            const uint8_t *src0 = in + (((long long)n * a.cbs + cb0) * a.H * a.W + (long long)ih0 * a.W + iw0) * CB;
            for (int u = pt; u < a.units; u += PROD_THREADS)
            {
                const uint4 t = table[u];
                const int ih = ih0 + (int)(t.z >> 16), iw = iw0 + (int)(t.z & 0xffffu);
                uint8_t *dst = stage + t.x;
                if ((unsigned)ih < (unsigned)a.H && (unsigned)iw < (unsigned)a.W && n + (int)t.w < a.N)
                {
                    const uint8_t *src = src0 + t.y;
#pragma unroll 4
                    for (int b = 0; b < blocks; ++b, dst += block, src += plane)
                        cp_async16(dst, src);
                }
                else
                    for (int b = 0; b < blocks; ++b, dst += block)
                        *reinterpret_cast<uint4 *>(dst) = outside;
            }
            if (!a.resident && !a.in_order)
                fetch_slabs(stage + a.patch_bytes, cb0, blocks, pt, PROD_THREADS);
            else if (!a.resident && warp == EPI_WARPS)
                fetch_runs(stage + a.patch_bytes, cb0, blocks, &full[st]);
            cp_async_commit();
            if (i >= ahead)
            {
                if (ahead == 3) cp_async_wait<3>();
                else if (ahead == 2) cp_async_wait<2>();
                else cp_async_wait<1>();
                finish();
            }
            if (++st == a.stages) { st = 0; used ^= 1; }
            if (++chunk == a.chunks) { chunk = 0; tile += gridDim.x; }
        }
        cp_async_wait<0>();
        if (ok)
            for (int left = min(total, ahead); left > 0; --left)
                finish();
    }
    else
    {
        // ---------------- issuers: tiles in turn ----------------
        const int me = warp - EPI_WARPS - PROD_WARPS;
        const uint32_t idesc = make_idesc(2 /*s32*/, 0, 0, 0 /*A K-major*/, 1 /*B MN-major*/, BM, NCOLS);
        const uint32_t block16 = (uint32_t)(a.planes * a.E), zero16 = a.o_zero >> 4;
        // a step's two operands; `x` entries from the stage's first
        auto step = [&](uint32_t stage16, uint32_t x0, uint32_t x1) {
            return make_smem_desc(smem_u32(smem), 0, 8 * CB, 0) + ((uint64_t)(x1 - x0) << 16) + (uint64_t)(stage16 + x0);
        };
        uint32_t nine[9]; // (the descriptors' other halves are all the same: fewer instructions in front of an MMA)
        if (NINE)
#pragma unroll
            for (int p = 0; p < 9; ++p)
            {
                const int s0 = 2 * p, s1 = 2 * p + 1;
                nine[p] = (uint32_t)step(0, a.operand[s0 % 9] + (s0 / 9) * block16, a.operand[s1 % 9] + (s1 / 9) * block16);
            }
        bool ok = __all_sync(0xffffffffu, mbar_wait(&filter_full, 0, status, 65));
        const uint32_t a_high = (uint32_t)(make_smem_desc(0, 0, 8 * CB, 0) >> 32), b_high = (uint32_t)(make_smem_desc(0, 0, a.run, 0) >> 32);
        // Whoever waits on a stage has to see every one of its phases: with one stage a tile and an even number of stages, a stage is
        // always the same issuer's; else one of them does all the work.
        const int issuers = a.chunks == 1 ? ISSUERS : 1;
        int st = me;
        uint32_t turn = 0;
        for (int i = me < issuers ? me : my_tiles; i < my_tiles && ok; i += issuers)
        {
            const int buf = i & 1;
            const uint32_t d = tmem + (uint32_t)(buf * NCOLS);
            if (i >= 2)
                ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], ((i >> 1) - 1) & 1, status, 63));
            bool first = true;
            for (int chunk = 0; chunk < a.chunks && ok; ++chunk)
            {
                ok = __all_sync(0xffffffffu, mbar_wait(&full[st], turn, status, 64));
                if (!ok)
                    break;
                tc_fence_after_sync();
                const int blocks = min(a.cc, a.cbs - chunk * a.cc);
                const uint32_t stage16 = (uint32_t)st * (a.stage_bytes >> 4);
                const uint32_t fb = a.resident ? a.o_filter + (uint32_t)(chunk * a.cc * a.taps * SLAB) : st * a.stage_bytes + a.patch_bytes;
                const uint64_t db = make_smem_desc(smem_u32(smem) + fb, 8 * CB, a.run, 0);
                if (elect_one())
                {
                    uint32_t acc = first ? 0u : 1u;
                    if (NINE)
                    {
                        uint32_t at = stage16, b = (uint32_t)db;
                        for (int cb = 0; cb + 1 < blocks; cb += 2, at += 2 * block16, b += 18 * (SLAB >> 4))
                        {
#pragma unroll
                            for (int p = 0; p < 9; ++p)
                                tc_mma_i8(d, desc_of(nine[p] + at, a_high), desc_of(b + (uint32_t)(p * 2 * (SLAB >> 4)), b_high), idesc, p == 0 ? acc : 1u);
                            acc = 1u;
                        }
                        if (blocks & 1)
                        {
#pragma unroll
                            for (int p = 0; p < 4; ++p)
                                tc_mma_i8(d, desc_of(nine[p] + at, a_high), desc_of(b + (uint32_t)(p * 2 * (SLAB >> 4)), b_high), idesc, p == 0 ? acc : 1u);
                            const uint32_t x = (uint32_t)(blocks - 1) * block16 + a.operand[8];
                            tc_mma_i8(d, step(stage16, x, zero16 - stage16), desc_of(b + (uint32_t)(8 * (SLAB >> 4)), b_high), idesc, 1u);
                        }
                    }
                    else
                    {
                        const int slabs = blocks * a.taps;
                        int t = 0;
                        uint32_t cb16 = 0;
                        for (int s = 0; s < slabs; s += 2)
                        {
                            const uint32_t x0 = a.operand[t] + cb16;
                            if (++t == a.taps) { t = 0; cb16 += block16; }
                            const uint32_t x1 = s + 1 < slabs ? a.operand[t] + cb16 : zero16 - stage16;
                            if (++t == a.taps) { t = 0; cb16 += block16; }
                            tc_mma_i8(d, step(stage16, x0, x1), db + (uint64_t)(s * (SLAB >> 4)), idesc, s == 0 ? acc : 1u);
                        }
                    }
                    tc_commit(&empty[st]);
                    if (chunk == a.chunks - 1)
                        tc_commit(&acc_full[buf]);
                }
                __syncwarp();
                first = false;
                st += issuers;
                if (st >= a.stages) { st -= a.stages; turn ^= 1; }
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == EPI_WARPS + PROD_WARPS)
        tmem_dealloc(tmem, TMEM_COLS);
}

template <int NT, bool NINE>
int launch_patch(const PatchArgs &a, const uint8_t *in, const uint8_t *filt, const int32_t *bias, uint8_t *out, cudaStream_t st)
{
    auto kern = conv_u8_patch_kernel<NT, NINE>;
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
    const int nblocks = (a.K + NT - 1) / NT;
    int gx = std::max(1, num_sms() / nblocks);
    if (gx > a.tiles)
        gx = a.tiles;
    kern<<<dim3((unsigned)gx, (unsigned)nblocks), THREADS, a.smem, st>>>(a, in, filt, bias, out, status);
    return launched("conv_u8_patch_kernel");
}

// Shared memory of a plan with NT output channels a CTA; false if it does not fit.
bool fit(PatchArgs &a, int NT)
{
    const uint32_t block = (uint32_t)(a.planes * a.E * CB), slab_run = (uint32_t)(a.taps * SLAB), groups = NT / CB + 1;
    auto plan = [&](bool resident, int cc, int stages) {
        const unsigned long long filter = (unsigned long long)groups * slab_run * (resident ? a.cbs : cc);
        if (filter > SMEM_LIMIT || (unsigned long long)block * cc > SMEM_LIMIT) // (what follows is in 32 bits)
            return false;
        a.resident = resident; a.cc = cc; a.stages = stages; a.chunks = (a.cbs + cc - 1) / cc;
        a.run = slab_run * (uint32_t)(resident ? a.cbs : cc);
        a.patch_bytes = block * cc;
        a.stage_bytes = (a.patch_bytes + (resident ? 0 : groups * a.run) + 127) & ~127u;
        a.o_filter = a.stage_bytes * stages;
        a.o_table = a.o_filter + (resident ? groups * a.run : 0);
        a.o_table = (a.o_table + 15) & ~15u;
        a.o_zero = a.o_table + (uint32_t)a.units * 16; // behind every stage: a descriptor's distance is not negative
        a.smem = a.o_zero + BM * CB + 512;                            // an odd step reads a slab past its last one
        return a.smem <= (uint32_t)SMEM_LIMIT;
    };
    // Tiles of one stage: an even number of stages (see the issuers).
    if (plan(true, a.cbs, 4) || plan(true, a.cbs, 2))
        return true;
    for (int cc = (a.cbs - 1) & ~1; cc >= 2; cc -= 2)
        if (plan(true, cc, 3))
            return true;
    for (int cc = std::min(4, (a.cbs + 1) & ~1); cc >= 2; cc -= 2)
        for (int stages = 4; stages >= 3; --stages)
            if ((a.cbs > cc || stages == 4) && plan(false, cc, stages))
                return true;
    return plan(false, 2, 2);
}
// Where conv_u8_ring.cu is the shorter way.  Its tiles are 128 outputs each and no junk; here small images under large windows leave
// few outputs a tile, and a filter that does not stay is fetched for each of them again.
//   Cycles of a step of 32 bytes: here 100 a tile while the filter stays, else what its bytes take, by bulk copies or 16 at a time, but not
// less than 1.6 for every 16 bytes of pixels; there 800 for the first tile of an SM, which waits for its gathers, and 650 for a tile more, with
// zero points that want further columns 1350 and 1400 (to 1700); with some room for what this leaves out.
// us, there and here: 64 -> 64 7x7 with a stride of two at 8x17, 1024 images 55 and 113; 192 -> 192 3x3 / 2 at 20x11, 256 images 34 and 58;
// 192 -> 192 7x7 / 2 at 23x23, 64 images 130 and 152; 256 -> 256 1x3 / 2 at 8x8, 1024 images 18.6 and 24.4; but 96 -> 48 7x7 / 2 at
// 6x6, 1024 images 63 and 53.
//   Launches of a few steps: the sums of the filter, which padding with a byte other than zero needs, take longer than the ring's
// steps: 16 -> 32 1x3 / 2 at 25x19 4.2 and 5.2, 32 -> 16 2x2 / 2 at 7x9, 8 images 4.3 and 5.1; 16 -> 96 2x2 / 2 at 3x3, 16 images 5.5 and 5.0.
// Windows that meet a pixel once or twice, few channels: 32 -> 16 2x2 / 2 at 25x25, 1024 images 14.8 and 19.9, 32 -> 32 2x2 at 18x18, 256 images
// 9.1 and 10.7, 16 -> 64 2x2 at 11x11 (1.8 times as many tiles), 1024 images 15.2 and 17.7.
// Of 2000 random layers some 40 were slower here than there by more than 2 %, behind this line 6, by 9 % at most.
bool ring_is_shorter(const PatchArgs &a, int nt, const int32_t *bias)
{
    if ((reinterpret_cast<uintptr_t>(bias) & 15) != 0)
        return false; // which the ring does not take
    const bool plain = a.zero_filt == -128 && (a.zero_in == 0 || a.zero_in == -128);
    const int few = a.taps * ((a.cbs + 1) / 2); // the ring's steps
    const bool little = a.planes == 4 && few <= 6 && a.K <= 32;
    const int sms = num_sms(), blocks = (a.K + nt - 1) / nt, side = std::max(1, sms / blocks);
    const long long rounds = (a.tiles + side - 1) / side, ring = ((long long)a.N * a.Ho * a.Wo + BM - 1) / BM;
    if (rounds == 1)
        return plain && a.zero_in != 0 && ((a.K <= 64 && few <= 4) || little);
    if (plain && (little || (a.zero_in != 0 && few <= 4 && (a.planes == 4 || a.K <= 32))))
        return true;
    if (few <= 4 && a.tiles > 1.3 * ring)
        return true;
    const double step = a.resident ? 100. : a.in_order ? std::max(105., 2.5 * nt) : std::max(165., 4.2 * nt);
    const double here = rounds * std::max(step, 3.2 * a.units / a.taps), tiles = (double)ring * ((a.K + 127) / 128) / sms;
    return here > (plain ? std::max(840., 680. * tiles) : std::max(1750., 1800. * tiles));
}
} // namespace

namespace sb
{
// Returns -1 when the layer is not covered by this kernel, otherwise a SMALL_B200_* code.
int conv2d_u8_patch(const small_b200_layer *L, const uint8_t *in, const uint8_t *filt, const int32_t *bias, uint8_t *out, cudaStream_t st)
{
    PatchArgs a{};
    a.N = L->N; a.H = L->H; a.W = L->W; a.C = L->C; a.K = L->K; a.Fh = L->Fh; a.Fw = L->Fw;
    a.sw = L->stride; a.sh = row_stride(L); a.pad_t = L->pad_t; a.pad_l = L->pad_l;
    a.taps = a.Fh * a.Fw;
    if (L->accumulate || a.C % CB != 0 || a.K % CB != 0 || a.C <= 0 || a.K <= 0 || a.taps < 2 || a.taps > MAX_TAPS || a.sw < 1 || a.sw > 2 ||
        a.sh < 1 || a.sh > 2 || a.pad_t < 0 || a.pad_l < 0 || L->zero_in > 0 || L->zero_in < -255)
        return -1;
    if (((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(filt) | reinterpret_cast<uintptr_t>(out)) & 15) != 0)
        return -1;
    a.Ho = out_dim(a.H, L->pad_t, L->pad_b, a.Fh, a.sh);
    a.Wo = out_dim(a.W, L->pad_l, L->pad_r, a.Fw, a.sw);
    if (a.N <= 0 || a.Ho <= 0 || a.Wo <= 0)
        return SMALL_B200_OK;
    a.cbs = a.C / CB;
    if ((long long)a.C * a.H * a.W >= 1 << 30)
        return -1; // 32-bit offsets inside an image
    a.zero_in = L->zero_in; a.zero_filt = L->zero_filt;
    a.lshift = L->lshift; a.rshift = L->rshift; a.mult = L->multiplier; a.k_zero = L->k_zero;
    a.outside = (uint32_t)(-L->zero_in) * 0x01010101u;
    a.planes = a.sh * a.sw;
    // Outputs of a tile: the split of a row into parts, and the rows (or whole images) of such a part that fit 128 GEMM rows, which
    // leave the fewest tiles.
    const int more_r = (a.Fh - 1) / a.sh, more_c = (a.Fw - 1) / a.sw;
    long long best = -1;
    for (int parts = 1; parts <= a.Wo; ++parts)
    {
        const int TW = (a.Wo + parts - 1) / parts, PW = TW + more_c;
        if (TW > BM)
            continue;
        const int rows = (BM - TW) / PW + 1, TH = std::min(rows, a.Ho), RI = TH + more_r;
        int ni = parts == 1 && TH == a.Ho ? std::min((rows - TH) / RI + 1, a.N) : 1;
        ni = (int)std::min<long long>(ni, 0xffffffffll / ((long long)a.C * a.H * a.W)); // 32-bit offsets inside a tile's images
        const int tx = (a.Wo + TW - 1) / TW, ty = (a.Ho + TH - 1) / TH;
        const long long tiles = (long long)tx * ty * ((a.N + ni - 1) / ni);
        if (best >= 0 && tiles >= best)
        {
            if (TW <= 8)
                break;
            continue;
        }
        best = tiles;
        a.TW = TW; a.PW = PW; a.TH = TH; a.RI = RI; a.ni = ni; a.tiles_x = tx; a.tiles_y = ty;
    }
    if (best < 0 || best > 0x3fffffff)
        return -1;
    a.tiles = (int)best;
    a.rows_in = (a.TH - 1) * a.sh + a.Fh; a.cols_in = (a.TW - 1) * a.sw + a.Fw;
    a.units = a.ni * a.rows_in * a.cols_in;
    const int patch_rows = std::max(a.ni * a.RI, a.ni * ((a.rows_in + a.sh - 1) / a.sh));
    a.E = std::max(BM + more_r * a.PW + more_c, patch_rows * a.PW);
    if (a.planes * a.E > 0xffff)
        return -1;
    a.by_tiles_x.set(a.tiles_x); a.by_tiles_y.set(a.tiles_y); a.by_PW.set(a.PW); a.by_RI.set(a.RI); a.by_taps.set(a.taps);
    int order[MAX_TAPS], at[MAX_TAPS];
    for (int t = 0; t < a.taps; ++t)
    {
        const int kh = t / a.Fw, kw = t % a.Fw;
        order[t] = t;
        at[t] = ((kh % a.sh) * a.sw + kw % a.sw) * a.E + kh / a.sh * a.PW + kw / a.sw;
    }
    std::sort(order, order + a.taps, [&](int x, int y) { return at[x] < at[y]; });
    for (int r = 0; r < a.taps; ++r)
    {
        a.rank[order[r]] = (uint8_t)r;
        a.in_order = (r == 0 || a.in_order) && order[r] == r;
        a.operand[r] = (uint16_t)at[order[r]];
    }
    // As few blocks of output channels as possible (each fetches the pixels again), unless SMs would be left without a tile.
    int nt = 128;
    while (nt > 16 && (a.K + nt / 2 - 1) / (nt / 2) == (a.K + nt - 1) / nt)
        nt /= 2;
    while (nt > 16 && (long long)a.tiles * ((a.K + nt - 1) / nt) * 2 <= num_sms())
        nt /= 2;
    while (!fit(a, nt))
        if ((nt /= 2) < 16)
            return -1;
    if (ring_is_shorter(a, nt, bias))
        return -1;
#define SB_PATCH(NT_) return a.taps == 9 ? launch_patch<NT_, true>(a, in, filt, bias, out, st) : launch_patch<NT_, false>(a, in, filt, bias, out, st)
    switch (nt)
    {
    case 128: SB_PATCH(128);
    case 64: SB_PATCH(64);
    case 32: SB_PATCH(32);
    default: SB_PATCH(16);
    }
#undef SB_PATCH
}
} // namespace sb
