// conv_f16x3.cu -- fp32 dense convolution (stride 1) on the 5th-generation tensor cores, every fp32 operand as a
// pair of half-precision words with a block scale.
//
// Arithmetic.  v * 2^e = hi + lo * 2^-10 with hi = half(v * 2^e), lo = half((v * 2^e - hi) * 2^10), both truncated: 11 + 11
// bits, the very words of a 3xTF32 split (where the tensor core itself drops the low bits of a tf32 operand).  A product
// is a_lo*b_hi + a_hi*b_lo + a_hi*b_hi in fp32 tensor memory; the dropped a_lo*b_lo is below 2^-20 of it.  The cross terms are
// summed first, and the first a_hi*b_hi brings them down by 2^-10 (an operand of the instruction), or they have columns of
// their own.  Half precision has a narrow range, so the power of two 2^e belongs to a block.
//   * Filter: all of it, or one output channel where the filter's scale would take digits from one of its rows (a tap's
//     sixteen input channels).  A row keeps 22 bits of its largest weight, down to 2^-26 of the channel's largest; beneath
//     that an error below 2^-47 of the channel's largest is left.
//   * Activations: a tile's patch of 16 input channels.  Every pixel's sixteen values keep 22 bits of the largest of them,
//     however large the pixels beside it: the scale brings the patch's largest to 2^6 at least, 22 bits reach down
//     to 2^-13, a patch with a pixel below that gets the scale that brings its largest to 2^13, and a tile with a patch where
//     that does not do either is computed on the FMA pipe (plain_tile).
//   * An infinity is no pair (inf - inf): a tile with one in a patch goes the same way, and with one in the filter, or a NaN
//     (which the zeros of the padding must not meet), the layer does.  A NaN in the activations is its own pair.
// So an output channel, an image or a pixel is as good as if it stood alone: the words of a value that is in range do not
// depend on the power of two.  (With lo stored as it is, 22 bits ended at 2^-3 and an error of 2^-24 remained: an output channel 2^-12 of
// the largest kept half its digits.  All of this costs 0.5 to 1.5 %: Tiny-YOLOv2 on 64 images 1.625
// -> 1.635 ms, ResNet-8 on 1024 429 -> 435 us.)  Scales are undone in the FMA with which the
// accumulation warps add a partial sum to their fp32 registers.  kind::f16 covers 16 channels per instruction where
// kind::tf32 covers 8 at the same cost (N/2 cycles of the pipe, 128 + N operand rows of 32 bytes), so a layer needs half
// the instructions, half the operand traffic in shared memory and half the filter bytes of the 3xTF32 form this
// replaced: 1024 -> 1024 channels 3x3 on 64 images of 13x13 0.800 -> 0.439 ms, 16 -> 32 at 208x208 with the max
// pool 0.198 -> 0.168, 128 -> 256 at 26x26 0.122 -> 0.078.  Against fp64 the 9216-term sums of the first are off by
// 5.3e-7 of the largest (3xTF32: 7.3e-7; the fp32 loop nest of include/small/abstract_layer.hpp:1368-1823, whose
// FLOAT_CONV_TILE_C this replaces: 5.7e-6).
//
// GEMM orientation: D[k][pixel] = sum_c W[k][c] * X[pixel][c].  The output channels are the
// tensor core's M (one tile of 128, or 64 for layers with fewer channels), the pixels its N
// (64..256 per CTA); wide-N instructions are what keeps the pipe busy.  The tensor pipe bounds the wide layers (1024 -> 1024
// 3x3 on 16 images of 13x13: 89.6 % of the cycles an SM is active, L1 and shared memory 75 % of theirs), and on long runs the
// power cap.
//
// Layers with 16, 32 or 64 output channels turn the GEMM around (PIXM): 128 pixels are the M of one MMA
// and all output channels its N, D[pixel][k].  A thread of the accumulation warps owns one pixel with all
// its channels: its sums go to the packed output as 64-byte runs without any transposition.  Three threads issue
// the MMAs there.
// Variants of the pixel-major kernel (template arguments MERGED, POOL): for 16 / 32 output channels
// [W_hi | W_lo] is one operand of 2K columns (two MMAs per tap instead of three, TcArgs::merged); for 32 / 64 output
// channels on wide images a following 2x2 stride-2 max pool can run in the epilogue (TcArgs::pool).
//
// Implicit GEMM without im2col ("linear shift"):
//   For one image and one block of 16 input channels, TMA copies a patch of the packed
//   activations [rows][PW columns][16 ch] (64 bytes per pixel) into shared memory.
//   PW = W + max(pad_l, pad_r): the zero column(s) that TMA's out-of-bounds fill produces at the
//   left edge of every row also serve as the right padding of the row above.  Splitter warps turn every
//   64-byte row into its 32 bytes of hi and 32 bytes of lo halves, in place and in the 64-byte swizzle, and that IS a
//   K-major operand of the tensor core: rows of 64 bytes, 8-pixel groups 512 bytes apart; the hardware applies the
//   swizzle to absolute shared-memory addresses, so a descriptor may start at any pixel.  Output pixel (r, c) is GEMM
//   column m = r*PW + c, and filter tap (kh, kw) of that pixel sits at patch entry m + kh*PW + kw: consecutive pixels
//   are consecutive rows for EVERY tap, so a tap only moves the descriptor's start address by 64 bytes
//   per pixel.  Columns with c >= Wo are junk and are not stored.
//   The filter [K/16][C/16][tap][16 c][16 k] is re-laid once per set of weights into
//   [K/MT][C/16][tap][c/8][hi k | lo k][8 c] (prepare_filter_kernel), MT = output channels per CTA: the K-major
//   canonical layout, hi and lo rows of a chunk one behind the other.  The taps of a group are then one contiguous run
//   that arrives by one bulk copy.
#include "tc_common.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <cstring>

namespace
{
using namespace sb;

constexpr int W_STAGES_MAX = 6; // filter stages, each one group of taps (a kernel row)
__host__ __device__ constexpr int x_slots_max(bool merged) { return merged ? 4 : 3; }
constexpr int BOX_PX = 32; // widest box of a TMA load: 256 elements of 8 bytes
constexpr int WIDE_WORDS = 32; // a CTA's tiles, a bit each: a launch has at most 1024 for every CTA
constexpr int SCALE_RING = 16; // patches whose block scale is remembered: slots + unflushed accumulator buffers, rounded up

struct TcArgs
{
    int N, C, K, H, W, Ho, Wo, Fh, Fw, pad_t, pad_l;
    int cbs, taps;
    int PW, PR;        // patch width / rows
    int NPX;           // pixels (GEMM columns) per CTA: 64, 128, 192 or 256
    int px_tiles;      // CTAs along the pixel axis per image
    int tiled;         // 0: tiles are ranges of full-width rows; 1: TH x TW pixel tiles
    int TW, TH, tiles_x; // tiled mode: valid columns / rows of a tile, tiles per row of tiles
    int MT;            // output channels per CTA (tensor-core M): 128 or 64
    int WR;            // channel rows a filter stage has room for: MT, or K in pixel-major tiles (N = K rows are read)
    int k_tiles;       // ceil(K / MT)
    int x_slots, w_stages;
    int pixm;          // 1: pixels on the tensor core's M, output channels on its N (K = 32 or 64)
    int tbufs;         // accumulator buffers in tensor memory: 2, or 4 when 4 * NPX <= 512 columns
    int group;         // filter taps summed in tensor memory before a flush
    // 1x1 layers: `cg` channel blocks travel as ONE patch of cg planes and are summed in tensor memory
    // as if they were the cg taps of a kernel row (cbs and taps then count these bundles: cbs = C/16/cg,
    // taps = group = cg).  A group of a 1x1 layer would otherwise be six MMAs, a third of the hand-overs
    // between the roles that a 3x3 kernel row pays for eighteen.  tap_step: descriptor units (16 bytes)
    // between the operand positions of two taps of a group: 4 (one pixel) or one plane of the patch.
    int cg, tap_step;
    // Output addressing in floats: pixel (r, c) of channel block kb lies at kb * o_kb_stride +
    // r * o_row_stride + c * 16 behind the image's first element.  Normally Ho*Wo*16 and Wo*16.
    // rows_view: a 1x1 layer on small images (H*W <= 64) is planned as ONE image whose rows are the
    // images of the batch (N' = 1, H' = N, W' = H*W): a 1x1 layer has no neighbourhoods, so a tile may
    // run across images and no tile is mostly empty (a 3x3-pixel image would fill 9 of a tile's 64
    // columns).  Only the strides differ: input rows are a whole image apart, and so are output rows.
    int rows_view;
    long long o_kb_stride, o_row_stride;
    // How a patch is fetched.  0: one TMA box of PW pixels x PR rows (x cg planes), zeros outside the image.  1: runs of
    // consecutive pixels by untiled bulk copies (1x1 layers have no halo): one run per plane of a tile (tiled), or one per
    // image row (rows_view with rows wider than a box).  x_row / x_plane: floats from a row / plane to the next.
    int runs;
    long long x_row, x_plane;
    int accumulate, act;
    float slope;
    unsigned smem_bytes;
    unsigned stage_off;  // byte offset of the output staging rows (0: they alias the operand buffers)
    int total_tiles;     // N * px_tiles * k_tiles
    int persistent;      // 1: one CTA per SM walks over the tiles; 0: one tile per CTA
    int ksplit;          // > 1: a cluster of that many CTAs shares a tile, each reduces a part of the channel blocks
    int tile_base;       // first tile of this launch (a layer may run as two launches, see the launch code)
    int w_resident;      // 1: every group of a tile has a filter stage of its own, loaded once per CTA (see fit_rings)
    // 16 or 32 output channels: a pixel-major MMA takes [W_hi | W_lo] (the rows lie one behind the other in every
    // 8-channel chunk) as ONE operand of 2K columns (the MERGED kernel, see its issuer).
    int merged;
    int split_sets;      // sets of splitters, 1 or 2 (see want_two_sets); with two the number of patch slots is even
    // Windows of at most nine taps are summed WHOLE in tensor memory where the stages fit (group = taps: at most nine
    // full-size accumulations, as many as one kernel row of two-word tf32 operands used to need): one flush and
    // one round of hand-overs per patch instead of one per kernel row.  row_skip: descriptor units from the last
    // tap of a kernel row to the first tap of the next one, beyond the one-pixel step.
    int row_skip;
    // 1: a 2x2 stride-2 max pool follows in the epilogue (pixel-major tiled plans only); the output strides
    // then describe the pooled tensor and `stage_off` locates the exchange rows of the pooling step
    int pool;
    FastDiv by_px_tiles, by_N, by_tiles_x, by_PW;
};

// Output channels per CTA, a function of K alone so that filter preparation and the
// convolution agree.
__host__ __device__ inline int pick_mt(int K) { return K >= 128 ? 128 : 64; }

// What the word behind the largest magnitudes says: channels have scales of their own; sums are to be made on the FMA pipe.
constexpr uint32_t OWN_SCALES = 1, PLAIN_FILTER = 2;

// Magnitudes of the filter's finite values as bits (without the sign, floats compare like integers): of every output channel the
// largest, behind those the largest of all, the word above, a place for the filter's scale, and of every channel the
// least of a row's largest (a row: a slab's sixteen input channels; ones of zeros do not count), complemented: 0 is none.
// blockIdx.y: block of 16 channels, its values [slab][16 c][16 k]; a thread takes rows of one channel.
__global__ void __launch_bounds__(256) filter_max_kernel(int slabs, const float *__restrict__ w, uint32_t *__restrict__ top)
{
    const int K = gridDim.y * CB, k = blockIdx.y * CB + (threadIdx.x & 15);
    uint32_t m = 0, least = 0;
    for (int slab = blockIdx.x * 16 + (threadIdx.x >> 4); slab < slabs; slab += gridDim.x * 16)
    {
        const float *row = w + ((long long)blockIdx.y * slabs + slab) * CB * CB + (threadIdx.x & 15);
        uint32_t r = 0;
#pragma unroll
        for (int c = 0; c < CB; ++c)
        {
            const uint32_t b = __float_as_uint(__ldg(row + c * CB)) & 0x7fffffffu;
            if (b >= 0x7f800000u)
                top[K + 1] = PLAIN_FILTER;
            else
                r = max(r, b);
        }
        m = max(m, r);
        least = max(least, r ? ~r : 0u);
    }
    if (m)
    {
        atomicMax(top + k, m);
        atomicMax(top + K, m);
        atomicMax(top + K + 3 + k, least);
    }
}

// The second word of a pair is stored 2^LO_SHIFT times its value.  It is below an ulp of the first, 2^-10 of a value that
// half precision holds, so it stays below 65536 -- and keeps its 11 bits wherever the first word keeps its own.
constexpr int LO_SHIFT = 10;
constexpr float LO_UP = 1 << LO_SHIFT, LO_DOWN = 1.f / LO_UP;
// A pair has its 22 bits from FAINT = 2^-13 on: its last bit is then 2^-34, the least that the second word can hold.
constexpr float FAINT = 1.f / 8192;
// Magnitudes up to which a sum of 2^20 products stays finite, and with it what the tensor core makes of it: 2^45 for the
// filter, a scale of 2^-48 (magnitudes of 2^61 at least) for a patch.
constexpr uint32_t LARGE_FILTER = (127u + 45) << 23;
constexpr float LARGE_DOWN = 281474976710656.f; // 2^48
// The least inverse scale of a channel that is undone in one factor with the patch's (2^-110 at least): 2^-30, and 2^-20 with 32 output
// channels, where cross terms are added by a factor of their own, LO_DOWN times that product.
__device__ __forceinline__ float least_down(int K) { return K == 32 ? LO_UP / (1 << 30) : 1.f / (1 << 30); }
constexpr uint32_t FAINT_SEEN = 0x7fffffffu; // the splitters' word for a patch with a row below that

// Block scale of a set of operands whose largest magnitude has the bits `top`: the power of two that brings it
// into [2^13, 2^14), and its inverse.  Exponents are held to where both, and LO_UP times the first, are normal numbers.
__device__ __forceinline__ float scale_up(uint32_t top)
{
    const uint32_t e = max(top >> 23, 30u);
    return __uint_as_float((267u - e) << 23);
}
__device__ __forceinline__ float scale_down(uint32_t top)
{
    const uint32_t e = max(top >> 23, 30u);
    return __uint_as_float((e - 13u) << 23);
}

// packed filter [K/16][slab][16 c][16 k] -> half-precision pairs [K/MT][slab][c/8][hi kv | lo kv][8 c]; kv = MT
// except in a last, partial tile (K % MT channels).  down[k] = the inverse of channel k's block scale, down[2 K + 1] holds
// OWN_SCALES if it isn't the same for all of them (beside PLAIN_FILTER, set before), down[2 K + 2] = the inverse of the filter's scale.
__global__ void __launch_bounds__(256)
prepare_filter_kernel(long long n, int slabs, int MT, int K, const float *__restrict__ w, const uint32_t *__restrict__ top,
                      __half *__restrict__ pairs, float *__restrict__ down)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const int k16 = (int)(i & 15), c = (int)((i >> 4) & 15);
    const long long t = i >> 8;            // kb16 * slabs + slab
    const int slab = (int)(t % slabs);
    const int k = (int)(t / slabs) * 16 + k16;
    const int tile = k / MT;
    const int kv = (K - tile * MT) < MT ? (K - tile * MT) : MT;
    const long long o = ((long long)tile * MT * slabs * 16 + (long long)slab * kv * 16) * 2 +
                        (long long)(c >> 3) * kv * 16 + (long long)(k - tile * MT) * 8 + (c & 7);
    // The filter's scale, or the channel's own where one of its rows would be faint at the filter's.  Channels that share a
    // scale cost the pixel-major kernel nothing; one that does not, a multiplication per output.
    const uint32_t all = top[K], least = ~top[K + 3 + k];
    const bool own = top[k] && __uint_as_float(least) * scale_up(all) < FAINT;
    const uint32_t t0 = own ? top[k] : all;
    if (slab == 0 && c == 0)
    {
        down[k] = scale_down(t0);
        // What the two scales are together has to be a number, and what the sums are: channels so small (2^-17, or 2^-7) have theirs
        // undone apart from the patch's, and a filter so large (2^45) is left to the FMA pipe.
        if (own || (top[k] && down[k] < least_down(K)))
            atomicOr(reinterpret_cast<uint32_t *>(down) + 2 * K + 1, OWN_SCALES);
        if (top[k] >= LARGE_FILTER)
            atomicOr(reinterpret_cast<uint32_t *>(down) + 2 * K + 1, PLAIN_FILTER);
        if (k == 0)
            down[2 * K + 2] = scale_down(all);
    }
    const float v = w[i] * scale_up(t0);
    const __half h = __float2half_rz(v);
    pairs[o] = h;
    pairs[o + (long long)kv * 8] = fabsf(v) <= 65504.f ? __float2half_rz((v - __half2float(h)) * LO_UP) : __float2half_rz(0.f);
}

// Tensor-core accumulation truncates: every MMA adds into the fp32 accumulator with
// round-toward-zero, a one-sided error that grows with the number of accumulations (measured
// here: 3e-5 of the output range after 1700 MMAs).  So tensor memory only ever holds the sum
// of one group of taps (a window of up to nine, or a kernel row) of one channel block, its small cross terms first;
// eight accumulation warps pull these partial sums out with tcgen05.ld and add them into fp32 registers with
// round-to-nearest, while the tensor core already works on the next groups in the other
// accumulator buffers of tensor memory (two of 192 or 256 columns, four when a buffer needs at
// most 128).
//
// warp 0: TMA producer, warps 1..2 (pixel-major 1..3): MMA issuers, warps 4..11: accumulation +
// epilogue (lane quarter = warp % 4, pixel half = (warp - 4) / 4), warps 12..15: operand
// splitters, and in the MERGED kernels with two sets of them warps 16..19 (below).
//
// The unit of the filter pipeline is a GROUP of taps: one bulk copy and one
// tcgen05.commit, which frees the filter stage for the producer and hands the partial sums to
// the accumulation warps.
//
// MERGED kernels (16 or 32 output channels) can have a second set of splitters, warps 16..19: the sets take the patches in turn.  A
// set takes 2100 to 3700 cycles a patch, a chain of a few hundred instructions, where the MMAs of a tile need 1400 to 2000:
// with one set it was the splitters that such a layer waited for.
constexpr int ACC_WARPS = 8;
constexpr int FIRST_ACC_WARP = 4;
constexpr int FIRST_SPLIT_WARP = 12;
constexpr int SPLIT_THREADS = 128;
__host__ __device__ constexpr int num_threads(int split_sets) { return split_sets == 2 ? 640 : 512; }
constexpr int COLS_PER_THREAD = 128;
__host__ __device__ constexpr int num_issuers(bool pixm) { return pixm ? 3 : 2; } // they take groups in turn

// Two fp32 values times their block scale as two pairs of half-precision words: hi = v,
// lo = (v - hi) * 2^LO_SHIFT, both cut to 11 bits as a tf32 operand is.  (Rounded to nearest the 9216-term sums come out at 3.0e-7 of the
// largest instead of 5.3e-7, but then results drift from the 3xTF32 form's by more than either is off: 2.5e-5 of a
// YOLO head, whose box sizes are exponentials, against 2e-6 with the same words.)
// up_lo = up * LO_UP.  (v - hi) * LO_UP in one fma on the half-precision word itself: as many instructions as without the factor.
__device__ __forceinline__ void split2(float a, float b, float up, float up_lo, uint32_t &hi, uint32_t &lo)
{
    static_assert(LO_SHIFT == 10, "0xE400 is -2^10 in half precision");
    asm("{\n\t.reg .f32 x, y;\n\t.reg .f16 h, g, m;\n\t"
        "mul.rn.f32 x, %2, %4;\n\tmul.rn.f32 y, %3, %4;\n\tcvt.rz.f16x2.f32 %0, y, x;\n\t"
        "mov.b32 {h, g}, %0;\n\tmov.b16 m, 0xE400;\n\t"
        "mul.rn.f32 x, %2, %5;\n\tmul.rn.f32 y, %3, %5;\n\tfma.rn.f32.f16 x, h, m, x;\n\tfma.rn.f32.f16 y, g, m, y;\n\t"
        "cvt.rz.f16x2.f32 %1, y, x;\n\t}"
        : "=&r"(hi), "=r"(lo) : "f"(a), "f"(b), "f"(up), "f"(up_lo));
}
// Largest magnitude (as bits) of the finite ones among eight values; `inf` is set if there is an infinity among them.
__device__ __forceinline__ uint32_t finite_max(const float4 *v, bool &inf)
{
    const uint4 a = *reinterpret_cast<const uint4 *>(v), b = *reinterpret_cast<const uint4 *>(v + 1);
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        m = max(m, w[i] & 0x7fffffffu);
    if (m >= 0x7f800000u)
    {
        m = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
        {
            const uint32_t u = w[i] & 0x7fffffffu;
            inf = inf || u == 0x7f800000u;
            m = max(m, u < 0x7f800000u ? u : 0u);
        }
    }
    return m;
}
__device__ __forceinline__ float max_abs(const float4 v)
{
    return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
}
// Largest of the splitter threads' values; `words` is used again only after another call.
template <int SPLIT_SETS>
__device__ __forceinline__ uint32_t split_reduce(uint32_t m, uint32_t *words, int w, int lane, int set)
{
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0)
        words[w] = m;
    if (SPLIT_SETS == 1)
        asm volatile("bar.sync 2, 128;" ::: "memory");
    else
        asm volatile("bar.sync %0, 128;" ::"r"(2 + set) : "memory");
    const uint4 t = *reinterpret_cast<const uint4 *>(words);
    return max(max(t.x, t.y), max(t.z, t.w));
}
// U pieces of 8 channels (piece u = half u & 1 of patch row u / 2; u, u + 128, ...) into hi and lo halves, in place.
// Returns the largest magnitude of those that belong to the patch (`valid` rows of the first plane, `valid2` of the
// second, `entries` further on); `least` becomes the least bits - 1 of a piece's largest magnitude (a piece of zeros: 2^32 - 1).  Neither the reads nor the writes are predicated -- rows behind the patch hold whatever
// the slot held before and are never stored from -- because the predicates cost more than the work: 1090 cycles for
// 256 rows by four warps one predicated piece at a time, 950 four at a time, 440 without the predicates (shared memory
// delivers about 74 bytes per cycle to loads and stores, which makes 430 the floor).
template <int U>
__device__ __forceinline__ float split_pieces(float4 *piece, int u0, float up, uint32_t entries, int valid, int valid2, uint32_t &least)
{
    const float up_lo = up * LO_UP;
    float4 v[U][2];
    float fm = 0.f;
#pragma unroll
    for (int q = 0; q < U; ++q)
    {
        const int u = u0 + q * SPLIT_THREADS, late = (u >> 2) & 1;
        v[q][0] = piece[2 * u + late];
        v[q][1] = piece[2 * u + 1 - late];
    }
    __syncwarp(); // a row belongs to two lanes: both have read it
#pragma unroll
    for (int q = 0; q < U; ++q)
    {
        const int u = u0 + q * SPLIT_THREADS, sw = (u >> 2) & 3, late = sw & 1, h = u & 1, r = u >> 1;
        uint4 hi, lo; // of the chunks in the order they were read
        split2(v[q][0].x, v[q][0].y, up, up_lo, hi.x, lo.x);
        split2(v[q][0].z, v[q][0].w, up, up_lo, hi.y, lo.y);
        split2(v[q][1].x, v[q][1].y, up, up_lo, hi.z, lo.z);
        split2(v[q][1].z, v[q][1].w, up, up_lo, hi.w, lo.w);
        float top = fmaxf(max_abs(v[q][0]), max_abs(v[q][1]));
        top = (r < valid || (uint32_t)(r - (int)entries) < (uint32_t)valid2) ? top : 0.f;
        fm = fmaxf(fm, top);
        least = __viaddmin_u32(__float_as_uint(top), 0xffffffffu, least);
        uint4 *row = reinterpret_cast<uint4 *>(piece + (2 * u & ~3));
        // late rows: chunks read in the other order, lo half written first
        row[(h + 2 * late) ^ sw] = late ? make_uint4(lo.z, lo.w, lo.x, lo.y) : hi;
        row[(h + 2 - 2 * late) ^ sw] = late ? make_uint4(hi.z, hi.w, hi.x, hi.y) : lo;
    }
    return fm;
}

// What the rows (a pixel's sixteen channels) of a patch hold that are this thread's to look at: the largest finite
// magnitude, and the least bits - 1 of a row's largest one (2^32 - 1: none but zeros; 0 where there is an infinity, so that the
// row counts as faint).  Once per CTA, and for patches that do not fit the scale at hand.
__device__ __forceinline__ uint2 look_at_rows(const float4 *piece, int sid, int total, uint32_t entries, int valid, int valid2)
{
    uint2 seen = make_uint2(0u, 0xffffffffu);
    for (int u = sid; u < total; u += SPLIT_THREADS)
    {
        bool inf = false;
        uint32_t row = finite_max(piece + 2 * u, inf);
        row = max(row, __shfl_xor_sync(0xffffffffu, row, 1)); // the row's other piece
        if ((u >> 1) < valid || (uint32_t)((u >> 1) - (int)entries) < (uint32_t)valid2)
        {
            seen.x = max(seen.x, row);
            seen.y = min(seen.y, inf ? 0u : row - 1u);
        }
    }
    return seen;
}

// One tile of work: an image, a range of pixels and a block of MT output channels.
struct Tile
{
    int n, kt, kv;             // image, channel tile, channels this tile really has
    int row_base, col_base;    // first patch row / column in image coordinates (before padding)
    int m_local0;              // first GEMM column inside the patch
    int tw_valid, th_valid;    // real outputs per patch row / patch rows that hold outputs
};

__device__ __forceinline__ Tile decode_tile(const TcArgs &a, int t)
{
    // Pixel tile fastest, then the image, channel tile slowest.  The CTAs that run at the same time then
    // share one or two filter slices (a slice of a 1024 -> 1024 3x3 layer is 4.7 MB),
    // which stay in L2 while every image's tiles pass over them, and the activations of the whole batch
    // (44 MB there) stay in L2 from one slice to the next; neighbouring tiles of an image, whose patches
    // share their halo rows, still run side by side.  With the channel tile fastest, every 9 images streamed
    // all of the filter again (with tf32 words, 541 MB of DRAM reads for 126 MB of algorithmic bytes; 166 MB
    // now, and the layer 3 % faster).
    Tile T;
    const int t1 = a.by_px_tiles.div(t), pt = t - t1 * a.px_tiles;
    T.kt = a.by_N.div(t1);
    T.n = t1 - T.kt * a.N;
    if (!a.tiled)
    {
        const int m0 = pt * a.NPX;
        T.row_base = a.by_PW.div(m0); T.col_base = 0; T.m_local0 = m0 - T.row_base * a.PW;
        T.tw_valid = a.Wo; T.th_valid = a.Ho;
    }
    else
    {
        const int ty = a.by_tiles_x.div(pt), tx = pt - ty * a.tiles_x;
        T.row_base = ty * a.TH; T.col_base = tx * a.TW; T.m_local0 = 0;
        T.tw_valid = (a.Wo - T.col_base) < a.TW ? (a.Wo - T.col_base) : a.TW; T.th_valid = a.TH;
    }
    T.kv = (a.K - T.kt * a.MT) < a.MT ? (a.K - T.kt * a.MT) : a.MT;
    return T;
}

// A CTA walks over tiles blockIdx.x, blockIdx.x + gridDim.x, ...  With a grid of one CTA per SM the
// roles run ahead of one another across tile boundaries: the producer, the splitters and the MMA
// issuer start the next tile while the accumulation warps still write the previous one out, which
// hides the start-up and the epilogue of a tile (half the life of a CTA on layers with few channel
// blocks).  All ring positions and barrier phases therefore count patches and groups over the whole
// life of the CTA.  With one tile per CTA (grid = number of tiles) the loop runs once and the
// output staging may alias the operand buffers (stage_off = 0).
// PERSIST = false: exactly one tile per CTA, known at compile time.
#define SB_TILE_LOOP(cond_extra) \
    for (int t = first_tile, once_ = 0; (PERSIST ? (t < a.total_tiles) : (once_ == 0)) && (cond_extra); t += tile_step, ++once_)

// Sums of two output channels k, k + 1 at four outputs (r, c) of image n over the channel blocks (or bundles) [cb0, cb1),
// from the activations as they are and the filter's two words: fp32 products, sixteen to a sum, and those added up in fp64.
__device__ __forceinline__ void plain_sums(const TcArgs &a, const float *in, const __half *filt, const float *filt_down, int n, int k,
                                           const int *r, const int *c, int cb0, int cb1, float2 *out)
{
    const int kt = k / a.MT, kv = min(a.MT, a.K - kt * a.MT), taps = a.Fh * a.Fw;
    const __half *wq = filt + ((long long)kt * a.MT * a.cbs * a.taps + (long long)cb0 * a.taps * kv) * 32 + (k - kt * a.MT) * 8;
    const float2 down2 = __ldg(reinterpret_cast<const float2 *>(filt_down + k));
    const float down[2] = {down2.x, down2.y};
    double sum[4][2]; // [output][channel]
#pragma unroll
    for (int i = 0; i < 8; ++i)
        sum[i >> 1][i & 1] = 0.0;
#pragma unroll 1
    for (int step = 0; step < (cb1 - cb0) * a.taps; ++step, wq += kv * 32)
    {
        const int block = step / taps, tap = step - block * taps, kh = tap / a.Fw, kw = tap - kh * a.Fw;
        const float *plane = in + (long long)((n * a.cbs + cb0) * a.cg + block) * a.x_plane;
        const float4 *x[4];
        float part[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            const int row = r[i] + kh - a.pad_t, col = c[i] + kw - a.pad_l;
            const bool inside = (uint32_t)row < (uint32_t)a.H && (uint32_t)col < (uint32_t)a.W;
            x[i] = inside ? reinterpret_cast<const float4 *>(plane + (long long)row * a.x_row + (long long)col * CB) : nullptr;
            part[i][0] = part[i][1] = 0.f;
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) // four input channels
        {
            float4 v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                v[i] = x[i] ? __ldg(x[i] + h) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int q = 0; q < 2; ++q)
            {
                const uint2 *w = reinterpret_cast<const uint2 *>(wq + (h >> 1) * kv * 16 + q * 8 + (h & 1) * 4);
                const uint2 hi = __ldg(w), lo = __ldg(w + kv * 2);
                const float2 h0 = __half22float2(*reinterpret_cast<const __half2 *>(&hi.x)), h1 = __half22float2(*reinterpret_cast<const __half2 *>(&hi.y));
                const float2 l0 = __half22float2(*reinterpret_cast<const __half2 *>(&lo.x)), l1 = __half22float2(*reinterpret_cast<const __half2 *>(&lo.y));
                const float w0 = fmaf(l0.x, LO_DOWN, h0.x) * down[q], w1 = fmaf(l0.y, LO_DOWN, h0.y) * down[q];
                const float w2 = fmaf(l1.x, LO_DOWN, h1.x) * down[q], w3 = fmaf(l1.y, LO_DOWN, h1.y) * down[q];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    part[i][q] = fmaf(v[i].w, w3, fmaf(v[i].z, w2, fmaf(v[i].y, w1, fmaf(v[i].x, w0, part[i][q]))));
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (x[i]) // a tap in the padding adds nothing, whatever the filter holds
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    sum[i][q] += (double)part[i][q];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        out[i] = make_float2((float)sum[i][0], (float)sum[i][1]);
}
// The outputs of a tile that met a wide patch (see the splitters), by the accumulation warps on the FMA pipe: a thread makes two
// channels of four GEMM columns, 32 apart, or of the four pixels of a pooled one.  Such a tile takes 8 (16
// channels) to 140 times (1024) as long as another one: images whose pixels are 2^26 apart within a tile are not what this kernel is for, but their results
// are as good as any.  A launch with a split reduction leaves the sums of the CTA's channel blocks in its staging rows.
template <bool SPLIT, bool POOL>
__device__ __noinline__ void plain_tile(const TcArgs &a, const Tile T, const float *in, const __half *filt, const float *filt_down,
                                           const float *bias, float *out, float act_ns, int warp, int lane, int cb0, int cb1, float *stage, int pitch)
{
    const int cols = POOL ? a.PW >> 1 : a.PW, px = POOL ? (a.TH >> 1) * cols : a.NPX, each = POOL ? 32 : 128;
#pragma unroll 1
    for (int k = warp * 2; k < T.kv; k += ACC_WARPS * 2)
#pragma unroll 1
        for (int p0 = 0; p0 < px; p0 += each)
        {
            const int kg = T.kt * a.MT + k;
            int r[4], c[4];
            bool live[4];
            float2 v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
            {
                const int p = p0 + lane + (POOL ? 0 : 32 * i), ml = POOL ? p : T.m_local0 + p, rl = ml / cols, cl = ml - rl * cols;
                r[i] = T.row_base + (POOL ? 2 * rl + (i >> 1) : rl);
                c[i] = T.col_base + (POOL ? 2 * cl + (i & 1) : cl);
                live[i] = p < px && c[i] - T.col_base < T.tw_valid && (POOL || rl < T.th_valid) && r[i] < a.Ho;
                if (!live[i])
                    c[i] = -0x8000; // outside the image for every tap
            }
            plain_sums(a, in, filt, filt_down, T.n, kg, r, c, cb0, cb1, v);
            const float2 b = bias && cb0 == 0 ? __ldg(reinterpret_cast<const float2 *>(bias + kg)) : make_float2(0.f, 0.f);
            if (POOL)
                v[0] = make_float2(fmaxf(fmaxf(v[0].x, v[1].x), fmaxf(v[2].x, v[3].x)), fmaxf(fmaxf(v[0].y, v[1].y), fmaxf(v[2].y, v[3].y)));
#pragma unroll
            for (int i = 0; i < (POOL ? 1 : 4); ++i)
                if (live[i])
                {
                    float2 y = make_float2(v[i].x + b.x, v[i].y + b.y);
                    float2 *o = reinterpret_cast<float2 *>(stage + (size_t)(p0 + lane + 32 * i) * pitch + k);
                    if (!SPLIT)
                    {
                        o = reinterpret_cast<float2 *>(out + ((long long)T.n * (a.K / CB) + kg / CB) * a.o_kb_stride +
                                                       (long long)(POOL ? r[i] >> 1 : r[i]) * a.o_row_stride +
                                                       (long long)(POOL ? c[i] >> 1 : c[i]) * CB + kg % CB);
                        if (a.accumulate)
                            y = make_float2(y.x + o->x, y.y + o->y);
                        y = make_float2(apply_act_ns(y.x, act_ns), apply_act_ns(y.y, act_ns));
                    }
                    *o = y;
                }
        }
}

// LATE: the accumulation warps work out where their pixel goes behind the sums, and fetch nothing ahead (see the launch).
template <bool PERSIST, bool SPLIT, bool PIXM = false, bool MERGED = false, bool POOL = false, int SPLIT_SETS = 1, bool LATE = false>
__global__ void __launch_bounds__(num_threads(SPLIT_SETS), 1)
conv_f16x3_kernel(const __grid_constant__ CUtensorMap map_x, const float *__restrict__ in, const __half *__restrict__ filt,
                  const float *__restrict__ filt_down, const __grid_constant__ TcArgs a, const float *__restrict__ bias, float *__restrict__ out, int *status)
{
    constexpr int NUM_THREADS = num_threads(SPLIT_SETS), X_SLOTS_MAX = x_slots_max(MERGED);
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t x_full[X_SLOTS_MAX], x_ready[X_SLOTS_MAX], x_empty[X_SLOTS_MAX];
    __shared__ __align__(8) uint64_t w_full[W_STAGES_MAX], g_done[W_STAGES_MAX];
    __shared__ __align__(8) uint64_t t_full[4], t_empty[4];
    __shared__ __align__(8) uint64_t peer_staged, peer_done; // split reduction: hand-over between the two CTAs
    __shared__ uint32_t tmem_base_s;
    __shared__ __align__(8) uint64_t x_redo[SPLIT_SETS]; // a patch fetched again because its block scale did not fit
    __shared__ float patch_down[SCALE_RING];   // inverse of the block scale of each patch in flight
    static_assert(WIDE_WORDS == 32, "a lane each");
    __shared__ uint32_t wide_tiles[WIDE_WORDS]; // bit i: the CTA's tile i has a wide patch (see the splitters)
    __shared__ __align__(16) uint32_t split_top[SPLIT_SETS][3][4];      // the splitter warps' maxima of the patch at hand
    __shared__ int acc_failed; // an accumulation warp gave up on a wait: all eight leave at the same tile

    const uint32_t entries = (uint32_t)a.PR * a.PW;
    const uint32_t x_bytes = entries * 64 * (uint32_t)a.cg;     // one patch [plane][entry][16 floats]
    const uint32_t x_part = (x_bytes + 4095u) & ~4095u;         // a patch slot: whole passes of the splitters (64 rows each)
    uint8_t *sX = smem;                                              // [slot][entry][64 B, 64-byte swizzle]
    uint8_t *sW = sX + (size_t)a.x_slots * x_part;                  // [stage][tap in group][c/8][hi kv | lo kv][16 B]
    const uint32_t w_stage = (uint32_t)a.group * a.WR * 64;         // bytes of one filter stage

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint32_t tmem_cols = 32;
    while ((int)tmem_cols < (PIXM ? a.tbufs * (a.NPX >> 7) * a.K * (MERGED ? 2 : 1) : a.tbufs * a.NPX))
        tmem_cols <<= 1;

    // Split reduction (one tile per CTA only): the CTAs of a cluster take a part of the channel blocks each, leave their
    // sums in shared memory at the end, and each adds up and stores its share of the tile.
    constexpr bool split = SPLIT && !PERSIST;
    const int crank = split ? (int)cluster_ctarank() : 0, S = split ? a.ksplit : 1;
    const int cb_begin = split ? crank * a.cbs / S : 0;
    const int cbs_l = split ? (crank + 1) * a.cbs / S - cb_begin : a.cbs; // channel blocks this CTA reduces
    const int steps = a.cbs * a.taps;
    const int groups_per_cb = a.taps / a.group, groups = cbs_l * groups_per_cb;
    const int first_tile = a.tile_base + (split ? blockIdx.x / (unsigned)S : blockIdx.x), tile_step = gridDim.x;

    // patch number pc / group number gc count over every tile of this CTA
    // pixels of a tile's patch that a copy delivers, per plane: every entry of a box (zeros outside the image), or
    // what lies inside the image where the patch is fetched as runs
    auto patch_rows = [&](const Tile &T) -> int {
        if (!a.runs)
            return (int)entries;
        if (a.tiled)
            return min(a.PW, a.W - T.col_base);
        return min(a.PR, a.H - T.row_base) * a.PW;
    };
    auto fetch_patch = [&](const Tile &T, int cb, int slot, uint64_t *bar) {
        uint8_t *dst = sX + (size_t)slot * x_part;
        const int plane = (T.n * a.cbs + cb_begin + cb) * a.cg;
        if (!a.runs)
        {
            mbar_expect_tx(bar, x_bytes);
            tma_load_3d(dst, &map_x, (T.col_base - a.pad_l) * 8, T.row_base - a.pad_t, plane, bar);
            return;
        }
        const uint32_t bytes = (uint32_t)patch_rows(T) * 64;
        mbar_expect_tx(bar, bytes * (uint32_t)a.cg);
        for (int p = 0; p < a.cg; ++p)
        {
            const float *src = in + (long long)(plane + p) * a.x_plane + (long long)T.row_base * a.x_row + (long long)T.col_base * CB;
            uint8_t *d = dst + (size_t)p * entries * 64;
            if (a.tiled)
                tma_load_1d(d, src, bytes, bar);
            else
                for (uint32_t done = 0; done < bytes; done += (uint32_t)a.PW * 64, src += a.x_row)
                    tma_load_1d(d + done, src, (uint32_t)a.PW * 64, bar);
        }
    };
    auto issue_patch = [&](const Tile &T, int cb, int slot) { fetch_patch(T, cb, slot, &x_full[slot]); };
    auto reload_patch = [&](const Tile &, int t, int cb, int slot, uint64_t *redo) {
        fetch_patch(decode_tile(a, t), cb, slot, redo);
    };
    auto issue_filter = [&](const Tile &T, int g, int st) {
        // the group's taps are contiguous, [tap][c/8][hi kv | lo kv][8 c]: one run; a partial last tile (kv < MT)
        // simply is a shorter one, and the MMA descriptors take 2 * kv * 16 bytes as the chunk stride
        const size_t off = (size_t)T.kt * a.MT * steps * 32 + (size_t)(g + cb_begin * groups_per_cb) * a.group * T.kv * 32;
        mbar_expect_tx(&w_full[st], (uint32_t)a.group * T.kv * 64);
        tma_load_1d(sW + (size_t)st * w_stage, filt + off, (uint32_t)a.group * T.kv * 64, &w_full[st]);
    };

    if (warp == 0)
    {
        if (lane == 0)
        {
            acc_failed = 0;
            for (int i = 0; i < X_SLOTS_MAX; ++i)
            {
                mbar_init(&x_full[i], 1); mbar_init(&x_ready[i], 1); mbar_init(&x_empty[i], PIXM ? 3 : 2);
            }
            for (int i = 0; i < W_STAGES_MAX; ++i)
            {
                mbar_init(&w_full[i], 1); mbar_init(&g_done[i], 1);
            }
            for (int i = 0; i < 4; ++i) { mbar_init(&t_full[i], 1); mbar_init(&t_empty[i], ACC_WARPS); }
            for (int i = 0; i < SPLIT_SETS; ++i)
                mbar_init(&x_redo[i], 1);
            mbar_init(&peer_staged, ACC_WARPS * S); mbar_init(&peer_done, ACC_WARPS * S);
            fence_barrier_init();
            // The first patch and the first filter stage only need their barriers: their round
            // trip to memory overlaps the tensor-memory allocation and the CTA-wide barrier.
            const Tile T = decode_tile(a, first_tile);
            issue_patch(T, 0, 0);
            issue_filter(T, 0, 0);
        }
        __syncwarp();
        tmem_alloc(&tmem_base_s, tmem_cols);
        tmem_relinquish();
    }
    if (tid >= NUM_THREADS - WIDE_WORDS)
        wide_tiles[tid - (NUM_THREADS - WIDE_WORDS)] = 0;
    tc_fence_before_sync();
    if (split)
        cluster_sync_all(); // the peer's barriers exist before anybody can arrive on them
    else
        __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_base_s;

    if (warp < FIRST_ACC_WARP || warp >= FIRST_SPLIT_WARP)
    {
        // The launch has 512 x 128 registers; the roles' shares add up to that at most (setmaxnreg draws on nothing else):
        // 128 x 88 + 256 x 168 + 128 x 88, pixel-major tiles 128 x 112 + 256 x 144 + 128 x 112.  (The least share also bounds
        // the function that is called for wide tiles: with 88 for the issuing warps it and its callers spilled, 16 -> 32 channels at
        // 208x208 with the pool 186 us, 168 with 112.)
        if (SPLIT_SETS == 2 && warp >= FIRST_SPLIT_WARP)
            asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        else if (SPLIT_SETS == 2)
            asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
        else if (PIXM)
            asm volatile("setmaxnreg.dec.sync.aligned.u32 112;");
        else
            asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
        if (warp == 0 && lane == 0)
        {
            // ---------------- producer ----------------
            bool ok = true;
            // Patches run ahead of the filter stages where a slot is free: a patch is a tiled copy of
            // a few hundred 64-byte rows from memory and takes several thousand cycles, more than
            // the MMAs of a tile with one or two channel blocks.  The look-ahead never waits (a wait
            // here would hold back the filter stages); only the patch of the group at hand does.
            // The patch cursor (p_t, p_cb) walks the same (tile, channel block) sequence as everybody else.
            // Ring positions are counters that wrap (here and in the other roles): a division by a ring's depth is some
            // forty instructions of straight-line code in every step of every role.
            int pc = 1, q = 0;             // patches issued (patch 0 already is), patches the groups have entered
            int slot = a.x_slots > 1 ? 1 : 0; // where patch pc goes, and the parity of the slot's last release
            uint32_t freed = a.x_slots > 1 ? 1 : 0;
            int p_t = first_tile, p_cb = 1;
            Tile PT = decode_tile(a, p_t); // decoded once per tile
            auto step_cursor = [&]() {
                if (p_cb == cbs_l)
                {
                    p_cb = 0;
                    p_t += tile_step;
                    if (PERSIST && p_t < a.total_tiles)
                        PT = decode_tile(a, p_t);
                }
            };
            step_cursor();
            auto next_patch = [&]() {
                issue_patch(PT, p_cb, slot);
                ++pc;
                ++p_cb;
                if (++slot == a.x_slots) { slot = 0; freed ^= 1; }
                step_cursor();
            };
            int st = 0;
            uint32_t w_freed = 1; // parity of the filter stage's last release; the first round finds all stages free
            bool w_first = true, first = true;
            SB_TILE_LOOP(ok)
            {
                const Tile T = decode_tile(a, t);
                int in_cb = 0;
                for (int g = 0; g < groups && ok; ++g)
                {
                    if (in_cb == 0)
                    {
                        if (pc <= q) // the look-ahead has not reached this group's patch: now it must go
                        {
                            if (pc >= a.x_slots) // all issuers' MMAs on the slot's previous patch are done
                                ok = mbar_wait(&x_empty[slot], freed, status, 11);
                            if (!ok)
                                break;
                            next_patch();
                        }
                        ++q;
                    }
                    if (++in_cb == groups_per_cb)
                        in_cb = 0;
                    while (pc < q - 1 + a.x_slots && (PERSIST ? p_t < a.total_tiles : p_t == first_tile) &&
                           (pc < a.x_slots || mbar_test(&x_empty[slot], freed)))
                        next_patch();
                    if (a.w_resident && !w_first)
                        continue; // the whole filter is in shared memory since the CTA's first tile
                    if (!w_first)
                        ok = mbar_wait(&g_done[st], w_freed, status, 12);
                    if (!ok)
                        break;
                    if (!first) // filter stage 0 already is on its way
                        issue_filter(T, g, st);
                    first = false;
                    if (++st == a.w_stages) { st = 0; w_first = false; w_freed ^= 1; }
                }
            }
        }
        else if (warp >= 1 && warp <= (PIXM ? 3 : 2))
        {
            // ---------------- MMA issuers ----------------
            // All descriptor fields except the 16-byte-granular start address are fixed per CTA,
            // and a new operand position is one 64-bit add on a precomputed descriptor.  A = filter
            // tap (M = channels), B = patch shifted by the tap (N = pixels).
            // The warps stay together and an elected lane issues: the operands then live in uniform registers, 42 cycles for
            // an MMA of few columns where a lane on its own took 56 to 60 (ResNet-8 at 1024 images 440 -> 429 us).
            // Issuing one MMA costs a thread about as long as the tensor pipe needs for it
            // (measured: one thread sustains an N = 192 MMA every 122 cycles, the pipe takes 96;
            // two threads together reach the 96), and whatever the thread does between two groups
            // (three barrier waits of about 200 cycles each, the commit) is idle tensor time on top.
            // Two threads therefore take the groups in turn, one per tensor-memory buffer: while
            // one waits for its filter stage and its buffer, the other one's MMAs keep the pipe
            // busy.  The groups are independent sums, so the two threads need no order between them.
            // Pixel-major tiles (PIXM: M = 128 pixels, N = all 32 or 64 output channels) have cheap
            // MMAs (N/2 cycles each), so a third thread joins to keep up with the pipe.
            constexpr int NISS = num_issuers(PIXM);
            const int me = warp - 1; // this thread issues the groups with g % NISS == me
            int turn = 0;            // g % NISS
            const bool own_t_full = PIXM || a.tbufs > a.w_stages;
            const int mtiles = a.NPX >> 7; // PIXM: blocks of 128 pixels per tile
            const int tb_mask = a.tbufs - 1, tb_shift = a.tbufs == 4 ? 2 : 1; // group g sums in buffer g % tbufs
            bool ok = true;
            // patch: rows of 64 bytes (one pixel's 16 channels) in the 64-byte swizzle the bulk copy
            // wrote; 8-pixel groups are 512 bytes apart; a pixel further is 4 descriptor units
            const uint64_t x_desc_base = make_smem_desc(smem_u32(sX), 16, 512, 4);
            const uint32_t idesc = make_idesc(1 /*f32*/, 0 /*f16*/, 0 /*f16*/, 0 /*A K-major*/, 0 /*B K-major*/,
                                              PIXM ? 128u : (uint32_t)a.MT, PIXM ? (uint32_t)a.K : (uint32_t)a.NPX);
            const uint32_t idesc_wide = make_idesc(1, 0, 0, 0, 0, 128u, 2u * (uint32_t)a.K); // MERGED: N = [hi | lo]
            const uint64_t x_lo_off = 2; // a pixel's row: 32 bytes of hi halves, 32 bytes of lo halves
            const uint64_t tap_step = (uint64_t)a.tap_step;
            const uint64_t w_stage_step = (uint64_t)w_stage >> 4;
            const uint64_t x_slot_step = (uint64_t)x_part >> 4;
            int slot = 0, xphase = 0, st = 0, wphase = 0, g = 0; // g counts groups over all tiles
            uint64_t x_slot_off = 0, w_stage_off = 0;
            SB_TILE_LOOP(ok)
            {
                // Of a tile the issuing threads need only its first GEMM column inside the patch and the channels
                // of its channel tile; 2-D pixel tiles of a layer with one channel tile always start at column 0
                // with all K channels, and the decode (three integer divisions per tile, for every issuing
                // thread and every tile, its own or not) is issue time taken from the MMAs.
                Tile T;
                if (a.tiled && a.k_tiles == 1)
                {
                    T.m_local0 = 0; T.kv = a.K;
                }
                else
                    T = decode_tile(a, t);
                const uint64_t x_desc0 = x_desc_base + (uint64_t)T.m_local0 * 4;
                // filter stage: [tap][c/8][kv hi rows | kv lo rows][16 B], kv = channels of this tile
                const uint64_t w_desc0 = make_smem_desc(smem_u32(sW), (uint32_t)T.kv * 32, 128, 0);
                const uint64_t w_tap = (uint64_t)T.kv * 4, w_lo_off = (uint64_t)T.kv;
                for (int cb = 0; cb < cbs_l && ok; ++cb)
                {
                    ok = __all_sync(0xffffffffu, mbar_wait(&x_ready[slot], xphase, status, 13));
                    if (!ok)
                        break;
                    uint64_t x_row = x_desc0 + x_slot_off; // patch position of tap (kh, 0)
                    for (int gi = 0; gi < groups_per_cb && ok; ++gi, ++g)
                    {
                        if (turn == me)
                        {
                            // resident stages complete phase 0 once and stay there; every issuer still has
                            // to observe that itself the first time it uses a stage (with 1, 2, 4 or 5
                            // stages a stage is not always the same thread's), and a completed phase
                            // answers at once
                            ok = mbar_wait(&w_full[st], a.w_resident ? 0u : (uint32_t)wphase, status, 14);
                            if (ok && g > tb_mask)
                                ok = mbar_wait(&t_empty[g & tb_mask], ((g >> tb_shift) - 1) & 1, status, 16);
                            ok = __all_sync(0xffffffffu, ok);
                            if (!ok)
                                break;
                            tc_fence_after_sync();
                            if (elect_one())
                            {
                                uint64_t wh = w_desc0 + w_stage_off, xh = x_row;
                                if (PIXM && MERGED)
                                {
                                    // [W_hi | W_lo] is one operand of 2K columns: x_hi times it gives the hi*hi sums in
                                    // columns [0, K) and one cross term in [K, 2K), x_lo * W_hi adds the other cross
                                    // term there.  Two instructions per tap and 128 pixels instead of three, the 128-pixel
                                    // operand read from shared memory twice instead of three times, and the small terms
                                    // never meet a full-size accumulator; the accumulation warps add the two halves.
                                    const uint32_t d0 = tmem + (uint32_t)((g & tb_mask) * mtiles * 2 * a.K);
                                    int kw = 0;
                                    for (int tp = 0; tp < a.group; ++tp, wh += w_tap, xh += tap_step)
                                    {
                                        for (int mt = 0; mt < mtiles; ++mt)
                                        {
                                            const uint64_t xa = xh + (uint64_t)mt * 512;
                                            const uint32_t d = d0 + (uint32_t)(mt * 2 * a.K);
                                            tc_mma_f16(d, xa, wh, idesc_wide, tp == 0 ? 0u : 1u);
                                            tc_mma_f16(d + (uint32_t)a.K, xa + x_lo_off, wh, idesc, 1u);
                                        }
                                        if (++kw == a.Fw) // on to the next patch row (0 where a group is one row)
                                        {
                                            kw = 0;
                                            xh += (uint64_t)a.row_skip;
                                        }
                                    }
                                }
                                else if (PIXM)
                                {
                                    const uint32_t d0 = tmem + (uint32_t)((g & tb_mask) * mtiles * a.K);
                                    // The small cross terms of the whole group first, the hi*hi terms last: the
                                    // tensor core adds into its accumulator with truncation, an error of one ulp OF
                                    // THE ACCUMULATOR per MMA, so only the MMAs issued while it holds full-size sums
                                    // (one per tap instead of three) contribute a full-size error.
                                    uint64_t wh2 = wh, xh2 = xh;
                                    int kw = 0, kw2 = 0;
                                    for (int tp = 0; tp < a.group; ++tp, wh += w_tap, xh += tap_step)
                                    {
                                        const uint64_t wl = wh + w_lo_off;
                                        for (int mt = 0; mt < mtiles; ++mt)
                                        {
                                            const uint64_t xa = xh + (uint64_t)mt * 512; // 128 pixels on
                                            const uint32_t d = d0 + (uint32_t)(mt * a.K);
                                            tc_mma_f16(d, xa, wl, idesc, tp == 0 ? 0u : 1u);
                                            tc_mma_f16(d, xa + x_lo_off, wh, idesc, 1u);
                                        }
                                        if (++kw == a.Fw) { kw = 0; xh += (uint64_t)a.row_skip; }
                                    }
                                    // the cross terms are 2^LO_SHIFT times too large: the first of the others mends that
                                    for (int mt = 0; mt < mtiles; ++mt)
                                        tc_mma_f16_rescaled<LO_SHIFT>(d0 + (uint32_t)(mt * a.K), xh2 + (uint64_t)mt * 512, wh2, idesc);
                                    for (int tp = 1; tp < a.group; ++tp)
                                    {
                                        wh2 += w_tap; xh2 += tap_step;
                                        if (++kw2 == a.Fw) { kw2 = 0; xh2 += (uint64_t)a.row_skip; }
                                        for (int mt = 0; mt < mtiles; ++mt)
                                            tc_mma_f16(d0 + (uint32_t)(mt * a.K), xh2 + (uint64_t)mt * 512, wh2, idesc, 1u);
                                    }
                                }
                                else
                                {
                                    const uint32_t d = tmem + (uint32_t)((g & tb_mask) * a.NPX);
                                    uint64_t wh2 = wh, xh2 = xh; // cross terms first, hi*hi last (see the pixel-major loop)
                                    int kw = 0, kw2 = 0;
                                    for (int tp = 0; tp < a.group; ++tp, wh += w_tap, xh += tap_step)
                                    {
                                        tc_mma_f16(d, wh + w_lo_off, xh, idesc, tp == 0 ? 0u : 1u);
                                        tc_mma_f16(d, wh, xh + x_lo_off, idesc, 1u);
                                        if (++kw == a.Fw) { kw = 0; xh += (uint64_t)a.row_skip; }
                                    }
                                    tc_mma_f16_rescaled<LO_SHIFT>(d, wh2, xh2, idesc);
                                    for (int tp = 1; tp < a.group; ++tp)
                                    {
                                        wh2 += w_tap; xh2 += tap_step;
                                        if (++kw2 == a.Fw) { kw2 = 0; xh2 += (uint64_t)a.row_skip; }
                                        tc_mma_f16(d, wh2, xh2, idesc, 1u);
                                    }
                                }
                                // the stage is free for the producer and the group's partial sums are
                                // complete for the accumulation warps: one commit serves both while the
                                // accumulator ring is no deeper than the filter ring (a waiter must not fall
                                // two phases behind its barrier)
                                tc_commit(&g_done[st]);
                                if (own_t_full)
                                    tc_commit(&t_full[g & tb_mask]);
                            }
                            __syncwarp();
                        }
                        if (++turn == NISS)
                            turn = 0;
                        x_row += (uint64_t)(a.group == a.Fw ? a.PW : 1) * 4;
                        w_stage_off += w_stage_step;
                        if (++st == a.w_stages) { st = 0; wphase ^= 1; w_stage_off = 0; }
                    }
                    if (elect_one())
                        tc_commit(&x_empty[slot]); // all issuers: the slot is free once the MMAs of each are done
                    __syncwarp();
                    x_slot_off += x_slot_step;
                    if (++slot == a.x_slots) { slot = 0; xphase ^= 1; x_slot_off = 0; }
                }
            }
        }
        else if (warp >= FIRST_SPLIT_WARP)
        {
            // ---------------- operand splitters ----------------
            // The copy left rows of 64 bytes (16 channels of a pixel).  Each is replaced in place by its hi and lo
            // halves, 32 bytes each, in the 64-byte swizzle the MMAs read (16-byte chunk j of row i at chunk
            // j ^ ((i >> 1) & 3)).  A thread takes 8 channels at a time, neighbouring lanes a row; rows 2, 3 of every
            // four touch their two chunks in the other order, so that neither the reads nor the writes of a warp
            // meet in a bank.
            // The block scale: a CTA starts from its first patch's largest magnitude (brought to 2^13..2^14) and keeps the
            // power of two as long as every patch's largest scaled magnitude stays in [2^6, 65504); the pass that converts
            // also finds that magnitude.  (Finding it first took as long as the conversion: a second pass over shared
            // memory and a barrier in front of every patch.)  A patch outside the range is fetched and converted again, and so is
            // one with a faint piece, whose largest magnitude is not zero but below FAINT when scaled (pieces, not whole
            // rows: a row is two lanes').  Then rows are looked at: a patch with a faint row at the scale that is its
            // own, one 2^-26 of its largest, makes its tile a wide one.
            // Two sets take the patches in turn, each with a scale of its own; a slot is always the same set's, or, where their number is
            // odd, one set takes all patches.
            const int set = SPLIT_SETS > 1 ? (warp - FIRST_SPLIT_WARP) >> 2 : 0, sid = tid - (FIRST_SPLIT_WARP + 4 * set) * 32;
            const bool in_turn = SPLIT_SETS > 1 && !(a.x_slots & 1);
            bool ok = set == 0 || in_turn, known = false;
            int slot = 0, scale_at = 0, whose = 0;
            uint32_t phase = 0, turn = 0;
            uint32_t redone = 0;
            uint32_t limit = 0;
            float up = 1.f, down = 1.f;
            SB_TILE_LOOP(ok)
            {
                Tile T = {};
                if (a.runs)
                    T = decode_tile(a, t);
                const int valid = patch_rows(T), valid2 = a.cg > 1 ? valid : 0; // pixels of the first / second plane
                const int total = (int)(x_part >> 5); // pieces, whole passes of the warps: the slot has room for them
                for (int cb = 0; cb < cbs_l && ok; ++cb)
                {
                    if (in_turn)
                    {
                        const bool mine = whose == set;
                        whose ^= 1;
                        if (!mine)
                        {
                            scale_at = (scale_at + 1) % SCALE_RING;
                            if (++slot == a.x_slots) { slot = 0; phase ^= 1; }
                            continue;
                        }
                    }
                    ok = mbar_wait(&x_full[slot], phase, status, 17);
                    if (!ok)
                        break;
                    float4 *piece = reinterpret_cast<float4 *>(sX + (size_t)slot * x_part);
                    uint32_t m = 0;
                    for (int round = 0; round < 2; ++round)
                    {
                        if (!known)
                        {
                            const uint2 seen = look_at_rows(piece, sid, total, entries, valid, valid2);
                            m = seen.x;
                            m = split_reduce<SPLIT_SETS>(m, split_top[set][2], warp - FIRST_SPLIT_WARP - 4 * set, lane, set);
                            up = scale_up(m);
                            down = scale_down(m);
                            limit = down >= LARGE_DOWN ? 0u : 0xffffffffu;
                            if (!limit || (seen.y != 0xffffffffu && __uint_as_float(seen.y + 1u) * up < FAINT))
                                atomicOr(&wide_tiles[once_ >> 5], 1u << (once_ & 31));
                        }
                        float fm = 0.f;
                        uint32_t least = 0xffffffffu;
                        int base = sid;
                        constexpr int AT_ONCE = SPLIT_SETS == 2 ? 2 : 4; // (registers: two sets of splitters have 72 a thread)
                        for (; base + (AT_ONCE - 1) * SPLIT_THREADS < total; base += AT_ONCE * SPLIT_THREADS)
                            fm = fmaxf(fm, split_pieces<AT_ONCE>(piece, base, up, entries, valid, valid2, least));
                        for (; base < total; base += SPLIT_THREADS)
                            fm = fmaxf(fm, split_pieces<1>(piece, base, up, entries, valid, valid2, least));
                        fence_proxy_async();
                        const bool faint = least != 0xffffffffu && __uint_as_float(least + 1u) * up < FAINT;
                        m = split_reduce<SPLIT_SETS>(faint ? FAINT_SEEN : __float_as_uint(fm * up), split_top[set][turn], warp - FIRST_SPLIT_WARP - 4 * set, lane, set);
                        // 0: all zero; not below 65504: would have overflowed (or an infinity in the input, which no
                        // scale helps: it stays one), or a faint row was seen
                        if (!known || m == 0 || (m >= 0x42800000u && m < 0x477fe000u))
                            break;
                        if (sid == 0)
                            reload_patch(T, t, cb, slot, &x_redo[set]);
                        ok = mbar_wait(&x_redo[set], redone & 1, status, 18);
                        ++redone;
                        if (!ok)
                            break;
                        known = false;
                        m = 0;
                    }
                    known = m - 1u < limit; // an all-zero patch says nothing about the next one; a large one's scale is not kept
                    if (sid == 0)
                    {
                        patch_down[scale_at] = down;
                        mbar_arrive(&x_ready[slot]);
                    }
                    turn ^= 1;
                    scale_at = (scale_at + 1) % SCALE_RING;
                    if (++slot == a.x_slots) { slot = 0; phase ^= 1; }
                }
            }
        }
    }
    else
    {
        if (!PIXM)
            asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
        else if (SPLIT_SETS == 1)
            asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
        else
            asm volatile("setmaxnreg.inc.sync.aligned.u32 128;");
        const float act_ns = act_neg_scale(a.act, a.slope); // activation: v > 0 ? v : v * act_ns
        // Whether tile i of this CTA is wide; known when its last sums are.  What is stored for such a tile is overwritten at
        // the end, so it matters here only where the output is also an input.
        if (__ldg(reinterpret_cast<const uint32_t *>(filt_down) + 2 * a.K + 1) & PLAIN_FILTER)
        {
            wide_tiles[lane] = 0xffffffffu; // all of them; every warp for itself
            __syncwarp();
        }
        auto is_wide = [&](int i) { return ((*reinterpret_cast<volatile uint32_t *>(&wide_tiles[i >> 5]) >> (i & 31)) & 1u) != 0; };
        if (PIXM)
        {
            // ---------------- accumulation + epilogue, pixel-major ----------------
            // A thread owns one pixel (its tensor-memory lane) and all K <= 64 output channels of it:
            // the running sums need 64 registers, a flush is one or two loads, and the epilogue
            // writes 64 contiguous bytes per channel block straight from the registers (a warp
            // covers 32 consecutive pixels: no transposition through shared memory, no barrier).
            const bool own_scales = __ldg(reinterpret_cast<const uint32_t *>(filt_down) + 2 * a.K + 1) & OWN_SCALES;
            const float w_down = own_scales ? 1.f : __ldg(filt_down + 2 * a.K + 2);
            const int quarter = warp & 3, mt = (warp - FIRST_ACC_WARP) >> 2;
            const int mtiles = a.NPX >> 7;
            const bool active = mt < mtiles, sectors = whole_sectors(out);
            const size_t plane = (size_t)a.o_kb_stride;
            bool ok = true;
            int gc = 0, pc = 0; // groups flushed, patches they came from
            for (int t = first_tile, once_ = 0; (PERSIST ? (t < a.total_tiles) : (once_ == 0)) && ok; t += tile_step, ++once_, ++pc)
            {
                const Tile T = decode_tile(a, t);
                // the bias seeds the sums (these loads overlap the wait for the first group), unless channels have scales of their own
                constexpr int ACC = MERGED ? 32 : 64; // output channels a thread can hold
                float acc[ACC];
#pragma unroll
                for (int c4 = 0; c4 < ACC / 4; ++c4)
                {
                    const float4 b = (bias && !own_scales && c4 * 4 < a.K) ? __ldg(reinterpret_cast<const float4 *>(bias) + c4)
                                                                           : make_float4(0.f, 0.f, 0.f, 0.f);
                    acc[4 * c4] = b.x; acc[4 * c4 + 1] = b.y; acc[4 * c4 + 2] = b.z; acc[4 * c4 + 3] = b.w;
                }
                int rl, cl, r, c; // this thread's pixel, of the patch and of the output
                bool live;
                float *o;
                auto locate = [&]() {
                    const int ml = T.m_local0 + mt * 128 + quarter * 32 + lane;
                    rl = a.by_PW.div(ml); cl = ml - rl * a.PW; r = T.row_base + rl; c = T.col_base + cl;
                    live = !POOL && active && cl < T.tw_valid && rl < T.th_valid && r < a.Ho;
                    o = out + (size_t)T.n * (a.K / CB) * plane + (size_t)r * a.o_row_stride + (size_t)c * CB;
                };
                if (!LATE)
                {
                    locate();
                    if (!POOL && a.accumulate && live) // on its way to L2 while the sums are made
                        for (int kb = 0; kb * CB < a.K; ++kb)
                            asm volatile("prefetch.global.L2 [%0];" ::"l"(o + (size_t)kb * plane));
                }
                int in_cb = 0;
                for (int g = 0; g < groups && ok; ++g, ++gc)
                {
                    if (in_cb == groups_per_cb) { in_cb = 0; ++pc; }
                    ++in_cb;
                    const int tb = gc & 3;
                    ok = mbar_wait(&t_full[tb], (gc >> 2) & 1, status, 15, 1u << 24);
                    if (!ok)
                        break;
                    tc_fence_after_sync();
                    // the group's sums are those of operands scaled by powers of two: undone here, in the same FMA
                    const float down = *reinterpret_cast<volatile float *>(&patch_down[pc % SCALE_RING]) * w_down;
                    if (active)
                    {
                        const uint32_t tbase = tmem + ((uint32_t)(quarter * 32) << 16) +
                                               (uint32_t)((tb * mtiles + mt) * a.K * (MERGED ? 2 : 1));
                        if (MERGED)
                        {
                            // columns [0, K): the hi*hi sums, [K, 2K): the cross terms of the same channels
                            uint32_t v[32];
                            tmem_ld32(tbase, v);
                            tmem_ld_wait();
                            if (a.K == 16)
                            {
#pragma unroll
                                for (int e = 0; e < 16; ++e)
                                    acc[e] = fmaf(fmaf(__uint_as_float(v[16 + e]), LO_DOWN, __uint_as_float(v[e])), down, acc[e]);
                            }
                            else
                            {
#pragma unroll
                                for (int e = 0; e < 32; ++e)
                                    acc[e] = fmaf(__uint_as_float(v[e]), down, acc[e]);
                                tmem_ld32(tbase + 32u, v);
                                tmem_ld_wait();
#pragma unroll
                                for (int e = 0; e < 32; ++e)
                                    acc[e] = fmaf(__uint_as_float(v[e]), down * LO_DOWN, acc[e]);
                            }
                        }
                        else // K = 64
                        {
#pragma unroll
                        for (int piece = 0; piece < 2; ++piece)
                            if (piece * 32 < a.K)
                            {
                                uint32_t v[32];
                                tmem_ld32(tbase + (uint32_t)(piece * 32), v);
                                tmem_ld_wait();
#pragma unroll
                                for (int e = 0; e < 32; ++e)
                                    acc[piece * 32 + e] = fmaf(__uint_as_float(v[e]), down, acc[piece * 32 + e]);
                            }
                        }
                    }
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(&t_empty[tb]);
                }
                if (LATE)
                    locate();
                if (own_scales)
#pragma unroll
                    for (int c4 = 0; c4 < ACC / 4; ++c4)
                        if (c4 * 4 < a.K)
                        {
                            const float4 b = bias ? __ldg(reinterpret_cast<const float4 *>(bias) + c4) : make_float4(0.f, 0.f, 0.f, 0.f);
                            const float4 d = __ldg(reinterpret_cast<const float4 *>(filt_down) + c4);
                            acc[4 * c4] = fmaf(acc[4 * c4], d.x, b.x); acc[4 * c4 + 1] = fmaf(acc[4 * c4 + 1], d.y, b.y);
                            acc[4 * c4 + 2] = fmaf(acc[4 * c4 + 2], d.z, b.z); acc[4 * c4 + 3] = fmaf(acc[4 * c4 + 3], d.w, b.w);
                        }
                if (POOL)
                {
                    // 2x2 max pool, stride 2, on the sums in registers (K = 32 or 64: a thread holds ACC = K
                    // sums).  Tiles have even heights and widths and an even patch width, so the horizontal
                    // neighbour of pixel (rl, cl) is the next lane of the same warp: the even lane of a pair keeps
                    // the lower half of the channels of BOTH pixels' maximum, the odd lane the upper half (one
                    // shuffle per kept channel).  The vertical neighbour is PW lanes further on, in another warp:
                    // odd rows leave their halves in shared memory, even rows pick them up behind a barrier of the
                    // eight accumulation warps, apply the activation (monotonic, so it commutes with the maximum;
                    // the launch code checks that) and store their half of the pooled pixel.  A first barrier
                    // keeps a warp from writing into the exchange rows while a slower one still reads the previous
                    // tile's.  Every instruction here competes with the MMA-issuing threads for the issue slots of
                    // the four schedulers, which is why the work is split between the lanes of a pair.
                    // Every warp comes to the first barrier at every tile; a warp whose wait ran out says so
                    // before it and all leave together (see the channel-major epilogue).
                    constexpr int HALF = ACC / 2;
                    const int upper = lane & 1;
                    float *xrow = reinterpret_cast<float *>(smem + a.stage_off) +
                                  ((size_t)(rl >> 1) * (a.PW >> 1) + (cl >> 1)) * (ACC + 4) + upper * HALF;
                    if (!ok)
                        *reinterpret_cast<volatile int *>(&acc_failed) = 1;
                    asm volatile("bar.sync 1, 256;" ::: "memory");
                    if (*reinterpret_cast<volatile int *>(&acc_failed))
                        ok = false;
                    if (ok)
                    {
                        float keep[HALF];
                        if (active)
                        {
#pragma unroll
                            for (int e = 0; e < HALF; ++e)
                            {
                                const float mine = upper ? acc[HALF + e] : acc[e], theirs = upper ? acc[e] : acc[HALF + e];
                                keep[e] = fmaxf(mine, __shfl_xor_sync(0xffffffffu, theirs, 1));
                            }
                            if ((rl & 1) && rl < a.TH)
                            {
#pragma unroll
                                for (int j = 0; j < HALF / 4; ++j)
                                    reinterpret_cast<float4 *>(xrow)[j] = make_float4(keep[4 * j], keep[4 * j + 1], keep[4 * j + 2], keep[4 * j + 3]);
                            }
                        }
                        asm volatile("bar.sync 1, 256;" ::: "memory");
                        const int c0 = T.col_base + (cl & ~1);
                        if (active && !(rl & 1) && (cl & ~1) < T.tw_valid && rl < a.TH && r < a.Ho)
                        {
                            float *o = out + ((size_t)T.n * (a.K / CB) + (size_t)upper * (HALF / CB)) * plane +
                                       (size_t)(r >> 1) * a.o_row_stride + (size_t)(c0 >> 1) * CB;
#pragma unroll
                            for (int j = 0; j < HALF / 4; ++j)
                            {
                                const float4 y = reinterpret_cast<const float4 *>(xrow)[j]; // row rl + 1 shares the slot
                                keep[4 * j] = apply_act_ns(fmaxf(keep[4 * j], y.x), act_ns);
                                keep[4 * j + 1] = apply_act_ns(fmaxf(keep[4 * j + 1], y.y), act_ns);
                                keep[4 * j + 2] = apply_act_ns(fmaxf(keep[4 * j + 2], y.z), act_ns);
                                keep[4 * j + 3] = apply_act_ns(fmaxf(keep[4 * j + 3], y.w), act_ns);
                                if (j & 1)
                                    store8(o + (size_t)(j >> 2) * plane + (j & 2) * 4, keep + 4 * j - 4, sectors);
                            }
                        }
                    }
                }
                else if (ok && live && !(a.accumulate && is_wide(once_)))
                {
                    if (a.accumulate)
#pragma unroll
                        for (int c4 = 0; c4 < ACC / 4; ++c4)
                            if (c4 * 4 < a.K)
                            {
                                const float4 old = *(reinterpret_cast<const float4 *>(o + (size_t)(c4 >> 2) * plane) + (c4 & 3));
                                acc[4 * c4] += old.x; acc[4 * c4 + 1] += old.y; acc[4 * c4 + 2] += old.z; acc[4 * c4 + 3] += old.w;
                            }
#pragma unroll
                    for (int k8 = 0; k8 < ACC / 8; ++k8)
                        if (k8 * 8 < a.K)
                        {
#pragma unroll
                            for (int e = 0; e < 8; ++e)
                                acc[8 * k8 + e] = apply_act_ns(acc[8 * k8 + e], act_ns);
                            store8(o + (size_t)(k8 >> 1) * plane + (k8 & 1) * 8, acc + 8 * k8, sectors);
                        }
                }
            }
        }
        else
        {
        // ---------------- accumulation + epilogue ----------------
        const int quarter = warp & 3;                    // TMEM lanes [32*quarter, 32*quarter+32)
        const int phalf = (warp - FIRST_ACC_WARP) >> 2;  // which half of the tile's pixels
        const int my_cols = a.NPX / 2;                   // 32, 64, 96 or 128
        const int col0 = phalf * my_cols;
        // 128-channel tile: lane l of quarter q holds channel 32q + l; 64-channel tile: channel
        // 16q + l in lanes 0..15 of each quarter
        const int k_local = (a.MT == 128) ? quarter * 32 + lane : quarter * 16 + lane;
        const bool lane_has_row = (a.MT == 128) || (lane < 16);
        // Output staging rows of MT + 16 floats (free of bank conflicts both for the channel-wise
        // writes and for the float4 reads); a persistent CTA stages 32 pixels of each half at a time.
        const int pitch = a.MT + 16;
        float *stage = reinterpret_cast<float *>(smem + a.stage_off);
        const int psub = lane >> 2, q4 = lane & 3; // 8 pixels x 4 float4 per warp and step
        const size_t plane = (size_t)a.o_kb_stride;
        bool ok = true;
        int gc = 0, pc = 0; // groups flushed, patches they came from
        int st = 0;
        uint32_t st_phase = 0;
        for (int t = first_tile, once_ = 0; (PERSIST ? (t < a.total_tiles) : (once_ == 0)) && ok; t += tile_step, ++once_, ++pc)
        {
            const Tile T = decode_tile(a, t);
            // the bias of this thread's channel seeds its sums (rank 0 only when several CTAs share a tile)
            const bool has_channel = lane_has_row && k_local < T.kv;
            const float seed = (bias && crank == 0 && has_channel) ? __ldg(bias + T.kt * a.MT + k_local) : 0.f;
            const float w_down = has_channel ? __ldg(filt_down + T.kt * a.MT + k_local) : 0.f;
            float acc[COLS_PER_THREAD];
#pragma unroll
            for (int c = 0; c < COLS_PER_THREAD; ++c)
                acc[c] = 0.f;
            int in_cb = 0;
            for (int g = 0; g < groups && ok; ++g, ++gc)
            {
                if (in_cb == groups_per_cb) { in_cb = 0; ++pc; }
                ++in_cb;
                const int tb = gc & (a.tbufs - 1);
                if (a.tbufs > a.w_stages)
                    ok = mbar_wait(&t_full[tb], (gc >> (a.tbufs == 4 ? 2 : 1)) & 1, status, 15, 1u << 24);
                else
                    {
                    ok = mbar_wait(&g_done[st], st_phase, status, 15, 1u << 24);
                    if (++st == a.w_stages) { st = 0; st_phase ^= 1; }
                }
                if (!ok)
                    break;
                tc_fence_after_sync();
                const float down = *reinterpret_cast<volatile float *>(&patch_down[pc % SCALE_RING]);
                const uint32_t tbase = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(tb * a.NPX + col0);
#pragma unroll
                for (int piece = 0; piece < COLS_PER_THREAD / 32; ++piece)
                {
                    if (piece * 32 < my_cols)
                    {
                        uint32_t v[32];
                        tmem_ld32(tbase + (uint32_t)(piece * 32), v);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 32; ++e)
                            acc[piece * 32 + e] = fmaf(__uint_as_float(v[e]), down, acc[piece * 32 + e]);
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(&t_empty[tb]);
            }
            // Epilogue (the other roles are already at work on the next tile): a thread owns one
            // channel of up to 128 pixels, the packed output wants 16 channels of one pixel together.
            const int kbs = T.kv / CB; // channel blocks this tile really has
            float *obase = out + ((size_t)T.n * (a.K / CB) + (size_t)T.kt * (a.MT / CB)) * plane + q4 * 4;
            if (!PERSIST)
            {
                // one tile per CTA: every operand buffer is dead, the whole tile is staged at once
                if (ok && lane_has_row)
                {
                    float *srow = stage + (size_t)col0 * pitch + k_local;
                    if (a.MT == 128)
                    {
#pragma unroll
                        for (int e = 0; e < COLS_PER_THREAD; ++e)
                            if (e < my_cols)
                                srow[e * 144] = fmaf(acc[e], w_down, seed);
                    }
                    else
                    {
#pragma unroll
                        for (int e = 0; e < COLS_PER_THREAD; ++e)
                            if (e < my_cols)
                                srow[e * 80] = fmaf(acc[e], w_down, seed);
                    }
                }
                asm volatile("bar.sync 1, 256;" ::: "memory"); // the eight accumulation warps
                if (split && ok && is_wide(0))
                {
                    // this CTA's part of the sums, in place of what it staged (each wide CTA of the cluster its own)
                    plain_tile<true, false>(a, T, in, filt, filt_down, bias, out, act_ns, warp - FIRST_ACC_WARP, lane, cb_begin, cb_begin + cbs_l, stage, pitch);
                    __syncwarp();
                }
                if (split)
                {
                    // Every warp tells every CTA of the cluster that its sums are staged; when all have, the units of the
                    // tile (8 pixels x 16 channels) go round over the warps of the cluster, each of which adds up the
                    // S staged parts in rank order and stores.  Nobody leaves before all have read.
                    if (lane < S)
                    {
                        asm volatile("fence.acq_rel.cluster;" ::: "memory");
                        mbar_arrive_remote(map_to_cta(&peer_staged, (uint32_t)lane));
                    }
                    __syncwarp();
                    ok = mbar_wait_cluster(&peer_staged, 0, status, 20) && ok;
                    const int pgs = a.NPX / 8, units = pgs * kbs;
                    for (int u = crank * ACC_WARPS + warp - FIRST_ACC_WARP; ok && u < units; u += S * ACC_WARPS)
                    {
                        const int kb = u / pgs, px = (u - kb * pgs) * 8 + psub;
                        const int ml = T.m_local0 + px;
                        const int rl = a.by_PW.div(ml), cl = ml - rl * a.PW;
                        const int r = T.row_base + rl, c = T.col_base + cl;
                        if (cl < T.tw_valid && rl < T.th_valid && r < a.Ho)
                        {
                            const float *sp = stage + (size_t)px * pitch + kb * CB + q4 * 4;
                            float4 part[8]; // all loads out together: a round trip to another SM takes about 1000 cycles
#pragma unroll
                            for (int q = 0; q < 8; ++q)
                                if (q < S)
                                    part[q] = ld_cluster_f4(map_to_cta(sp, (uint32_t)q));
                            float4 x = part[0];
#pragma unroll
                            for (int q = 1; q < 8; ++q)
                                if (q < S)
                                {
                                    x.x += part[q].x; x.y += part[q].y; x.z += part[q].z; x.w += part[q].w;
                                }
                            float *o = obase + (size_t)r * a.o_row_stride + (size_t)c * CB + (size_t)kb * plane;
                            if (a.accumulate)
                            {
                                const float4 s4 = *reinterpret_cast<const float4 *>(o);
                                x.x += s4.x; x.y += s4.y; x.z += s4.z; x.w += s4.w;
                            }
                            x.x = apply_act_ns(x.x, act_ns); x.y = apply_act_ns(x.y, act_ns);
                            x.z = apply_act_ns(x.z, act_ns); x.w = apply_act_ns(x.w, act_ns);
                            *reinterpret_cast<float4 *>(o) = x;
                        }
                    }
                    __syncwarp();
                    if (lane < S)
                        mbar_arrive_remote(map_to_cta(&peer_done, (uint32_t)lane));
                    __syncwarp();
                    mbar_wait_cluster(&peer_done, 0, status, 21);
                }
                else if (ok && !(a.accumulate && is_wide(0)))
                {
                    for (int pg = warp - FIRST_ACC_WARP; pg < a.NPX / 8; pg += ACC_WARPS)
                    {
                        const int px = pg * 8 + psub;
                        const int ml = T.m_local0 + px;
                        const int rl = a.by_PW.div(ml), cl = ml - rl * a.PW;
                        const int r = T.row_base + rl, c = T.col_base + cl;
                        if (cl < T.tw_valid && rl < T.th_valid && r < a.Ho)
                        {
                            const float *sp = stage + (size_t)px * pitch + q4 * 4;
                            float *o = obase + (size_t)r * a.o_row_stride + (size_t)c * CB;
#pragma unroll
                            for (int kb = 0; kb < 8; ++kb)
                              if (kb < kbs)
                            {
                                float4 x = *reinterpret_cast<const float4 *>(sp + kb * CB);
                                float *ok_ = o + (size_t)kb * plane;
                                if (a.accumulate)
                                {
                                    const float4 s4 = *reinterpret_cast<const float4 *>(ok_);
                                    x.x += s4.x; x.y += s4.y; x.z += s4.z; x.w += s4.w;
                                }
                                x.x = apply_act_ns(x.x, act_ns); x.y = apply_act_ns(x.y, act_ns);
                                x.z = apply_act_ns(x.z, act_ns); x.w = apply_act_ns(x.w, act_ns);
                                *reinterpret_cast<float4 *>(ok_) = x;
                            }
                        }
                    }
                }
            }
            else
            {
#pragma unroll
            for (int piece = 0; piece < COLS_PER_THREAD / 32; ++piece)
            {
                if (piece * 32 < my_cols) // uniform over the CTA
                {
                    if (ok && lane_has_row)
                    {
                        float *srow = stage + (size_t)(phalf * 32) * pitch + k_local;
                        if (a.MT == 128)
                        {
#pragma unroll
                            for (int e = 0; e < 32; ++e)
                                srow[e * 144] = fmaf(acc[piece * 32 + e], w_down, seed);
                        }
                        else
                        {
#pragma unroll
                            for (int e = 0; e < 32; ++e)
                                srow[e * 80] = fmaf(acc[piece * 32 + e], w_down, seed);
                        }
                    }
                    // The give-up decision is made for the CTA, not per warp: the named barrier below
                    // needs all eight warps at every tile, so a warp whose wait ran out says so before
                    // the barrier and everybody reads it after, and all leave the tile loop together.
                    if (!ok)
                        *reinterpret_cast<volatile int *>(&acc_failed) = 1;
                    asm volatile("bar.sync 1, 256;" ::: "memory"); // the eight accumulation warps
                    if (*reinterpret_cast<volatile int *>(&acc_failed))
                        ok = false;
                    if (ok && !(a.accumulate && is_wide(once_)))
                    {
                        // staged row s holds pixel (s / 32) * my_cols + piece * 32 + s % 32 of the tile
                        const int s_row = (warp - FIRST_ACC_WARP) * 8 + psub;
                        const int px = (s_row >> 5) * my_cols + piece * 32 + (s_row & 31);
                        const int ml = T.m_local0 + px;
                        const int rl = a.by_PW.div(ml), cl = ml - rl * a.PW;
                        const int r = T.row_base + rl, c = T.col_base + cl;
                        if (cl < T.tw_valid && rl < T.th_valid && r < a.Ho)
                        {
                            const float *sp = stage + (size_t)s_row * pitch + q4 * 4;
                            float *o = obase + (size_t)r * a.o_row_stride + (size_t)c * CB;
#pragma unroll
                            for (int kb = 0; kb < 8; ++kb)
                              if (kb < kbs)
                            {
                                float4 x = *reinterpret_cast<const float4 *>(sp + kb * CB);
                                float *ok_ = o + (size_t)kb * plane;
                                if (a.accumulate)
                                {
                                    const float4 s4 = *reinterpret_cast<const float4 *>(ok_);
                                    x.x += s4.x; x.y += s4.y; x.z += s4.z; x.w += s4.w;
                                }
                                x.x = apply_act_ns(x.x, act_ns); x.y = apply_act_ns(x.y, act_ns);
                                x.z = apply_act_ns(x.z, act_ns); x.w = apply_act_ns(x.w, act_ns);
                                *reinterpret_cast<float4 *>(ok_) = x;
                            }
                        }
                    }
                    asm volatile("bar.sync 1, 256;" ::: "memory"); // before the staging rows are reused
                }
            }
            }
        }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0)
        tmem_dealloc(tmem, tmem_cols);
    // Wide tiles, when everything else is done: nobody waits for these warps any more, and in the middle of the tile loop the
    // code for them costs every other tile registers (ResNet-8 at 1024 images 426 us without it, 432 with a call here, 464
    // with it in the loop).
    if (!split && __any_sync(0xffffffffu, wide_tiles[lane]) && warp >= FIRST_ACC_WARP && warp < FIRST_SPLIT_WARP)
    {
        const float act_ns = act_neg_scale(a.act, a.slope);
        for (int i = 0, t = first_tile; i < WIDE_WORDS * 32 && t < a.total_tiles; ++i, t += tile_step)
        {
            if (wide_tiles[i >> 5] >> (i & 31) & 1u)
                plain_tile<false, POOL>(a, decode_tile(a, t), in, filt, filt_down, bias, out, act_ns, warp - FIRST_ACC_WARP, lane, 0, a.cbs, nullptr, 0);
            if (!PERSIST)
                break;
        }
    }
}

// Two sets of splitters where the conversion of the patches sets the pace: more than three patches a CTA, one after the
// other (16 -> 32 channels at 208x208, 32 images: 86.4 us with one set, 81.6 with two; 64 -> 32 at 52x52, 64 images 41.4
// and 37.3; with two patches a CTA, 16 -> 16 at 32x32, 32 images, 8.3 and 8.6).  One set, whose patch slots need not be an even number
// (three for two: 128 -> 32 with the pool at 112x112, 16 images 130.5 -> 111.0, 64 -> 32 5x5 with the pool at 64x64, 64 images
// 154.7 -> 147.1, 32 -> 16 1x1 onto what is there at 112x112, 16 images 17.2 -> 16.8) and whose kernel leaves the accumulation
// warps more registers, where those also read what is there (16 -> 16 at 32x32, 1024 images onto the shortcut: 80 and
// 85), and before a pool, which makes them the slower ones while the input comes from L2 (16 -> 32 at 208x208, 16 images
// 43.2 and 44.6; 64 images, 177 MB from memory, 152.2 and 146.6) or a tile is two patches and two groups (32 -> 32 3x3 at 58x340, 256
// images 508.6 and 548.5, at 240x200, 64 images 297.7 and 304.8).
bool want_two_sets(const TcArgs &a)
{
    constexpr long long L2_BYTES = 126ll << 20;
    const long long tiles = (long long)a.N * a.px_tiles * a.k_tiles, blocks = std::min<long long>(tiles, num_sms());
    return a.merged && !a.accumulate && (a.cbs > 1 || tiles > 3 * blocks) &&
           (!a.pool || ((long long)a.N * a.C * a.H * a.W * (long long)sizeof(float) > L2_BYTES && (a.cbs != 2 || a.group != a.taps)));
}

// Picks ring depths for the patch / filter sizes already in `a`.  Narrow layers run persistent (one
// CTA per SM walks over the tiles, roles overlap across tiles), which needs the output staging rows
// next to the operand buffers; the others keep the deepest rings and let the staging alias them.  need_two: only accept plans with two patches in flight.
bool fit_rings(TcArgs &a, bool need_two)
{
    a.row_skip = (a.cg == 1 && a.group != a.Fw) ? (a.PW - a.Fw) * 4 : 0;
    const size_t limit = 226 * 1024;
    const int entries = a.PR * a.PW;
    const size_t x_part = ((size_t)entries * 64 * a.cg + 4095) & ~(size_t)4095;
    a.WR = a.pixm ? a.K : a.MT;
    a.split_sets = want_two_sets(a) ? 2 : 1; // (pixel-major tiles: always persistent)
    const size_t w_part = (size_t)a.WR * 64 * a.group; // one filter stage
    const size_t staging = (size_t)64 * (a.MT + 16) * 4; // 32 pixels of each half of the tile
    // {patch slots, filter stages (>= 2: a commit serves both rings)}
    static const int pref[][2] = {{4, 6}, {4, 3}, {3, 6}, {3, 4}, {3, 3}, {2, 3}, {3, 2}, {2, 2}, {1, 3}, {1, 2}};
    const int issuers = num_issuers(a.pixm);
    // persistent where it pays and fits: narrow layers (64-channel tiles: small filter stages and
    // staging rows, little work per tile); wide ones need the shared memory for deeper rings
    // Pixel-major persistent tiles whose whole filter fits: one stage per group of a tile, loaded once
    // per CTA.  The filter ring otherwise puts a bulk copy's round trip to L2 into every group's chain
    // of hand-overs (producer waits for the stage, copies, the issuer waits for the copy), and for
    // these layers that chain, not the MMAs, sets the pace (16 -> 32 channels at 208x208: 0.22 ms
    // with no MMA issued at all, 0.30 ms with them).
    a.w_resident = 0;
    // pooled epilogue: exchange rows, one slot of K + 4 floats per pair of columns of every odd row
    const size_t pool_rows = a.pool ? (size_t)(a.TH / 2) * (a.PW / 2) * (a.K + 4) * 4 : 0;
    if (a.pixm && a.k_tiles == 1 && a.cg == 1)
    {
        const int stages = a.cbs * (a.taps / a.group);
        if (stages <= W_STAGES_MAX)
            for (int xs = x_slots_max(a.merged); xs >= 2; xs -= a.split_sets)
            {
                const size_t ops = (size_t)xs * x_part + (size_t)stages * w_part;
                const size_t smem = ops + pool_rows;
                if (smem <= limit)
                {
                    a.x_slots = xs; a.w_stages = stages; a.smem_bytes = (unsigned)smem; a.tbufs = 4;
                    a.persistent = 1; a.stage_off = (unsigned)ops; a.w_resident = 1;
                    return true;
                }
            }
    }
    for (int any = a.split_sets == 2 ? 0 : 1; any < 2; ++any) // two sets of splitters want an even number of slots
    for (int persistent = (a.MT == 64 ? 1 : 0); persistent >= (a.pixm ? 1 : 0); --persistent)
        for (const auto &p : pref)
        {
            // A wait by parity takes a phase two further on for done, so an issuer has to see every fill of a stage it waits
            // on: a stage is always the same issuer's.  (Waiting for the MMAs of a stage's last fill as well lets any number serve, but
            // 64 -> 64 channels 7x7 at 28x28, 64 images, then takes 99.6 us instead of 90.6, 256 -> 256 at 14x14 118 instead of 105,
            // and ResNet-8 on 1024 images 2 % longer for the test alone.)
            if (p[1] % issuers)
                continue;
            // Four slots serve two sets of splitters, each with its next patch on the way while the MMAs read its last one (two
            // slots and four, us: 256 -> 32 channels 3x3 at 23x94, 128 images 330 and 280; 64 -> 32 7x7 at 96x135, 64 images 667 and 624; 128 -> 16
            // 1x1 at 184x22, 32 images 29.3 and 24.0).  Six filter stages beside them only where a group is a whole window: 128 -> 32 3x3
            // at 13x8, 128 images 17.4 with six and 17.9 with three, but 256 -> 16 5x5 at 92x81, 64 images 851 and 742.
            if (p[0] == 4 && (a.split_sets != 2 || any || (p[1] == 6 && a.group != a.taps)))
                continue;
            const int xs = p[0] < a.cbs || persistent ? p[0] : a.cbs;
            if (!any && (xs & 1))
                continue;
            if (need_two && xs < 2 && a.cbs >= 2)
                continue;
            const size_t ops = (size_t)xs * x_part + (size_t)p[1] * w_part;
            const size_t full = (size_t)a.NPX * (a.MT + 16) * 4; // one tile per CTA stages the whole tile
            const size_t smem = persistent ? ops + (a.pixm ? pool_rows : staging) : (ops > full ? ops : full);
            if (smem <= limit)
            {
                a.x_slots = xs; a.w_stages = p[1]; a.smem_bytes = (unsigned)smem;
                a.tbufs = (a.pixm || 4 * a.NPX <= 512) ? 4 : 2;
                a.persistent = persistent; a.stage_off = persistent ? (unsigned)ops : 0u;
                return true;
            }
        }
    return false;
}

// Wide images: TH x TW pixel tiles.  A tile's patch is (TH + Fh) x (TW + Fw - 1) pixels, so the
// halo stays small (a range of full-width rows of a 208-wide image drags two whole rows of halo
// along for every 256 outputs).  GEMM column j of a tile is patch-linear: row j / PW, column j % PW,
// columns >= TW of each patch row are junk.
bool plan_tiled(const small_b200_layer *L, TcArgs &a, int cap)
{
    double best = 0.0;
    int best_tw = 0, best_th = 0;
    const int gran = a.pixm ? 128 : 64;
    for (int tw = 8; tw <= a.Wo && tw + a.Fw - 1 <= BOX_PX; tw += (a.pool ? 2 : 1))
    {
        const int pw = tw + a.Fw - 1;
        int th = (cap - tw) / pw + 1;
        if (th > a.Ho)
            th = a.Ho;
        if (a.pool && (th &= ~1) == 0) // pooled epilogue: pairs of rows and of columns stay inside a tile
            continue;
        const int npx = ((th - 1) * pw + tw + gran - 1) / gran * gran;
        const long long tiles = (long long)((a.Wo + tw - 1) / tw) * ((a.Ho + th - 1) / th);
        const double eff = (double)a.Wo * a.Ho / ((double)tiles * npx);
        if (eff > best + 1e-9)
        {
            best = eff; best_tw = tw; best_th = th;
        }
    }
    if (!best_tw)
        return false;
    a.tiled = 1; a.TW = best_tw; a.TH = best_th;
    a.PW = a.TW + a.Fw - 1;
    a.PR = a.TH + a.Fh; // one row more than the taps reach: the junk tail of the last row reads it
    if (a.PR > 256)
        return false;
    a.NPX = ((a.TH - 1) * a.PW + a.TW + gran - 1) / gran * gran;
    a.tiles_x = (a.Wo + a.TW - 1) / a.TW;
    a.px_tiles = a.tiles_x * ((a.Ho + a.TH - 1) / a.TH);
    // the last GEMM column's last tap must stay inside the patch
    if ((a.NPX - 1) + (a.Fh - 1) * a.PW + (a.Fw - 1) >= a.PR * a.PW)
        a.PR = ((a.NPX - 1) + (a.Fh - 1) * a.PW + (a.Fw - 1)) / a.PW + 1;
    return fit_rings(a, false);
}

// Tiling and shared-memory plan of one layer; false when the shape is not covered.
bool plan_as_g(const small_b200_layer *L, TcArgs &a, bool pixm, bool pool, bool whole, bool rows_view, int npx_cap)
{
    if (!L || L->stride != 1 || row_stride(L) != 1 || L->C % CB != 0 || L->K % CB != 0 || L->C <= 0 || L->K <= 0)
        return false;
    if (L->H <= 0 || L->W <= 0 || L->Fh <= 0 || L->Fw <= 0 || L->Fw > 16 || L->Fh > 16)
        return false;
    a = TcArgs{};
    a.N = L->N; a.C = L->C; a.K = L->K; a.H = L->H; a.W = L->W; a.Fh = L->Fh; a.Fw = L->Fw;
    a.pad_t = L->pad_t; a.pad_l = L->pad_l;
    a.x_row = (long long)a.W * CB; a.x_plane = (long long)a.H * a.W * CB;
    a.Ho = out_dim(L->H, L->pad_t, L->pad_b, L->Fh, 1);
    a.Wo = out_dim(L->W, L->pad_l, L->pad_r, L->Fw, 1);
    a.cbs = L->C / CB; a.taps = L->Fh * L->Fw;
    a.accumulate = L->accumulate; a.act = L->act; a.slope = L->slope;
    a.PW = L->W + (L->pad_l > L->pad_r ? L->pad_l : L->pad_r);
    a.MT = pick_mt(a.K);
    a.k_tiles = (a.K + a.MT - 1) / a.MT;
    a.group = a.Fw; // one kernel row per flush: taps = Fh * Fw is a multiple of it
    a.cg = 1; a.tap_step = 4;
    // few output channels: pixels on the tensor core's M (see the kernel's PIXM paths)
    a.pixm = pixm ? 1 : 0;
    a.merged = (pixm && a.K <= 32) ? 1 : 0;
    a.row_skip = 0;
    if (whole)
    {
        // the whole window in one group (TcArgs::row_skip): at most 3x3
        if (a.Fh < 2 || a.taps > 9)
            return false;
        a.group = a.taps;
    }
    a.pool = pool ? 1 : 0;
    if (pool)
    {
        // only the pixel-major tiled plan has the pooled epilogue; even sizes and an even patch width
        if (!pixm || a.accumulate || a.Ho % 2 || a.Wo % 2 || a.Fw % 2 == 0 || a.Ho == 0 || a.Wo == 0 ||
            L->W + (L->pad_l > L->pad_r ? L->pad_l : L->pad_r) <= 64)
            return false;
        return plan_tiled(L, a, npx_cap);
    }
    if (a.Ho == 0 || a.Wo == 0)
        return true;
    // 1x1 layer: two channel blocks per patch and per group (see TcArgs::cg)
    const bool pointwise = a.taps == 1 && !L->pad_t && !L->pad_b && !L->pad_l && !L->pad_r;
    if (a.taps == 1 && a.cbs % 2 == 0)
    {
        a.cg = 2; a.cbs /= 2; a.taps = 2; a.group = 2;
    }
    if (pointwise && !rows_view)
    {
        // no neighbourhoods: an image is one row of pixels, a tile a run of NPX of them
        a.W *= a.H; a.H = 1; a.Wo = a.W; a.Ho = 1;
        a.tiled = 1; a.TH = 1; a.PR = 1; a.runs = 1;
        const int gran = a.pixm ? 128 : 64, tiles_cap = (a.W + npx_cap - 1) / npx_cap;
        for (int npx = ((a.W + tiles_cap - 1) / tiles_cap + gran - 1) / gran * gran; npx >= gran; npx -= gran)
        {
            a.NPX = a.TW = a.PW = npx;
            a.tiles_x = a.px_tiles = (a.W + npx - 1) / npx;
            if (a.cg > 1)
                a.tap_step = npx * 4;
            if (fit_rings(a, npx > 128))
                return true;
        }
        return false;
    }
    if (rows_view)
    {
        a.x_row = (long long)a.C * a.W; a.x_plane = (long long)a.W * CB;
        a.runs = a.PW > BOX_PX ? 1 : 0;
    }
    else if (a.PW > BOX_PX)
    {
        if (a.cg > 1) // a padded 1x1 layer: one channel block at a time
        {
            a.cbs *= 2; a.cg = 1; a.taps = 1; a.group = 1;
        }
        return plan_tiled(L, a, npx_cap);
    }
    // GEMM columns of one image: the last valid one is (Ho-1)*PW + Wo-1
    const int m_img = (a.Ho - 1) * a.PW + a.Wo;
    const int tiles_cap = (m_img + npx_cap - 1) / npx_cap;
    const int gran = a.pixm ? 128 : 64;
    int npx_first = ((m_img + tiles_cap - 1) / tiles_cap + gran - 1) / gran * gran;
    // First pass: only plans that keep two patches in flight (a layer with few channel blocks
    // per CTA otherwise waits for every patch's load and split), even at a narrower tile;
    // second pass: anything that fits.
    for (int pass = 0; pass < 2; ++pass)
        for (int npx = npx_first; npx >= (pass == 0 ? 128 : gran); npx -= gran)
        {
            a.NPX = npx;
            a.px_tiles = (m_img + npx - 1) / npx;
            const int need = (a.PW - 1) + npx + (a.Fh - 1) * a.PW + (a.Fw - 1);
            a.PR = (need + a.PW - 1) / a.PW;
            if (a.cg > 1)
            {
                // the planes of a patch lie back to back: each must keep the phase of the 64-byte
                // swizzle (a multiple of eight 64-byte rows)
                while ((a.PR * a.PW) % 8)
                    ++a.PR;
                a.tap_step = a.PR * a.PW * 4;
            }
            if (a.PR > 256)
                continue;
            if (fit_rings(a, pass == 0))
                return true;
        }
    return false;
}
bool plan_as(const small_b200_layer *L, TcArgs &a, bool pixm, bool pool, bool rows_view, int npx_cap)
{
    // pixel-major: whole-window groups only where the filter stays resident in shared memory; channel-major: where
    // two stages of a whole window and two patches fit
    if (plan_as_g(L, a, pixm, pool, true, rows_view, npx_cap) && (a.Ho == 0 || a.Wo == 0 || (pixm ? a.w_resident : a.x_slots >= 2)))
        return true;
    return plan_as_g(L, a, pixm, pool, false, rows_view, npx_cap);
}
bool plan_shape(const small_b200_layer *L, TcArgs &a, bool rows_view, int npx_cap)
{
    const bool want_pixm = L && (L->K == 16 || L->K == 32 || L->K == 64);
    if (want_pixm && plan_as(L, a, true, false, rows_view, 256))
        return true;
    return plan_as(L, a, false, false, rows_view, npx_cap);
}
bool plan(const small_b200_layer *L, TcArgs &a, int npx_cap = 256)
{
    if (L && L->Fh == 1 && L->Fw == 1 && L->stride == 1 && !L->pad_t && !L->pad_b && !L->pad_l && !L->pad_r &&
        L->N > 1 && L->H > 0 && L->W > 0 && (long long)L->H * L->W <= 64)
    {
        small_b200_layer V = *L; // the batch as the rows of one image (TcArgs::rows_view)
        V.N = 1; V.H = L->N; V.W = L->H * L->W;
        if (plan_shape(&V, a, true, npx_cap))
        {
            a.rows_view = 1;
            a.o_kb_stride = (long long)V.W * CB;
            a.o_row_stride = (long long)(L->K / CB) * V.W * CB;
            return true;
        }
    }
    if (!plan_shape(L, a, false, npx_cap))
        return false;
    a.o_kb_stride = (long long)a.Ho * a.Wo * CB;
    a.o_row_stride = (long long)a.Wo * CB;
    return true;
}
// The convolution with the 2x2 stride-2 max pool `pool` in its epilogue; the strides describe the pooled tensor.
bool plan_pooled(const small_b200_layer *L, const small_b200_layer *pool, TcArgs &a)
{
    if (!L || !pool || !(L->K == 32 || L->K == 64) || L->accumulate)
        return false;
    // the activation is applied after the maximum: it must not decrease (ReLU, or LeakyReLU with a slope >= 0)
    if (L->act == SMALL_B200_ACT_LEAKY && !(L->slope >= 0.f))
        return false;
    if (pool->Fh != 2 || pool->Fw != 2 || pool->stride != 2 || row_stride(pool) != 2 || pool->pad_t || pool->pad_b ||
        pool->pad_l || pool->pad_r)
        return false;
    if (!plan_as(L, a, true, true, false, 256))
        return false;
    if (pool->H != a.Ho || pool->W != a.Wo || pool->C != L->K || pool->N != L->N)
        return false;
    a.o_kb_stride = (long long)(a.Ho / 2) * (a.Wo / 2) * CB;
    a.o_row_stride = (long long)(a.Wo / 2) * CB;
    return true;
}

int run_tc(const small_b200_layer *L, const small_b200_layer *pool, const float *in, const float *filt_prepared,
           const float *bias, float *out, void *stream);
} // namespace

extern "C"
{
int small_b200_conv2d_f32_tf32x3_supported(const small_b200_layer *L)
{
    TcArgs a;
    return plan(L, a) ? 1 : 0;
}

int small_b200_conv2d_f32_tf32x3_preferred(const small_b200_layer *L)
{
    TcArgs a;
    if (!L || L->C < 16 || !plan(L, a))
        return 0;
    // tiles that run across the images of a batch (1x1 layers on small images, dense heads) are full
    // whatever the image size; otherwise an image must give a tile something to do
    if (a.rows_view)
        return (long long)L->N * L->H * L->W >= 256 ? 1 : 0;
    return (long long)a.Ho * a.Wo >= 9 ? 1 : 0;
}

int small_b200_filter_prepare_tf32x3(const small_b200_layer *L, const float *filt, float *prepared, void *stream)
{
    if (!L || L->C % CB != 0 || L->K % CB != 0 || L->C <= 0 || L->K <= 0 || L->Fh <= 0 || L->Fw <= 0)
        return fail(SMALL_B200_INVALID_ARGUMENT, "Conv2D<float> (3xTF32) ERROR: shape not covered by the tensor-core path.");
    const long long n = (long long)L->K * L->C * L->Fh * L->Fw;
    // [0, n) floats: the half-precision pairs; behind them, for each output channel, the inverse of its block scale and its
    // largest magnitude, then what filter_max_kernel says (n is 16 K at least, and the caller provides 2 n)
    uint32_t *top = reinterpret_cast<uint32_t *>(prepared + n + L->K);
    SB_CUDA(cudaMemsetAsync(top, 0, (2 * (size_t)L->K + 3) * sizeof(uint32_t), as_stream(stream)));
    const long long blocks = (n + 255) / 256;
    const int slabs = (L->C / CB) * L->Fh * L->Fw, max_blocks = (slabs + 63) / 64;
    filter_max_kernel<<<dim3((unsigned)(max_blocks < 64 ? max_blocks : 64), (unsigned)(L->K / CB)), 256, 0, as_stream(stream)>>>(slabs, filt, top);
    if (int rc = launched("filter_max_kernel"))
        return rc;
    prepare_filter_kernel<<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(
        n, slabs, pick_mt(L->K), L->K, filt, top, reinterpret_cast<__half *>(prepared), prepared + n);
    return launched("prepare_filter_kernel");
}

int small_b200_conv2d_f32_tf32x3(const small_b200_layer *L, const float *in, const float *filt_prepared,
                                 const float *bias, float *out, void *stream)
{
    return run_tc(L, nullptr, in, filt_prepared, bias, out, stream);
}

int small_b200_conv2d_maxpool_f32_tf32x3_supported(const small_b200_layer *conv, const small_b200_layer *pool)
{
    TcArgs a;
    return plan_pooled(conv, pool, a) ? 1 : 0;
}

int small_b200_conv2d_maxpool_f32_tf32x3(const small_b200_layer *conv, const small_b200_layer *pool, const float *in,
                                         const float *filt_prepared, const float *bias, float *out, void *stream)
{
    if (!conv || !pool)
        return fail(SMALL_B200_INVALID_ARGUMENT, "Conv2D+MaxPool2D<float> (3xTF32) ERROR: null layer.");
    return run_tc(conv, pool, in, filt_prepared, bias, out, stream);
}
} // extern "C"

namespace
{
// Cycles of one channel block (or bundle) of a channel-major tile: its MMAs (32 + N/4 cycles each for their operands, N/2
// for the pipe), the filter stage's way into shared memory (about 40 bytes per cycle), or the splitters' passes.
double block_cycles(const TcArgs &a)
{
    const double mma = 3.0 * a.taps * (a.NPX / 2 > 32 + a.NPX / 4 ? a.NPX / 2 : 32 + a.NPX / 4);
    const double filter = a.taps * a.MT * 64 / 40.0;
    const double split = 600 + 1100.0 * a.PR * a.PW * a.cg / 256;
    return mma > filter ? (mma > split ? mma : split) : (filter > split ? filter : split);
}
// How a channel-major layer is cut: tile width (plans of at most 256, 192, 128, 64 pixels), how many CTAs of a cluster
// share a tile's reduction, and the same for the tiles of a last, partial wave where that runs as a launch of its own
// behind the full ones (rem_split, 0: one launch).  Small batches leave most SMs idle without it: 1024 -> 1024
// channels on one 13x13 image are 8 tiles of 192 pixels.  The estimate counts whole waves of CTAs; the fixed costs are
// those of starting a CTA (8000 cycles from its first instruction to its first finished sums, most of it cold code and
// the first filter stage) and of the exchange between the CTAs of a cluster (2000 until all are there, 4000 to 7000 to
// read the parts from the other SMs at some 13 bytes per cycle); a second launch costs another start.
// One image: conv8 of Tiny-YOLOv2 (1024 -> 1024 at 13x13) 62 -> 25 us, conv7 56 -> 19, conv6 33 -> 13, conv5 24 -> 13.
struct Cut
{
    int npx_cap, split, rem_split;
};
int configure()
{
    static PerDeviceOnce configured;
    int dev;
    if (configured.needed(&dev))
    {
#define SB_SMEM(...) SB_CUDA(cudaFuncSetAttribute(conv_f16x3_kernel<__VA_ARGS__>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024))
        SB_SMEM(true, false);
        SB_SMEM(true, false, true);
        SB_SMEM(true, false, true, false, true);
        SB_SMEM(true, false, true, true);
        SB_SMEM(true, false, true, true, true);
        SB_SMEM(true, false, true, true, false, 2);
        SB_SMEM(true, false, true, true, true, 2);
        SB_SMEM(true, false, true, true, false, 1, true);
        SB_SMEM(true, false, true, true, false, 2, true);
        SB_SMEM(false, false);
        SB_SMEM(false, true);
#undef SB_SMEM
        configured.mark(dev);
    }
    return SMALL_B200_OK;
}
// Clusters of S such CTAs (one per SM) that the current device runs at a time: they may not cross the borders of its
// groups of SMs (148 SMs: 74 pairs, 33 clusters of 4, 22 of 6, 15 of 8).
int resident_clusters(int S)
{
    static std::atomic<int> known[64][9];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64)
        dev = 0;
    int n = known[dev][S].load(std::memory_order_relaxed);
    if (n)
        return n;
    n = num_sms() / S;
    if (S > 1)
    {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)S); cfg.blockDim = dim3(num_threads(1));
        cfg.dynamicSmemBytes = 226 * 1024;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr; cfg.numAttrs = 1;
        int q = 0;
        if (cudaOccupancyMaxActiveClusters(&q, conv_f16x3_kernel<false, true>, &cfg) == cudaSuccess && q > 0)
            n = q;
        else
            cudaGetLastError();
    }
    known[dev][S].store(n, std::memory_order_relaxed);
    return n;
}
Cut choose_cut(const small_b200_layer *L)
{
    const double start = 8000, exchange = 6000;
    const long long sms = num_sms();
    static const int widths[] = {1, 2, 3, 4, 6, 8};
    Cut best{256, 1, 0};
    double best_cost = 0;
    int last_npx = 0;
    for (int cap = 256; cap >= 64; cap -= 64)
    {
        TcArgs a;
        if (!plan(L, a, cap) || a.pixm || a.persistent || a.NPX == last_npx)
            continue;
        last_npx = a.NPX;
        const long long tiles = (long long)a.N * a.px_tiles * a.k_tiles;
        const double t = block_cycles(a);
        for (int S : widths)
        {
            if (S > a.cbs)
                break;
            const long long room = resident_clusters(S);
            const double each = t * ((a.cbs + S - 1) / S) + start + (S > 1 ? exchange : 0);
            const double cost = ((tiles + room - 1) / room) * each;
            // a finer cut has to promise something: the exchange is an estimate
            if (best_cost == 0 || cost < 0.95 * best_cost)
            {
                best_cost = cost; best = Cut{cap, S, 0};
            }
            const long long full = tiles / sms, rem = tiles % sms;
            if (S > 1 && full > 0 && rem > 0)
            {
                const double mixed = full * (t * a.cbs + start) + ((rem + room - 1) / room) * each + start;
                if (mixed < 0.95 * best_cost)
                {
                    best_cost = mixed; best = Cut{cap, 1, S};
                }
            }
        }
    }
    return best;
}

int run_tc(const small_b200_layer *L, const small_b200_layer *pool, const float *in, const float *filt_prepared,
           const float *bias, float *out, void *stream)
{
    if (int rc = check_window_layer(L, "Conv2D<float>", true, 2))
        return rc;
    if (int rc = configure())
        return rc;
    TcArgs a;
    const Cut cut = pool ? Cut{256, 1, 0} : choose_cut(L);
    if (pool ? !plan_pooled(L, pool, a) : !plan(L, a, cut.npx_cap))
        return fail(SMALL_B200_INVALID_ARGUMENT, pool ? "Conv2D+MaxPool2D<float> (3xTF32) ERROR: shape not covered by the fused tensor-core path."
                                                      : "Conv2D<float> (3xTF32) ERROR: shape not covered by the tensor-core path.");
    if (a.N == 0 || a.Ho == 0 || a.Wo == 0)
        return SMALL_B200_OK;

    CUtensorMap mx;
    {
        // activations [N*cbs][H][W][8 x 8 bytes]: whole rows of the image are the innermost dimension.  (A map with a
        // pixel's 64 bytes innermost moves one 64-byte row per 9 to 12 cycles, whatever memory delivers.)
        const uint64_t dims[3] = {(uint64_t)a.W * 8, (uint64_t)a.H, (uint64_t)a.N * a.cbs * a.cg};
        const uint64_t strides[2] = {(uint64_t)a.x_row * 4, (uint64_t)a.x_plane * 4};
        const uint32_t box[3] = {(uint32_t)a.PW * 8, (uint32_t)a.PR, (uint32_t)a.cg};
        if (a.runs)
            memset(&mx, 0, sizeof(mx));
        else if (int rc = make_tensor_map(&mx, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, in, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE))
            return rc;
    }
    int *status = device_status_ptr();
    if (!status)
        return fail(SMALL_B200_CUDA_ERROR, "device status word not available");
    const long long tiles = (long long)a.N * a.px_tiles * a.k_tiles;
    if (tiles > 0x7fffffffLL)
        return fail(SMALL_B200_INVALID_ARGUMENT, "Conv2D<float> (3xTF32) ERROR: too many tiles.");
    a.total_tiles = (int)tiles;
    a.by_px_tiles.set(a.px_tiles); a.by_N.set(a.N); a.by_tiles_x.set(a.tiled ? a.tiles_x : 1); a.by_PW.set(a.PW);
    long long blocks = tiles;
    if (a.persistent && blocks > num_sms())
        blocks = num_sms();
    a.ksplit = (a.pixm || a.persistent) ? 1 : cut.split;
    blocks *= a.ksplit;
    const __half *filt = reinterpret_cast<const __half *>(filt_prepared);
    const float *filt_down = filt_prepared + (size_t)a.K * a.C * a.Fh * a.Fw;
    auto launch_split = [&](const TcArgs &ta, long long nblocks) -> int {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)nblocks); cfg.blockDim = dim3(num_threads(1));
        cfg.dynamicSmemBytes = ta.smem_bytes; cfg.stream = as_stream(stream);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)ta.ksplit; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr; cfg.numAttrs = 1;
        SB_CUDA(cudaLaunchKernelEx(&cfg, conv_f16x3_kernel<false, true>, mx, in, filt, filt_down, ta, bias, out, status));
        return SMALL_B200_OK;
    };
    if (!a.pixm && !a.persistent && cut.rem_split)
    {
        const long long full = tiles / num_sms() * num_sms(), rem = tiles - full;
        TcArgs a1 = a;
        a1.tile_base = 0;
        conv_f16x3_kernel<false, false><<<(unsigned)full, num_threads(1), a.smem_bytes, as_stream(stream)>>>(mx, in, filt, filt_down, a1, bias, out, status);
        if (int rc = launched("conv_f16x3_kernel"))
            return rc;
        TcArgs a2 = a;
        a2.tile_base = (int)full; a2.ksplit = cut.rem_split;
        if (int rc = launch_split(a2, a2.ksplit * rem))
            return rc;
        return launched("conv_f16x3_kernel");
    }
    const long long room = a.persistent ? blocks * WIDE_WORDS * 32 : tiles; // tiles of a launch (wide_tiles)
    for (long long base = 0; base < tiles; base += room)
    {
    a.tile_base = (int)base; a.total_tiles = (int)std::min(tiles, base + room);
    const unsigned grid = (unsigned)(a.persistent ? std::min(blocks, tiles - base) : blocks);
    // Tiles of many patches: LATE, since what the other form keeps in registers over the sums costs more in every group than the
    // epilogue then gains.  us, the other form and this: onto what is there 256 -> 16 channels 3x3 at 43x162, 64 images 428 and 414, 128 -> 16
    // at 52x30, one image 20.4 and 19.1; but 16 -> 16 at 112x112, 256 images 178 and 207, 64 -> 64 1x1 at 32x32, 1024 images 133 and 159.
    const bool two = a.split_sets == 2, late = a.cg == 1 && a.cbs > 4;
#define SB_LAUNCH_PIXM(M, P, SETS, LATE) \
    conv_f16x3_kernel<true, false, true, M, P, SETS, LATE><<<grid, num_threads(SETS), a.smem_bytes, as_stream(stream)>>>(\
        mx, in, filt, filt_down, a, bias, out, status)
    if (a.pool && two)
        SB_LAUNCH_PIXM(true, true, 2, false);
    else if (a.pool && a.merged)
        SB_LAUNCH_PIXM(true, true, 1, false);
    else if (a.pool)
        SB_LAUNCH_PIXM(false, true, 1, false);
    else if (two && late)
        SB_LAUNCH_PIXM(true, false, 2, true);
    else if (two)
        SB_LAUNCH_PIXM(true, false, 2, false);
    else if (a.merged && late)
        SB_LAUNCH_PIXM(true, false, 1, true);
    else if (a.merged)
        SB_LAUNCH_PIXM(true, false, 1, false);
    else if (a.pixm)
        SB_LAUNCH_PIXM(false, false, 1, false);
#undef SB_LAUNCH_PIXM
    else if (a.persistent)
        conv_f16x3_kernel<true, false><<<grid, num_threads(1), a.smem_bytes, as_stream(stream)>>>(mx, in, filt, filt_down, a, bias, out, status);
    else if (a.ksplit > 1)
    {
        if (int rc = launch_split(a, blocks))
            return rc;
    }
    else
        conv_f16x3_kernel<false, false><<<grid, num_threads(1), a.smem_bytes, as_stream(stream)>>>(mx, in, filt, filt_down, a, bias, out, status);
    if (int rc = launched("conv_f16x3_kernel"))
        return rc;
    }
    return SMALL_B200_OK;
}
} // namespace

extern "C" int small_b200_conv2d_f32_tf32x3_cut(const small_b200_layer *L, int *cut)
{
    if (!L || !cut || !small_b200_conv2d_f32_tf32x3_supported(L))
        return fail(SMALL_B200_INVALID_ARGUMENT, "Conv2D<float> (3xTF32) ERROR: shape not covered by the tensor-core path.");
    if (int rc = configure()) // the clusters that fit are counted with the kernel's shared memory
        return rc;
    const Cut c = choose_cut(L);
    cut[0] = c.npx_cap; cut[1] = c.split; cut[2] = c.rem_split;
    return SMALL_B200_OK;
}

// ---------------------------------------------------------------------------------------------
// The same tensor-core convolution for callers that must not allocate device memory.
//
// small_b200_conv2d_f32_tf32x3 needs scratch from its caller: the filter re-laid for the tensor
// core, with its scales.  Some callers cannot provide it: code that runs inside
// a region where cudaMalloc is forbidden or would synchronise the device (a real-time loop, a
// plug-in that only ever receives its input and output pointers, a host that has handed all of
// its device memory to another allocator).  For them the scratch lives in this fixed array
// inside the library image.  Every GPU that loads the library carries these 16 MiB until the
// process exits, which is why the limit is modest.
constexpr size_t STATIC_SCRATCH_FLOATS = (size_t)4 << 20; // 4 Mi floats = 16 MiB
static __device__ __align__(256) float g_static_scratch[STATIC_SCRATCH_FLOATS];

namespace
{
// In host code `g_static_scratch` is only a stand-in for the device symbol, not an address a
// kernel could use; the device address is looked up once per device, with that device current.
int static_scratch_ptr(float **ptr)
{
    static float *ptrs[64] = {nullptr};
    int dev = 0;
    SB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64)
        return fail(SMALL_B200_CUDA_ERROR, "device index out of range for the static scratch table");
    if (!ptrs[dev])
    {
        float *p = nullptr;
        SB_CUDA(cudaGetSymbolAddress((void **)&p, g_static_scratch));
        ptrs[dev] = p;
    }
    *ptr = ptrs[dev];
    return SMALL_B200_OK;
}
} // namespace

extern "C" int small_b200_conv2d_f32_tf32x3_noalloc(const small_b200_layer *L, const float *in,
                                                    const float *filt, const float *bias, float *out,
                                                    void *stream)
{
    if (int rc = check_window_layer(L, "Conv2D<float>", true, 2))
        return rc;
    if (!small_b200_conv2d_f32_tf32x3_supported(L))
        return fail(SMALL_B200_INVALID_ARGUMENT,
                    "Conv2D<float> (3xTF32, no-alloc) ERROR: shape not covered by the tensor-core path.");
    const size_t filt_elems = (size_t)L->K * L->C * L->Fh * L->Fw;
    const size_t need = 2 * filt_elems; // what small_b200_filter_prepare_tf32x3 asks for
    if (need > STATIC_SCRATCH_FLOATS)
        return fail(SMALL_B200_INVALID_ARGUMENT,
                    "Conv2D<float> (3xTF32, no-alloc) ERROR: this call needs " + std::to_string(need * 4) +
                        " bytes of scratch (2 x K*C*Fh*Fw filter elements, 4 bytes each) but the "
                        "built-in scratch holds " + std::to_string(STATIC_SCRATCH_FLOATS * 4) +
                        " bytes; use small_b200_conv2d_f32_tf32x3 with caller-provided scratch.");
    float *scratch = nullptr;
    if (int rc = static_scratch_ptr(&scratch))
        return rc;
    float *prepared = scratch;
    // Nothing in the scratch has to start from zero: the region this call reads is completely
    // rewritten for the sizes of this call before the convolution reads it.
    if (int rc = small_b200_filter_prepare_tf32x3(L, filt, prepared, stream))
        return rc;
    return small_b200_conv2d_f32_tf32x3(L, in, prepared, bias, out, stream);
}
