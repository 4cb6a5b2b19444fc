// fp32 convolution on the tensor cores: every operand as three bf16 parts, partial sums added in fp32.
//
// An fp32 value of 2^-110 or more is b1 + b2 + b3 exactly, each part the bf16 nearest to what the parts before leave (8 + 8 + 8 bits);
// a smaller one up to 2^-134, half of the smallest bf16.  A product is then nine bf16 products, exact in fp32; the three of them
// below 2^-24 of it are left out:
//     x w = x1 w1 + (x1 w2 + x2 w1) + (x2 w2 + x1 w3 + x3 w1) + O(2^-25).
// The tensor core truncates its sums, so it never adds for long: the products of one K block of 32, smallest first, go to a fresh
// accumulator, and the running sums are kept in registers, fp32 additions rounded to nearest.  The result is nearer to a double-
// precision convolution than the FFMA chain's (conv_simt.cu); both errors stand in the table at thb_conv_f32_splits.
//
// What bounds it is the rate of the multiplies, twelve per K block, of 45 cycles for 64 columns and 64 for 128 (768 cycles a K block
// of a 128 x 128 tile; 880 measured, 212 TFLOP/s on a 3x3 128->128 layer @28x28 of 64 images against 46 for the FFMA kernel).
// The operands: raw activations arrive in shared memory, are split on their way to TENSOR memory, from where the multiplies read
// them, and are not written back; the weights' parts were laid out once, a stage after the other, for untiled copies.
//   4 or 8 warps  add the accumulator of every K block to their registers, 64 columns each
//   8 warps       split, four every other K block: a thread owns a pixel row = TMEM lane; without a 32-channel slab (first layers)
//                 they gather the row's 16-byte chunks from global memory themselves, a K block of theirs ahead
//   1 warp        copies activations: 128 rows of 32 channels a K block (tiled or im2col-mode TMA)
//   1 warp        copies weight parts, ahead of griddepcontrol.wait (no launch of a forward writes them)
//   2 warps       issue the multiplies, every other K block each (one alone: 1330 cycles a K block)
// Launches of few tiles share a tile's K blocks among the 2, 4 or 8 CTAs of a cluster, which push their partial columns to the
// owner as in conv_few_tc.cu.  The result passes through shared memory, so that global memory is read (residual) and written in
// rows of 16-byte chunks.
//
// The parts are those of weights times a power of two, one for each channel (weight_units_kernel): no fp32 weight loses a bit then, and
// the sums stay far from the ends of the range.  Some sums the parts may spoil all the same; those outputs are computed again by FFMA
// from the fp32 weights (exact4):
//   - a sum that is not finite: infinity times a zero part, a value that rounds to an infinite part;
//   - a sum so small that the 2^-134 an activation may have lost show in its bits;
//   - a sum of zero, if its activations have subnormal numbers among them: below 2^-134 all of their parts are zero;
//   - every sum of a channel with weights of 2^26 or more.
// To look at every sum costs 0 to 2.5 % (3x3 64->64 @56x56, 64 images 100.3 -> 102.1 us; 1x1 64->256 @56x56, 16 images 36.2 -> 36.9; tiles
// of 128 channels the same).  What is found is slow: a blank input takes 2.5 to 6 times the time of an ordinary one, one of 1e-35 a hundred.
//
// Every mbarrier wait is bounded; one that runs out records a code in *status and the CTA drains.
#include <cuda.h>
#include <string.h>
#include "common.cuh"
#include "conv_maps.cuh"

namespace {

constexpr int BM = 128, BK = 32;
constexpr int A_BYTES = BM * BK * 4;
constexpr int RECV_ROWS = BM + 1;  // (padded: a warp's reads of several column groups meet in no bank)

// A tile is 128 pixels x 64 NT channels.  NT = 2: one CTA to an SM, a multiply of 128 columns takes little longer than one of 64.
// NT = 1 (layers of 64 channels, launches of few tiles): two CTAs to an SM, each half of the tensor memory.  GATHER: the activations do not come by TMA.
template <int NT, bool GATHER> struct Cfg {
    static constexpr int BN = 64 * NT, BPART = BN * BK * 2, B_BYTES = 3 * BPART;
    // Stages of raw activations (gather: two a group), an even number: a stage then belongs to one of the two splitting groups, which
    // sees every phase of its barrier.  With an odd one a group sees every other phase, all of one parity, and passes a stage whose
    // copy for the OTHER group has not landed yet (copies land out of order: a later one had).
    static constexpr int RA = 4;
    // Stages of weight parts, an even number: a barrier of the ring then serves the K blocks of one parity only, and the other
    // parity's multiplies cannot carry it a phase further than someone still waits for.
    static constexpr int RB = NT == 2 ? 6 : 4;
    static constexpr int NA = NT == 2 ? 4 : 2;                              // operands in tensor memory, next to two accumulators
    static constexpr int A_COL = 2 * BN, TMEM_COLS = 256 * NT;
    static constexpr int CONV = 4 * NT, MISC = CONV + 8, NTHREADS = (MISC + 4) * 32;  // first warps of the groups
    static constexpr int RECV_BYTES = (BN / 4) * RECV_ROWS * 16;
    static constexpr int SMEM = 1024 + RA * A_BYTES + RB * B_BYTES;
    static_assert(RECV_BYTES <= RB * B_BYTES, "the partial sums take the place of the weight stages");
    static_assert(RA % 2 == 0 && RB % 2 == 0 && RB >= NA && SMEM <= 227 * 1024, "stages");
    static_assert(NT == 2 || (2 * (SMEM + 1024) <= 228 * 1024 && 3 * (SMEM + 1024) > 228 * 1024), "two CTAs to an SM, not three");
    static_assert(A_COL + 64 * NA <= TMEM_COLS, "tensor memory");
};

struct F32Params {
    const float *x, *w;
    float *y;
    const int *kinfo;
    int P, H, W, in_ld, oW, oHW, dH, dW, padH, padW, kW, Cout, Cout_pad, out_ld, n_kchunks, nkb, n_tiles;
    const float *scale, *shift, *slope, *res;
    int res_ld;
    float self_coef, res_coef;
    int act_kind;
    float act_th, act_val, act_alpha;
    int mode, slabs;   // 0: gathered; 1: activations are a plain matrix; 2: im2col-mode copies, `slabs` slabs of 32 channels per tap
    int splits, pdl, test_withhold;
    int halves;        // NT = 1 on weights laid out for 128 channels: a tile's parts are halves of theirs
    const uint8_t *parts;  // the weights' parts, one stage after another: [column tile][K block][part][64 rows of 64 bytes, swizzled]
    const float *units;    // per channel what its sums are in units of (negative: it has no weights but zero); then per channel the smallest ordinary sum
    int *status;
    long long wait_limit;
};

__device__ __forceinline__ void report(int *status, int code) { *reinterpret_cast<volatile int *>(status) = code; }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void st_cluster_v4(uint32_t smem, uint32_t rank, float a, float b, float c, float d)
{
    uint32_t at;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem), "r"(rank));
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// untiled copy of `bytes` (a multiple of 16, both addresses too), no multicast
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// the parts of two values, the first in the low half of each word
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ void split_pair(float lo, float hi, uint32_t &p1, uint32_t &p2, uint32_t &p3)
{
    p1 = bf16_pair(lo, hi);
    lo -= __uint_as_float(p1 << 16);
    hi -= __uint_as_float(p1 & 0xffff0000u);
    p2 = bf16_pair(lo, hi);
    p3 = bf16_pair(lo - __uint_as_float(p2 << 16), hi - __uint_as_float(p2 & 0xffff0000u));
}
// eight elements of a row into the three parts of a TMEM operand
__device__ __forceinline__ void split_store(uint32_t taddr, const float4 &a, const float4 &b)
{
    uint32_t p1[4], p2[4], p3[4];
    split_pair(a.x, a.y, p1[0], p2[0], p3[0]);
    split_pair(a.z, a.w, p1[1], p2[1], p3[1]);
    split_pair(b.x, b.y, p1[2], p2[2], p3[2]);
    split_pair(b.z, b.w, p1[3], p2[3], p3[3]);
    tmem_st4(taddr, p1);
    tmem_st4(taddr + 16, p2);
    tmem_st4(taddr + 32, p3);
}

// twice an fp32's bits less one, as an unsigned number: in the order of the magnitudes, but for zero, which is above them all
__device__ __forceinline__ uint32_t magnitude(float v) { return 2 * __float_as_uint(v) - 1; }
// the largest and the smallest magnitude of four values (the largest: NaN if one of them is)
__device__ __forceinline__ float max4(float a, float b, float c, float d)
{
    float m;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
    asm("max.NaN.abs.f32 %0, %1, %2, %2;" : "=f"(m) : "f"(m), "f"(d));
    return m;
}
__device__ __forceinline__ float min4(float a, float b, float c, float d)
{
    float m;
    asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
    asm("min.abs.f32 %0, %1, %2, %2;" : "=f"(m) : "f"(m), "f"(d));
    return m;
}

// Four channels of one pixel: y = act(self * (sum * scale + shift) + res_coef * residual), channels >= Cout zero.
struct Affine4 {
    float sc[4], sh[4];
    __device__ __forceinline__ Affine4(const F32Params &p, int c0)
    {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const bool in = c0 + j < p.Cout;
            sc[j] = in ? (p.scale ? p.scale[c0 + j] : 1.f) : 0.f;
            sh[j] = in ? (p.shift ? p.shift[c0 + j] : 0.f) : 0.f;
        }
    }
    __device__ __forceinline__ void store(const F32Params &p, int pm, int c0, const float4 &s, const float4 &r) const
    {
        float v[4] = {s.x, s.y, s.z, s.w};
        const float rr[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            v[j] = v[j] * sc[j] + sh[j];
            if (p.res) v[j] = p.self_coef * v[j] + p.res_coef * rr[j];
            if (p.act_kind == THB_ACT_THRESHOLD) v[j] = v[j] > p.act_th ? v[j] : p.act_val;
        }
        if (p.act_kind > THB_ACT_THRESHOLD) {
#pragma unroll 1
            for (int j = 0; j < 4; j++) {  // (a loop: the general activation four times over is a thousand instructions)
                const float t = thb_apply_act(v[0], p.act_kind, p.act_th, p.act_val, p.act_alpha, p.slope && c0 + j < p.Cout ? p.slope[c0 + j] : 0.f);
                v[0] = v[1]; v[1] = v[2]; v[2] = v[3]; v[3] = t;
            }
        }
        *reinterpret_cast<float4 *>(p.y + (size_t)pm * p.out_ld + c0) =
            make_float4(v[0], c0 + 1 < p.Cout ? v[1] : 0.f, c0 + 2 < p.Cout ? v[2] : 0.f, c0 + 3 < p.Cout ? v[3] : 0.f);
    }
};

// The activations of one pixel's sums, four at a time, zeros outside the image
struct Patch {
    const F32Params &p;
    int n, ih0, iw0;
    __device__ __forceinline__ Patch(const F32Params &p, int pm) : p(p), n(pm / p.oHW)
    {
        const int rem = pm - n * p.oHW, oh = rem / p.oW;
        ih0 = oh * p.dH - p.padH;
        iw0 = (rem - oh * p.oW) * p.dW - p.padW;
    }
    __device__ __forceinline__ float4 chunk(int g) const
    {
        const int ki = __ldg(p.kinfo + g), ih = ih0 + ((ki >> 24) & 0x7f), iw = iw0 + ((ki >> 16) & 0xff);
        if (ki < 0 || (unsigned)ih >= (unsigned)p.H || (unsigned)iw >= (unsigned)p.W) return make_float4(0.f, 0.f, 0.f, 0.f);
        return *reinterpret_cast<const float4 *>(p.x + ((size_t)(n * p.H + ih) * p.W + iw) * p.in_ld + (ki & 0xffff) * 4);
    }
};

// Four channels of one pixel by FFMA from the fp32 weights: chains of 32 products, whose sums are added.
__device__ __forceinline__ float4 exact4(const F32Params &p, int pm, int c0)
{
    const Patch patch(p, pm);
    float s[4] = {0.f, 0.f, 0.f, 0.f}, t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int g = 0; g < p.n_kchunks; g++) {
        float4 v = patch.chunk(g);
#pragma unroll 1
        for (int e = 0; e < 4; e++) {
            const float4 wv = *reinterpret_cast<const float4 *>(p.w + (size_t)(g * 4 + e) * p.Cout_pad + c0);
            t[0] = fmaf(v.x, wv.x, t[0]); t[1] = fmaf(v.x, wv.y, t[1]);
            t[2] = fmaf(v.x, wv.z, t[2]); t[3] = fmaf(v.x, wv.w, t[3]);
            v.x = v.y; v.y = v.z; v.z = v.w;
        }
        if ((g & 7) == 7 || g == p.n_kchunks - 1) {
#pragma unroll
            for (int j = 0; j < 4; j++) { s[j] += t[j]; t[j] = 0.f; }
        }
    }
    return make_float4(s[0], s[1], s[2], s[3]);
}

// A warp: are there subnormal numbers among the activations of one pixel's sums?
__device__ __forceinline__ bool subnormals(const F32Params &p, int pm, int lane)
{
    const Patch patch(p, pm);
    uint32_t least = ~0u;
#pragma unroll 2
    for (int g = lane; g < p.n_kchunks; g += 32) {
        const float4 v = patch.chunk(g);
        least = min(min(least, min(magnitude(v.x), magnitude(v.y))), min(magnitude(v.z), magnitude(v.w)));
    }
    return __any_sync(~0u, least < 2 * 0x00800000u - 1);
}

// A warp's rows that have a sum which is not ordinary (bits of `rare`: a thread's rows r0, r0 + step, ...): those sums computed again
// or not, and stored.  G lanes share a row.
__device__ __forceinline__ void store_rare(const F32Params &p, const uint8_t *part, unsigned rare, int r0, int step, int S, int G, int m0, int c0)
{
    const int lane = threadIdx.x & 31;
    for (unsigned any = __reduce_or_sync(~0u, rare); any; any &= any - 1) {
        const int k = __ffs(any) - 1, r = r0 + k * step;
        const bool mine = rare >> k & 1;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        bool spoilt = false, zero = false;
        if (mine) {
            const float4 u4 = *reinterpret_cast<const float4 *>(p.units + c0), l4 = *reinterpret_cast<const float4 *>(p.units + p.Cout_pad + c0);
            const float u[4] = {u4.x, u4.y, u4.z, u4.w}, l[4] = {l4.x, l4.y, l4.z, l4.w};
            for (int q = 0; q < S; q++) {
                const float4 t = *reinterpret_cast<const float4 *>(part + (q * G * RECV_ROWS + r) * 16);
                v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float m = fabsf(v[i]);
                zero |= m == 0.f && u[i] > 0.f;
                spoilt |= m != 0.f && !(m >= l[i] && m < INFINITY);
                v[i] *= fabsf(u[i]);
            }
        }
        if (__any_sync(~0u, zero))
            for (int first = 0; first < 32; first += G) {  // the warp's rows number k: G lanes each
                const bool here = zero && lane / G == first / G;
                if (__any_sync(~0u, here)) spoilt |= subnormals(p, m0 + __shfl_sync(~0u, r, first), lane) && here;
            }
        if (!mine) continue;
        const float4 rv = p.res ? *reinterpret_cast<const float4 *>(p.res + (size_t)(m0 + r) * p.res_ld + c0) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 sums = make_float4(v[0], v[1], v[2], v[3]);
        if (spoilt) sums = exact4(p, m0 + r, c0);
        Affine4(p, c0).store(p, m0 + r, c0, sums, rv);
    }
}

template <int NT, bool GATHER>
__global__ void __launch_bounds__(Cfg<NT, GATHER>::NTHREADS, 3 - NT) conv_f32_kernel(const __grid_constant__ CUtensorMap tmapA, const __grid_constant__ F32Params p)
{
    using C = Cfg<NT, GATHER>;
    constexpr int BN = C::BN, RA = C::RA, RB = C::RB, NA = C::NA, BPART = C::BPART, B_BYTES = C::B_BYTES, TMEM_COLS = C::TMEM_COLS;
    constexpr int W_A = C::MISC, W_B = C::MISC + 1, W_MMA = C::MISC + 2;
    constexpr uint32_t IDESC = make_idesc(1u, 1u, BN);
    extern __shared__ __align__(1024) uint8_t smem[];
    // raw activations there; read; K block i may be multiplied (stage i % RB: weights there, operand in TMEM, accumulator free);
    // multiplied.  One wait and one commit a K block: each costs the multiplying thread a hundred cycles.
    uint64_t *fullA = reinterpret_cast<uint64_t *>(smem), *emptyA = fullA + RA, *go = emptyA + RA, *done = go + RB;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + RB);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    volatile int *issued = abort_flag + 1;  // copies issued: activations, weights
    uint8_t *ringB = smem + 1024, *ringA = ringB + RB * B_BYTES, *recv = ringB;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int S = p.splits;
    const int rank = S > 1 ? (int)(blockIdx.x % S) : 0, tile = S > 1 ? (int)(blockIdx.x / S) : (int)blockIdx.x;
    const int m0 = (tile / p.n_tiles) * BM, n0 = (tile % p.n_tiles) * BN;
    const int kb0 = (int)((long)p.nkb * rank / S), nkb = (int)((long)p.nkb * (rank + 1) / S) - kb0;

    if (tid == 0) {
        for (int s = 0; s < RA; s++) { mbar_init(smem_u32(&fullA[s]), 1); mbar_init(smem_u32(&emptyA[s]), 4); }
        for (int s = 0; s < RB; s++) { mbar_init(smem_u32(&go[s]), 5 + 4 * NT); mbar_init(smem_u32(&done[s]), 1); }
        *abort_flag = issued[0] = issued[1] = 0;
        fence_barrier_init();
        fence_proxy_async_smem();
    }
    if (!GATHER && warp == W_A && lane == 0) tma_prefetch_desc(&tmapA);
    if (warp == W_MMA) {
        tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (p.pdl) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (p.pdl && warp != W_B) asm volatile("griddepcontrol.wait;" ::: "memory");

    auto give_up = [&](int code) {
        report(p.status, code);
        *abort_flag = 1;
    };
    // The sums go by way of shared memory: column group c / 4 of the tile belongs to rank c / W, slot [rank][group][row] there.
    const int wshift = (NT == 2 ? 7 : 6) - (S == 1 ? 0 : S == 2 ? 1 : S == 4 ? 2 : 3), W = 1 << wshift, G = W >> 2;
    // the end of the main loop, for every warp: afterwards the stages of all CTAs of the cluster are free
    auto leave = [&]() {
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (*abort_flag && warp == W_A) {
            // a wait ran out: copies still on their way must land before their stages are used again or the CTA leaves (a weight
            // stage's barrier may miss other arrivals and then never completes: 2 ms are a thousand times what a copy takes)
            for (int i = max(issued[0] - RA, 0); i < issued[0]; i++) mbar_wait_bounded(smem_u32(&fullA[i % RA]), (i / RA) & 1, 4000000);
            for (int i = max(issued[1] - RB, 0); i < issued[1]; i++) mbar_wait_bounded(smem_u32(&go[i % RB]), (i / RB) & 1, 4000000);
        }
        __syncthreads();
        if (warp == W_MMA) tmem_dealloc(tmem, TMEM_COLS);
        if (S > 1) {
            cluster_arrive();
            cluster_wait();
        }
    };
    // every part of the sums has arrived
    auto gathered = [&]() {
        if (S > 1) {
            __syncwarp();
            cluster_arrive();
            cluster_wait();
        } else
            __syncthreads();
    };
    const int row = tid & 127;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    bool have = true;

    if (warp < C::CONV) {
        // group `half` adds columns 64 half .. + 63
        if (NT == 1) asm volatile("setmaxnreg.inc.sync.aligned.u32 88;");
        const int half = warp >> 2;
        float acc[64];
#pragma unroll
        for (int i = 0; i < 64; i++) acc[i] = 0.f;
        if (lane == 0) {
            mbar_arrive(smem_u32(&go[0]));
            mbar_arrive(smem_u32(&go[1]));
        }
        int s = 0, s2 = 2;  // stages of K blocks i and i + 2
        uint32_t ph = 0;
        for (int i = 0; i < nkb; i++) {
            const int b = i & 1;
            have = mbar_wait_bounded(smem_u32(&done[s]), ph, p.wait_limit);
            if (!have && lane == 0) give_up(2);
            have = __all_sync(0xffffffffu, have);
            if (!have) break;
            tc_fence_after();
#pragma unroll
            for (int q = 0; q < 8; q++) {
                uint32_t v[8];
                tmem_ld8(tmem + lanes + b * BN + half * 64 + q * 8, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; j++) acc[q * 8 + j] += __uint_as_float(v[j]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&go[s2]));
            if (++s == RB) { s = 0; ph ^= 1; }
            if (++s2 == RB) s2 = 0;
        }
        leave();
        uint8_t *at = recv + (size_t)row * 16;
        if (S == 1) {
#pragma unroll
            for (int q = 0; q < 16; q++)
                *reinterpret_cast<float4 *>(at + (half * 16 + q) * RECV_ROWS * 16) = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
        } else {
#pragma unroll
            for (int q = 0; q < 16; q++) {
                const int c = half * 64 + 4 * q;
                st_cluster_v4(smem_u32(at + (rank * G + ((c >> 2) & (G - 1))) * RECV_ROWS * 16), c >> wshift, acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
            }
        }
        gathered();
        return;
    }
    if (warp >= C::MISC) {
        if (NT == 1) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == W_A) {
            if (!GATHER && lane == 0) {
                int iw = 0, ih = 0, in = 0, tap_w = 0, tap_h = 0, slab = 0;
                if (p.mode == 2) {
                    in = m0 / p.oHW;
                    const int rem = m0 - in * p.oHW, oh = rem / p.oW;
                    ih = oh * p.dH - p.padH;
                    iw = (rem - oh * p.oW) * p.dW - p.padW;
                    const int tap = kb0 / p.slabs;
                    slab = kb0 - tap * p.slabs;
                    tap_h = tap / p.kW;
                    tap_w = tap - tap_h * p.kW;
                }
                int s = 0;
                uint32_t ph = 0;
                for (int i = 0; i < nkb; i++) {
                    if (i >= RA && !mbar_wait_bounded(smem_u32(&emptyA[s]), ph ^ 1, p.wait_limit)) {
                        give_up(3);
                        break;
                    }
                    if (p.test_withhold && i == nkb - 1) break;
                    const uint32_t bar = smem_u32(&fullA[s]), dst = smem_u32(ringA + s * A_BYTES);
                    mbar_arrive_expect_tx(bar, A_BYTES);
                    if (p.mode == 1) tma_load_2d(dst, &tmapA, bar, (kb0 + i) * BK, m0);
                    else {
                        tma_load_im2col_4d(dst, &tmapA, bar, slab * BK, iw, ih, in, (uint16_t)tap_w, (uint16_t)tap_h);
                        if (++slab == p.slabs) {
                            slab = 0;
                            if (++tap_w == p.kW) { tap_w = 0; tap_h++; }
                        }
                    }
                    issued[0] = i + 1;
                    if (++s == RA) { s = 0; ph ^= 1; }
                }
            }
            __syncwarp();
        } else if (warp == W_B) {
            if (lane == 0) {
                const int ct = tile % p.n_tiles;
                const bool halves = NT == 1 && p.halves;
                const uint8_t *src = halves ? p.parts + ((size_t)(ct >> 1) * p.nkb + kb0) * (2 * B_BYTES) + (ct & 1) * BPART
                                            : p.parts + ((size_t)ct * p.nkb + kb0) * B_BYTES;
                int s = 0;
                uint32_t ph = 0;
                for (int i = 0; i < nkb; i++) {
                    if (i >= RB && !mbar_wait_bounded(smem_u32(&done[s]), ph ^ 1, p.wait_limit)) {
                        give_up(3);
                        break;
                    }
                    const uint32_t bar = smem_u32(&go[s]), dst = smem_u32(ringB + s * B_BYTES);
                    mbar_arrive_expect_tx(bar, B_BYTES);
                    if (halves)
                        for (int part = 0; part < 3; part++) bulk_load(dst + part * BPART, src + (size_t)i * (2 * B_BYTES) + part * (2 * BPART), BPART, bar);
                    else
                        bulk_load(dst, src + (size_t)i * B_BYTES, B_BYTES, bar);
                    issued[1] = i + 1;
                    if (++s == RB) { s = 0; ph ^= 1; }
                }
            }
            __syncwarp();
        } else {
            // two multiplying warps, every other K block each: what one spends on its wait, its commit and its loop (400 cycles, half
            // of a K block's multiplies) the other's multiplies cover
            const int first = warp - W_MMA;
            const bool leader = elect_one();
            int s = first;
            uint32_t ph = 0;
            for (int i = first; i < nkb; i += 2) {
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&go[s]), ph, p.wait_limit))) {
                    if (leader) give_up(4);
                    break;
                }
                tc_fence_after();
                const uint32_t sb = smem_u32(ringB + s * B_BYTES), d = tmem + first * BN, a = tmem + C::A_COL + (i & (NA - 1)) * 64;
                uint64_t w[3];
#pragma unroll
                for (int part = 0; part < 3; part++) w[part] = make_sw64_kmajor_desc(sb + part * BPART);
                constexpr int pa[6] = {2, 0, 1, 1, 0, 0}, pw[6] = {0, 2, 1, 0, 1, 0};  // smallest products first
                if (leader) {
#pragma unroll
                    for (int t = 0; t < 6; t++)
#pragma unroll
                        for (int k = 0; k < 2; k++) tc_mma_f16_ta(d, a + pa[t] * 16 + k * 8, w[pw[t]] + 2 * k, IDESC, (t | k) != 0);
                    tc_commit(smem_u32(&done[s]));
                }
                __syncwarp();
                s += 2;
                if (s >= RB) { s -= RB; ph ^= 1; }
            }
        }
        leave();
        gathered();
        return;
    }
    {
        // group 0 the even K blocks, group 1 the odd ones (one group alone paced the tile: 1000 cycles a K block)
        const int group = (warp - C::CONV) >> 2, pm = m0 + row;
        // gather: this row's position at tap (0, 0), and the words of the group's next block, one a lane
        int ih0 = 0, iw0 = 0, pix = -1, words = -1;
        auto words_of = [&](int i) {
            const int g = (kb0 + i) * 8 + (lane & 7);
            return i < nkb && g < p.n_kchunks ? __ldg(p.kinfo + g) : -1;
        };
        auto gather = [&](int i, int stage) {  // the row's 128 bytes of K block i, zeros outside the image; nobody else reads them
            const int mine = words;
            words = words_of(i + 2);
            const uint32_t dst = smem_u32(ringA + stage * A_BYTES + row * 128);
#pragma unroll 2
            for (int q = 0; q < 8; q++) {
                const int ki = __shfl_sync(0xffffffffu, mine, q);
                const int ih = ih0 + ((ki >> 24) & 0x7f), iw = iw0 + ((ki >> 16) & 0xff);
                const bool in = ki >= 0 && pix >= 0 && (unsigned)ih < (unsigned)p.H && (unsigned)iw < (unsigned)p.W;
                cp_async16_ca(dst + ((q ^ (row & 7)) << 4), in ? p.x + (size_t)(pix + ih * p.W + iw) * p.in_ld + (ki & 0xffff) * 4 : p.x, in ? 16u : 0u);
            }
            cp_async_commit();
        };
        if (GATHER) {
            if (pm < p.P) {
                const int n = pm / p.oHW, rem = pm - n * p.oHW, oh = rem / p.oW;
                ih0 = oh * p.dH - p.padH;
                iw0 = (rem - oh * p.oW) * p.dW - p.padW;
                pix = n * p.H * p.W;
            }
            words = words_of(group);
            gather(group, group);
        }
        int sa = group, s = group, s2 = group;  // stages of the raw activations, of K block i and of K block i - NA
        uint32_t pa = 0, ph2 = 0;
        for (int i = group; i < nkb; i += 2) {
            if (GATHER) {
                gather(i + 2, sa ^ 2);
                cp_async_wait<1>();
            } else {
                have = mbar_wait_bounded(smem_u32(&fullA[sa]), pa, p.wait_limit);
            }
            if (i >= NA) {
                have = mbar_wait_bounded(smem_u32(&done[s2]), ph2, p.wait_limit) && have;
                s2 += 2;
                if (s2 >= RB) { s2 -= RB; ph2 ^= 1; }
            }
            if (!__all_sync(0xffffffffu, have)) {
                if (lane == 0) give_up(5);
                break;
            }
            tc_fence_after();
            const uint8_t *src = ringA + sa * A_BYTES + row * 128;
            const uint32_t taddr = tmem + lanes + C::A_COL + (i & (NA - 1)) * 64;
            // (kept a loop: unrolled, the instructions of the three groups displace one another in the instruction cache)
#pragma unroll 1
            for (int q = 0; q < 4; q++) {
                const float4 a = *reinterpret_cast<const float4 *>(src + (((2 * q) ^ (row & 7)) << 4));
                const float4 b = *reinterpret_cast<const float4 *>(src + (((2 * q + 1) ^ (row & 7)) << 4));
                split_store(taddr + q * 4, a, b);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(smem_u32(&go[s]));
                if (!GATHER) mbar_arrive(smem_u32(&emptyA[sa]));
            }
            s += 2;
            if (s >= RB) s -= RB;
            if (GATHER) sa ^= 2;
            else {
                sa += 2;
                if (sa >= RA) { sa -= RA; pa ^= 1; }
            }
        }
        if (GATHER) cp_async_wait<0>();
    }
    // A thread stores four channels of every step-th row.  Their constants are read while the last multiplies run.
    const int t2 = tid - C::CONV * 32, step = 256 >> (wshift - 2), g = t2 & (G - 1), c0 = n0 + rank * W + g * 4;
    const int r0 = t2 >> (wshift - 2), rows = c0 < p.Cout ? min(BM, p.P - m0) : 0;
    Affine4 f(p, c0);
    const float4 unit = *reinterpret_cast<const float4 *>(p.units + c0), least = *reinterpret_cast<const float4 *>(p.units + p.Cout_pad + c0);
    // the units go into the scales where that loses nothing (they are 2^-100 at least); elsewhere no sum is ordinary
    const bool folded = min(min(magnitude(f.sc[0]), magnitude(f.sc[1])), min(magnitude(f.sc[2]), magnitude(f.sc[3]))) > magnitude(0x1p-26f);
    const bool idle = unit.x < 0.f || unit.y < 0.f || unit.z < 0.f || unit.w < 0.f;  // a channel without weights: its zeros are ordinary
    const float ordinary = !folded ? INFINITY : idle ? 0.f : max4(least.x, least.y, least.z, least.w);
    f.sc[0] *= fabsf(unit.x); f.sc[1] *= fabsf(unit.y); f.sc[2] *= fabsf(unit.z); f.sc[3] *= fabsf(unit.w);
    leave();
    gathered();
    if (*abort_flag) return;

    const uint8_t *part = recv + (size_t)g * RECV_ROWS * 16;
    unsigned rare = 0;  // the thread's rows that have a sum which is not ordinary
#pragma unroll 1
    for (int r = r0, k = 0; r < rows; r += 2 * step, k += 2) {
        float4 rv[2], v[2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            rv[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (p.res && r + j * step < rows) rv[j] = *reinterpret_cast<const float4 *>(p.res + (size_t)(m0 + r + j * step) * p.res_ld + c0);
        }
#pragma unroll
        for (int j = 0; j < 2; j++) v[j] = *reinterpret_cast<const float4 *>(part + min(r + j * step, BM - 1) * 16);
        for (int q = 1; q < S; q++) {
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const float4 u = *reinterpret_cast<const float4 *>(part + (q * G * RECV_ROWS + min(r + j * step, BM - 1)) * 16);
                v[j].x += u.x; v[j].y += u.y; v[j].z += u.z; v[j].w += u.w;
            }
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
            if (r + j * step >= rows) continue;
            if (min4(v[j].x, v[j].y, v[j].z, v[j].w) >= ordinary && max4(v[j].x, v[j].y, v[j].z, v[j].w) < INFINITY)
                f.store(p, m0 + r + j * step, c0, v[j], rv[j]);
            else
                rare |= 1u << (k + j);
        }
    }
    if (idle) {
        // (in a loop of its own: the instructions would slow the loop above down, 3 to 7 %)
        const float4 u = *reinterpret_cast<const float4 *>(p.units + c0), l = *reinterpret_cast<const float4 *>(p.units + p.Cout_pad + c0);
#pragma unroll 1
        for (int r = r0, k = 0; r < rows; r += step, k++) {
            float4 v = *reinterpret_cast<const float4 *>(part + r * 16);
            for (int q = 1; q < S; q++) {
                const float4 t = *reinterpret_cast<const float4 *>(part + (q * G * RECV_ROWS + r) * 16);
                v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
            }
            if ((u.x > 0.f && fabsf(v.x) < l.x) || (u.y > 0.f && fabsf(v.y) < l.y) || (u.z > 0.f && fabsf(v.z) < l.z) || (u.w > 0.f && fabsf(v.w) < l.w)) rare |= 1u << k;
        }
    }
    if (__any_sync(~0u, rare)) store_rare(p, part, rare, r0, step, S, G, m0, c0);
}

// fp32 weights [Ktot][Cout_pad] -> F32Params.units, 32 channels to a block of 32 x 32 threads.  A channel of largest weight 2^e (to
// 2^(e + 1)) is multiplied by 2^39, or more to bring it to 1, up to 2^100: its smallest weights, 2^-149, then come to 2^-110 or more,
// and a product that vanishes, below 2^-165, vanishes in fp32 as well.  Its sums are trusted while what 2^16 activations may have lost,
// 2^(-134 + 16) of its scaled weights, is below a quarter of their last bit; and from 2^-90 on, lest parts of products vanish.
__global__ void weight_units_kernel(const float *w, int Ktot, int Cout_pad, float *units)
{
    __shared__ float most[32][33];
    const int c = blockIdx.x * 32 + threadIdx.x;
    float m = 0.f;
#pragma unroll 4
    for (int k = threadIdx.y; k < Ktot; k += 32) m = fmaxf(m, fabsf(w[(size_t)k * Cout_pad + c]));
    most[threadIdx.y][threadIdx.x] = m;
    __syncthreads();
    if (threadIdx.y) return;
    for (int i = 1; i < 32; i++) m = fmaxf(m, most[i][threadIdx.x]);
    const int e = m == 0.f ? -39 : m < 0x1p26f ? ilogbf(m) : 26, up = max(39, min(100, -e));
    units[c] = m == 0.f ? -0x1p-39f : ldexpf(1.f, -up);
    units[Cout_pad + c] = e == 26 ? INFINITY : ldexpf(1.f, max(e + up - 91, -90));
}

// fp32 weights [Ktot][Cout_pad] -> F32Params.parts, zeros behind Ktot: 64 channels of one K block
__global__ void split_weights_kernel(const float *w, const float *units, int Ktot, int nkb, int Cout_pad, int BN, uint8_t *out)
{
    __shared__ float t[32][65];
    const int kb = blockIdx.x, n0 = blockIdx.y * 64;
    for (int i = threadIdx.x; i < 32 * 64; i += 256) {
        const int k = i / 64, n = i % 64;
        t[k][n] = kb * 32 + k < Ktot ? w[(size_t)(kb * 32 + k) * Cout_pad + n0 + n] * (1.f / fabsf(units[n0 + n])) : 0.f;
    }
    __syncthreads();
    const int part = BN * 64;  // bytes
    uint8_t *stage = out + ((size_t)(n0 / BN) * nkb + kb) * 3 * part + (n0 % BN) * 64;
    for (int i = threadIdx.x; i < 64 * 16; i += 256) {
        const int n = i >> 4, q = i & 15;  // a word: two values
        uint32_t p1, p2, p3;
        split_pair(t[2 * q][n], t[2 * q + 1][n], p1, p2, p3);
        const int at = n * 64 + (((q >> 2) ^ ((n >> 1) & 3)) << 4) + (q & 3) * 4;  // 64-byte swizzle
        *reinterpret_cast<uint32_t *>(stage + at) = p1;
        *reinterpret_cast<uint32_t *>(stage + part + at) = p2;
        *reinterpret_cast<uint32_t *>(stage + 2 * part + at) = p3;
    }
}


// How the activation operand is loaded (F32Params.mode), -1: not by this kernel
int operand_mode(const thb_conv_desc *d)
{
    if (d->kH == 1 && d->kW == 1 && d->dH == 1 && d->dW == 1 && d->padH == 0 && d->padW == 0 && d->oH == d->H && d->oW == d->W && d->Cin_pad % BK == 0) return 1;
    if (d->Cin_pad % BK == 0 && thb_im2col_ok(d)) return 2;
    return d->Cin_pad <= 16 ? 0 : -1;
}

int k_blocks(const thb_conv_desc *d) { return (d->Ktot_pad + BK - 1) / BK; }

// Channels of a tile as the weights are laid out (a property of the layer, not of the batch).  Reductions of fewer than four K
// blocks are mostly prologue and epilogue, which two small CTAs on an SM overlap: 1x1 64->256 @56x56, 16 images 45 -> 37 us, 64->512
// @28x28 25 -> 20; from 128 channels on it is even (128->512: 25.5 / 25.5), 3x3 128->128 of 64 images 95 -> 70 with 128.
int tile_n(const thb_conv_desc *d) { return d->Cout_pad % 128 == 0 && k_blocks(d) >= 4 ? 128 : 64; }

// Channels of a launch's tiles.  Where CTAs of 64 channels, as many parts a tile, take half of the SMs at most, a CTA takes half of a
// tile the weights are laid out for: a K block's multiplies take 540 cycles instead of 768, and beside its 113 KB of shared memory and
// half of the tensor memory the next launch of the chain sets itself up.  us of kernels, tiles of 128 / this / 64 up to all SMs:
// AlexNet, 1 image 117 / 115 / 112, 2 images 133 / 133 / 142; ResNet-50, 1 image 579 / 566 / 557, 4 images 658 / 658 / 668; ResNet-18,
// 3 images 267 / 263 / 276.
int launch_n(const thb_conv_desc *d, int splits, long sms)
{
    const long tiles = ((long)d->N * d->oH * d->oW + BM - 1) / BM * (d->Cout_pad / 64);
    return tile_n(d) == 128 && tiles * splits * 2 > sms ? 128 : 64;
}

template <int NT, bool GATHER> int launch(const CUtensorMap &a, const F32Params &p, cudaStream_t st)
{
    using C = Cfg<NT, GATHER>;
    const auto kern = conv_f32_kernel<NT, GATHER>;
    static bool set[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !set[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
        if (e != cudaSuccess) return thb_note_launch(e, "conv_f32_kernel attributes");
        if (dev >= 0 && dev < 64) set[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(((p.P + BM - 1) / BM) * p.n_tiles * p.splits));
    cfg.blockDim = dim3(C::NTHREADS);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (p.splits > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)p.splits;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        n++;
    }
    if (p.pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        n++;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    const cudaError_t le = cudaLaunchKernelEx(&cfg, kern, a, p);
    return thb_note_launch(le != cudaSuccess ? le : cudaGetLastError(), "conv_f32_kernel");
}

}  // namespace

extern "C" int thb_conv_f32_supported(const thb_conv_desc *d)
{
    // (from 64 products a sum on: with fewer, the FFMA chain's error is the smaller one)
    return d->dtype == THB_F32 && d->kH * d->kW * d->Cin >= 64 && !d->x2 && !d->in_row_pitch && d->Cout_pad % 64 == 0 && operand_mode(d) >= 0 && d->kH <= 127 && d->kW <= 255;
}

static size_t parts_bytes(const thb_conv_desc *d) { return (size_t)d->Cout_pad * k_blocks(d) * 3 * BK * 2; }

extern "C" size_t thb_conv_f32_split_bytes(const thb_conv_desc *d) { return parts_bytes(d) + 2 * d->Cout_pad * sizeof(float); }

extern "C" int thb_conv_f32_split_weights(const thb_conv_desc *d, void *w_split, thb_stream s)
{
    if (!thb_conv_f32_supported(d)) return THB_ERR_UNSUPPORTED;
    if (!d->w || !w_split) return THB_ERR_ARG;
    float *units = (float *)((uint8_t *)w_split + parts_bytes(d));
    weight_units_kernel<<<d->Cout_pad / 32, dim3(32, 32), 0, (cudaStream_t)s>>>((const float *)d->w, d->Ktot_pad, d->Cout_pad, units);
    const int rc = THB_LAUNCH_CHECK("weight_units_kernel");
    if (rc != THB_OK) return rc;
    split_weights_kernel<<<dim3(k_blocks(d), d->Cout_pad / 64), 256, 0, (cudaStream_t)s>>>((const float *)d->w, units, d->Ktot_pad, k_blocks(d),
                                                                                                d->Cout_pad, tile_n(d), (uint8_t *)w_split);
    return THB_LAUNCH_CHECK("split_weights_kernel");
}

// The reduction split while that leaves at most one CTA to an SM and at least four K blocks to a CTA; tiles of 64 channels (two CTAs fit
// an SM) once more where at least eight are left.  (Split on to two CTAs an SM at four K blocks each, us of kernels before / now:
// AlexNet, 2 images 137 / 133; ResNet-18, 3 images 292 / 263; ResNet-50, 3 images 634 / 604.  Never on to two: AlexNet, 8 images 232.)
// Measured, us in 1 / 2 / 4 / 8 parts (* the rule's choice; before: the FFMA kernel's own rule) and the relative error (2-norm,
// against double precision) of the choice / of the FFMA kernel:
//   7x7/2 3->64 @225x225, 9 images            52*                      before  85    7.5e-8 / 1.5e-7
//   3x3 64->64 @57x57, 9 images               21* / 26 / 37 / 65       before  61    9.9e-8 / 4.3e-7
//   3x3 128->128 @29x29, 9 images             24 / 17* / 25 / 44       before  62    9.1e-8 / 4.3e-7
//   3x3 256->256 @15x15, 9 images             39 / 24 / 18* / 37       before  60    9.7e-8 / 3.0e-7
//   3x3 512->512 @8x8, 9 images               69 / 40 / 26* / 34       before  88    1.1e-7 / 4.2e-7
//   1x1/2 64->128 @57x57, 9 images           6.4* / 7.9                before  9.5   6.0e-8 / 8.0e-8
//   1x1 64->256 @56x56, 16 images             37* / 75                 before  48    6.4e-8 / 1.4e-7
//   1x1 256->1024 @14x14, 16 images           21* / 28                 before  53    8.0e-8 / 2.9e-7
//   11x11/4 3->64 @224x224, 1 image           18 / 14 / 12* / 12       before  12    8.3e-8 / 1.1e-7
//   5x5 64->192 @27x27, 1 image               29 / 18 / 13 / 13*       before  27    9.4e-8 / 2.0e-7
//   3x3 384->256 @13x13, 1 image              53 / 31 / 20 / 15*       before  17    1.1e-7 / 2.7e-7
//   3x3 512->512 @7x7, 1 image                67 / 38 / 23 / 16*       before  20    1.1e-7 / 2.3e-7
//   6x6 256->4096 @18x25, 1 image            146* / 151 / 146 / 196    before 681    3.1e-7 / 6.1e-7 (of 512 channels)
//   512->1000 of 9 rows                       11 / 9.8 / 8.7 / 8.8*    before 7.5    8.5e-8 / 1.6e-7
extern "C" int thb_conv_f32_splits(const thb_conv_desc *d)
{
    const long sms = thb_conv_launch_knobs().sms, tiles = ((long)d->N * d->oH * d->oW + BM - 1) / BM * (d->Cout_pad / tile_n(d));
    const int nkb = k_blocks(d);
    int S = 1;
    while (S < 8 && (tiles * 2 * S <= sms ? nkb >= 4 * S : tile_n(d) == 64 && tiles * S <= sms && nkb >= 16 * S)) S *= 2;
    return S;
}

extern "C" int thb_conv_f32_fwd(const thb_conv_desc *d, const void *w_split, const void *x, void *y, thb_stream s)
{
    if (!d->w || !d->kinfo || !w_split || !x || !y || !d->status) return THB_ERR_ARG;
    if (!thb_conv_f32_supported(d)) return THB_ERR_UNSUPPORTED;
    if (d->in_ld < d->Cin_pad || d->in_ld % 4 || d->out_ld % 4 || (d->res && d->res_ld % 4)) return THB_ERR_ARG;
    F32Params p;
    memset(&p, 0, sizeof(p));
    p.x = (const float *)x; p.w = (const float *)d->w; p.y = (float *)y; p.kinfo = d->kinfo;
    p.P = d->N * d->oH * d->oW;
    p.H = d->H; p.W = d->W; p.in_ld = d->in_ld; p.oW = d->oW; p.oHW = d->oH * d->oW;
    p.dH = d->dH; p.dW = d->dW; p.padH = d->padH; p.padW = d->padW; p.kW = d->kW;
    p.Cout = d->Cout; p.Cout_pad = d->Cout_pad; p.out_ld = d->out_ld;
    p.n_kchunks = d->Ktot_pad / 4; p.nkb = k_blocks(d);
    p.scale = d->scale; p.shift = d->shift; p.slope = d->act.kind == THB_ACT_PRELU ? d->act.slope : nullptr;
    p.res = (const float *)d->res; p.res_ld = d->res_ld; p.self_coef = d->self_coef; p.res_coef = d->res_coef;
    p.act_kind = d->act.kind; p.act_th = d->act.threshold; p.act_val = d->act.value; p.act_alpha = d->act.alpha;
    if (p.P <= 0) return THB_OK;
    const ThbConvLaunch kn = thb_conv_launch_knobs();
    p.pdl = kn.pdl; p.wait_limit = kn.wait_limit; p.test_withhold = kn.test_withhold;
    p.status = d->status;
    p.mode = operand_mode(d);
    p.slabs = d->Cin_pad / BK;
    p.splits = d->splits > 0 ? d->splits : thb_conv_f32_splits(d);
    if (p.splits != 1 && p.splits != 2 && p.splits != 4 && p.splits != 8) return THB_ERR_ARG;
    while (p.splits > p.nkb) p.splits /= 2;
    const int bn = launch_n(d, p.splits, kn.sms);
    p.n_tiles = d->Cout_pad / bn;
    p.halves = bn < tile_n(d);
    p.parts = (const uint8_t *)w_split;
    p.units = (const float *)(p.parts + parts_bytes(d));
    CUtensorMap a = {};
    if (p.mode && !thb_activation_tmap(d, x, p.mode, &a)) return thb_note_launch(cudaErrorUnknown, "conv_f32: tensor map");
    const cudaStream_t st = (cudaStream_t)s;
    if (bn == 128) return p.mode ? launch<2, false>(a, p, st) : launch<2, true>(a, p, st);
    return p.mode ? launch<1, false>(a, p, st) : launch<1, true>(a, p, st);
}
