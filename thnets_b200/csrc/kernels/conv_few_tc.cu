// Tensor-core convolution for launches of few tiles (16-bit types, uint8): small batches, the late stages of a network.
//
// What bounds such a layer is not arithmetic or bandwidth but the chain of one tile: with 8 images or fewer a ResNet layer
// is 1 to 100 tiles, the persistent kernel (conv_tc.cu) runs one of them per SM, and a K block costs the SM's copy engine
// about 0.33 us (an im2col box of 128 rows) however idle the other SMs are: 72 K blocks of a 3x3 512->512 layer took 30 us.
// Here
//   * a tile is 128 pixels x 64 channels, one CTA works on one tile only, and two CTAs fit an SM;
//   * the K blocks of a tile are shared by the S = 1, 2, 4 or 8 CTAs of a thread-block cluster.  Each pushes the columns of
//     its fp32 partial tile to the CTA that owns them, through distributed shared memory, and every owner adds the S parts
//     in rank order and finishes its 64 / S channels (no atomics, no scratch in global memory, no second launch);
//   * weights and activations are loaded by two different warps, and since weights do not depend on the kernel before, their
//     loads start ahead of griddepcontrol.wait, under that kernel's tail;
//   * the epilogue goes from registers to global memory.
// Measured: the tables at thb_conv_few_splits and thb_conv_few_supported.  ResNet-18, 1 image: 305 -> 155 us of kernels;
// ResNet-50, 8 images: 727 -> 480 us.
//
// Every mbarrier wait is bounded; one that runs out records a code in *status and the CTA drains (all its threads still
// reach both cluster barriers, so that its peers end too).
#include <cuda.h>
#include <string.h>
#include "common.cuh"
#include "conv_maps.cuh"

namespace {

constexpr int BM = 128, BN = 64;
constexpr int NTHREADS = 224;  // 4 epilogue warps, activation producer, weight producer, MMA issuer
constexpr int A_BYTES = BM * 128, B_BYTES = BN * 128, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int MAX_STAGES = 8;
constexpr int BAR_BYTES = 1024;
constexpr int RECV_BYTES = BM * BN * 4;  // the partial columns a CTA receives, its own included

struct FewParams {
    uint8_t *y;
    float *y_nchw;             // not null: the result goes here as NCHW floats (device or pinned host memory) instead of to y
    const int *prev_status;    // with y_nchw: the status word of the launches before, passed on to `status` when set
    const uint8_t *res;
    const float *scale, *shift, *slope;
    int P, oW, oHW, dH, dW, padH, padW, kW, Cout, out_ld, res_ld, nkb, n_tiles;
    float self_coef, res_coef;
    int act_kind;
    float act_th, act_val, act_alpha;
    int mode;                  // 1: activations are a plain matrix; 2: im2col-mode copies, `slabs` 128-byte slabs per tap
    int slabs, tma_kw, tma_padw;
    int nkb1, a2_mode, a2_d;   // second activation operand from K block nkb1 on (1: plain matrix, 2: sampled every a2_d pixels)
    int half, ntaps;           // a tap (a kernel row stored with its padding) is half a K block: two copies of 64-byte rows a block
    int splits, stages, pdl;
    // uint8: zero-point correction, requantisation, bias and Threshold as in the persistent kernel (conv_tc.cu)
    int H, W, kH, Cin, a_off, b_off, c_off, c_mult, c_shift, tail_start, relu_thr, relu_val, ca, cb, res_addend;
    int classes, tbl_bytes;    // border classes of the kernel window, and the bytes their table takes
    const int *wsat, *bias_add, *csum;
    int *csum_out;
    int test_withhold;         // tests only: the last K block's activations are never delivered
    int *status;
    long long wait_limit;
};

// (a plain store: the word may lie in pinned host memory)
__device__ __forceinline__ void report(int *status, int code) { *reinterpret_cast<volatile int *>(status) = code; }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_addr(uint32_t smem, uint32_t rank)
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem), "r"(rank));
    return a;
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

template <int KIND> __device__ __forceinline__ uint32_t pack2(float a, float b)
{
    if (KIND == 0) {
        __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<uint32_t *>(&h);
    }
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&h);
}
template <int KIND> __device__ __forceinline__ float2 unpack2(uint32_t v)
{
    if (KIND == 0) return __half22float2(*reinterpret_cast<__half2 *>(&v));
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162 *>(&v));
}

// Per-channel constants of the tile in shared memory: scale and shift (times self_coef when a residual is fused), slope.
struct Consts {
    float sc[BN], sh[BN], sl[BN];
};

// Eight channels of one pixel, the first of them channel c of the tile: y = act(acc * scale + shift + res_coef * residual),
// channels >= Cout zero.  The operations and their order are those of the persistent kernel's epilogue: the same bits.
// ACT: 0 none, 1 plain ReLU, 2 anything.  The variant is chosen once per tile: with the general activation inlined in every
// chunk the epilogue was bound by instruction fetch (0.8 us per chunk of eight channels).
template <int KIND, int ACT>
__device__ __forceinline__ uint4 finish8(const float (&acc)[8], const uint4 &rv, int c, int left, const Consts &k, const FewParams &p)
{
    const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
    uint32_t ow[4];
#pragma unroll
    for (int h = 0; h < 4; h++) {
        float v[2];
        const float2 rr = unpack2<KIND>(rw[h]);
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int i = 2 * h + e;
            v[e] = fmaf(acc[i], k.sc[c + i], k.sh[c + i]);
            if (p.res) v[e] = fmaf(p.res_coef, e ? rr.y : rr.x, v[e]);
            if (ACT == 1) v[e] = fmaxf(v[e], 0.f);
            if (ACT == 2) v[e] = thb_apply_act(v[e], p.act_kind, p.act_th, p.act_val, p.act_alpha, k.sl[c + i]);
            if (i >= left) v[e] = 0.f;
        }
        ow[h] = pack2<KIND>(v[0], v[1]);
    }
    return make_uint4(ow[0], ow[1], ow[2], ow[3]);
}

// The thread's pixel, straight from its TMEM lane (no split): 64 channels.
template <int KIND, int ACT>
__device__ __forceinline__ void finish_tmem(uint32_t taddr, const uint4 (&rv)[BN / 8], uint8_t *dst, bool real, int left, const Consts &k,
                                            const FewParams &p)
{
#pragma unroll(ACT == 2 ? 1 : 8)
    for (int j = 0; j < BN / 8; j++) {
        uint32_t a[8];
        tmem_ld8(taddr + j * 8, a);
        tmem_ld_wait();
        float acc[8];
#pragma unroll
        for (int i = 0; i < 8; i++) acc[i] = __uint_as_float(a[i]);
        uint4 res = rv[0];
#pragma unroll
        for (int q = 1; q < BN / 8; q++)  // (constant indices keep the residual in registers)
            if (q == j) res = rv[q];
        const uint4 o = finish8<KIND, ACT>(acc, res, j * 8, left - j * 8, k, p);
        if (real && j * 8 < left) *reinterpret_cast<uint4 *>(dst + j * 16) = o;
    }
}

// The same for a network's last convolution, whose result leaves as NCHW floats (rounded through the 16-bit type like any
// other): a warp's lanes are 32 neighbouring pixels of a plane, so every channel is a coalesced 128-byte store.
template <int KIND, int ACT>
__device__ __forceinline__ void finish_nchw(uint32_t taddr, const uint4 (&rv)[BN / 8], float *dst, size_t plane, bool real, int left, const Consts &k,
                                            const FewParams &p)
{
#pragma unroll 1
    for (int j = 0; j < BN / 8 && j * 8 < left; j++) {
        uint32_t a[8];
        tmem_ld8(taddr + j * 8, a);
        tmem_ld_wait();
        float acc[8];
#pragma unroll
        for (int i = 0; i < 8; i++) acc[i] = __uint_as_float(a[i]);
        uint4 res = rv[0];
#pragma unroll
        for (int q = 1; q < BN / 8; q++)
            if (q == j) res = rv[q];
        const uint4 o = finish8<KIND, ACT>(acc, res, j * 8, left - j * 8, k, p);
        const uint32_t w[4] = {o.x, o.y, o.z, o.w};
        if (real) {
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const float2 v = unpack2<KIND>(w[h]);
                if (j * 8 + 2 * h < left) dst[(j * 8 + 2 * h) * plane] = v.x;
                if (j * 8 + 2 * h + 1 < left) dst[(j * 8 + 2 * h + 1) * plane] = v.y;
            }
        }
    }
}

// The same for the W = 64 / S channels this CTA owns, summing the S parts its peers (and itself) left in `recv`.
template <int KIND, int ACT>
__device__ __forceinline__ void finish_parts(const uint8_t *recv, int S, int W, int c_local, const uint4 (&rv)[BN / 8], uint8_t *dst, int left,
                                             int row, const Consts &k, const FewParams &p)
{
#pragma unroll 1
    for (int j = 0; j < W / 8 && j * 8 < left; j++) {
        float acc[8];
#pragma unroll
        for (int i = 0; i < 8; i++) acc[i] = 0.f;
        const float4 *part = reinterpret_cast<const float4 *>(recv) + (size_t)(2 * j) * BM + row;
        for (int r = 0; r < S; r++, part += (W >> 2) * BM) {
            const float4 u = part[0], v = part[BM];
            acc[0] += u.x; acc[1] += u.y; acc[2] += u.z; acc[3] += u.w;
            acc[4] += v.x; acc[5] += v.y; acc[6] += v.z; acc[7] += v.w;
        }
        uint4 res = rv[0];
#pragma unroll
        for (int q = 1; q < BN / 16; q++)  // (W <= 32 here)
            if (q == j) res = rv[q];
        *reinterpret_cast<uint4 *>(dst + j * 16) = finish8<KIND, ACT>(acc, res, c_local + j * 8, left - j * 8, k, p);
    }
}

// Eight channels of one pixel in uint8: zero-point correction (the border class's table word times c_mult, the row's own term),
// gemmlowp requantisation, the reference's saturating bias add with its tail quirk, the fused residual and the Threshold -- the
// integer arithmetic of the persistent kernel's u8_chunk32.
struct U8Row {
    uint32_t rc;
    int tailmask, thr, shift;
};
__device__ __forceinline__ uint2 finish8_u8(const int (&acc)[8], const int *t, const int *b, const U8Row &e, const uint2 &rv, int left,
                                            const FewParams &p)
{
    uint32_t ow[2] = {0, 0};
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int sres = (int)((uint32_t)acc[i] * (uint32_t)p.c_mult + (uint32_t)t[i] + e.rc) >> e.shift;
        const int q = min(max(sres, 0), 255), t2 = q + b[i];
        int v = max(min(max(t2, 0), 255), t2 & e.tailmask);
        if (p.res) {
            const int r = (int)(((i < 4 ? rv.x : rv.y) >> (8 * (i & 3))) & 255u);
            v = min(max(p.ca * v + p.cb * r + p.res_addend, 0), 255);
        }
        v = v > e.thr ? v : p.relu_val;
        if (i < left) ow[i >> 2] |= (uint32_t)v << (8 * (i & 3));
    }
    return make_uint2(ow[0], ow[1]);
}

template <int KIND>
__global__ void __launch_bounds__(NTHREADS) conv_few_kernel(const __grid_constant__ CUtensorMap tmapW, const __grid_constant__ CUtensorMap tmapA,
                                                            const __grid_constant__ CUtensorMap tmapA2, const FewParams p)
{
    constexpr uint32_t IDESC = make_idesc(KIND == 2 ? 2u : 1u, KIND == 1 ? 1u : 0u, BN);
    constexpr int KE = KIND == 2 ? 128 : 64;  // elements of a K block
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem), *empty = full + MAX_STAGES, *acc_full = empty + MAX_STAGES;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    Consts &consts = *reinterpret_cast<Consts *>(smem + 192);
    static_assert(192 + sizeof(Consts) <= BAR_BYTES, "barriers and constants share the first kilobyte");
    // (every CTA of a cluster has the same layout, so an offset into this one's receive buffer fits its peers' too)
    uint8_t *recv = smem + BAR_BYTES;
    uint8_t *ring = recv + (p.splits > 1 ? RECV_BYTES : 0);
    int *tbl = reinterpret_cast<int *>(ring), *bias = reinterpret_cast<int *>(smem + 192);  // uint8
    if (KIND == 2) ring += p.tbl_bytes;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int S = p.splits, nst = p.stages;
    const int rank = S > 1 ? (int)(blockIdx.x % S) : 0, tile = S > 1 ? (int)(blockIdx.x / S) : (int)blockIdx.x;
    const int m0 = (tile / p.n_tiles) * BM, n0 = (tile % p.n_tiles) * BN;
    const int kb0 = (int)((long)p.nkb * rank / S), kb1 = (int)((long)p.nkb * (rank + 1) / S);

    if (tid == 0) {
        for (int s = 0; s < nst; s++) {
            mbar_init(smem_u32(&full[s]), 2);  // the two producers
            mbar_init(smem_u32(&empty[s]), 1);
        }
        mbar_init(smem_u32(acc_full), 1);
        *abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async_smem();
    }
    if (KIND == 2) {
        // T[class][channel] = b_off * (sum of the channel's weights over the taps inside the image) * c_mult
        const int ncc = 1 + 2 * p.padW, satw = p.kW + 1, satn = (p.kH + 1) * satw;
        for (int i = tid; i < p.classes * BN; i += NTHREADS) {
            const int k = i / BN, c = min(n0 + i % BN, p.Cout - 1), rc = k / ncc, cc = k - rc * ncc;
            const int r0 = rc <= p.padH ? rc : 0, r1 = rc > p.padH ? p.kH - (rc - p.padH) : p.kH;
            const int s0 = cc <= p.padW ? cc : 0, s1 = cc > p.padW ? p.kW - (cc - p.padW) : p.kW;
            const int *t = p.wsat + (size_t)c * satn;
            tbl[i] = (int)((uint32_t)(p.b_off * (__ldg(t + r1 * satw + s1) - __ldg(t + r0 * satw + s1) - __ldg(t + r1 * satw + s0) +
                                                 __ldg(t + r0 * satw + s0))) * (uint32_t)p.c_mult);
        }
        if (tid < BN) bias[tid] = p.bias_add ? __ldg(p.bias_add + min(n0 + tid, p.Cout - 1)) : 0;
    } else if (tid < BN) {  // (weights, like the packed matrix: no launch of the forward writes them)
        const float self = p.res ? p.self_coef : 1.f;
        consts.sc[tid] = (p.scale ? __ldg(p.scale + n0 + tid) : 1.f) * self;
        consts.sh[tid] = (p.shift ? __ldg(p.shift + n0 + tid) : 0.f) * self;
        consts.sl[tid] = p.slope ? __ldg(p.slope + n0 + tid) : 0.f;
    }
    if (warp == 4 && lane == 0) {
        tma_prefetch_desc(&tmapA);
        if (p.nkb1) tma_prefetch_desc(&tmapA2);
    }
    if (warp == 5 && lane == 0) tma_prefetch_desc(&tmapW);
    if (warp == 6) {
        tmem_alloc(smem_u32(tmem_slot), BN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (S > 1) cluster_arrive();  // (the wait is ahead of the first store to a peer)
    if (p.pdl) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // weights are not written by any launch of the forward: their producer does not wait for the kernel before
    if (p.pdl && warp != 5) asm volatile("griddepcontrol.wait;" ::: "memory");

    uint4 rv[BN / 8];
    uint2 r8[BN / 8];   // uint8
    U8Row u8 = {0, 0, -1, 0};
    const int *trow = tbl;
    const int row = tid;  // epilogue threads: pixel row of the tile = TMEM lane
    const int pm = m0 + row;
    const int wshift = S == 1 ? 6 : S == 2 ? 5 : S == 4 ? 4 : 3, W = 1 << wshift, c_first = n0 + rank * W, cout8 = (p.Cout + 7) & ~7;  // the channels this CTA finishes
    const int act = p.act_kind == THB_ACT_NONE ? 0 : p.act_kind == THB_ACT_THRESHOLD && p.act_th == 0.f && p.act_val == 0.f ? 1 : 2;
    bool have = false;

    if (p.prev_status && blockIdx.x == 0 && tid == 0) {
        const int before = *p.prev_status;
        if (before) report(p.status, before);
    }
    if (warp < 4) {
        // the residual of this thread's pixel, asked for before the accumulator is awaited
#pragma unroll
        for (int j = 0; j < BN / 8; j++) {
            rv[j] = make_uint4(0, 0, 0, 0);
            if (KIND != 2 && p.res && pm < p.P && j * 8 < W && c_first + j * 8 < cout8)
                rv[j] = __ldg(reinterpret_cast<const uint4 *>(p.res + ((size_t)pm * p.res_ld + c_first + j * 8) * 2));
        }
        if (KIND == 2) {
#pragma unroll
            for (int j = 0; j < BN / 8; j++) {
                r8[j] = make_uint2(0, 0);
                if (p.res && pm < p.P && j * 8 < W && c_first + j * 8 < cout8)
                    r8[j] = __ldg(reinterpret_cast<const uint2 *>(p.res + (size_t)pm * p.res_ld + c_first + j * 8));
            }
            const int pc = min(pm, p.P - 1), n = pc / p.oHW, rem = pc - n * p.oHW, oh = rem / p.oW, ow = rem - oh * p.oW;
            const int ihb = oh * p.dH - p.padH, iwb = ow * p.dW - p.padW;
            const int r0 = max(0, -ihb), r1 = min(p.kH, p.H - ihb), s0 = max(0, -iwb), s1 = min(p.kW, p.W - iwb);
            const int cb = p.kH - r1, cr = p.kW - s1;  // (clipped on one side at most: the launcher checks)
            trow = tbl + ((r0 > 0 ? r0 : cb > 0 ? p.padH + cb : 0) * (1 + 2 * p.padW) + (s0 > 0 ? s0 : cr > 0 ? p.padW + cr : 0)) * BN + rank * W;
            const int *cs = p.csum + ((size_t)n * p.H + ihb) * p.W + iwb;
            int xsum = 0;
            if (p.kH <= 4 && p.kW <= 4) {
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const int r = i >> 2, q = i & 3;
                    xsum += r >= r0 && r < r1 && q >= s0 && q < s1 ? __ldg(cs + r * p.W + q) : 0;
                }
            } else
                for (int r = r0; r < r1; r++)
                    for (int q = s0; q < s1; q++) xsum += __ldg(cs + r * p.W + q);
            const int corr = p.a_off * (xsum + p.b_off * (r1 - r0) * (s1 - s0) * p.Cin);
            u8.shift = max(p.c_shift, 0);
            u8.rc = (uint32_t)(corr + p.c_off) * (uint32_t)p.c_mult + (p.c_shift >= 1 ? 1u << (p.c_shift - 1) : 0u);
            u8.tailmask = rem < p.tail_start ? 0 : 255;
            u8.thr = p.relu_thr;
        }
        have = mbar_wait_bounded(smem_u32(acc_full), 0, p.wait_limit);
        if (!have) {
            if (lane == 0) report(p.status, 2);
            *abort_flag = 1;
        }
        have = __all_sync(0xffffffffu, have);
        tc_fence_after();
    } else if (warp == 4) {
        if (lane == 0) {
            int iw = 0, ih = 0, in = 0, tap_w = 0, tap_h = 0, slab = 0;
            if (p.mode == 2) {
                in = m0 / p.oHW;
                const int rem = m0 - in * p.oHW, oh = rem / p.oW;
                ih = oh * p.dH - p.padH;
                iw = (rem - oh * p.oW) * p.dW - p.tma_padw;
                const int tap = KIND == 2 && p.half ? 2 * kb0 : kb0 / p.slabs;
                slab = KIND == 2 && p.half ? 0 : kb0 - tap * p.slabs;
                tap_h = tap / p.tma_kw;
                tap_w = tap - tap_h * p.tma_kw;
            } else if (p.a2_mode == 2) {
                in = m0 / p.oHW;
                const int rem = m0 - in * p.oHW, oh = rem / p.oW;
                ih = oh * p.a2_d;
                iw = (rem - oh * p.oW) * p.a2_d;
            }
            int s = 0;
            uint32_t ph = 0;
            for (int kb = kb0; kb < kb1; kb++) {
                if (kb - kb0 >= nst && !mbar_wait_bounded(smem_u32(&empty[s]), ph ^ 1, p.wait_limit)) {
                    report(p.status, 3);
                    *abort_flag = 1;
                    break;
                }
                if (p.test_withhold && kb == kb1 - 1) break;
                const uint32_t bar = smem_u32(&full[s]), dst = smem_u32(ring + s * STAGE_BYTES);
                if (KIND == 2 && p.half) {
                    const int nh = 2 * kb + 1 < p.ntaps ? 2 : 1;
                    mbar_arrive_expect_tx(bar, (uint32_t)(nh * (A_BYTES / 2)));
                    for (int h = 0; h < nh; h++) {
                        tma_load_im2col_4d(dst + h * (A_BYTES / 2), &tmapA, bar, 0, iw, ih, in, (uint16_t)tap_w, (uint16_t)tap_h);
                        if (++tap_w == p.tma_kw) { tap_w = 0; tap_h++; }
                    }
                    if (++s == nst) { s = 0; ph ^= 1; }
                    continue;
                }
                mbar_arrive_expect_tx(bar, A_BYTES);
                if (p.nkb1 && kb >= p.nkb1) {
                    if (p.a2_mode == 1) tma_load_2d(dst, &tmapA2, bar, (kb - p.nkb1) * KE, m0);
                    else tma_load_im2col_4d(dst, &tmapA2, bar, (kb - p.nkb1) * KE, iw, ih, in, 0, 0);
                } else if (p.mode == 1) {
                    tma_load_2d(dst, &tmapA, bar, kb * KE, m0);
                } else {
                    tma_load_im2col_4d(dst, &tmapA, bar, slab * KE, iw, ih, in, (uint16_t)tap_w, (uint16_t)tap_h);
                    if (++slab == p.slabs) {
                        slab = 0;
                        if (++tap_w == p.tma_kw) { tap_w = 0; tap_h++; }
                    }
                }
                if (++s == nst) { s = 0; ph ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == 5) {
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            for (int kb = kb0; kb < kb1; kb++) {
                if (kb - kb0 >= nst && !mbar_wait_bounded(smem_u32(&empty[s]), ph ^ 1, p.wait_limit)) {
                    report(p.status, 3);
                    *abort_flag = 1;
                    break;
                }
                const uint32_t bar = smem_u32(&full[s]);
                const uint32_t dst = smem_u32(ring + s * STAGE_BYTES + A_BYTES);
                if (KIND == 2 && p.half) {
                    const int nh = 2 * kb + 1 < p.ntaps ? 2 : 1;
                    mbar_arrive_expect_tx(bar, (uint32_t)(nh * (B_BYTES / 2)));
                    for (int h = 0; h < nh; h++) tma_load_2d(dst + h * (B_BYTES / 2), &tmapW, bar, (2 * kb + h) * (KE / 2), n0);
                } else {
                    mbar_arrive_expect_tx(bar, B_BYTES);
                    tma_load_2d(dst, &tmapW, bar, kb * KE, n0);
                }
                if (++s == nst) { s = 0; ph ^= 1; }
            }
        }
        __syncwarp();
    } else {
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            bool alive = true;
            for (int kb = kb0; kb < kb1; kb++) {
                if (!mbar_wait_bounded(smem_u32(&full[s]), ph, p.wait_limit)) {
                    report(p.status, 4);
                    *abort_flag = 1;
                    alive = false;
                    break;
                }
                tc_fence_after();
                const uint32_t sa = smem_u32(ring + s * STAGE_BYTES), sb = sa + A_BYTES;
                if (KIND == 2 && p.half) {
                    const int nh = 2 * kb + 1 < p.ntaps ? 2 : 1;
                    for (int h = 0; h < nh; h++) {
                        const uint64_t ad = make_sw64_kmajor_desc(sa + h * (A_BYTES / 2)), bd = make_sw64_kmajor_desc(sb + h * (B_BYTES / 2));
#pragma unroll
                        for (int k = 0; k < 2; k++) {
                            if (KIND == 2) tc_mma_i8(tmem_base, ad + 2 * k, bd + 2 * k, IDESC, ((kb - kb0) | h | k) != 0);
                            else tc_mma_f16(tmem_base, ad + 2 * k, bd + 2 * k, IDESC, ((kb - kb0) | h | k) != 0);
                        }
                    }
                } else {
                    const uint64_t ad = make_sw128_kmajor_desc(sa), bd = make_sw128_kmajor_desc(sb);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        if (KIND == 2) tc_mma_i8(tmem_base, ad + 2 * k, bd + 2 * k, IDESC, ((kb - kb0) | k) != 0);
                        else tc_mma_f16(tmem_base, ad + 2 * k, bd + 2 * k, IDESC, ((kb - kb0) | k) != 0);
                    }
                }
                if (kb + nst < kb1) tc_commit(smem_u32(&empty[s]));
                if (++s == nst) { s = 0; ph ^= 1; }
            }
            if (alive) tc_commit(smem_u32(acc_full));
        }
        __syncwarp();
    }
    if (S > 1) {
        __syncwarp();
        cluster_wait();  // every CTA of the cluster has started
        if (have) {
#pragma unroll
            for (int half = 0; half < BN; half += 32) {
                uint32_t a[32];
                __syncwarp();
                tmem_ld32(tmem_base + ((uint32_t)(warp * 32) << 16) + half, a);
                tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    // columns half + 4q .. + 3 belong to CTA `owner`; slot [rank][column group][row] of its buffer
                    const int c = half + 4 * q, owner = c >> wshift, g = (c & (W - 1)) >> 2;
                    const uint32_t at = smem_u32(recv + (size_t)((rank * (W >> 2) + g) * BM + row) * 16);
                    st_cluster_v4(cluster_addr(at, owner), a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
                }
            }
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        if constexpr (KIND == 2) {
            if (have && pm < p.P) {
                uint32_t rowsum = 0;
                const int left = p.Cout - c_first, left16 = ((p.Cout + 15) & ~15) - c_first;
#pragma unroll 1
                for (int j = 0; j < W / 8 && j * 8 < left16; j++) {
                    int acc[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) acc[i] = 0;
                    const int4 *part = reinterpret_cast<const int4 *>(recv) + (size_t)(2 * j) * BM + row;
                    for (int r = 0; r < S; r++, part += (W >> 2) * BM) {
                        const int4 u = part[0], v = part[BM];
                        acc[0] += u.x; acc[1] += u.y; acc[2] += u.z; acc[3] += u.w;
                        acc[4] += v.x; acc[5] += v.y; acc[6] += v.z; acc[7] += v.w;
                    }
                    uint2 res = r8[0];
#pragma unroll
                    for (int q = 1; q < BN / 16; q++)
                        if (q == j) res = r8[q];
                    const uint2 o = finish8_u8(acc, trow + j * 8, bias + rank * W + j * 8, u8, res, left - j * 8, p);
                    *reinterpret_cast<uint2 *>(p.y + (size_t)pm * p.out_ld + c_first + j * 8) = o;
                    rowsum = __dp4a(o.x, 0x01010101u, __dp4a(o.y, 0x01010101u, rowsum));
                }
                if (p.csum_out && left > 0) atomicAdd(p.csum_out + pm, (int)rowsum);
            }
        } else if constexpr (KIND != 2) if (have && pm < p.P) {
            uint8_t *dst = p.y + ((size_t)pm * p.out_ld + c_first) * 2;
            const int left = p.Cout - c_first;
            if (act == 0) finish_parts<KIND, 0>(recv, S, W, rank * W, rv, dst, left, row, consts, p);
            else if (act == 1) finish_parts<KIND, 1>(recv, S, W, rank * W, rv, dst, left, row, consts, p);
            else finish_parts<KIND, 2>(recv, S, W, rank * W, rv, dst, left, row, consts, p);
        }
    } else if constexpr (KIND == 2) {
        if (have) {
            const uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16);
            uint32_t rowsum = 0;
            const int left = p.Cout - n0, left16 = ((p.Cout + 15) & ~15) - n0;
            __syncwarp();
#pragma unroll 1
            for (int j = 0; j < BN / 8 && j * 8 < left16; j++) {
                uint32_t a[8];
                tmem_ld8(taddr + j * 8, a);
                tmem_ld_wait();
                int acc[8];
#pragma unroll
                for (int i = 0; i < 8; i++) acc[i] = (int)a[i];
                uint2 res = r8[0];
#pragma unroll
                for (int q = 1; q < BN / 8; q++)
                    if (q == j) res = r8[q];
                const uint2 o = finish8_u8(acc, trow + j * 8, bias + j * 8, u8, res, left - j * 8, p);
                if (pm < p.P) *reinterpret_cast<uint2 *>(p.y + (size_t)pm * p.out_ld + n0 + j * 8) = o;
                rowsum = __dp4a(o.x, 0x01010101u, __dp4a(o.y, 0x01010101u, rowsum));
            }
            if (p.csum_out && pm < p.P) {
                if (p.n_tiles == 1) p.csum_out[pm] = (int)rowsum;
                else atomicAdd(p.csum_out + pm, (int)rowsum);  // (the buffer was cleared before the launch)
            }
        }
    } else if (have && p.y_nchw) {
        const uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16);
        const bool real = pm < p.P;
        const int img = pm / p.oHW;
        float *dst = p.y_nchw + ((size_t)img * p.Cout + n0) * p.oHW + (pm - img * p.oHW);
        __syncwarp();
        if (act == 0) finish_nchw<KIND, 0>(taddr, rv, dst, p.oHW, real, p.Cout - n0, consts, p);
        else if (act == 1) finish_nchw<KIND, 1>(taddr, rv, dst, p.oHW, real, p.Cout - n0, consts, p);
        else finish_nchw<KIND, 2>(taddr, rv, dst, p.oHW, real, p.Cout - n0, consts, p);
    } else if (have) {
        const uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16);
        uint8_t *dst = p.y + ((size_t)pm * p.out_ld + n0) * 2;
        const bool real = pm < p.P;
        __syncwarp();
        if (act == 0) finish_tmem<KIND, 0>(taddr, rv, dst, real, p.Cout - n0, consts, p);
        else if (act == 1) finish_tmem<KIND, 1>(taddr, rv, dst, real, p.Cout - n0, consts, p);
        else finish_tmem<KIND, 2>(taddr, rv, dst, real, p.Cout - n0, consts, p);
    }
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && warp == 4 && lane == 0) {
        // a wait ran out: copies still on their way must land before the CTA may leave
        const int n = kb1 - kb0 < nst ? kb1 - kb0 : nst;
        for (int s = 0; s < n; s++) mbar_wait_bounded(smem_u32(&full[s]), ((kb1 - kb0 - 1 - s) / nst) & 1, p.wait_limit);
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 6) tmem_dealloc(tmem_base, BN);
}

// How the activation operand is loaded: 0 not at all (a gather would be needed), else FewParams.mode and its companions.
int operand_mode(const thb_conv_desc *d, FewParams &p, int &tmap_mode)
{
    const bool plain = d->kH == 1 && d->kW == 1 && d->dH == 1 && d->dW == 1 && d->padH == 0 && d->padW == 0 && d->oH == d->H && d->oW == d->W;
    const int bke = d->dtype == THB_U8 ? 128 : 64;
    p.slabs = d->Cin_pad / bke;
    p.tma_kw = d->kW;
    p.tma_padw = d->padW;
    p.half = 0;
    p.ntaps = d->kH * d->kW;
    if (d->in_row_pitch) {
        if (!thb_im2col_ok(d) || d->dW != 1) return 0;
        p.slabs = 1;
        p.tma_kw = 1;
        p.tma_padw = 0;
        p.ntaps = d->kH;
        if (d->kW * d->Cin_pad == bke && d->Ktot_pad == d->kH * bke) {
            tmap_mode = 3;
            return 2;
        }
        p.half = 1;
        tmap_mode = 5;
        return d->dtype == THB_U8 && d->kW * d->Cin_pad * 2 == bke && d->Ktot_pad == (d->kH + 1) / 2 * bke ? 2 : 0;
    }
    tmap_mode = plain ? 1 : 2;
    if (plain) return 1;
    if (!thb_im2col_ok(d)) return 0;
    if (d->dtype == THB_U8 && d->Cin_pad * 2 == bke && d->Ktot_pad == (p.ntaps + 1) / 2 * bke) {
        p.half = 1;
        tmap_mode = 4;
        return 2;
    }
    return d->Cin_pad % bke == 0 && d->Ktot_pad == d->kH * d->kW * d->Cin_pad ? 2 : 0;
}

long tiles_of(const thb_conv_desc *d) { return (((long)d->N * d->oH * d->oW + BM - 1) / BM) * ((d->Cout_pad + BN - 1) / BN); }

bool eligible(const thb_conv_desc *d)
{
    if (d->dtype == THB_U8) {
        // (the table of border classes needs windows that are clipped on one side at most, by no more than the padding)
        if (d->x2 || d->acc_out || d->in_ld % 16 || d->out_ld % 16 || (d->res && d->res_ld % 16)) return false;
        if (d->H < d->kH || d->W < d->kW || d->padH >= d->kH || d->padW >= d->kW || (1 + 2 * d->padH) * (1 + 2 * d->padW) > 25) return false;
        if ((d->oH - 1) * d->dH + d->kH - d->H > 2 * d->padH || (d->oW - 1) * d->dW + d->kW - d->W > 2 * d->padW) return false;
    } else if (d->dtype != THB_F16 && d->dtype != THB_BF16) return false;
    else if ((d->Cout_pad % BN && d->Cout_pad != 32) || d->acc_out || d->csum_out || d->splitk_scratch) return false;
    else if (d->in_ld % 8 || d->out_ld % 8 || (d->res && d->res_ld % 8)) return false;
    FewParams p;
    int tm;
    const int mode = operand_mode(d, p, tm), allowed = thb_conv_launch_knobs().a_tma;
    return mode != 0 && (allowed < 0 || allowed == 2 || mode <= allowed);
}

template <int KIND>
int launch(const CUtensorMap *w, const CUtensorMap *a, const CUtensorMap *a2, const FewParams &p, int ctas, int smem, cudaStream_t st)
{
    static bool set[64];
    int dev = 0;
    cudaGetDevice(&dev);
    auto kern = conv_few_kernel<KIND>;
    if (dev >= 0 && dev < 64 && !set[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
        if (e != cudaSuccess) return thb_note_launch(e, "conv_few_kernel attributes");
        set[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(NTHREADS);
    cfg.dynamicSmemBytes = (size_t)smem;
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
    const cudaError_t le = cudaLaunchKernelEx(&cfg, kern, *w, *a, *a2, p);
    return thb_note_launch(le != cudaSuccess ? le : cudaGetLastError(), "conv_few_kernel");
}

}  // namespace

// How many CTAs should share the reduction of each tile of this convolution in conv_few_kernel (1: none need to).  Measured, us
// per launch in a chain of launches (the persistent kernel / no split / split in 2 / 4 / 8):
//   3x3 512->512 @7x7,  1 image,  8 tiles of 72 K blocks   28.9 / 25.4 / 15.2 / 9.6 / 7.3
//   3x3 256->256 @14x14, 1 image, 8 tiles of 36            17.0 / 14.4 /  9.8 / 7.1 / 5.7
//   1x1 1024->256 @14x14, 1 image, 8 tiles of 16           10.0 /  8.0 /  6.5 / 5.2 / 4.8
//   1x1 256->1024 @14x14, 1 image, 32 tiles of 4            6.3 /  4.7 /  4.9 / 6.1
//   3x3 256->256 @14x14, 8 images, 52 tiles of 36          17.3 / 15.6 / 11.2 / 9.0 / 15.0
//   3x3 128->128 @28x28, 8 images, 98 tiles of 18          12.9 / 10.0 /  8.7 / 14.1
//   1x1 512->128 @28x28, 8 images, 98 tiles of 8            8.9 /  6.5 /  7.0
// So: eight K blocks or more, at least two of them to a CTA, up to one CTA per SM -- two per SM where four K blocks stay, but
// not in clusters of eight.
// uint8: the caller says with `splits` (1 included) that this kernel takes the convolution, since it has to clear csum_out when
// several CTAs add to a pixel's sum; 0 here: it should not.
extern "C" int thb_conv_few_splits(const thb_conv_desc *d)
{
    const ThbConvLaunch kn = thb_conv_launch_knobs();
    const int u8 = d->dtype == THB_U8;
    if (kn.few_tiles == 0 || !eligible(d) || (!u8 && d->Cout_pad % BN)) return !u8;
    const long tiles = tiles_of(d);
    const int nkb = d->Ktot_pad / (u8 ? 128 : 64);
    if (u8 && tiles > (kn.few_tiles >= 0 ? kn.few_tiles : 4L * kn.sms)) return 0;
    int S = 1;
    while (S < 8 && nkb >= 8 && nkb / (2 * S) >= 2 && tiles * 2 * S <= (S < 4 && nkb / (2 * S) >= 4 ? 2 : 1) * (long)kn.sms) S *= 2;
    return S;
}

// Does this convolution belong to conv_few_kernel?  A split one does.  Otherwise small CTAs beat the persistent kernel up to
// about four of them per SM (8 images, tiles / persistent / here: 1x1 512->2048 @7x7, 128: 9.0 / 7.0; 256->1024 @14x14, 208:
// 7.9 / 5.7; 128->512 @28x28, 392: 8.3 / 6.2; 64->256 @56x56, 784: 9.5 / 11.1), and the patch kernel up to one.
extern "C" int thb_conv_few_supported(const thb_conv_desc *d)
{
    if (d->dtype == THB_U8) return d->splits >= 1 && eligible(d);
    if (!eligible(d) || d->Cout_pad % BN) return 0;
    if (d->splits > 1) return 1;
    const ThbConvLaunch kn = thb_conv_launch_knobs();
    const long most = kn.few_tiles >= 0 ? kn.few_tiles : (d->kH * d->kW > 1 && thb_conv_patch_supported(d) ? 1 : 4) * (long)kn.sms;
    return tiles_of(d) <= most;
}

static int few_fwd(const thb_conv_desc *d, const void *x, void *y, float *y_nchw, const int *prev_status, int *status, thb_stream s)
{
    if (!d->w || !status || !x || !(y || y_nchw)) return THB_ERR_ARG;
    FewParams p;
    memset(&p, 0, sizeof(p));
    int tmap_mode = 0;
    p.mode = operand_mode(d, p, tmap_mode);
    if (!p.mode || !eligible(d)) return THB_ERR_UNSUPPORTED;
    p.y = (uint8_t *)y;
    p.y_nchw = y_nchw;
    p.prev_status = prev_status;
    p.res = (const uint8_t *)d->res; p.res_ld = d->res_ld;
    p.scale = d->scale; p.shift = d->shift; p.slope = d->act.kind == THB_ACT_PRELU ? d->act.slope : nullptr;
    p.P = d->N * d->oH * d->oW; p.oW = d->oW; p.oHW = d->oH * d->oW;
    p.dH = d->dH; p.dW = d->dW; p.padH = d->padH; p.padW = d->padW; p.kW = d->kW;
    p.Cout = d->Cout; p.out_ld = d->out_ld;
    const int u8 = d->dtype == THB_U8;
    p.nkb = d->Ktot_pad / (u8 ? 128 : 64);
    p.H = d->H; p.W = d->W; p.kH = d->kH; p.Cin = d->Cin;
    if (u8) {
        if (!d->wsat || !d->csum) return THB_ERR_ARG;
        p.a_off = d->a_offset; p.b_off = d->b_offset; p.c_off = d->c_offset; p.c_mult = d->c_mult; p.c_shift = d->c_shift;
        p.tail_start = d->tail_start;
        p.relu_thr = d->relu_thr < 0 ? -1 : d->relu_thr;
        p.relu_val = d->relu_val;
        p.wsat = d->wsat; p.bias_add = d->bias_add; p.csum = d->csum; p.csum_out = d->csum_out;
        p.classes = (1 + 2 * d->padH) * (1 + 2 * d->padW);
        p.tbl_bytes = (p.classes * BN * 4 + 1023) & ~1023;
        if (d->res) {
            p.ca = (int)d->self_coef; p.cb = (int)d->res_coef;
            if ((p.ca != 1 && p.ca != -1) || (p.cb != 1 && p.cb != -1) || (float)p.ca != d->self_coef || (float)p.cb != d->res_coef) return THB_ERR_UNSUPPORTED;
            const int twice = -(p.ca + p.cb - 1) * 255;  // floor(-(ca + cb - 1) * 127.5), as thb_u8_combine
            p.res_addend = twice >= 0 ? twice / 2 : -((-twice + 1) / 2);
        }
    }
    p.n_tiles = (d->Cout_pad + BN - 1) / BN;  // (32 padded channels: the copy fills the missing weight rows with zeros)
    p.self_coef = d->self_coef; p.res_coef = d->res_coef;
    p.act_kind = d->act.kind; p.act_th = d->act.threshold; p.act_val = d->act.value; p.act_alpha = d->act.alpha;
    p.status = status;
    if (p.P <= 0) return THB_OK;
    p.splits = d->splits > 1 ? d->splits : 1;
    if (p.splits != 1 && p.splits != 2 && p.splits != 4 && p.splits != 8) return THB_ERR_ARG;
    if (p.splits > p.nkb) return THB_ERR_ARG;
    const ThbConvLaunch kn = thb_conv_launch_knobs();
    p.pdl = kn.pdl; p.wait_limit = kn.wait_limit; p.test_withhold = kn.test_withhold;
    const CUtensorMap *w = thb_weights_tmap(d, BN, p.half ? 64 : 128), *a, *a2;
    if (d->x2) {
        const int cin2 = d->Cin - d->cin1;
        if (d->res || p.mode != 1 || d->in_row_pitch || d->cin1 <= 0 || d->cin1 % 64 || cin2 <= 0 || cin2 % 64 || d->x2_d < 1 || d->x2_d > 8 ||
            d->Cin_pad != d->Cin || (d->x2_H - 1) / d->x2_d + 1 != d->oH || (d->x2_W - 1) / d->x2_d + 1 != d->oW)
            return THB_ERR_UNSUPPORTED;
        p.nkb1 = d->cin1 / 64;
        p.a2_d = d->x2_d;
        p.a2_mode = d->x2_d == 1 ? 1 : 2;
        a = thb_matrix_tmap(x, p.P, d->cin1, d->in_ld, d->dtype, 64);
        if (p.a2_mode == 1) a2 = thb_matrix_tmap(d->x2, p.P, cin2, d->x2_ld, d->dtype, 64);
        else {
            thb_conv_desc d2;
            memset(&d2, 0, sizeof(d2));
            d2.dtype = d->dtype;
            d2.N = d->N; d2.H = d->x2_H; d2.W = d->x2_W; d2.Cin = d2.Cin_pad = cin2; d2.in_ld = d->x2_ld;
            d2.kH = d2.kW = 1; d2.dH = d2.dW = d->x2_d; d2.oH = d->oH; d2.oW = d->oW;
            a2 = thb_activation_tmap(&d2, d->x2, 2);
        }
    } else
        a = a2 = thb_activation_tmap(d, x, tmap_mode);
    if (!w || !a || !a2) return thb_note_launch(cudaErrorUnknown, "conv_few: tensor map");
    const int per = (p.nkb + p.splits - 1) / p.splits;
    const int ctas = ((p.P + BM - 1) / BM) * p.n_tiles * p.splits;
    // stages: as many as fit the CTAs an SM gets.  Clusters always leave room for two CTAs to an SM, or a GPC holds too few of
    // them at once (ResNet-18 on 4 images: 193 us with a fourth stage, 168 with three)
    p.stages = kn.few_stages > 0 ? kn.few_stages : p.splits > 1 || ctas > 2 * kn.sms ? 3 : ctas > kn.sms ? 4 : 5;
    if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
    if (p.stages > per) p.stages = per;
    const int smem = 1024 + BAR_BYTES + (p.splits > 1 ? RECV_BYTES : 0) + p.tbl_bytes + p.stages * STAGE_BYTES;
    cudaStream_t st = (cudaStream_t)s;
    return u8 ? launch<2>(w, a, a2, p, ctas, smem, st) : d->dtype == THB_F16 ? launch<0>(w, a, a2, p, ctas, smem, st) : launch<1>(w, a, a2, p, ctas, smem, st);
}

extern "C" int thb_conv_few_fwd(const thb_conv_desc *d, const void *x, void *y, thb_stream s)
{
    return few_fwd(d, x, y, nullptr, nullptr, d->status, s);
}

extern "C" int thb_conv_nchw_supported(const thb_conv_desc *d)
{
    thb_conv_desc one = *d;
    one.splits = 0;
    return d->dtype != THB_U8 && eligible(&one) && !d->x2;
}

extern "C" int thb_conv_nchw_fwd(const thb_conv_desc *d, const void *x, float *y, int *status_out, thb_stream s)
{
    if (!thb_conv_nchw_supported(d) || !status_out) return THB_ERR_UNSUPPORTED;
    thb_conv_desc one = *d;
    one.splits = 0;
    return few_fwd(&one, x, nullptr, y, d->status, status_out, s);
}
