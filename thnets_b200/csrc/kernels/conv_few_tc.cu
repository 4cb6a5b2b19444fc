// Tensor-core convolution for launches of few tiles (16-bit types, uint8): small batches, the late stages of a network.
//
// What bounds such a layer is not arithmetic or bandwidth but the chain of one tile: with 8 images or fewer a ResNet layer
// is 1 to 100 tiles, the persistent kernel (conv_tc.cu) runs one of them per SM, and a K block costs the SM's copy engine
// about 0.33 us (an im2col box of 128 rows) however idle the other SMs are: 72 K blocks of a 3x3 512->512 layer took 30 us.
// Here
//   * a tile is 128 pixels x 64 channels, one CTA works on one tile only, and two CTAs fit an SM;
//   * the K blocks of a tile are shared by the S = 1, 2, 4 or 8 CTAs of a thread-block cluster.  Each pushes the columns of
//     its fp32 partial tile to the CTA that owns them, through distributed shared memory (stores that the owner's barrier
//     counts: a cluster barrier behind them took 1100 to 2900 cycles), and every owner adds the S parts in rank order and
//     finishes its 64 / S channels (no atomics, no scratch in global memory, no second launch);
//   * weights and activations are loaded by two different warps, and since weights do not depend on the kernel before, their
//     loads start ahead of griddepcontrol.wait, under that kernel's tail, as does everything that is worked out from parameters;
//   * the epilogue passes the accumulator through shared memory to a thread per row and eight channels, whose constants stay in
//     registers and whose rows leave and arrive whole (a thread per row took 3900 cycles a tile, 1600 now).
// Measured: the tables at thb_conv_few_splits and thb_conv_few_supported.  Calls: ResNet-18 fp16, 1 image 179 -> 160 us; ResNet-50
// fp16, 8 images 537 -> 510; ResNet-18 uint8, 1 image 206 -> 184.  What is left of a launch's 4 to 6 us: 2 us from the last store to
// the next launch's first load, 0.5 us to its first K block, the K blocks, 1.5 us of exchange and epilogue.
//
// Every mbarrier wait is bounded; one that runs out records a code in *status and the CTA drains (all its threads still
// reach both cluster barriers; its peers' waits for its part run out like any other).
#include <cuda.h>
#include <string.h>
#include "common.cuh"
#include "conv_maps.cuh"

namespace {

constexpr int BM = 128, BN = 64;
// EW epilogue warps (4 or 8), an activation producer, a weight producer, an MMA issuer
constexpr int nthreads(int ew) { return (ew + 3) * 32; }
constexpr int A_BYTES = BM * 128, B_BYTES = BN * 128, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int MAX_STAGES = 8;
// ahead of the tiles: barriers, from 192 on the per-channel constants; uint8: bias addends, per-row terms from 448 on, then the table
constexpr int U8_ROWS = 448, U8_TABLE = U8_ROWS + BM * 8;
__host__ __device__ constexpr int header_bytes(bool u8, int tbl_bytes) { return u8 ? (U8_TABLE + tbl_bytes + 1023) & ~1023 : 1024; }
// Partial sums by way of shared memory: groups of four columns, the rows of a group after one another and one row of padding, so
// that neither a warp's 32 rows of a group nor its reads of several groups meet in a bank.
constexpr int RECV_ROWS = BM + 1, RECV_BYTES = (BN / 4) * RECV_ROWS * 16;

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
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_addr(uint32_t smem, uint32_t rank)
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem), "r"(rank));
    return a;
}
// 16 bytes into the shared memory of a CTA of the cluster, counted by a barrier there
__device__ __forceinline__ void st_async_v4(uint32_t addr, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%2, %3, %4, %5}, [%1];" ::"r"(addr), "r"(bar), "r"(a),
                 "r"(b), "r"(c), "r"(d)
                 : "memory");
}
template <int EW> __device__ __forceinline__ void epi_bar_sync() { asm volatile("bar.sync 1, %0;" ::"n"(EW * 32) : "memory"); }

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

// Eight channels of one pixel: y = act(acc * scale + shift + res_coef * residual), channels >= Cout zero.  The operations and
// their order are those of the persistent kernel's epilogue: the same bits.  ACT: 0 none, 1 plain ReLU, 2 anything.
template <int KIND, int ACT>
__device__ __forceinline__ uint4 finish8(const float (&acc)[8], const uint4 &rv, const float (&sc)[8], const float (&sh)[8], const float *sl, int left,
                                         const FewParams &p)
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
            v[e] = fmaf(acc[i], sc[i], sh[i]);
            if (p.res) v[e] = fmaf(p.res_coef, e ? rr.y : rr.x, v[e]);
            if (ACT == 1) v[e] = fmaxf(v[e], 0.f);
            if (ACT == 2) v[e] = thb_apply_act(v[e], p.act_kind, p.act_th, p.act_val, p.act_alpha, sl[i]);
            if (i >= left) v[e] = 0.f;
        }
        ow[h] = pack2<KIND>(v[0], v[1]);
    }
    return make_uint4(ow[0], ow[1], ow[2], ow[3]);
}

// A network's last convolution, whose result leaves as NCHW floats (rounded through the 16-bit type like any other), straight
// from the thread's TMEM lane: a warp's lanes are 32 neighbouring pixels of a plane, so every channel is a coalesced 128-byte
// store.  Two groups of four warps take every other eight channels.
template <int KIND, int ACT>
__device__ __forceinline__ void finish_nchw(uint32_t taddr, const uint8_t *res, float *dst, size_t plane, bool real, int left, const Consts &k,
                                            int first, int step, const FewParams &p)
{
#pragma unroll 1
    for (int j = first; j < BN / 8 && j * 8 < left; j += step) {
        uint32_t a[8];
        tmem_ld8(taddr + j * 8, a);
        tmem_ld_wait();
        float acc[8], sc[8], sh[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            acc[i] = __uint_as_float(a[i]);
            sc[i] = k.sc[j * 8 + i];
            sh[i] = k.sh[j * 8 + i];
        }
        uint4 rv = make_uint4(0, 0, 0, 0);
        if (p.res && real) rv = __ldg(reinterpret_cast<const uint4 *>(res + j * 16));
        const uint4 o = finish8<KIND, ACT>(acc, rv, sc, sh, k.sl + j * 8, left - j * 8, p);
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

// Eight columns of one row, the sum of the S parts in rank order: `part` points at the first part's first group of four.
template <typename T> struct vec4;
template <> struct vec4<float> { typedef float4 type; };
template <> struct vec4<int> { typedef int4 type; };
template <typename T> __device__ __forceinline__ void sum_parts(const uint8_t *part, int S, int stride, T (&acc)[8])
{
    typedef typename vec4<T>::type V;
    const V u0 = *reinterpret_cast<const V *>(part), v0 = *reinterpret_cast<const V *>(part + RECV_ROWS * 16);
    acc[0] = u0.x; acc[1] = u0.y; acc[2] = u0.z; acc[3] = u0.w;
    acc[4] = v0.x; acc[5] = v0.y; acc[6] = v0.z; acc[7] = v0.w;
    for (int r = 1; r < S; r++) {
        part += stride;
        const V u = *reinterpret_cast<const V *>(part), v = *reinterpret_cast<const V *>(part + RECV_ROWS * 16);
        acc[0] += u.x; acc[1] += u.y; acc[2] += u.z; acc[3] += u.w;
        acc[4] += v.x; acc[5] += v.y; acc[6] += v.z; acc[7] += v.w;
    }
}

// The items (row, eight channels) of an epilogue thread: eight channels of those this CTA finishes, rows r0, r0 + rows, ...  The
// residual of the first four is there already.
template <int KIND, int ACT>
__device__ __forceinline__ void finish_rows(const uint8_t *part, int S, int stride, int r0, int rows, uint4 (&rv)[4], int m0, const float *sc_, const float *sh_,
                                            const float *sl, int left, const uint8_t *res, uint8_t *dst, const FewParams &p)
{
    float sc[8], sh[8];
#pragma unroll
    for (int i = 0; i < 8; i++) { sc[i] = sc_[i]; sh[i] = sh_[i]; }
#pragma unroll 1
    for (int r = r0; r < BM;) {
#pragma unroll
        for (int i = 0; i < 4; i++, r += rows) {
            if (r >= BM || m0 + r >= p.P) return;
            float acc[8];
            sum_parts(part, S, stride, acc);
            part += rows * 16;
            *reinterpret_cast<uint4 *>(dst + (size_t)r * p.out_ld * 2) = finish8<KIND, ACT>(acc, rv[i], sc, sh, sl, left, p);
        }
        if (p.res) {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (r + i * rows < BM && m0 + r + i * rows < p.P) rv[i] = __ldg(reinterpret_cast<const uint4 *>(res + (size_t)(r + i * rows) * p.res_ld * 2));
        }
    }
}

// Eight channels of one pixel in uint8: zero-point correction (the border class's table word times c_mult, the row's own term),
// gemmlowp requantisation, the reference's saturating bias add with its tail quirk, the fused residual and the Threshold -- the
// integer arithmetic of the persistent kernel's u8_chunk32.
struct U8Row {
    uint32_t rc;
    int trow;  // the border class's row of the table, its sign bit set where the reference's tail quirk does not apply
};
__device__ __forceinline__ uint2 finish8_u8(const int (&acc)[8], const int *tbl, const int (&b)[8], const U8Row &e, int shift, int thr, const uint2 &rv, int left,
                                            const FewParams &p)
{
    const int tailmask = e.trow < 0 ? 0 : 255;
    const int4 *t4 = reinterpret_cast<const int4 *>(tbl + (e.trow & 0x7fffffff));
    const int4 ta = t4[0], tb = t4[1];
    const int t[8] = {ta.x, ta.y, ta.z, ta.w, tb.x, tb.y, tb.z, tb.w};
    uint32_t ow[2] = {0, 0};
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int sres = (int)((uint32_t)acc[i] * (uint32_t)p.c_mult + (uint32_t)t[i] + e.rc) >> shift;
        const int q = min(max(sres, 0), 255), t2 = q + b[i];
        int v = max(min(max(t2, 0), 255), t2 & tailmask);
        if (p.res) {
            const int r = (int)(((i < 4 ? rv.x : rv.y) >> (8 * (i & 3))) & 255u);
            v = min(max(p.ca * v + p.cb * r + p.res_addend, 0), 255);
        }
        v = v > thr ? v : p.relu_val;
        if (i < left) ow[i >> 2] |= (uint32_t)v << (8 * (i & 3));
    }
    return make_uint2(ow[0], ow[1]);
}

template <int KIND, int EW>
__global__ void __launch_bounds__(nthreads(EW), EW == 8 ? 2 : 3) conv_few_kernel(const __grid_constant__ CUtensorMap tmapW, const __grid_constant__ CUtensorMap tmapA,
                                                               const __grid_constant__ CUtensorMap tmapA2, const __grid_constant__ FewParams p)
{
    constexpr uint32_t IDESC = make_idesc(KIND == 2 ? 2u : 1u, KIND == 1 ? 1u : 0u, BN);
    constexpr int KE = KIND == 2 ? 128 : 64;  // elements of a K block
    constexpr int EPI = EW * 32, NT = EPI + 96, W_A = EW, W_B = EW + 1, W_MMA = EW + 2;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem), *empty = full + MAX_STAGES, *acc_full = empty + MAX_STAGES, *recv_full = acc_full + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(recv_full + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    Consts &consts = *reinterpret_cast<Consts *>(smem + 192);
    static_assert((2 * MAX_STAGES + 2) * 8 + 8 <= 192 && 192 + sizeof(Consts) <= 1024, "barriers and constants share the first kilobyte");
    U8Row *row_terms = reinterpret_cast<U8Row *>(smem + U8_ROWS);  // uint8
    // (every CTA of a cluster has the same layout, so an offset into this one's receive buffer fits its peers' too; unsplit, the
    // sums of the CTA itself take the place of its stages, which are free by then)
    uint8_t *recv = smem + header_bytes(KIND == 2, p.tbl_bytes);
    int *tbl = reinterpret_cast<int *>(smem + U8_TABLE), *bias = reinterpret_cast<int *>(smem + 192);  // uint8
    uint8_t *ring = recv + (p.splits > 1 ? (RECV_BYTES + 1023) / 1024 * 1024 : 0);

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
        mbar_init(smem_u32(recv_full), 1);
        *abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async_smem();
        if (S > 1) mbar_arrive_expect_tx(smem_u32(recv_full), min(BM, p.P - m0) * BN * 4);  // what the S CTAs push: the tile's real rows
    }
    if (KIND == 2) {
        // T[class][channel] = b_off * (sum of the channel's weights over the taps inside the image) * c_mult
        const int ncc = 1 + 2 * p.padW, satw = p.kW + 1, satn = (p.kH + 1) * satw;
        for (int i = tid; i < p.classes * BN; i += NT) {
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
    if (warp == W_A && lane == 0) {
        tma_prefetch_desc(&tmapA);
        if (p.nkb1) tma_prefetch_desc(&tmapA2);
    }
    if (warp == W_B && lane == 0) tma_prefetch_desc(&tmapW);
    if (warp == W_MMA) {
        tmem_alloc(smem_u32(tmem_slot), BN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (S > 1) cluster_arrive();  // (the wait is ahead of the first store to a peer)
    if (p.pdl) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // weights are not written by any launch of the forward: their producer does not wait for the kernel before; the others do once
    // they have worked out what they need
    auto launch_wait = [&]() { if (p.pdl) asm volatile("griddepcontrol.wait;" ::: "memory"); };

    if (warp >= W_A) {
        if (warp == W_A) {
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
                launch_wait();
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
        } else if (warp == W_B) {
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
            // (the whole warp waits and steps, one elected thread issues: addresses stay in uniform registers)
            const bool leader = elect_one();
            launch_wait();
            int s = 0;
            uint32_t ph = 0;
            bool alive = true;
            for (int kb = kb0; kb < kb1; kb++) {
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&full[s]), ph, p.wait_limit))) {
                    if (leader) {
                        report(p.status, 4);
                        *abort_flag = 1;
                    }
                    alive = false;
                    break;
                }
                tc_fence_after();
                const uint32_t sa = smem_u32(ring + s * STAGE_BYTES), sb = sa + A_BYTES;
                if (KIND == 2 && p.half) {
                    const int nh = 2 * kb + 1 < p.ntaps ? 2 : 1;
                    if (leader) {
                        for (int h = 0; h < nh; h++) {
                            const uint64_t ad = make_sw64_kmajor_desc(sa + h * (A_BYTES / 2)), bd = make_sw64_kmajor_desc(sb + h * (B_BYTES / 2));
#pragma unroll
                            for (int k = 0; k < 2; k++) {
                                if (KIND == 2) tc_mma_i8(tmem_base, ad + 2 * k, bd + 2 * k, IDESC, ((kb - kb0) | h | k) != 0);
                                else tc_mma_f16(tmem_base, ad + 2 * k, bd + 2 * k, IDESC, ((kb - kb0) | h | k) != 0);
                            }
                        }
                    }
                } else {
                    const uint64_t ad = make_sw128_kmajor_desc(sa), bd = make_sw128_kmajor_desc(sb);
                    if (leader) {
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            if (KIND == 2) tc_mma_i8(tmem_base, ad + 2 * k, bd + 2 * k, IDESC, ((kb - kb0) | k) != 0);
                            else tc_mma_f16(tmem_base, ad + 2 * k, bd + 2 * k, IDESC, ((kb - kb0) | k) != 0);
                        }
                    }
                }
                if (leader && kb + nst < kb1) tc_commit(smem_u32(&empty[s]));
                __syncwarp();
                if (++s == nst) { s = 0; ph ^= 1; }
            }
            if (alive && leader) tc_commit(smem_u32(acc_full));
            __syncwarp();
        }
        if (S > 1) {
            cluster_wait();
            cluster_arrive_relaxed();
        }
    } else {
        // ---- epilogue: the accumulator by way of shared memory to the CTA that finishes its columns, there a thread per row and
        // eight channels, so that residual and result pass in whole rows (the thread that owns a row used to finish all of its
        // channels: 3900 cycles of instructions and scattered 16-byte stores against 1600 now) ----
        const int row = tid & 127, grp = warp >> 2;  // TMEM lane; eight warps: columns 32 grp .. + 31, four: all
        // this CTA finishes W = 64 / S channels, 1 << cshift items a row
        const int sshift = S == 1 ? 0 : S == 2 ? 1 : S == 4 ? 2 : 3, wshift = 6 - sshift, W = 1 << wshift, cshift = 3 - sshift;
        const int c_local = rank * W + (tid & ((1 << cshift) - 1)) * 8, c_first = n0 + c_local, cout8 = (p.Cout + 7) & ~7;
        const int r0 = tid >> cshift, rows = EPI >> cshift;
        const int act = p.act_kind == THB_ACT_NONE ? 0 : p.act_kind == THB_ACT_THRESHOLD && p.act_th == 0.f && p.act_val == 0.f ? 1 : 2;
        launch_wait();
        if (p.prev_status && blockIdx.x == 0 && tid == 0) {
            const int before = *p.prev_status;
            if (before) report(p.status, before);
        }
        // the residual of this thread's items, asked for before the accumulator is awaited
        uint4 rv[4];
        uint2 r8[32 / EW];   // uint8
        const uint8_t *res = p.res + ((size_t)m0 * p.res_ld + c_first) * (KIND == 2 ? 1 : 2);
#pragma unroll
        for (int i = 0; i < (KIND == 2 ? 32 / EW : 4); i++) {
            const int r = r0 + i * rows;
            const bool real = p.res && !p.y_nchw && r < BM && m0 + r < p.P && c_first < cout8;
            if (KIND == 2) r8[i] = real ? __ldg(reinterpret_cast<const uint2 *>(res + (size_t)r * p.res_ld)) : make_uint2(0, 0);
            else rv[i] = real ? __ldg(reinterpret_cast<const uint4 *>(res + (size_t)r * p.res_ld * 2)) : make_uint4(0, 0, 0, 0);
        }
        if (KIND == 2 && grp == 0) {
            const int pc = min(m0 + row, p.P - 1), n = pc / p.oHW, rem = pc - n * p.oHW, oh = rem / p.oW, ow = rem - oh * p.oW;
            const int ihb = oh * p.dH - p.padH, iwb = ow * p.dW - p.padW;
            const int w0 = max(0, -ihb), w1 = min(p.kH, p.H - ihb), s0 = max(0, -iwb), s1 = min(p.kW, p.W - iwb);
            const int cb = p.kH - w1, cr = p.kW - s1;  // (clipped on one side at most: the launcher checks)
            const int *cs = p.csum + ((size_t)n * p.H + ihb) * p.W + iwb;
            int xsum = 0;
            if (p.kH <= 4 && p.kW <= 4) {
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const int r = i >> 2, q = i & 3;
                    xsum += r >= w0 && r < w1 && q >= s0 && q < s1 ? __ldg(cs + r * p.W + q) : 0;
                }
            } else
                for (int r = w0; r < w1; r++)
                    for (int q = s0; q < s1; q++) xsum += __ldg(cs + r * p.W + q);
            const int corr = p.a_off * (xsum + p.b_off * (w1 - w0) * (s1 - s0) * p.Cin);
            U8Row t;
            t.rc = (uint32_t)(corr + p.c_off) * (uint32_t)p.c_mult + (p.c_shift >= 1 ? 1u << (p.c_shift - 1) : 0u);
            t.trow = ((w0 > 0 ? w0 : cb > 0 ? p.padH + cb : 0) * (1 + 2 * p.padW) + (s0 > 0 ? s0 : cr > 0 ? p.padW + cr : 0)) * BN;
            if (rem < p.tail_start) t.trow |= (int)0x80000000u;
            row_terms[row] = t;
        }
        bool have = mbar_wait_bounded(smem_u32(acc_full), 0, p.wait_limit);
        if (!have) {
            if (lane == 0) report(p.status, 2);
            *abort_flag = 1;
        }
        have = __all_sync(0xffffffffu, have);
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
        const bool nchw = KIND != 2 && p.y_nchw;  // (never split)
        if (nchw) {
            if constexpr (KIND != 2) if (have) {
                const int pm = m0 + row, img = pm / p.oHW;
                const bool real = pm < p.P;
                float *dst = p.y_nchw + ((size_t)img * p.Cout + n0) * p.oHW + (pm - img * p.oHW);
                const uint8_t *nres = p.res + ((size_t)pm * p.res_ld + n0) * 2;
                if (act == 0) finish_nchw<KIND, 0>(taddr, nres, dst, p.oHW, real, p.Cout - n0, consts, grp, EW / 4, p);
                else if (act == 1) finish_nchw<KIND, 1>(taddr, nres, dst, p.oHW, real, p.Cout - n0, consts, grp, EW / 4, p);
                else finish_nchw<KIND, 2>(taddr, nres, dst, p.oHW, real, p.Cout - n0, consts, grp, EW / 4, p);
            }
        } else {
            if (S > 1) cluster_wait();  // every CTA of the cluster has started
            if (have) {
                uint8_t *at = recv + (size_t)row * 16;
                const uint32_t bar = smem_u32(recv_full);
#pragma unroll 1
                for (int c0 = EW == 8 ? grp * 32 : 0; c0 < (EW == 8 ? grp * 32 + 32 : 64); c0 += 32) {
                    uint32_t a[32];
                    tmem_ld32(taddr + c0, a);
                    tmem_ld_wait();
                    if (S == 1) {
#pragma unroll
                        for (int q = 0; q < 8; q++)
                            *reinterpret_cast<uint4 *>(at + (c0 / 4 + q) * RECV_ROWS * 16) = make_uint4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
                    } else if (m0 + row < p.P) {
                        // columns c .. c + 3 belong to CTA c / W; slot [rank][column group][row] of its buffer
#pragma unroll
                        for (int q = 0; q < 8; q++) {
                            const int c = c0 + 4 * q, owner = c >> wshift, g = (c & (W - 1)) >> 2;
                            st_async_v4(cluster_addr(smem_u32(at + (rank * (W >> 2) + g) * RECV_ROWS * 16), owner), cluster_addr(bar, owner), a[4 * q],
                                        a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
                        }
                    }
                }
            }
            __syncwarp();
            if (S > 1) {
                cluster_arrive_relaxed();  // (waited for at the end: no CTA leaves before its peers have pushed what they will)
                // (also without an accumulator of its own, whose part is then missing: what the peers have pushed lands meanwhile.  At the
                // end of the kernel, for such a CTA alone, the wait cost registers: ResNet-50 on 8 images 431.3 -> 432.7 to 441 us)
                if (!mbar_wait_bounded(smem_u32(recv_full), 0, p.wait_limit) && have) {
                    report(p.status, 5);
                    *abort_flag = 1;
                    have = false;
                }
                have = __all_sync(0xffffffffu, have);
            }
            if (S == 1 || KIND == 2) epi_bar_sync<EW>();
            if constexpr (KIND == 2) {
                if (have) {
                    const int left = p.Cout - c_first, shift = max(p.c_shift, 0), thr = p.relu_thr;
                    const bool write = c_first < ((p.Cout + 15) & ~15);
                    const uint8_t *part = recv + (size_t)(2 * (tid & ((1 << cshift) - 1)) * RECV_ROWS + r0) * 16;
                    int b[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) b[i] = bias[c_local + i];
#pragma unroll
                    for (int i = 0; i < 32 / EW; i++) {
                        const int r = r0 + i * rows, pm = m0 + r;
                        if (r >= BM) break;  // (the same for a whole warp)
                        int acc[8];  // (rows beyond the last pixel: whatever lies there, never stored)
                        sum_parts(part + i * rows * 16, S, (2 << cshift) * RECV_ROWS * 16, acc);
                        const U8Row t = row_terms[r];
                        const uint2 o = finish8_u8(acc, tbl + c_local, b, t, shift, thr, r8[i], left, p);
                        if (write && pm < p.P) *reinterpret_cast<uint2 *>(p.y + (size_t)pm * p.out_ld + c_first) = o;
                        if (p.csum_out) {
                            // the lanes of a row add up its bytes
                            int sum = (int)__dp4a(o.x, 0x01010101u, __dp4a(o.y, 0x01010101u, 0u));
                            for (int d = 1; d < 1 << cshift; d <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
                            if (pm < p.P && !(tid & ((1 << cshift) - 1))) {
                                if (p.n_tiles == 1 && S == 1) p.csum_out[pm] = sum;
                                else atomicAdd(p.csum_out + pm, sum);  // (the buffer was cleared before the launch)
                            }
                        }
                    }
                }
            } else {
                if (have && c_first < cout8) {
                    const int left = p.Cout - c_first, stride = (2 << cshift) * RECV_ROWS * 16;
                    const uint8_t *part = recv + (size_t)(2 * (tid & ((1 << cshift) - 1)) * RECV_ROWS + r0) * 16;
                    uint8_t *dst = p.y + ((size_t)m0 * p.out_ld + c_first) * 2;
                    const float *sc = consts.sc + c_local, *sh = consts.sh + c_local, *sl = consts.sl + c_local;
                    if (act == 0) finish_rows<KIND, 0>(part, S, stride, r0, rows, rv, m0, sc, sh, sl, left, res, dst, p);
                    else if (act == 1) finish_rows<KIND, 1>(part, S, stride, r0, rows, rv, m0, sc, sh, sl, left, res, dst, p);
                    else finish_rows<KIND, 2>(part, S, stride, r0, rows, rv, m0, sc, sh, sl, left, res, dst, p);
                }
            }
        }
    }
    if (S > 1) cluster_wait();
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && warp == W_A && lane == 0) {
        // a wait ran out: copies still on their way must land before the CTA may leave
        const int n = kb1 - kb0 < nst ? kb1 - kb0 : nst;
        for (int s = 0; s < n; s++) mbar_wait_bounded(smem_u32(&full[s]), ((kb1 - kb0 - 1 - s) / nst) & 1, p.wait_limit);
    }
    __syncthreads();
    tc_fence_after();
    if (warp == W_MMA) tmem_dealloc(tmem_base, BN);
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

template <int KIND, int EW>
int launch(const CUtensorMap &w, const CUtensorMap &a, const CUtensorMap &a2, const FewParams &p, int ctas, int smem, cudaStream_t st)
{
    static bool set[64];
    int dev = 0;
    cudaGetDevice(&dev);
    const auto kern = conv_few_kernel<KIND, EW>;
    if (dev >= 0 && dev < 64 && !set[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
        if (e != cudaSuccess) return thb_note_launch(e, "conv_few_kernel attributes");
        set[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(nthreads(EW));
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
    const cudaError_t le = cudaLaunchKernelEx(&cfg, kern, w, a, a2, p);
    return thb_note_launch(le != cudaSuccess ? le : cudaGetLastError(), "conv_few_kernel");
}

}  // namespace

// How many CTAs should share the reduction of each tile of this convolution in conv_few_kernel (1: none need to).  Measured, us
// per launch in a chain of launches (the persistent kernel / no split / split in 2 / 4 / 8; * the rule's choice):
//   3x3 512->512 @7x7,  1 image,  8 tiles of 72 K blocks   25.2 / 22.7 / 13.4 / 8.6 / 6.2*
//   3x3 256->256 @14x14, 1 image, 8 tiles of 36            14.8 / 13.3 /  9.3 / 6.8 / 5.7*
//   3x3 128->128 @28x28, 1 image, 14 tiles of 18            9.8 /  8.6 /  7.0 / 5.8* / 6.4
//   1x1 1024->256 @14x14, 1 image, 8 tiles of 16            8.9 /  7.3 /  6.3 / 5.3* / 5.2
//   1x1 512->2048 @7x7, 1 image, 32 tiles of 8              6.7 /  5.3 /  4.5* / 4.9 / 6.1
//   1x1 256->1024 @14x14, 1 image, 32 tiles of 4            5.6 /  4.4* / 5.5 / 6.2
//   3x3 256->256 @14x14, 4 images, 28 tiles of 36          15.1 / 13.6 / 10.1 / 8.8 / 7.6*
//   3x3 256->256 @14x14, 8 images, 52 tiles of 36          15.2 / 13.7 / 10.6 / 9.3* / 14.0
//   3x3 512->512 @7x7,  8 images, 32 tiles of 72           25.6 / 23.6 / 15.4 / 11.4 / 9.4*
//   3x3 128->128 @28x28, 8 images, 98 tiles of 18          11.1 /  9.0 /  8.5* / 13.5
//   1x1 1024->256 @14x14, 8 images, 52 tiles of 16          9.2 /  7.7 /  7.5* / 7.7
//   1x1 512->128 @28x28, 8 images, 98 tiles of 8            7.5 /  5.8* / 6.9
//   uint8 3x3 256->256 @14x14, 1 image, 8 tiles of 18      10.0 / 10.4 /  7.9 / 5.9 / 5.4*
//   uint8 1x1 2048->512 @7x7, 16 images, 56 tiles of 16     9.7 /  9.5 /  8.9 / 7.7* / 13.2
// So: four K blocks to a CTA (uint8 two), eight (four) where two CTAs share an SM -- four in clusters of eight, of which there are
// never more than the SMs hold at once.
// uint8: the caller says with `splits` (1 included) that this kernel takes the convolution, since it has to clear csum_out when
// several CTAs add to a pixel's sum; 0 here: it should not.
extern "C" int thb_conv_few_splits(const thb_conv_desc *d)
{
    const ThbConvLaunch kn = thb_conv_launch_knobs();
    const int u8 = d->dtype == THB_U8;
    if (kn.few_tiles == 0 || !eligible(d) || (!u8 && d->Cout_pad % BN)) return !u8;
    const long tiles = tiles_of(d);
    const int nkb = d->Ktot_pad / (u8 ? 128 : 64);
    if (u8 && tiles > (kn.few_tiles >= 0 ? kn.few_tiles : 2L * kn.sms)) return 0;
    int S = 1;
    while (S < 8) {
        const long ctas = tiles * 2 * S;
        const int part = nkb / (2 * S);  // K blocks left to a CTA
        if (part < (u8 ? 2 : 4) || ctas > (S == 4 ? 7 * (long)kn.sms / 4 : 2 * (long)kn.sms) || (ctas > kn.sms && part < (u8 || S == 4 ? 4 : 8))) break;
        S *= 2;
    }
    return S;
}

// Does this convolution belong to conv_few_kernel?  A split one does.  Otherwise small CTAs beat the persistent kernel while all of
// them are resident, three to an SM (tiles / persistent / here, us: 1x1 512->128 @28x28, 392: 11.1 / 9.7; 3x3 256->256 @14x14, 392:
// 28.5 / 20.7; 3x3 128->128 @28x28, 454: 18.1 / 22.3; 3x3 256->256 @14x14, 588: 30.1 / 35.5), and the patch kernel up to one.
// uint8 (thb_conv_few_splits): two to an SM (3x3 256->256 @14x14, 296: 14.1 / 13.9; 256->1024, 400: 9.7 / 11.0).
extern "C" int thb_conv_few_supported(const thb_conv_desc *d)
{
    if (d->dtype == THB_U8) return d->splits >= 1 && eligible(d);
    if (!eligible(d) || d->Cout_pad % BN) return 0;
    if (d->splits > 1) return 1;
    const ThbConvLaunch kn = thb_conv_launch_knobs();
    const long most = kn.few_tiles >= 0 ? kn.few_tiles : (d->kH * d->kW > 1 && thb_conv_patch_supported(d) ? 1 : 3) * (long)kn.sms;
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
        p.tbl_bytes = p.classes * BN * 4;
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
    CUtensorMap w, a, a2;
    bool ok = thb_weights_tmap(d, BN, p.half ? 64 : 128, &w);
    if (d->x2) {
        const int cin2 = d->Cin - d->cin1;
        if (d->res || p.mode != 1 || d->in_row_pitch || d->cin1 <= 0 || d->cin1 % 64 || cin2 <= 0 || cin2 % 64 || d->x2_d < 1 || d->x2_d > 8 ||
            d->Cin_pad != d->Cin || (d->x2_H - 1) / d->x2_d + 1 != d->oH || (d->x2_W - 1) / d->x2_d + 1 != d->oW)
            return THB_ERR_UNSUPPORTED;
        p.nkb1 = d->cin1 / 64;
        p.a2_d = d->x2_d;
        p.a2_mode = d->x2_d == 1 ? 1 : 2;
        ok = ok && thb_matrix_tmap(x, p.P, d->cin1, d->in_ld, d->dtype, 64, &a);
        if (p.a2_mode == 1) ok = ok && thb_matrix_tmap(d->x2, p.P, cin2, d->x2_ld, d->dtype, 64, &a2);
        else {
            thb_conv_desc d2;
            memset(&d2, 0, sizeof(d2));
            d2.dtype = d->dtype;
            d2.N = d->N; d2.H = d->x2_H; d2.W = d->x2_W; d2.Cin = d2.Cin_pad = cin2; d2.in_ld = d->x2_ld;
            d2.kH = d2.kW = 1; d2.dH = d2.dW = d->x2_d; d2.oH = d->oH; d2.oW = d->oW;
            ok = ok && thb_activation_tmap(&d2, d->x2, 2, &a2);
        }
    } else {
        ok = ok && thb_activation_tmap(d, x, tmap_mode, &a);
        a2 = a;
    }
    if (!ok) return thb_note_launch(cudaErrorUnknown, "conv_few: tensor map");
    const int per = (p.nkb + p.splits - 1) / p.splits;
    const int ctas = ((p.P + BM - 1) / BM) * p.n_tiles * p.splits;
    // stages: as many as fit the CTAs an SM gets.  Clusters always leave room for two CTAs to an SM, or a GPC holds too few of
    // them at once (ResNet-18 on 4 images: 193 us with a fourth stage, 168 with three)
    p.stages = kn.few_stages > 0 ? kn.few_stages : p.splits > 1 || ctas > 2 * kn.sms ? 3 : ctas > kn.sms ? 4 : 5;
    if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
    if (p.stages > per) p.stages = per;
    const int recv = (RECV_BYTES + 1023) / 1024 * 1024, room = p.stages * STAGE_BYTES;
    const int smem = 1024 + header_bytes(u8, p.tbl_bytes) + (p.splits > 1 ? recv + room : room > recv ? room : recv);
    cudaStream_t st = (cudaStream_t)s;
    // eight epilogue warps where one tile's chain is the launch; four where three CTAs share an SM and overlap
    if (p.splits > 1 || ctas <= 2 * kn.sms)
        return u8 ? launch<2, 8>(w, a, a2, p, ctas, smem, st) : d->dtype == THB_F16 ? launch<0, 8>(w, a, a2, p, ctas, smem, st) : launch<1, 8>(w, a, a2, p, ctas, smem, st);
    return u8 ? launch<2, 4>(w, a, a2, p, ctas, smem, st) : d->dtype == THB_F16 ? launch<0, 4>(w, a, a2, p, ctas, smem, st) : launch<1, 4>(w, a, a2, p, ctas, smem, st);
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
