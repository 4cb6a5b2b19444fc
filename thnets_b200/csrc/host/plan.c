/*
 * Execution planner and runtime of a converted network.
 *
 * The reference's engines swap one function pointer per module and allocate every activation on
 * every forward (cudnn/cudnn_basic.c:189-303, thapi.c:203-210, :405-416).  Here a network becomes,
 * once per input shape and per GPU, a list of kernel launches over two resident arenas:
 *   1. shape inference over the flat model (ranks and sizes as the reference's operators produce them);
 *   2. fusion: convolution/Linear + BatchNorm + two-input CAddTable + Threshold/PReLU collapse into one
 *      launch when each intermediate has a single consumer; BatchNorm + activation otherwise;
 *   3. liveness-based packing of all activations into one arena; weights packed and uploaded once;
 *   4. a batch is cut into contiguous slices, one per GPU; every GPU runs the whole list on its slice
 *      and the slices of the result are gathered by peer copies into GPU 0 (nothing is reduced).
 * Activations are channels-innermost ([N][H][W][ld]); the API's NCHW fp32 tensors are converted at the
 * two ends by the pre/postprocess kernels.
 */
#include <cuda_runtime_api.h>
#ifdef __SSE2__
#include <emmintrin.h>
#endif
#include <omp.h>
#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>
#include "thb_internal.h"

static char g_error[512];
const char *thb_engine_error(void) { return g_error; }
void thb_set_error(const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_error, sizeof(g_error), fmt, ap);
    va_end(ap);
    if (th_debug) fprintf(stderr, "thb200: %s\n", g_error);
}
#define CU(call)                                                                                   \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) {                                                                   \
            thb_set_error("%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
            return -1;                                                                             \
        }                                                                                          \
    } while (0)

void *thb_host_alloc_pinned(size_t bytes)
{
    void *p = 0;
    if (cudaHostAlloc(&p, bytes ? bytes : 1, cudaHostAllocPortable) != cudaSuccess) return 0;
    return p;
}
void thb_host_free_pinned(void *p)
{
    if (p) cudaFreeHost(p);
}

/* ------------------------------------------------------------------------------------------------ */
typedef struct {
    int N, C, H, W, rank;
    int flat, fC, fH, fW; /* flat: logical [N, C] view of a channels-innermost [N, fH, fW, fC] tensor */
} shape;

typedef struct {
    int buf;   /* activation buffer id, -1: not materialised */
    int ld;    /* pixel stride in elements */
    int coff;  /* channel offset inside the buffer */
    shape s;
    int csum_buf;        /* u8 mode: 1 + the buffer holding this tensor's per-pixel channel sums once a convolution asked for them; 0: none yet */
    float q_sub, q_mult; /* u8 mode */
    int q_dyn;           /* u8 mode: the scale is measured per forward (network input) */
    int row_pitch, pad_left; /* rows stored with horizontal zero padding (the staged network input only), else 0 */
} value;

typedef struct {
    size_t bytes, offset;
    int first, last;
    int zeroed; /* cleared before every forward, all such buffers at once (they lie at the arena's start) */
} abuf;

enum step_kind {
    ST_CONV, ST_GEMV, ST_MAXPOOL, ST_AVGPOOL, ST_AFFINE, ST_U8THR, ST_U8COMBINE, ST_COMBINE, ST_COPY, ST_SOFTMAX, ST_COL2IM,
    ST_CSUM, ST_TO_NCHW, ST_UPSAMPLE, ST_ZEROPAD, ST_REFLECTPAD, ST_SLICEC, ST_CMAX, ST_LOGSOFTMAX, ST_NORMALIZE, ST_UNPOOL, ST_FROM_NCHW
};

typedef struct {
    int kind, dtype;
    int scratch_buf; /* fp32 partial tiles of a convolution whose K blocks are split over several CTAs (-1: none) */
    int nin, in_buf[8], in_ld[8], in_coff[8];
    int out_buf, out_ld, out_coff;
    int aux_buf; /* csum scratch (conv u8) */
    int aux2_buf; /* conv u8: channel sums of its OUTPUT, written by the convolution itself for the next one (-1: none) */
    float coef[8];
    int N, H, W, C, oH, oW, kH, kW, dH, dW, padH, padW, flag;
    long pixels;
    const float *scale, *shift, *bias;
    thb_act act;
    float beta;
    int thr, val;
    thb_conv_desc conv;
    thb_tmap *tmap;
    const void *w; /* gemv weights */
    const void *w_split; /* conv fp32: the weights' parts for the tensor-core kernel (NULL: the kernel on the FP32 units) */
    int K, M;
    int dyn_quant; /* conv u8 whose input scale is only known per forward (first layer) */
    /* u8 conv constants needed to derive the per-forward parameters */
    float w_sub, w_mult, out_sub, out_mult;
    int flops_node; /* model node index of the conv (profiling) */
    int dual;       /* convolution with a second activation operand (in_buf[1]) instead of a residual */
    long out_pixels; int out_C; /* extent of the output tensor (th_minmax) */
    long in_off0, out_off0; /* element offsets added to the first input / the output (slices and joins along the batch dimension) */
    int pool_k, pool_pad, pool_oH, pool_oW; /* pool_k > 0: the max pooling that follows runs inside the convolution launch */
    double flops_extra; /* FLOPs of the second convolution computed by the same launch */
} step;

typedef struct instance {
    int device, slice_n, slice_off;
    cudaStream_t stream;
    cudaEvent_t ev0, ev1;
    cudaStream_t wb_stream; /* carries the copy of the normalised input back to the caller, beside the forward (made on first use) */
    cudaEvent_t ev_wb;
    int wb_pending;
    size_t device_bytes; /* allocated by the plan: activations, staging, result (weights belong to the engine) */
    void **allocs;
    int nallocs, capallocs;
    void **hostmem; /* host arrays the launches' descriptors point to */
    int nhost, caphost;
    unsigned char *arena;
    size_t arena_bytes, zero_bytes; /* the first zero_bytes of the arena are cleared before every forward */
    float *d_in;          /* staged NCHW fp32 input */
    unsigned char *d_img; /* staged u8 HWC images */
    float *d_out;         /* NCHW fp32 result */
    float *d_minmax;
    float h_minmax[2];    /* host copy of the slice's input extremes (uint8 engine) */
    int *d_status;
    int *h_status;        /* pinned: the boundary kernel out leaves a copy of *d_status here with every result */
    abuf *bufs;
    int nbufs;
    step *steps;
    int nsteps;
    value in_val, out_val;
    shape out_shape;
    long out_count;
    float last_ms;
    /* the planned launches as one CUDA graph: captured from the second forward on (the first runs them directly,
     * which also sets every kernel's attributes), replayed with a single launch afterwards */
    cudaGraphExec_t graph;
    int runs, graph_state; /* graph_state: 0 not tried, 1 usable, -1 capture failed or switched off */
    int graph_from;        /* first launch inside the graph (the ones before it are issued directly every forward) */
    int graph_launches;    /* kernel launches one replay stands for */
    /* Sliced start: a large batch is copied in `slices` parts on a stream of its own, and the first `prefix` launches run on
     * each part as it arrives (set up by choose_slices; 0: the launches wait for the whole batch) */
    int prefix, slices;
    int head; /* the last launch is a convolution that can leave its result as NCHW floats: no boundary kernel out */
    double hidden_us; /* modelled gain */
    cudaStream_t copy_stream;
    cudaEvent_t ev_slice[8];
    int input_s2d; /* the network input is staged space-to-depth by this factor, the stride of the first convolution (0: as it is) */
    int input_neigh; /* uint8 engine, 3x3 / stride 1 / pad 1 first convolution on a three-plane float batch: the boundary kernel
                      * stages every pixel's 27 quantised neighbours as the channels of that pixel (taps outside the image: the
                      * byte of 0.0), and the layer runs as a 1x1 convolution over them -- no gather, no border classes */
    int input_pad16; /* the network input is staged with 16 channels per pixel (zeros behind the real ones) for a stride-1
                      * first convolution, which then runs as a 16-channel convolution through the patch kernel */
} instance;

/* What an engine keeps per input shape: the planned launches and activation memory of every GPU (`inst`) and, once a
 * host-input forward was pipelined, of its sub-batches.  Weights are not in here: they belong to the engine (wblob). */
typedef struct shape_plan {
    int N, C, H, W, rank, cp;
    int built; /* GPUs used, 0: not built */
    instance inst[8];
    /* Host-input forwards are pipelined: the batch slice of each GPU is cut into `chunks` sub-batches, each with its own
     * plan instance and stream on that GPU, so that the host-to-device copy of one sub-batch runs under the kernels of
     * the one before it.  Built on the first such forward; chunk c of GPU g is pipe[g * chunks + c]. */
    instance pipe[32];
    int chunks, pipe_built, pipe_chunks;
    const unsigned char *cut; /* boundaries of the sub-batches in sixteenths (sub_batch_cuts), NULL: thb_slice_sub_batches */
    int peer_gather;
    int no_split; /* planned without second copies of fp32 weights: with them it did not fit */
    unsigned long long used; /* forward counter of the last use */
} shape_plan;

/* Packed weights and per-channel constants in device memory, kept by the engine and found again by what they were made
 * from: every plan of the same network on a device (a sub-batch, another batch size, another image size) shares them. */
typedef struct {
    int device, key[20];
    void *ptr;
    float meta[2]; /* uint8 weights: their quantisation */
} wblob;

/* Plans kept per engine.  A program whose last batch is short, or that alternates between a few image sizes, comes back
 * to a shape it used before: planning again costs milliseconds (a hundred allocations and the graph capture) against
 * hundreds of microseconds for the forward.  Bounded in number and, so that rarely used shapes do not pin device memory,
 * in bytes: plans beyond MAX_PLAN_BYTES are dropped least recently used first, whatever their number. */
enum { MAX_PLANS = 4 };
static const size_t MAX_PLAN_BYTES = (size_t)12 << 30;

struct thb_engine {
    thb_model *model;
    int mode, dtype, ngpus;
    float range;
    int strict_math;
    shape_plan *plans[MAX_PLANS];
    shape_plan *cur; /* the plan of the last forward (or the one being built) */
    unsigned long long clock;
    wblob *blobs;
    int nblobs, capblobs;
    int out_of_memory; /* the last plan failed for want of device memory */
    float *h_out;
    size_t h_out_bytes;
    float *h_stage; /* pinned staging buffer for float batches that arrive in pageable host memory */
    size_t h_stage_bytes;
    float last_ms;
    int peer_gather;
    /* arguments of the last forward, for the device-resident timing loop */
    int honour_pads; /* THB200_HONOUR_PADS=1: ending pads, dilation, auto_pad and reflection padding of ONNX convolutions are computed */
    int whole_batch; /* the model has an operator that looks across the batch: one GPU, no sub-batches */
    int last_has_x, last_cp, last_bgr;
    float last_mean[3], last_std[3];
};

static int align_of(int dtype) { return thb_channel_align(dtype); }
static int esize_of(int dtype) { return dtype == THB_F32 ? 4 : dtype == THB_U8 ? 1 : 2; }
static int ru(int v, int m) { return (v + m - 1) / m * m; }

/* ---- device allocations owned by an instance ---- */
static void *dalloc(thb_engine *E, instance *I, size_t bytes)
{
    void *p = 0;
    const cudaError_t e = cudaMalloc(&p, bytes ? bytes : 16);
    if (e != cudaSuccess) {
        E->out_of_memory = e == cudaErrorMemoryAllocation;
        cudaGetLastError();
        thb_set_error("cudaMalloc of %zu bytes failed on device %d", bytes, I->device);
        return 0;
    }
    I->device_bytes += bytes;
    if (I->nallocs == I->capallocs) {
        I->capallocs = I->capallocs ? I->capallocs * 2 : 64;
        I->allocs = realloc(I->allocs, I->capallocs * sizeof(void *));
    }
    I->allocs[I->nallocs++] = p;
    return p;
}
/* host memory that lives as long as the instance */
static void host_keep(instance *I, void *p)
{
    if (I->nhost == I->caphost) {
        I->caphost = I->caphost ? I->caphost * 2 : 64;
        I->hostmem = realloc(I->hostmem, I->caphost * sizeof(void *));
    }
    I->hostmem[I->nhost++] = p;
}

/* ---- weights and constants, owned by the engine ---- */
enum blob_tag { BL_SCALE = 1, BL_SHIFT, BL_SLOPE, BL_BIAS, BL_FACTOR, BL_ADDEND, BL_GEMV, BL_CONV, BL_KINFO, BL_WSAT, BL_SPLIT };
enum { BLOB_KEY = sizeof(((wblob *)0)->key) / sizeof(int) };

static wblob *blob_find(thb_engine *E, int device, const int *key)
{
    for (int i = 0; i < E->nblobs; i++)
        if (E->blobs[i].device == device && !memcmp(E->blobs[i].key, key, sizeof(E->blobs[i].key))) return &E->blobs[i];
    return 0;
}
/* upload `bytes` (host NULL: only room for them) and keep them under `key` (on the instance's device, which is current) */
static wblob *blob_add(thb_engine *E, int device, const int *key, const void *host, size_t bytes)
{
    void *p = 0;
    const cudaError_t e = cudaMalloc(&p, bytes ? bytes : 16);
    if (e != cudaSuccess || (host && cudaMemcpy(p, host, bytes, cudaMemcpyHostToDevice) != cudaSuccess)) {
        E->out_of_memory = e == cudaErrorMemoryAllocation;
        cudaGetLastError();
        if (p) cudaFree(p);
        thb_set_error("upload of %zu bytes failed on device %d", bytes, device);
        return 0;
    }
    if (E->nblobs == E->capblobs) {
        E->capblobs = E->capblobs ? E->capblobs * 2 : 256;
        E->blobs = realloc(E->blobs, E->capblobs * sizeof(wblob));
    }
    wblob *b = &E->blobs[E->nblobs++];
    memset(b, 0, sizeof(*b));
    b->device = device;
    memcpy(b->key, key, sizeof(b->key));
    b->ptr = p;
    return b;
}

/* ---- shape rules ---- */
static int conv_out(int in, int k, int d, int pad) { return (in + 2 * pad - k) / d + 1; }
/* SpatialMaxPooling.c:196-210 / SpatialAveragePooling.c:120-139 */
static int pool_out(int in, int k, int d, int pad, int ceil_mode, int any_pad)
{
    int o = ceil_mode ? (int)ceilf((float)(in - k + 2 * pad) / d) + 1 : (int)floorf((float)(in - k + 2 * pad) / d) + 1;
    if (any_pad && (o - 1) * d >= in + pad) --o; /* the last window must start inside the image */
    return o;
}

typedef struct {
    thb_engine *E;
    instance *I;
    thb_model *M;
    value *val;
    int *uses;      /* consumer count per node (+1 for the output) */
    int *absorbed;  /* node folded into an earlier launch */
    int *leader;    /* node index at which the value of node i is produced */
    int capbufs, capsteps;
} planner;

static int new_buf(planner *P, size_t bytes)
{
    instance *I = P->I;
    if (I->nbufs == P->capbufs) {
        P->capbufs = P->capbufs ? P->capbufs * 2 : 64;
        I->bufs = realloc(I->bufs, P->capbufs * sizeof(abuf));
    }
    abuf *b = &I->bufs[I->nbufs];
    b->bytes = (bytes + 255) & ~(size_t)255;
    b->offset = 0;
    b->zeroed = 0;
    b->first = b->last = -1;
    return I->nbufs++;
}
static step *new_step(planner *P, int kind)
{
    instance *I = P->I;
    if (I->nsteps == P->capsteps) {
        P->capsteps = P->capsteps ? P->capsteps * 2 : 64;
        I->steps = realloc(I->steps, P->capsteps * sizeof(step));
    }
    step *s = &I->steps[I->nsteps++];
    memset(s, 0, sizeof(*s));
    s->kind = kind;
    s->dtype = P->E->dtype;
    s->out_buf = s->aux_buf = s->aux2_buf = s->scratch_buf = -1;
    for (int i = 0; i < 8; i++) s->in_buf[i] = -1;
    s->flops_node = -1;
    return s;
}
static void step_in(step *s, const value *v)
{
    s->in_buf[s->nin] = v->buf;
    s->in_ld[s->nin] = v->ld;
    s->in_coff[s->nin] = v->coff;
    s->nin++;
}
/* fresh dense activation buffer for a value of shape `sh` */
static void materialise(planner *P, value *v, shape sh)
{
    int al = align_of(P->E->dtype);
    long pixels = (long)sh.N * sh.H * sh.W;
    v->s = sh;
    v->ld = ru(sh.C, al);
    v->coff = 0;
    v->buf = new_buf(P, (size_t)pixels * v->ld * esize_of(P->E->dtype));
}
static void step_out(step *s, const value *v)
{
    s->out_buf = v->buf;
    s->out_ld = v->ld;
    s->out_coff = v->coff;
    /* extent of the result, for the per-launch min/max report (th_minmax) */
    s->out_pixels = v->s.flat ? (long)v->s.N * v->s.fH * v->s.fW : (long)v->s.N * v->s.H * v->s.W;
    s->out_C = v->s.flat ? v->s.fC : v->s.C;
}

/* host-side value of one stored element (th_minmax report only) */
static float element_as_float(const void *p, long i, int dtype)
{
    if (dtype == THB_F32) return ((const float *)p)[i];
    if (dtype == THB_U8) return ((const unsigned char *)p)[i];
    unsigned short h = ((const unsigned short *)p)[i];
    unsigned int bits;
    if (dtype == THB_BF16) bits = (unsigned int)h << 16;
    else {
        const unsigned int sign = (h & 0x8000u) << 16, exp = (h >> 10) & 31, man = h & 1023;
        if (exp == 0) {
            float f = (float)man * (1.0f / 16777216.0f); /* subnormal: man * 2^-24 */
            return sign ? -f : f;
        }
        bits = exp == 31 ? sign | 0x7f800000u | (man << 13) : sign | ((exp + 112) << 23) | (man << 13);
    }
    float f;
    memcpy(&f, &bits, 4);
    return f;
}

/* Joining without a copy: when every launch that writes a value's buffer takes an output pitch (convolutions, pooling,
 * elementwise kernels) and every reader takes an input pitch and a channel offset (the concatenation itself,
 * convolutions, pooling), those launches are pointed at the value's channel slice of the joined buffer instead
 * (thb_conv_desc.in_ld / out_ld and the kernels' x_ld / y_ld exist for this), and the value's own buffer is never
 * allocated.  Returns 1 when done, 0 when the value has to be copied.  THB200_JOIN_COPY=1 keeps the copies (diagnostic). */
static int write_into_slice(planner *P, int node, value *v, int jbuf, int jld, int coff)
{
    const char *e = getenv("THB200_JOIN_COPY"); /* (read while planning, not per launch) */
    const int keep_copies = e && atoi(e);
    instance *I = P->I;
    if (keep_copies || node == P->M->output || v->buf < 0 || v->coff || v->row_pitch || v->s.flat || v->buf == I->in_val.buf)
        return 0;
    /* readers still to be planned will see the slice: all of them must be able to */
    for (int j = 0; j < P->M->nnodes; j++) {
        const thb_node *c = &P->M->nodes[j];
        for (int q = 0; q < c->nin; q++)
            if (c->in[q] == node && !(c->op == OP_CONCAT || c->op == OP_MAXPOOL || c->op == OP_AVGPOOL || (c->op == OP_CONV && q == 0)))
                return 0;
    }
    /* no other value may live in the buffer (views and aliases), launches of the same fused chain apart */
    for (int i = 0; i < P->M->nnodes; i++)
        if (i != node && P->val[i].buf == v->buf && !P->absorbed[i]) return 0;
    int writers = 0;
    for (int t = 0; t < I->nsteps; t++) {
        const step *s = &I->steps[t];
        for (int k = 0; k < s->nin; k++)
            if (s->in_buf[k] == v->buf) {
                /* an earlier reader: its first operand, through a kernel that takes pitch and offset */
                if (k != 0 || s->out_buf == v->buf || s->in_coff[0] || s->in_off0 || s->in_ld[0] != v->ld || s->dual ||
                    !(s->kind == ST_CONV || s->kind == ST_MAXPOOL || s->kind == ST_AVGPOOL || s->kind == ST_CSUM || s->kind == ST_COPY))
                    return 0;
                if (s->kind == ST_CONV && (s->conv.in_ld != v->ld || s->conv.in_row_pitch)) return 0;
            }
        if (s->aux_buf == v->buf || s->aux2_buf == v->buf) return 0;
        if (s->out_buf != v->buf) continue;
        if (s->out_coff || s->out_off0 || s->out_ld != v->ld) return 0;
        switch (s->kind) {
        case ST_CONV: case ST_MAXPOOL: case ST_AVGPOOL: case ST_AFFINE: case ST_COMBINE: case ST_U8COMBINE: case ST_U8THR:
        case ST_UPSAMPLE: case ST_COL2IM:
            writers++;
            break;
        default:
            return 0;
        }
    }
    if (!writers) return 0;
    for (int t = 0; t < I->nsteps; t++) {
        step *s = &I->steps[t];
        if (s->nin > 0 && s->in_buf[0] == v->buf) {
            s->in_buf[0] = jbuf; s->in_ld[0] = jld; s->in_coff[0] = coff;
            if (s->kind == ST_CONV) s->conv.in_ld = jld;
        }
        if (s->out_buf != v->buf) continue;
        s->out_buf = jbuf; s->out_ld = jld; s->out_coff = coff;
        if (s->kind == ST_CONV) s->conv.out_ld = jld;
    }
    v->buf = jbuf; v->ld = jld; v->coff = coff;
    return 1;
}

static int sole_consumer(planner *P, int node)
{
    if (P->uses[node] != 1 || node == P->M->output) return -1;
    for (int j = node + 1; j < P->M->nnodes; j++)
        for (int k = 0; k < P->M->nodes[j].nin; k++)
            if (P->M->nodes[j].in[k] == node) return j;
    return -1;
}

/* A small per-channel array on the device: `n` words padded with zeros to `padded`, shared by node, purpose and contents. */
static void *upload_words(planner *P, int node, int tag, const void *src, int n, int padded)
{
    unsigned *tmp = calloc(padded > 0 ? padded : 1, sizeof(unsigned));
    memcpy(tmp, src, sizeof(unsigned) * n);
    unsigned long long h = 1469598103934665603ull;
    for (int i = 0; i < padded; i++) h = (h ^ tmp[i]) * 1099511628211ull;
    const int key[BLOB_KEY] = {node, tag, n, padded, (int)h, (int)(h >> 32)};
    wblob *b = blob_find(P->E, P->I->device, key);
    if (!b) b = blob_add(P->E, P->I->device, key, tmp, sizeof(unsigned) * padded);
    free(tmp);
    return b ? b->ptr : 0;
}

static int fill_act(planner *P, thb_act *a, const thb_node *n, int C)
{
    const int node = (int)(n - P->M->nodes);
    a->kind = n->act_kind;
    a->threshold = n->act_threshold;
    a->value = n->act_value;
    a->alpha = n->act_alpha;
    a->slope = 0;
    if (n->act_kind == THB_ACT_PRELU) {
        /* the kernels read per-channel arrays in 16-byte groups and per 64-column block: a multiple of 64 floats */
        const int padded = ru(C, 64);
        float *tmp = calloc(padded, sizeof(float));
        if (!tmp || (n->nslope && n->nslope != C)) {
            free(tmp);
            thb_set_error("wrong number of input planes for PReLU (%d slopes, %d channels)", n->nslope, C);
            return -1;
        }
        for (int i = 0; i < C; i++) tmp[i] = n->nslope ? n->slope[i] : n->slope[0];
        a->slope = upload_words(P, node, BL_SLOPE, tmp, padded, padded);
        free(tmp);
        if (!a->slope) return -1;
    }
    return 0;
}

/* Where a planned convolution's weights come from and how they are laid out over the descriptor's Cout x Cin x kH x kW. */
enum { WS_PLAIN, WS_DECONV, WS_FLAT, WS_S2D, WS_NEIGH, WS_PAD16, WS_DILATED, WS_DUAL };
typedef struct {
    const thb_node *n;
    int bn, dual_conv, dual_bn, kind;
    float self_coef, res_coef; /* WS_DUAL */
    int permute_hw, ld;        /* WS_FLAT: positions per channel and stored channels of the flattened input */
    int s2d, s2d_padH, s2d_padW;
} wsource;

/* The weights in the descriptor's [Cout][Cin][kH][kW] order; a new array, or the node's own (then *owned = 0). */
static float *weights_oihw(const thb_model *M, const thb_conv_desc *d, const wsource *ws, int u8, int *owned)
{
    const thb_node *n = ws->n;
    const int kH = d->kH, kW = d->kW, Cin = d->Cin;
    float *fold = 0, *w = 0;
    const float *src = n->weight;
    if (u8 && ws->bn >= 0) {
        const size_t per = (size_t)n->Cin * n->kH * n->kW;
        src = fold = malloc(sizeof(float) * per * n->Cout);
#pragma omp parallel for schedule(static)
        for (int co = 0; co < n->Cout; co++)
            for (size_t k = 0; k < per; k++) fold[co * per + k] = n->weight[co * per + k] * M->nodes[ws->bn].scale[co];
    }
    *owned = 1;
    if (ws->kind == WS_PLAIN) {
        if (fold) return fold;
        *owned = 0;
        return n->weight;
    }
    const size_t count = (size_t)d->Cout * Cin * kH * kW;
    w = calloc(count ? count : 1, sizeof(float));
    switch (ws->kind) {
    case WS_DECONV: {
        /* column (kh*kW + kw)*Cp + co  <-  W[ci][co][kh][kw] */
        const int taps = n->kH * n->kW, Cp = d->Cout / taps;
        for (int ci = 0; ci < Cin; ci++)
            for (int co = 0; co < n->Cout; co++)
                for (int t = 0; t < taps; t++)
                    w[((size_t)t * Cp + co) * Cin + ci] = src[((size_t)ci * n->Cout + co) * taps + t];
        break;
    }
    case WS_FLAT:
#pragma omp parallel for schedule(static)
        for (int o = 0; o < n->Cout; o++)
            for (int k = 0; k < n->Cin; k++)
                w[(size_t)o * Cin + (size_t)(k % ws->permute_hw) * ws->ld + k / ws->permute_hw] = src[(size_t)o * n->Cin + k];
        break;
    case WS_S2D:
        /* W'[co][(ph*f + pw)*Cin + c][dh][dw] = W[co][c][f*(dh - pad') + ph + pad][...] where that row exists */
        for (int co = 0; co < n->Cout; co++)
            for (int c = 0; c < n->Cin; c++)
                for (int r = 0; r < n->kH; r++)
                    for (int q = 0; q < n->kW; q++) {
                        const int f = ws->s2d, tr = r - n->padH + f * ws->s2d_padH, tq = q - n->padW + f * ws->s2d_padW; /* >= 0 */
                        const int dh = tr / f, ph = tr % f, dw = tq / f, pw = tq % f;
                        w[(((size_t)co * Cin + (ph * f + pw) * n->Cin + c) * kH + dh) * kW + dw] =
                            src[(((size_t)co * n->Cin + c) * n->kH + r) * n->kW + q];
                    }
        break;
    case WS_NEIGH:
        /* W'[co][(r*3 + s)*3 + c] = W[co][c][r][s]: the order the boundary kernel stores a pixel's neighbours in */
        for (int co = 0; co < n->Cout; co++)
            for (int c = 0; c < 3; c++)
                for (int t = 0; t < 9; t++) w[(size_t)co * 27 + t * 3 + c] = src[((size_t)co * 3 + c) * 9 + t];
        break;
    case WS_PAD16:
        for (int co = 0; co < n->Cout; co++)
            memcpy(w + (size_t)co * 16 * kH * kW, src + (size_t)co * n->Cin * kH * kW, sizeof(float) * n->Cin * kH * kW);
        break;
    case WS_DILATED: {
        const int dlH = n->dlH > 0 ? n->dlH : 1, dlW = n->dlW > 0 ? n->dlW : 1;
        for (long oc = 0; oc < (long)n->Cout * Cin; oc++)
            for (int r = 0; r < n->kH; r++)
                for (int q = 0; q < n->kW; q++) w[(oc * kH + r * dlH) * kW + q * dlW] = src[(oc * n->kH + r) * n->kW + q];
        break;
    }
    case WS_DUAL: {
        const thb_node *c2 = &M->nodes[ws->dual_conv];
        const int c1n = n->Cin, c2n = c2->Cin;
        for (int co = 0; co < n->Cout; co++) {
            const float s1 = ws->self_coef * (ws->bn >= 0 ? M->nodes[ws->bn].scale[co] : 1.f);
            const float s2 = ws->res_coef * (ws->dual_bn >= 0 ? M->nodes[ws->dual_bn].scale[co] : 1.f);
            float *row = w + (size_t)co * (c1n + c2n);
            for (int ci = 0; ci < c1n; ci++) row[ci] = s1 * n->weight[(size_t)co * c1n + ci];
            for (int ci = 0; ci < c2n; ci++) row[c1n + ci] = s2 * c2->weight[(size_t)co * c2n + ci];
        }
        break;
    }
    }
    free(fold);
    return w;
}

/* The second copy of an fp32 convolution's weights, which sends it to the tensor cores; none, and so the kernel on the FP32 units,
 * where that one does not take the layer, where the device has no room for the copy, or none for the plan beside the copies, and
 * with THB200_NO_F32_TC=1. */
static const void *conv_split_weights(planner *P, const thb_conv_desc *d, const int *conv_key)
{
    thb_engine *E = P->E;
    const char *off = getenv("THB200_NO_F32_TC");
    if ((off && atoi(off)) || E->cur->no_split || !thb_conv_f32_supported(d)) return 0;
    int key[BLOB_KEY];
    memcpy(key, conv_key, sizeof(key));
    key[1] = BL_SPLIT;
    wblob *w = blob_find(E, P->I->device, key);
    if (w) return w->ptr;
    w = blob_add(E, P->I->device, key, 0, thb_conv_f32_split_bytes(d));
    if (!w) {
        E->out_of_memory = 0;
        return 0;
    }
    if (thb_conv_f32_split_weights(d, w->ptr, 0)) { /* (waited for at the end of the plan) */
        cudaFree(w->ptr);
        E->nblobs--;
        return 0;
    }
    return w->ptr;
}

/* Packed weights and gather table of a planned convolution: the engine's, when a plan with the same layout made them
 * before (another batch or image size nearly always has it), else packed here and uploaded. */
static int conv_weights(planner *P, step *s, thb_conv_desc *d, const wsource *ws)
{
    thb_engine *E = P->E;
    const int dev = P->I->device, node = (int)(ws->n - P->M->nodes), u8 = E->dtype == THB_U8;
    int key[BLOB_KEY] = {node, BL_CONV, ws->kind, ws->bn, ws->dual_conv, ws->dual_bn, ws->permute_hw, ws->ld, (ws->s2d * 16 + ws->s2d_padH) * 16 + ws->s2d_padW,
                         d->Cout, d->Cin, d->kH, d->kW, d->Cin_pad, d->Ktot_pad, d->Cout_pad, d->cin1, d->in_row_pitch ? d->in_ld : 0};
    wblob *w = blob_find(E, dev, key);
    if (!w) {
        const size_t wbytes = thb_conv_weight_bytes(d), kwords = thb_conv_kinfo_words(d);
        const size_t sat = (size_t)d->Cout * (d->kH + 1) * (d->kW + 1);
        void *packed = malloc(wbytes);
        int *kinfo = malloc(kwords * sizeof(int)), *wsat = 0, owned = 0;
        unsigned char *wq = 0;
        float *src = weights_oihw(P->M, d, ws, u8, &owned), sub = 0, mult = 0;
        if (u8) {
            /* lowp/lowp_basic.c:156-157: weights and bias quantised over their own ranges */
            const long wn = (long)d->Cout * d->Cin * d->kH * d->kW;
            wq = malloc(wn);
            thb_lowp_quantize(src, wn, wq, &sub, &mult);
            wsat = malloc(sizeof(int) * sat);
        }
        const int rc = thb_conv_pack_weights_host(d, u8 ? 0 : src, wq, packed, kinfo, wsat);
        int ok = !rc;
        if (ok) {
            key[1] = BL_KINFO;
            ok = blob_add(E, dev, key, kinfo, kwords * sizeof(int)) != 0;
        }
        if (ok && wsat) {
            key[1] = BL_WSAT;
            ok = blob_add(E, dev, key, wsat, sizeof(int) * sat) != 0;
        }
        if (ok) {
            /* last: its presence says that all of them are there */
            key[1] = BL_CONV;
            w = blob_add(E, dev, key, packed, wbytes);
            if (w) { w->meta[0] = sub; w->meta[1] = mult; }
        }
        if (owned) free(src);
        free(packed); free(kinfo); free(wsat); free(wq);
        if (rc) thb_set_error("weight packing failed (%d)", rc);
        if (!w) return -1;
    }
    d->w = w->ptr;
    s->w_sub = w->meta[0]; s->w_mult = w->meta[1];
    key[1] = BL_KINFO;
    d->kinfo = blob_find(E, dev, key)->ptr;
    key[1] = BL_WSAT;
    d->wsat = u8 ? blob_find(E, dev, key)->ptr : 0;
    if (d->dtype == THB_F32) {
        s->w_split = conv_split_weights(P, d, key);
        d->splits = s->w_split ? thb_conv_f32_splits(d) : thb_conv_simt_splits(d); /* (also on parts of the batch: a sliced start changes no sum) */
    }
    return 0;
}

/* Emit the launch(es) of a convolution / Linear / transposed convolution and whatever folds into it.
 * Returns the node whose value the launch produces. */
static int plan_gemm_group(planner *P, int i)
{
    thb_engine *E = P->E;
    instance *I = P->I;
    thb_model *M = P->M;
    thb_node *n = &M->nodes[i];
    const value *in = &P->val[n->in[0]];
    const int dtype = E->dtype, al = align_of(dtype);
    shape is = in->s, os = is;
    int is_linear = n->op == OP_LINEAR, is_deconv = n->op == OP_DECONV;
    /* first convolution of stride f on a space-to-depth input (see instance_build): rewritten as a stride-1 convolution
     * over f*f*Cin channels.  Input row f*oh - pad + r is block row oh + floor((r - pad)/f), phase (r - pad) mod f. */
    const int s2d = n->in[0] == 0 && n->op == OP_CONV ? I->input_s2d : 0, s2d_f = s2d ? s2d : 1;
    const int pad16 = I->input_pad16 && n->in[0] == 0 && n->op == OP_CONV;  /* 16 stored channels, zeros behind the real ones */
    const int neigh = I->input_neigh && n->in[0] == 0 && n->op == OP_CONV;  /* 27 neighbours per pixel: a 1x1 convolution */
    const int s2d_padH = (n->padH + s2d_f - 1) / s2d_f, s2d_padW = (n->padW + s2d_f - 1) / s2d_f;
    const int s2d_kH = (n->kH - 1 - n->padH) / s2d_f + s2d_padH + 1, s2d_kW = (n->kW - 1 - n->padW) / s2d_f + s2d_padW + 1;

    /* ---- geometry ---- */
    int kH = n->kH, kW = n->kW, Cin = n->Cin, H = is.H, W = is.W, in_ld = in->ld, permute_hw = 0;
    int honour = 0, ekH = n->kH, ekW = n->kW, padT = n->padH, padB = n->padH, padL = n->padW, padR = n->padW;
    value refl_val;
    if (is_linear) {
        long feat = is.flat ? (long)is.fC * is.fH * is.fW : (long)is.C * is.H * is.W;
        if (feat != n->Cin) { thb_set_error("Linear expects %d inputs, got %ld", n->Cin, feat); return -1; }
        if (is.flat || is.H * is.W > 1) {
            /* the features are an NCHW flatten of a channels-innermost tensor: permute the weight's K axis */
            int fH = is.flat ? is.fH : is.H, fW = is.flat ? is.fW : is.W;
            if (in->coff) { thb_set_error("Linear on a channel slice is not supported"); return -1; }
            permute_hw = fH * fW;
            Cin = permute_hw * in->ld;
            in_ld = Cin;
        }
        H = W = 1;
        os.rank = is.N == 1 ? 1 : 2;
        os.C = n->Cout; os.H = os.W = 1; os.flat = 0;
    } else if (is_deconv) {
        if (is.rank < 3) { thb_set_error("3D or 4D (batch mode) tensor is expected"); return -1; }
        if (is.C != n->Cin) { thb_set_error("input channels and nInputPlane dont match"); return -1; }
        os.C = n->Cout;
        os.H = (is.H - 1) * n->dH - 2 * n->padH + n->kH + n->adjH;
        os.W = (is.W - 1) * n->dW - 2 * n->padW + n->kW + n->adjW;
    } else if (neigh) {
        os.C = n->Cout;  /* same spatial size (3x3, pad 1, stride 1) */
        Cin = 27;
        kH = kW = 1;
    } else if (s2d) {
        /* the logical input is still [N, Cin, H, W]: output size from the original geometry */
        os.C = n->Cout;
        os.H = conv_out(E->cur->H, n->kH, s2d, n->padH);
        os.W = conv_out(E->cur->W, n->kW, s2d, n->padW);
        if (os.H < 1 || os.W < 1) { thb_set_error("Given input size: (%dx%dx%d). Output size is too small", n->Cin, E->cur->H, E->cur->W); return -1; }
        Cin = s2d == 2 ? 4 * n->Cin : in->ld; /* (stride 4: every stored channel, the unused ones with zero weights) */
        kH = s2d_kH; kW = s2d_kW;
    } else {
        if (is.rank < 3) { thb_set_error("convolution needs a 3D or 4D input"); return -1; }
        if (is.C != n->Cin) { thb_set_error("nInputPlane %d does not match input planes %d", n->Cin, is.C); return -1; }
        os.C = n->Cout;
        /* Ending pads that differ from the leading ones, dilation, auto_pad and reflection padding: the reference's ONNX
         * loader parses them and none of its engines reads them (SpatialConvolution.c:88-109, onnx.cc:677-690), so by
         * default they are ignored here too -- and said so.  THB200_HONOUR_PADS=1 computes what the ONNX model asks for:
         * auto_pad resolved from the input size, a reflection-padded copy of the input, the output size from both pads
         * (the kernels pad with zeros wherever a window leaves the image, so only the size changes), and a dilated
         * kernel written out with zeros between its taps. */
        const int dlH = n->dlH > 0 ? n->dlH : 1, dlW = n->dlW > 0 ? n->dlW : 1;
        const int nontrivial = n->op == OP_CONV && (n->pad2H != n->padH || n->pad2W != n->padW || dlH != 1 || dlW != 1 || n->autopad || n->refl_pad);
        if (nontrivial && !(E->honour_pads && dtype != THB_U8)) {
            static int told = 0;
            if (!told++)
                fprintf(stderr, "thb200: a convolution's ending pads / dilation / auto_pad / reflection padding are ignored, as by the "
                                "reference (THB200_HONOUR_PADS=1 honours them)\n");
        }
        if (nontrivial && E->honour_pads && dtype != THB_U8) {
            honour = 1;
            ekH = (kH - 1) * dlH + 1; ekW = (kW - 1) * dlW + 1;
            padT = n->padH; padB = n->pad2H; padL = n->padW; padR = n->pad2W;
            if (n->autopad) {
                /* SAME_UPPER (1): the odd pixel of padding goes to the end; SAME_LOWER (2): to the beginning */
                int th_ = ((is.H + n->dH - 1) / n->dH - 1) * n->dH + ekH - is.H, tw_ = ((is.W + n->dW - 1) / n->dW - 1) * n->dW + ekW - is.W;
                if (th_ < 0) th_ = 0;
                if (tw_ < 0) tw_ = 0;
                padT = n->autopad == 1 ? th_ / 2 : th_ - th_ / 2; padB = th_ - padT;
                padL = n->autopad == 1 ? tw_ / 2 : tw_ - tw_ / 2; padR = tw_ - padL;
            }
            if (n->refl_pad && (padT || padB || padL || padR)) {
                if (padT >= is.H || padB >= is.H || padL >= is.W || padR >= is.W) { thb_set_error("reflection padding larger than the image"); return -1; }
                shape ps = is;
                ps.H = is.H + padT + padB; ps.W = is.W + padL + padR;
                memset(&refl_val, 0, sizeof(refl_val));
                materialise(P, &refl_val, ps);
                step *rs = new_step(P, ST_REFLECTPAD);
                step_in(rs, in); step_out(rs, &refl_val);
                rs->N = is.N; rs->H = is.H; rs->W = is.W; rs->C = is.C;
                rs->padW = padL; rs->kW = padR; rs->padH = padT; rs->kH = padB;
                in = &refl_val;
                is = ps; H = is.H; W = is.W; in_ld = in->ld;
                padT = padB = padL = padR = 0;
            }
            os.H = (is.H + padT + padB - ekH) / n->dH + 1;
            os.W = (is.W + padL + padR - ekW) / n->dW + 1;
            kH = ekH; kW = ekW;
        } else {
            os.H = conv_out(is.H, kH, n->dH, n->padH);
            os.W = conv_out(is.W, kW, n->dW, n->padW);
        }
        if (os.H < 1 || os.W < 1) { thb_set_error("Given input size: (%dx%dx%d). Output size is too small", is.C, is.H, is.W); return -1; }
    }

    /* ---- what folds in ---- */
    int cur = i, bn = -1, comb = -1, act = -1, j;
    /* In uint8 mode a batch normalisation that follows is folded into the weights and the bias BEFORE they are
     * quantised (w' = w * scale[co], b' = b * scale[co] + shift[co], the algebra of the reference's ONNX loader,
     * onnx.cc:537-548): the reference's lowp engine itself refuses the module (lowp/lowp_basic.c:194-196). */
    if (!is_deconv && (j = sole_consumer(P, cur)) >= 0 && M->nodes[j].op == OP_BN) { bn = j; cur = j; }
    if (bn >= 0 && M->nodes[bn].C != n->Cout) { thb_set_error("batch-norm width mismatch"); return -1; }
    int res_node = -1;
    float self_coef = 1.f, res_coef = 0.f;
    /* uint8: the fused residual needs what thb_u8_combine needs (two tensors on the static range, coefficients +-1)
     * and the table-driven epilogue (at most 13 border classes, the image at least as large as the kernel) */
    const char *nofuse = getenv("THB200_U8_NO_FUSED_RESIDUAL");
    const int u8_res_ok = dtype == THB_U8 && !in->q_dyn && (1 + 2 * n->padH) * (1 + 2 * n->padW) <= 13 && H >= kH && W >= kW &&
                          n->padH < kH && n->padW < kW && !is_linear && !(nofuse && atoi(nofuse));
    if ((dtype != THB_U8 || u8_res_ok) && !is_deconv && (j = sole_consumer(P, cur)) >= 0 && M->nodes[j].op == OP_COMBINE && M->nodes[j].nin == 2) {
        int pos = M->nodes[j].in[0] == cur ? 0 : 1, other = M->nodes[j].in[1 - pos];
        const float c0 = M->nodes[j].coef[0], c1 = M->nodes[j].coef[1];
        const int u8_ok = dtype != THB_U8 || ((c0 == 1.f || c0 == -1.f) && (c1 == 1.f || c1 == -1.f) && !P->val[other].q_dyn &&
                                              P->val[other].q_sub == -E->range / 2 && P->val[other].q_mult == 255 / E->range);
        if (u8_ok && other != cur && other < i && P->val[other].buf >= 0 && !P->val[other].s.flat &&
            (long)P->val[other].s.C == os.C && P->val[other].s.H == os.H && P->val[other].s.W == os.W) {
            comb = j; cur = j; res_node = other;
            self_coef = M->nodes[j].coef[pos];
            res_coef = M->nodes[j].coef[1 - pos];
        }
    }
    /* Two 1x1 convolutions whose (batch-normalised) outputs meet in a two-input sum -- a bottleneck block's last
     * convolution and its projection shortcut -- run as ONE convolution over both inputs: the weights side by side
     * along K (each scaled by its batch-norm and its coefficient of the sum), one accumulator, neither addend written.
     * 16-bit tensor-core modes only; the second convolution must not have been planned yet and must be used nowhere else. */
    int dual_conv = -1, dual_bn = -1;
    {
        const char *nodual = getenv("THB200_NO_DUAL");
        if (comb < 0 && (dtype == THB_F16 || dtype == THB_BF16) && !is_deconv && !is_linear && !s2d && n->kH == 1 && n->kW == 1 &&
            n->dH == 1 && n->dW == 1 && n->padH == 0 && n->padW == 0 && n->Cin % 64 == 0 && n->Cout >= 64 && !in->row_pitch &&
            in->coff == 0 && !(nodual && atoi(nodual)) && (j = sole_consumer(P, cur)) >= 0 && M->nodes[j].op == OP_COMBINE &&
            M->nodes[j].nin == 2) {
            const int pos = M->nodes[j].in[0] == cur ? 0 : 1, other = M->nodes[j].in[1 - pos];
            int ob = -1, oc = other;
            if (other > cur && other < j && M->nodes[other].op == OP_BN && P->uses[other] == 1) { ob = other; oc = M->nodes[other].in[0]; }
            if (oc > cur && oc < j && P->uses[oc] == 1 && M->nodes[oc].op == OP_CONV && oc != M->output && other != M->output) {
                const thb_node *c2 = &M->nodes[oc];
                const value *v2 = &P->val[c2->in[0]];
                if (c2->kH == 1 && c2->kW == 1 && c2->padH == 0 && c2->padW == 0 && c2->dH == c2->dW && c2->dH >= 1 && c2->dH <= 8 &&
                    c2->Cout == n->Cout && c2->Cin % 64 == 0 && c2->in[0] <= i && v2->buf >= 0 && !v2->s.flat && v2->s.rank >= 3 &&
                    v2->s.C == c2->Cin && v2->coff == 0 && !v2->row_pitch && v2->s.N == is.N &&
                    conv_out(v2->s.H, 1, c2->dH, 0) == os.H && conv_out(v2->s.W, 1, c2->dW, 0) == os.W &&
                    (ob < 0 || M->nodes[ob].C == n->Cout)) {
                    dual_conv = oc; dual_bn = ob;
                    comb = j; cur = j;
                    self_coef = M->nodes[j].coef[pos];
                    res_coef = M->nodes[j].coef[1 - pos];
                }
            }
        }
    }
    if ((j = sole_consumer(P, cur)) >= 0 && M->nodes[j].op == OP_ACT &&
        (dtype != THB_U8 || M->nodes[j].act_kind == THB_ACT_THRESHOLD)) { act = j; cur = j; }
    for (int k = i + 1; k <= cur; k++)
        if (k == bn || k == comb || k == act || k == dual_conv || k == dual_bn) { P->absorbed[k] = 1; P->leader[k] = i; }
    /* A stride-2 max pooling as the only consumer of this convolution (after its batch-norm and activation) can run
     * inside the convolution's launch, which then stores the pooled tensor only: decided below, once the kernel
     * geometry is known (16-bit types, at most 64 output channels, stride-1 convolution). */
    int pool = -1;
    if ((dtype == THB_F16 || dtype == THB_BF16) && !is_linear && !is_deconv && comb < 0 && dual_conv < 0 && n->Cout <= 64 &&
        (j = sole_consumer(P, cur)) >= 0 && M->nodes[j].op == OP_MAXPOOL) {
        const thb_node *pn = &M->nodes[j];
        if (pn->kH == pn->kW && pn->dH == 2 && pn->dW == 2 && pn->padH == pn->padW) pool = j;
    }

    /* ---- per-channel scale / shift ---- */
    float *scale = 0, *shift = 0;
    float *scale_h = 0, *shift_h = 0; /* host copies, owned by the instance (thb_conv_desc.scale_host / shift_host) */
    if (dtype != THB_U8) {
        int Cp = ru(n->Cout, 64);
        float *hs = calloc(Cp, sizeof(float)), *hh = calloc(Cp, sizeof(float));
        for (int c = 0; c < n->Cout; c++) {
            float b = n->bias ? n->bias[c] : 0.f;
            hs[c] = bn >= 0 ? M->nodes[bn].scale[c] : 1.f;
            hh[c] = bn >= 0 ? M->nodes[bn].scale[c] * b + M->nodes[bn].shift[c] : b;
        }
        if (bn >= 0 && M->nodes[bn].C != n->Cout) { free(hs); free(hh); thb_set_error("batch-norm width mismatch"); return -1; }
        if (dual_conv >= 0) {
            /* both scales go into the weights (below); what is left is the sum of the two shifts */
            const thb_node *c2 = &M->nodes[dual_conv];
            for (int c = 0; c < n->Cout; c++) {
                const float b2 = c2->bias ? c2->bias[c] : 0.f;
                const float h2 = dual_bn >= 0 ? M->nodes[dual_bn].scale[c] * b2 + M->nodes[dual_bn].shift[c] : b2;
                hh[c] = self_coef * hh[c] + res_coef * h2;
                hs[c] = 1.f;
            }
        }
        if (bn >= 0 && dual_conv < 0) { scale = upload_words(P, i, BL_SCALE, hs, Cp, Cp); scale_h = hs; }
        if ((dual_conv >= 0 || bn >= 0 || n->bias) && !is_deconv) { shift = upload_words(P, i, BL_SHIFT, hh, Cp, Cp); shift_h = hh; }
        if (scale_h) host_keep(P->I, hs); else free(hs);
        if (shift_h) host_keep(P->I, hh); else free(hh);
    }

    value *out = &P->val[cur];

    /* ---- small-batch Linear: weight-streaming GEMV ---- */
    if (is_linear && dtype != THB_U8 && is.N <= 8) {
        materialise(P, out, os);
        step *s = new_step(P, ST_GEMV);
        step_in(s, in);
        step_out(s, out);
        /* weight rows are as long as the physical feature vector (channel padding included, zero weights there) */
        const int Kp = permute_hw ? Cin : in->ld;
        s->N = is.N; s->K = Kp; s->M = n->Cout; s->in_ld[0] = permute_hw ? in_ld : in->ld;
        s->scale = scale; s->shift = shift;
        if (act >= 0 && fill_act(P, &s->act, &M->nodes[act], n->Cout)) return -1;
        const int key[BLOB_KEY] = {i, BL_GEMV, Kp, permute_hw, in->ld};
        wblob *wb = blob_find(E, P->I->device, key);
        if (!wb) {
            const size_t es = esize_of(dtype);
            unsigned char *hw = calloc((size_t)n->Cout * Kp, es);
#pragma omp parallel for schedule(static)
            for (int o = 0; o < n->Cout; o++)
                for (int k = 0; k < n->Cin; k++) {
                    long dst = k;
                    if (permute_hw) { int c = k / permute_hw, hw_ = k % permute_hw; dst = (long)hw_ * in->ld + c; }
                    float v = n->weight[(size_t)o * n->Cin + k];
                    if (dtype == THB_F32) ((float *)hw)[(size_t)o * Kp + dst] = v;
                    else ((unsigned short *)hw)[(size_t)o * Kp + dst] = thb_float_to_half_bits(v, dtype == THB_BF16);
                }
            wb = blob_add(E, P->I->device, key, hw, (size_t)n->Cout * Kp * es);
            free(hw);
        }
        if (!wb) return -1;
        s->w = wb->ptr;
        s->flops_node = i;
        return cur;
    }

    /* ---- implicit-GEMM convolution launch ---- */
    int csum_buf = -1;
    if (dtype == THB_U8) {
        /* per-pixel channel sums of the input feed the zero-point correction of the convolution */
        /* (several convolutions reading one tensor share one pass; csum_buf holds buffer index + 1, 0 = none yet) */
        value *inw = &P->val[n->in[0]];
        if (inw->csum_buf > 0 && !is_linear) csum_buf = inw->csum_buf - 1;
        else {
            csum_buf = new_buf(P, sizeof(int) * (size_t)is.N * H * W);
            step *cs = new_step(P, ST_CSUM);
            step_in(cs, in);
            cs->in_ld[0] = in_ld;
            cs->pixels = (long)is.N * H * W; cs->C = Cin; cs->out_buf = csum_buf;
            cs->W = W; cs->oW = in->row_pitch; cs->padW = in->pad_left;
            if (!is_linear) inw->csum_buf = csum_buf + 1;
        }
    }
    step *s = new_step(P, ST_CONV);
    thb_conv_desc *d = &s->conv;
    s->aux_buf = csum_buf;
    d->dtype = dtype;
    d->N = is.N; d->H = H; d->W = W; d->Cin = Cin; d->in_ld = in_ld;
    d->in_row_pitch = in->row_pitch; d->in_pad_left = in->pad_left;
    d->kH = kH; d->kW = kW; d->dH = n->dH; d->dW = n->dW; d->padH = n->padH; d->padW = n->padW;
    if (neigh) d->padH = d->padW = 0;
    d->self_coef = 1.f; d->res_coef = 0.f; d->relu_thr = -1;
    int Cp_out = ru(n->Cout, al);
    wsource ws = {n, bn, dual_conv, dual_bn, WS_PLAIN, self_coef, res_coef, permute_hw, in->ld, s2d, s2d_padH, s2d_padW};
    float *b_fold = 0; /* uint8: bias with the batch normalisation folded in (the weights: conv_weights) */
    const float *bias_eff = n->bias;
    if (dtype == THB_U8 && bn >= 0) {
        b_fold = malloc(sizeof(float) * n->Cout);
        for (int co = 0; co < n->Cout; co++)
            b_fold[co] = (n->bias ? n->bias[co] * M->nodes[bn].scale[co] : 0.f) + M->nodes[bn].shift[co];
        bias_eff = b_fold;
    }
    if (is_deconv) {
        /* column matrix [N*H*W][kH*kW*Cp] */
        ws.kind = WS_DECONV;
        d->Cout = kH * kW * Cp_out; d->kH = d->kW = 1; d->dH = d->dW = 1; d->padH = d->padW = 0;
        d->oH = H; d->oW = W;
    } else if (is_linear) {
        d->Cout = n->Cout; d->oH = d->oW = 1;
        if (permute_hw && b_fold) { free(b_fold); thb_set_error("batch-norm after a flattened Linear is not supported in Lowp"); return -1; }
        if (permute_hw) ws.kind = WS_FLAT;
    } else if (s2d) {
        ws.kind = WS_S2D;
        d->Cout = n->Cout; d->oH = os.H; d->oW = os.W;
        d->dH = d->dW = 1; d->padH = s2d_padH; d->padW = s2d_padW;
    } else if (neigh) {
        ws.kind = WS_NEIGH;
        d->Cout = n->Cout; d->oH = os.H; d->oW = os.W;
    } else if (pad16) {
        /* the same convolution over 16 input channels, the added ones with zero weights */
        ws.kind = WS_PAD16;
        d->Cout = n->Cout; d->oH = os.H; d->oW = os.W;
        d->Cin = 16;
        d->BN = 64; /* (the patch kernel's tile, also below 33 output channels) */
    } else {
        d->Cout = n->Cout; d->oH = os.H; d->oW = os.W;
        if (honour) {
            d->padH = padT; d->padW = padL;
            /* dilation: the kernel written out at its full extent, zeros between the taps */
            if (ekH != n->kH || ekW != n->kW) ws.kind = WS_DILATED;
        }
    }
    if (dual_conv >= 0) {
        /* [Cout][cin1 + cin2] weights: each convolution's rows scaled by its batch-norm and its coefficient of the sum */
        const thb_node *c2 = &M->nodes[dual_conv];
        const value *v2 = &P->val[c2->in[0]];
        ws.kind = WS_DUAL;
        d->Cin = n->Cin + c2->Cin;
        d->cin1 = n->Cin;
        d->x2_ld = v2->ld; d->x2_H = v2->s.H; d->x2_W = v2->s.W; d->x2_d = c2->dH;
    }
    if (pool >= 0) d->BN = 64;
    if (thb_conv_geometry(d)) { free(b_fold); thb_set_error("unsupported convolution geometry %dx%d", kH, kW); return -1; }
    if (pool >= 0 && !thb_conv_maxpool_supported(d, M->nodes[pool].kH, 2, M->nodes[pool].padH)) {
        pool = -1;
        d->BN = 0;
        thb_conv_geometry(d);
    }
    if (dual_conv < 0 && in_ld < d->Cin_pad) { free(b_fold); thb_set_error("internal: input stride %d below padded channels %d", in_ld, d->Cin_pad); return -1; }
    /* Splitting a reduction over CTAs changes the order in which its fp32 partial sums are added, and whether a layer is
     * split depends on how many tiles the (sub-)batch gives it: with it, a batch sharded over GPUs or cut into sub-batches
     * no longer reproduces the whole batch bit for bit.  That identity is worth more than the few-tile layers' time, so
     * the 16-bit engines split only on request (THB200_SPLITK=1). */
    const char *ske = getenv("THB200_SPLITK");
    const int want_split = ske && atoi(ske);
    if (want_split && is_linear && (dtype == THB_F16 || dtype == THB_BF16) && d->BN < 128 && d->Cout >= 128) {
        /* A Linear on a batch of rows is a handful of tiles with a very long reduction.  The geometry rule narrows its tiles
         * so that more SMs get a share of the weights; where the reduction can be split over CTAs instead, wide tiles
         * move four times the weight bytes per barrier round (25088 -> 4096 on 32 rows: 135 -> about 40 us). */
        const int bn_narrow = d->BN;
        size_t bytes = 0;
        d->BN = 128;
        if (thb_conv_geometry(d) || thb_conv_splitk_plan(d, &bytes) < 2) {
            d->BN = bn_narrow;
            thb_conv_geometry(d);
        }
    }
    if (!want_split && pool < 0 && P->I->slice_n > 0 && is.N == P->I->slice_n && (dtype == THB_F16 || dtype == THB_BF16)) {
        /* Few tiles: the CTAs of a cluster share each tile's reduction.  The split follows from the batch of the whole call, so
         * that a GPU's slice of it, or a sub-batch, adds its partial sums in the same order as the whole batch on one GPU. */
        thb_conv_desc whole = *d;
        whole.N = E->cur->N;
        whole.out_ld = ru(d->Cout, al);
        d->splits = thb_conv_few_splits(&whole);
        if (d->splits < 2) d->splits = 0;
    }
    /* (integer sums: any split gives the same bytes) */
    if (dtype == THB_U8 && is.N == P->I->slice_n) {
        d->out_ld = ru(d->Cout, al);
        d->splits = thb_conv_few_splits(d);
    }
    if (want_split && pool < 0 && dual_conv < 0 && (dtype == THB_F16 || dtype == THB_BF16) && !thb_conv_patch_supported(d)) {
        /* a launch of few tiles: several CTAs share each tile's reduction, through an fp32 scratch that lives for this launch */
        size_t sk_bytes = 0;
        const int S = thb_conv_splitk_plan(d, &sk_bytes);
        if (S > 1) {
            d->splits = S;
            s->scratch_buf = new_buf(P, sk_bytes);
        }
    }

    if (conv_weights(P, s, d, &ws)) { free(b_fold); return -1; }
    if (dtype != THB_F32) {
        s->tmap = aligned_alloc(64, sizeof(thb_tmap));
        if (thb_conv_make_tmap(d, s->tmap)) { thb_set_error("TMA descriptor creation failed"); return -1; }
        d->tmap = s->tmap;
    }
    d->status = P->I->d_status;
    step_in(s, in);
    s->in_ld[0] = in_ld;
    s->flops_node = i;
    if (dual_conv >= 0) {
        step_in(s, &P->val[M->nodes[dual_conv].in[0]]);
        s->dual = 1;
        s->flops_extra = 2.0 * is.N * os.H * os.W * (double)n->Cout * M->nodes[dual_conv].Cin;
    }

    if (dtype == THB_U8) {
        if (!bias_eff) { thb_set_error("the lowp engine needs a bias on every convolution"); return -1; }
        unsigned char *bq = malloc(n->Cout);
        float b_sub, b_mult;
        thb_lowp_quantize(bias_eff, n->Cout, bq, &b_sub, &b_mult);
        free(b_fold);
        if (b_mult == 0) { free(bq); thb_set_error("an all-zero bias has no quantisation range in the lowp engine"); return -1; }
        float out_sub = -E->range / 2, out_mult = 255 / E->range; /* lowp_basic.c:137-138 */
        int *addend = malloc(sizeof(int) * n->Cout);
        thb_lowp_bias_addends(bq, n->Cout, b_sub, b_mult, out_mult, addend);
        d->bias_add = upload_words(P, i, BL_ADDEND, addend, n->Cout, n->Cout);
        free(addend); free(bq);
        s->out_sub = out_sub; s->out_mult = out_mult;
        int ohw = d->oH * d->oW;
        d->tail_start = ohw - ohw % 8;
        if (in->q_dyn) s->dyn_quant = 1;
        else {
            thb_lowp_gemm_params(s->w_sub, s->w_mult, in->q_sub, in->q_mult, out_sub, out_mult, &d->a_offset, &d->b_offset,
                                 &d->c_offset, &d->c_mult, &d->c_shift);
        }
        if (act >= 0) {
            /* lowp_Threshold.c:7-8: both bytes scaled with the (conv output) quantisation parameters */
            d->relu_thr = thb_lowp_scale_float(out_sub, out_mult, M->nodes[act].act_threshold);
            d->relu_val = thb_lowp_scale_float(out_sub, out_mult, M->nodes[act].act_value);
        }
        out->q_sub = out_sub; out->q_mult = out_mult;
        /* one column tile: the epilogue sees every output byte of a pixel and leaves their sum for the next convolution */
        const char *nocs = getenv("THB200_U8_NO_CSUM_OUT");
        if (!is_linear && !(nocs && atoi(nocs) == 1) && (d->Cout_pad == d->BN || !(nocs && atoi(nocs) == 2))) {
            s->aux2_buf = new_buf(P, sizeof(int) * (size_t)is.N * os.H * os.W);
            out->csum_buf = s->aux2_buf + 1;
            /* several column tiles add their shares, into a cleared buffer (a clearing launch in front of each of them was a
             * tenth of a ResNet-50 forward: 2.7 to 6 us, and every one breaks the programmatic launch chain) */
            P->I->bufs[s->aux2_buf].zeroed = d->splits ? (d->Cout_pad + 63) / 64 * d->splits > 1 : d->Cout_pad != d->BN;
        }
        if (res_node >= 0) {
            const value *rv = &P->val[res_node];
            step_in(s, rv);
            d->res_ld = rv->ld;
            d->self_coef = self_coef; d->res_coef = res_coef;
        }
    } else {
        d->scale = scale; d->shift = shift;
        d->scale_host = scale_h; d->shift_host = shift_h;
        if (act >= 0 && !is_deconv && fill_act(P, &d->act, &M->nodes[act], n->Cout)) return -1;
        if (res_node >= 0) {
            const value *rv = &P->val[res_node];
            step_in(s, rv);
            d->res_ld = rv->ld;
            d->self_coef = self_coef; d->res_coef = res_coef;
        }
    }

    if (is_deconv) {
        value cols;
        shape cs = is; cs.C = d->Cout;
        memset(&cols, 0, sizeof(cols));
        materialise(P, &cols, cs);
        s = &P->I->steps[P->I->nsteps - 1];
        step_out(s, &cols);
        s->conv.out_ld = cols.ld;
        materialise(P, out, os);
        step *g = new_step(P, ST_COL2IM);
        step_in(g, &cols);
        step_out(g, out);
        g->N = is.N; g->H = is.H; g->W = is.W; g->C = n->Cout; g->kH = kH; g->kW = kW; g->dH = n->dH; g->dW = n->dW;
        g->padH = n->padH; g->padW = n->padW; g->oH = os.H; g->oW = os.W;
        /* SpatialFullConvolution.c:229-238: the bias GEMM runs with beta = 11 whenever a bias exists */
        g->beta = E->strict_math ? 1.f : 11.f;
        if (n->bias) g->bias = upload_words(P, i, BL_BIAS, n->bias, n->Cout, ru(n->Cout, 64));
        if (act >= 0 && fill_act(P, &g->act, &M->nodes[act], n->Cout)) return -1;
        return cur;
    }
    if (pool >= 0) {
        const thb_node *pn = &M->nodes[pool];
        shape ps = os;
        ps.H = pool_out(os.H, pn->kH, 2, pn->padH, pn->ceil_mode, pn->padH || pn->padW);
        ps.W = pool_out(os.W, pn->kW, 2, pn->padW, pn->ceil_mode, pn->padH || pn->padW);
        if (ps.H < 1 || ps.W < 1) { thb_set_error("input image smaller than kernel size"); return -1; }
        P->absorbed[pool] = 1;
        P->leader[pool] = i;
        out = &P->val[pool];
        os = ps;
        cur = pool;
    }
    materialise(P, out, os);
    s = &P->I->steps[P->I->nsteps - 1];
    step_out(s, out);
    s->conv.out_ld = out->ld;
    if (pool >= 0) {
        s->pool_k = M->nodes[pool].kH; s->pool_pad = M->nodes[pool].padH; s->pool_oH = os.H; s->pool_oW = os.W;
    }
    return cur;
}

static int plan_node(planner *P, int i)
{
    thb_engine *E = P->E;
    thb_model *M = P->M;
    thb_node *n = &M->nodes[i];
    const int dtype = E->dtype, al = align_of(dtype);
    value *out = &P->val[i];
    const value *in = n->nin ? &P->val[n->in[0]] : 0;
    step *s;
    int j;

    if (dtype == THB_U8 && n->op != OP_CONV && n->op != OP_LINEAR && n->op != OP_ACT && n->op != OP_MAXPOOL &&
        n->op != OP_VIEW && n->op != OP_ALIAS && n->op != OP_AVGPOOL && !(n->op == OP_COMBINE && n->nin == 2)) {
        /* the reference's lowp conversion rejects these module types too (lowp_basic.c:160-208); beyond it, this engine
         * takes what a residual network needs: a batch normalisation folded into the convolution before it, the
         * two-input CAddTable / CSubTable and the average pooling, each on the static output quantisation */
        thb_set_error("operator %d not supported in Lowp", n->op);
        return -1;
    }
    switch (n->op) {
    case OP_CONV: case OP_LINEAR: case OP_DECONV:
        return plan_gemm_group(P, i) < 0 ? -1 : 0;
    case OP_BN: case OP_ACT: case OP_SCALE: {
        int act = -1, C = in->s.C;
        if (in->s.flat) { thb_set_error("elementwise operator on a flattened spatial tensor is not supported"); return -1; }
        value *dst = out;
        if (dtype == THB_U8) {
            if (n->act_kind != THB_ACT_THRESHOLD) { thb_set_error("only Threshold is supported in Lowp"); return -1; }
            materialise(P, out, in->s);
            out->q_sub = in->q_sub; out->q_mult = in->q_mult;
            s = new_step(P, ST_U8THR);
            step_in(s, in); step_out(s, out);
            s->pixels = (long)in->s.N * in->s.H * in->s.W; s->C = C;
            s->thr = thb_lowp_scale_float(in->q_sub, in->q_mult, n->act_threshold);
            s->val = thb_lowp_scale_float(in->q_sub, in->q_mult, n->act_value);
            if (in->q_dyn) { thb_set_error("Threshold directly on the network input is not supported in Lowp"); return -1; }
            return 0;
        }
        if (n->op == OP_BN && (j = sole_consumer(P, i)) >= 0 && M->nodes[j].op == OP_ACT) {
            act = j; P->absorbed[j] = 1; P->leader[j] = i; dst = &P->val[j];
        }
        materialise(P, dst, in->s);
        s = new_step(P, ST_AFFINE);
        step_in(s, in); step_out(s, dst);
        s->pixels = (long)in->s.N * in->s.H * in->s.W; s->C = C;
        if (n->op == OP_BN) {
            if (n->C != C) { thb_set_error("batch-norm over %d channels applied to %d", n->C, C); return -1; }
            s->scale = upload_words(P, i, BL_SCALE, n->scale, C, ru(C, 64));
            s->shift = upload_words(P, i, BL_SHIFT, n->shift, C, ru(C, 64));
            if (act >= 0 && fill_act(P, &s->act, &M->nodes[act], C)) return -1;
        } else if (n->op == OP_SCALE) {
            float *f = malloc(sizeof(float) * C);
            for (int c = 0; c < C; c++) f[c] = n->factor;
            s->scale = upload_words(P, i, BL_FACTOR, f, C, ru(C, 64));
            free(f);
        } else if (fill_act(P, &s->act, n, C))
            return -1;
        return 0;
    }
    case OP_MAXPOOL: case OP_AVGPOOL: {
        shape os = in->s;
        int kH = n->kH, kW = n->kW;
        if (in->s.rank < 3 || in->s.flat) { thb_set_error("3D or 4D (batch mode) tensor expected"); return -1; }
        if (n->op == OP_AVGPOOL) {
            if (kW == 0) kW = in->s.W;
            if (kH == 0) kH = in->s.H;
            if (!(kW / 2 >= n->padW && kH / 2 >= n->padH)) { thb_set_error("pad should be smaller than half of kernel size"); return -1; }
        }
        if (dtype == THB_U8 && n->op == OP_AVGPOOL && (n->padH || n->padW || in->q_dyn)) {
            thb_set_error("padded average pooling is not supported in Lowp");
            return -1;
        }
        os.H = pool_out(in->s.H, kH, n->dH, n->padH, n->ceil_mode, n->padH || n->padW);
        os.W = pool_out(in->s.W, kW, n->dW, n->padW, n->ceil_mode, n->padH || n->padW);
        if (os.H < 1 || os.W < 1) { thb_set_error("input image smaller than kernel size"); return -1; }
        materialise(P, out, os);
        out->q_sub = in->q_sub; out->q_mult = in->q_mult; out->q_dyn = in->q_dyn;
        s = new_step(P, n->op == OP_MAXPOOL ? ST_MAXPOOL : ST_AVGPOOL);
        step_in(s, in); step_out(s, out);
        s->N = in->s.N; s->H = in->s.H; s->W = in->s.W; s->C = in->s.C; s->kH = kH; s->kW = kW; s->dH = n->dH; s->dW = n->dW;
        s->padH = n->padH; s->padW = n->padW; s->oH = os.H; s->oW = os.W; s->flag = n->count_include_pad;
        if (dtype == THB_U8 && n->op == OP_MAXPOOL && thb_maxpool_sums_supported(in->s.C, kH, kW, in->ld, out->ld)) {
            /* the pixels' channel sums for the convolution behind it, from the values in hand */
            s->aux2_buf = new_buf(P, sizeof(int) * (size_t)os.N * os.H * os.W);
            out->csum_buf = s->aux2_buf + 1;
        }
        return 0;
    }
    case OP_COMBINE: {
        if (dtype == THB_U8) {
            const value *b = &P->val[n->in[1]];
            int act = -1;
            if (in->q_dyn || b->q_dyn || in->q_sub != b->q_sub || in->q_mult != b->q_mult ||
                in->q_sub != -E->range / 2 || in->s.flat || b->s.flat) {
                thb_set_error("CAddTable in Lowp needs two tensors on the static output quantisation");
                return -1;
            }
            if (b->s.C != in->s.C || b->s.H != in->s.H || b->s.W != in->s.W || b->s.N != in->s.N) {
                thb_set_error("Sum of tensors of different sizes");
                return -1;
            }
            if ((n->coef[0] != 1.f && n->coef[0] != -1.f) || (n->coef[1] != 1.f && n->coef[1] != -1.f)) {
                thb_set_error("only sums and differences are supported in Lowp");
                return -1;
            }
            value *dst = out;
            if ((j = sole_consumer(P, i)) >= 0 && M->nodes[j].op == OP_ACT && M->nodes[j].act_kind == THB_ACT_THRESHOLD) {
                act = j; P->absorbed[j] = 1; P->leader[j] = i; dst = &P->val[j];
            }
            materialise(P, dst, in->s);
            dst->q_sub = in->q_sub; dst->q_mult = in->q_mult;
            s = new_step(P, ST_U8COMBINE);
            step_in(s, in); step_in(s, b); step_out(s, dst);
            s->coef[0] = n->coef[0]; s->coef[1] = n->coef[1];
            s->pixels = (long)in->s.N * in->s.H * in->s.W; s->C = in->s.C;
            s->thr = -1; s->val = 0;
            if (act >= 0) {
                s->thr = thb_lowp_scale_float(in->q_sub, in->q_mult, M->nodes[act].act_threshold);
                s->val = thb_lowp_scale_float(in->q_sub, in->q_mult, M->nodes[act].act_value);
            }
            return 0;
        }
        materialise(P, out, in->s);
        s = new_step(P, ST_COMBINE);
        for (int k = 0; k < n->nin; k++) {
            const value *v = &P->val[n->in[k]];
            if (v->s.C != in->s.C || v->s.H != in->s.H || v->s.W != in->s.W || v->s.N != in->s.N) {
                thb_set_error("Sum of tensors of different sizes");
                return -1;
            }
            step_in(s, v);
            s->coef[k] = n->coef[k];
        }
        step_out(s, out);
        s->pixels = (long)in->s.N * in->s.H * in->s.W; s->C = in->s.C;
        return 0;
    }
    case OP_CONCAT: {
        /* JoinTable.c:43-44: dimension 1 of a 1-D or 3-D input means dimension 0; only the channel
         * (feature) dimension is supported here */
        int dim = n->dim;
        if (dim == 1 && (in->s.rank == 1 || in->s.rank == 3)) dim--;
        int chan_dim = (in->s.rank == 4 || in->s.rank == 2) ? 1 : 0;
        if (dim == 0 && chan_dim == 1) {
            /* JoinTable.c:46-57 / Concat.c:21-76 along the batch dimension: the inputs' images one after the other */
            if (P->I->slice_n != E->cur->N) { thb_set_error("concatenation along the batch dimension needs the whole batch on one GPU"); return -1; }
            shape os = in->s;
            os.N = 0;
            for (int k = 0; k < n->nin; k++) {
                const value *v = &P->val[n->in[k]];
                if (v->s.rank != in->s.rank || v->s.flat) { thb_set_error("Concatenation of tensors of different dimensionality"); return -1; }
                if (v->s.H != in->s.H || v->s.W != in->s.W || v->s.C != in->s.C) { thb_set_error("Concatenation of tensors of different sizes"); return -1; }
                os.N += v->s.N;
            }
            materialise(P, out, os);
            long img = 0;
            for (int k = 0; k < n->nin; k++) {
                const value *v = &P->val[n->in[k]];
                s = new_step(P, ST_COPY);
                step_in(s, v); step_out(s, out);
                s->pixels = (long)v->s.N * os.H * os.W; s->C = v->s.C;
                s->out_off0 = img * os.H * os.W * out->ld;
                img += v->s.N;
            }
            return 0;
        }
        if (dim != chan_dim) { thb_set_error("concatenation along dimension %d is not supported", n->dim); return -1; }
        shape os = in->s;
        os.C = 0;
        for (int k = 0; k < n->nin; k++) {
            const value *v = &P->val[n->in[k]];
            if (v->s.rank != in->s.rank) { thb_set_error("Concatenation of tensors of different dimensionality"); return -1; }
            if (v->s.H != in->s.H || v->s.W != in->s.W || v->s.N != in->s.N || v->s.flat) {
                thb_set_error("Concatenation of tensors of different sizes");
                return -1;
            }
            if (k < n->nin - 1 && v->s.C % al) {
                thb_set_error("concatenation of %d channels is not aligned to %d", v->s.C, al);
                return -1;
            }
            os.C += v->s.C;
        }
        materialise(P, out, os);
        int coff = 0;
        for (int k = 0; k < n->nin; k++) {
            value *v = &P->val[n->in[k]];
            const int C = v->s.C;
            if (!write_into_slice(P, n->in[k], v, out->buf, out->ld, coff)) {
                s = new_step(P, ST_COPY);
                step_in(s, v); step_out(s, out);
                s->out_coff = coff;
                s->pixels = (long)os.N * os.H * os.W; s->C = C;
            }
            coff += C;
        }
        return 0;
    }
    case OP_SOFTMAX: {
        if (in->s.flat) { thb_set_error("SoftMax on a flattened spatial tensor is not supported"); return -1; }
        materialise(P, out, in->s);
        s = new_step(P, ST_SOFTMAX);
        step_in(s, in); step_out(s, out);
        s->pixels = (long)in->s.N * in->s.H * in->s.W; s->C = in->s.C;
        return 0;
    }
    case OP_VIEW: {
        /* View.c:86-97: batch > 1 gives [batch, numElements], otherwise a 1-D tensor */
        long total = (long)in->s.N * in->s.C * in->s.H * in->s.W, per = n->numElements;
        long batch = in->s.rank == 4 || in->s.rank == 2 ? in->s.N : 1;
        if (per == -1) per = total / batch; else batch = total / per;
        if (batch != in->s.N || per * batch != total) { thb_set_error("View to %d elements does not keep the batch dimension", n->numElements); return -1; }
        *out = *in;
        out->s.rank = batch > 1 ? 2 : 1;
        if (in->s.flat) return 0;
        if (in->s.H * in->s.W > 1) {
            /* consumers that are Linear read the channels-innermost data through a permuted weight; anything
             * else (and the network output) gets the data reordered to the NCHW flatten it expects */
            int all_linear = i != M->output;
            for (int k = i + 1; k < M->nnodes && all_linear; k++)
                for (int q = 0; q < M->nodes[k].nin; q++)
                    if (M->nodes[k].in[q] == i && M->nodes[k].op != OP_LINEAR) all_linear = 0;
            if (all_linear && in->coff == 0 && dtype != THB_U8) {
                out->s.flat = 1; out->s.fC = in->s.C; out->s.fH = in->s.H; out->s.fW = in->s.W;
                out->s.C = (int)per; out->s.H = out->s.W = 1;
                return 0;
            }
            if (i == M->output) {
                /* the postprocess kernel emits NCHW order anyway: keep the spatial form, remember the rank */
                out->s.flat = 2;
                return 0;
            }
            shape os = in->s;
            os.C = (int)per; os.H = os.W = 1; os.rank = out->s.rank;
            materialise(P, out, os);
            out->q_sub = in->q_sub; out->q_mult = in->q_mult; out->q_dyn = in->q_dyn;
            s = new_step(P, ST_TO_NCHW);
            step_in(s, in); step_out(s, out);
            s->N = in->s.N; s->H = in->s.H; s->W = in->s.W; s->C = in->s.C;
            return 0;
        }
        out->s.C = (int)per; out->s.H = out->s.W = 1;
        return 0;
    }
    case OP_RESHAPE: {
        /* Reshape.c:22-36: the elements of each image, in the reference's (channel, row, column) order, become a
         * [C, H, W] map.  Without a batch dimension (3-D result) when batchMode is false, or absent while the tensor has
         * exactly numElements elements and its first dimension is not 1; with the input's batch in front otherwise. */
        if (dtype == THB_U8) { thb_set_error("Reshape is not supported in Lowp"); return -1; }
        const int rC = n->reshape[0], rH = n->reshape[1], rW = n->reshape[2];
        const long total = (long)in->s.N * in->s.C * in->s.H * in->s.W, per = (long)rC * rH * rW;
        const int size0 = in->s.rank == 4 || in->s.rank == 2 ? in->s.N : in->s.C;
        const int nonbatch = n->batch_mode == 0 || (n->batch_mode == -1 && total == n->numElements && size0 != 1);
        if (rC < 1 || rH < 1 || rW < 1 || per != n->numElements || per * in->s.N != total || (nonbatch && in->s.N != 1)) {
            thb_set_error("Reshape to %dx%dx%d does not fit %ld elements in %d image(s)", rC, rH, rW, total, in->s.N);
            return -1;
        }
        if (in->s.flat || in->s.H * in->s.W != 1) { thb_set_error("Reshape of a spatial tensor to three dimensions is not supported"); return -1; }
        shape os = in->s;
        os.C = rC; os.H = rH; os.W = rW; os.rank = nonbatch ? 3 : 4;
        materialise(P, out, os);
        s = new_step(P, ST_FROM_NCHW);
        step_in(s, in); step_out(s, out);
        s->N = in->s.N; s->H = rH; s->W = rW; s->C = rC;
        return 0;
    }
    case OP_UPSAMPLE: {
        /* Upsample.c:18-63 */
        if (in->s.rank < 3 || in->s.flat) { thb_set_error("Only 3D and 4D input is supported"); return -1; }
        shape os = in->s;
        os.H *= 2; os.W *= 2;
        materialise(P, out, os);
        s = new_step(P, ST_UPSAMPLE);
        step_in(s, in); step_out(s, out);
        s->N = in->s.N; s->H = in->s.H; s->W = in->s.W; s->C = in->s.C;
        return 0;
    }
    case OP_ZEROPAD: {
        /* SpatialZeroPadding.c:17-60 (negative pads crop) */
        if (in->s.rank < 3 || in->s.flat) { thb_set_error("input dimension must be 3 or 4"); return -1; }
        shape os = in->s;
        os.H = in->s.H + n->pad_t + n->pad_b; os.W = in->s.W + n->pad_l + n->pad_r;
        if (os.H < 1 || os.W < 1) { thb_set_error("zero padding leaves an empty tensor"); return -1; }
        materialise(P, out, os);
        s = new_step(P, ST_ZEROPAD);
        step_in(s, in); step_out(s, out);
        s->N = in->s.N; s->H = in->s.H; s->W = in->s.W; s->C = in->s.C;
        s->padW = n->pad_l; s->kW = n->pad_r; s->padH = n->pad_t; s->kH = n->pad_b;
        return 0;
    }
    case OP_SLICE: {
        /* Slice.c:34-39 + THFloatTensor_slice (thbasic.c:192-209): [from, to) along dimension `axis` of the tensor as the
         * reference ranks it ([N,C,H,W], [C,H,W], [N,C] or [C]) */
        if (in->s.flat) { thb_set_error("Slice of a flattened spatial tensor is not supported"); return -1; }
        const int rank = in->s.rank, ax = n->slice_axis;
        int which = -1; /* 0 batch, 1 channels, 2 rows, 3 columns */
        if (rank == 4) which = ax;
        else if (rank == 3) which = ax + 1;
        else if (rank == 2) which = ax;
        else if (rank == 1) which = ax == 0 ? 1 : -1;
        const int size = which == 0 ? in->s.N : which == 1 ? in->s.C : which == 2 ? in->s.H : which == 3 ? in->s.W : -1;
        if (which < 0 || which > 3 || (rank <= 2 && which > 1) || n->slice_from < 0 || n->slice_to <= n->slice_from || n->slice_to > size) {
            thb_set_error("Slice [%d, %d) along dimension %d does not fit the tensor", n->slice_from, n->slice_to, ax);
            return -1;
        }
        shape os = in->s;
        const int len = n->slice_to - n->slice_from;
        if (which == 1) {
            os.C = len;
            materialise(P, out, os);
            s = new_step(P, ST_SLICEC);
            step_in(s, in); step_out(s, out);
            s->pixels = (long)os.N * os.H * os.W; s->C = len; s->flag = n->slice_from;
        } else if (which == 0) {
            if (P->I->slice_n != E->cur->N) { thb_set_error("a slice along the batch dimension needs the whole batch on one GPU"); return -1; }
            os.N = len;
            materialise(P, out, os);
            s = new_step(P, ST_COPY);
            step_in(s, in); step_out(s, out);
            s->pixels = (long)len * os.H * os.W; s->C = os.C;
            s->in_off0 = (long)n->slice_from * os.H * os.W * in->ld;
        } else {
            if (which == 2) os.H = len; else os.W = len;
            materialise(P, out, os);
            s = new_step(P, ST_ZEROPAD);
            step_in(s, in); step_out(s, out);
            s->N = in->s.N; s->H = in->s.H; s->W = in->s.W; s->C = in->s.C;
            s->padW = which == 3 ? -n->slice_from : 0; s->kW = which == 3 ? n->slice_to - in->s.W : 0;
            s->padH = which == 2 ? -n->slice_from : 0; s->kH = which == 2 ? n->slice_to - in->s.H : 0;
        }
        return 0;
    }
    case OP_CMAX: {
        /* Cmax.c:20-68 (inputs of one shape; the reference also takes shorter later inputs, which nothing here produces) */
        if (n->nin > 8) { thb_set_error("Cmax of %d tensors is not supported", n->nin); return -1; }
        for (int k = 0; k < n->nin; k++) {
            const value *v = &P->val[n->in[k]];
            if (v->s.rank != in->s.rank) { thb_set_error("Cmax of tensors of different dimensionality"); return -1; }
            if (v->s.C != in->s.C || v->s.H != in->s.H || v->s.W != in->s.W || v->s.N != in->s.N || v->s.flat) {
                thb_set_error("Cmax of tensors of different sizes");
                return -1;
            }
        }
        materialise(P, out, in->s);
        s = new_step(P, ST_CMAX);
        for (int k = 0; k < n->nin; k++) step_in(s, &P->val[n->in[k]]);
        step_out(s, out);
        s->pixels = (long)in->s.N * in->s.H * in->s.W; s->C = in->s.C;
        return 0;
    }
    case OP_LOGSOFTMAX: {
        if (in->s.flat) { thb_set_error("LogSoftMax on a flattened spatial tensor is not supported"); return -1; }
        if (P->I->slice_n != E->cur->N && !E->strict_math) { thb_set_error("LogSoftMax as the reference computes it needs the whole batch on one GPU"); return -1; }
        materialise(P, out, in->s);
        s = new_step(P, ST_LOGSOFTMAX);
        step_in(s, in); step_out(s, out);
        s->pixels = (long)in->s.N * in->s.H * in->s.W; s->C = in->s.C;
        /* LogSoftMax.c:77 subtracts from the values at the start of the whole input; THB200_STRICT_MATH=1: from each position's own */
        s->flag = !E->strict_math;
        return 0;
    }
    case OP_NORMALIZE: {
        /* Normalize.c:12-44: per row of a 2-D tensor, over the whole tensor (batch included) otherwise */
        if (in->s.flat || in->coff || in->ld != ru(in->s.C, al)) { thb_set_error("Normalize needs a dense tensor"); return -1; }
        const int per_row = in->s.rank == 2;
        if (!per_row && P->I->slice_n != E->cur->N) { thb_set_error("Normalize over a whole batch tensor needs the batch on one GPU"); return -1; }
        materialise(P, out, in->s);
        s = new_step(P, ST_NORMALIZE);
        step_in(s, in); step_out(s, out);
        s->N = in->s.N; s->pixels = (long)in->s.H * in->s.W * in->ld; s->flag = per_row;
        s->aux_buf = new_buf(P, sizeof(float) * (size_t)(in->s.N > 0 ? in->s.N : 1));
        return 0;
    }
    case OP_UNPOOL: {
        /* SpatialMaxUnpooling.c:42-121: input 0 has the size of the pooling's output, the result that of its input */
        const value *xin = &P->val[n->in[1]];
        if (in->s.rank != 3 && in->s.rank != 4) { thb_set_error("3D or 4D (batch mode) tensor is expected"); return -1; }
        if (in->s.flat || xin->s.flat || xin->buf < 0) { thb_set_error("SpatialMaxUnpooling needs spatial tensors"); return -1; }
        const int oH = pool_out(xin->s.H, n->kH, n->dH, n->padH, n->ceil_mode, n->padH || n->padW);
        const int oW = pool_out(xin->s.W, n->kW, n->dW, n->padW, n->ceil_mode, n->padH || n->padW);
        if (in->s.H != oH || in->s.W != oW || in->s.C != xin->s.C || in->s.N != xin->s.N) {
            thb_set_error("Invalid input size w.r.t current indices size");
            return -1;
        }
        shape os = xin->s;
        os.rank = in->s.rank;
        materialise(P, out, os);
        s = new_step(P, ST_UNPOOL);
        step_in(s, in); step_in(s, xin); step_out(s, out);
        s->N = os.N; s->H = os.H; s->W = os.W; s->C = os.C; s->oH = oH; s->oW = oW;
        s->kH = n->kH; s->kW = n->kW; s->dH = n->dH; s->dW = n->dW; s->padH = n->padH; s->padW = n->padW;
        return 0;
    }
    case OP_ALIAS:
        *out = *in;
        return 0;
    }
    thb_set_error("internal: unknown operator %d", n->op);
    return -1;
}

/* Can launch `s` run on some of its images?  (The planned convolutions and poolings whose images are independent; what
 * they add is the image offset of every operand, exec_step.) */
static int sliceable(const instance *I, const step *s)
{
    switch (s->kind) {
    case ST_CONV: return s->conv.N == I->slice_n && s->scratch_buf < 0 && !s->in_off0 && !s->out_off0;
    case ST_MAXPOOL: return s->N == I->slice_n;
    case ST_CSUM: return s->pixels % I->slice_n == 0;
    default: return 0;
    }
}

/* Microseconds that a launch on the whole slice takes beyond LAUNCH_US, roughly: its share of the arithmetic (at 0.62 PFLOP/s in
 * the 16-bit modes, 0.75 in uint8, 100 TFLOP/s in fp32 on the tensor cores and 36 on the FP32 units, what the layers of a large batch reach on average) or of the bytes
 * (4.5 TB/s), whichever is more.  LAUNCH_US is every launch's fill, drain and partly filled wave (ResNet-18 and -50 on 1 to 256
 * images: within a fifth of 7 us a launch plus this). */
#define LAUNCH_US 7.0
#define PART_LAUNCH_US 8.5 /* ... of a launch on a part of the batch: issued directly, not from the graph */
static double model_us(const step *s)
{
    double elems = (double)s->out_pixels * s->out_C * 2, us = 0;
    if (s->kind == ST_CONV) {
        const thb_conv_desc *d = &s->conv;
        const double rate = s->dtype == THB_F32 ? (s->w_split ? 100e6 : 36e6) : s->dtype == THB_U8 ? 0.75e9 : 0.62e9; /* per microsecond */
        us = 2.0 * d->N * d->oH * d->oW * (double)d->Cout * d->Cin * d->kH * d->kW / rate;
        elems = (double)d->N * d->H * d->W * d->Cin + elems * (s->nin > 1 ? 1 : 0.5);
    }
    const double b = elems * esize_of(s->dtype) / 4.5e6;
    return us > b ? us : b;
}

/* The network's last launch as one that writes NCHW floats itself (thb_conv_nchw_fwd)?  For maps: a segmentation network's
 * classifier, whose scores are the largest tensor of the forward, written once instead of three times.  Not where the layer
 * shares its reduction among CTAs or is a Linear (one position per image: nothing to transpose). */
static int plan_head(const instance *I)
{
    const step *s = I->nsteps ? &I->steps[I->nsteps - 1] : 0;
    const char *off = getenv("THB200_NO_HEAD");
    if (!s || (off && atoi(off)) || s->kind != ST_CONV || s->dual || s->pool_k || s->scratch_buf >= 0 || s->conv.splits > 1 ||
        s->in_off0 || s->out_off0 || s->out_coff || s->out_buf != I->out_val.buf || I->out_val.coff || s->conv.Cout != I->out_val.s.C ||
        s->conv.oH * s->conv.oW < 32)
        return 0;
    return thb_conv_nchw_supported(&s->conv);
}

/* microseconds of a slice's input on its way to the device (measured: 55 GB/s from pinned memory) */
static double copy_in_us(const thb_engine *E, const instance *I)
{
    const shape_plan *p = E->cur;
    return (double)I->slice_n * p->H * p->W * (p->cp ? p->cp : 4.0 * p->C) / 50e3;
}

/* A batch of 256 pictures takes 0.7 ms to arrive, a fifth of a ResNet-50 forward.  The first launches of a network are the
 * ones with the most pixels, which lose nothing on a part of the batch: they follow the copy part by part, and the rest of the
 * network runs on the whole batch.  (Cutting the whole network into sub-batches instead repeats the fill and drain of all its
 * small layers: ResNet-50 on 96 + 160 pictures, 4.35 ms of kernels instead of 3.65.)  The number of parts and of launches are
 * those with the earliest end in a model: a part starts when it has arrived and the one before it has been through the launches,
 * each of which takes PART_LAUNCH_US and its share of model_us on it. */
static void choose_slices(thb_engine *E, instance *I)
{
    I->prefix = I->slices = 0;
    /* (a uint8 float batch: its range is known when the last of it has been staged, scanned or copied, and nothing starts before) */
    if ((E->dtype == THB_U8 && !E->cur->cp) || E->cur->cp == 2 || E->whole_batch || I->in_val.buf < 0) return;
    const char *off = getenv("THB200_NO_SLICES");
    if (off && atoi(off)) return;
    const double t_in = copy_in_us(E, I);
    double all = 0;
    for (int t = 0; t < I->nsteps; t++) all += LAUNCH_US + model_us(&I->steps[t]);
    const double whole = t_in + all;
    double best = whole - 20;
    for (int m = 2; m <= 8 && m <= I->slice_n / 2; m++) {
        double sliced = 0;
        for (int p = 1; p <= I->nsteps - I->head && sliceable(I, &I->steps[p - 1]); p++) {
            sliced += model_us(&I->steps[p - 1]);
            double end = 0;
            for (int c = 0; c < m; c++) {
                const double came = t_in * (2 * c + 1) / (2 * m - 1);
                end = (came > end ? came : end) + p * PART_LAUNCH_US + sliced * (c ? 2 : 1) / (2 * m - 1);
            }
            end += all - p * LAUNCH_US - sliced;
            if (end >= best) continue;
            best = end;
            I->prefix = p;
            I->slices = m;
            I->hidden_us = whole - end;
        }
    }
}

/* part c of a sliced start: the first one is half as large as the others, so that the kernels start early */
static void slice_part(const instance *I, int c, int *i0, int *cnt)
{
    const int w = 2 * I->slices - 1, n = I->slice_n;
    *i0 = c ? (int)((long)n * (2 * c - 1) / w) : 0;
    *cnt = (int)((long)n * (2 * c + 1) / w) - *i0;
}

/* liveness-based packing of the activation buffers into one arena */
static size_t pack_arena(instance *I)
{
    for (int t = 0; t < I->nsteps; t++) {
        step *s = &I->steps[t];
        int ids[12], n = 0;
        for (int k = 0; k < s->nin; k++) ids[n++] = s->in_buf[k];
        ids[n++] = s->out_buf;
        ids[n++] = s->aux_buf;
        ids[n++] = s->aux2_buf;
        ids[n++] = s->scratch_buf;
        for (int k = 0; k < n; k++)
            if (ids[k] >= 0) {
                abuf *b = &I->bufs[ids[k]];
                if (b->first < 0) b->first = t;
                b->last = t;
            }
    }
    /* a sliced start runs its launches part by part: whatever they touch is alive until the last part has run them all */
    for (int b = 0; b < I->nbufs; b++)
        if (I->prefix && I->bufs[b].last >= 0 && I->bufs[b].first < I->prefix) {
            I->bufs[b].first = 0;
            if (I->bufs[b].last < I->prefix - 1) I->bufs[b].last = I->prefix - 1;
        }
    /* the network input lives from the preprocess launch (before step 0); the output until the postprocess */
    if (I->in_val.buf >= 0) I->bufs[I->in_val.buf].first = -1;
    if (I->out_val.buf >= 0) I->bufs[I->out_val.buf].last = I->nsteps;
    size_t top = 0;
    for (int b = 0; b < I->nbufs; b++)
        if (I->bufs[b].zeroed) {
            I->bufs[b].offset = top;
            top += I->bufs[b].bytes;
        }
    I->zero_bytes = top;
    for (int b = 0; b < I->nbufs; b++) {
        abuf *B = &I->bufs[b];
        if (B->zeroed) continue;
        if (B->last < 0 && b != I->in_val.buf) { B->offset = 0; continue; }
        size_t off = I->zero_bytes;
        for (;;) {
            int moved = 0;
            for (int o = 0; o < b; o++) {
                abuf *O = &I->bufs[o];
                if (O->zeroed || (O->last < 0 && o != I->in_val.buf)) continue;
                int overlap_time = !(O->last < B->first || B->last < O->first);
                if (overlap_time && off < O->offset + O->bytes && O->offset < off + B->bytes) {
                    off = O->offset + O->bytes;
                    moved = 1;
                }
            }
            if (!moved) break;
        }
        B->offset = off;
        if (off + B->bytes > top) top = off + B->bytes;
    }
    return top;
}

static void instance_free(instance *I)
{
    if (!I->stream) return; /* (the first thing an instance has) */
    for (int i = 0; i < I->nhost; i++) free(I->hostmem[i]);
    free(I->hostmem);
    cudaSetDevice(I->device);
    if (I->stream) cudaStreamSynchronize(I->stream);
    for (int i = 0; i < I->nallocs; i++) cudaFree(I->allocs[i]);
    for (int i = 0; i < I->nsteps; i++) free(I->steps[i].tmap);
    if (I->graph) cudaGraphExecDestroy(I->graph);
    if (I->ev0) cudaEventDestroy(I->ev0);
    if (I->ev1) cudaEventDestroy(I->ev1);
    if (I->ev_wb) cudaEventDestroy(I->ev_wb);
    if (I->wb_stream) cudaStreamDestroy(I->wb_stream);
    if (I->copy_stream) { cudaStreamSynchronize(I->copy_stream); cudaStreamDestroy(I->copy_stream); }
    for (int c = 0; c < 8; c++)
        if (I->ev_slice[c]) cudaEventDestroy(I->ev_slice[c]);
    if (I->stream) cudaStreamDestroy(I->stream);
    thb_host_free_pinned(I->h_status);
    free(I->allocs); free(I->steps); free(I->bufs);
    memset(I, 0, sizeof(*I));
}

/* `sub`: -1 when the instance computes all of its GPU's images, else which of the pipelined sub-batches of them.  An earlier
 * sub-batch's kernels come first where two compete for the SMs: its result can leave while the later ones are computed. */
static int instance_build(thb_engine *E, instance *I, int device, int slice_off, int slice_n, int sub)
{
    thb_model *M = E->model;
    memset(I, 0, sizeof(*I));
    I->device = device; I->slice_off = slice_off; I->slice_n = slice_n;
    CU(cudaSetDevice(device));
    int prio_lo = 0, prio_hi = 0;
    CU(cudaDeviceGetStreamPriorityRange(&prio_lo, &prio_hi));
    const int prio = sub < 0 ? prio_lo : prio_hi + sub < prio_lo ? prio_hi + sub : prio_lo;
    CU(cudaStreamCreateWithPriority(&I->stream, cudaStreamNonBlocking, prio));
    CU(cudaEventCreate(&I->ev0));
    CU(cudaEventCreate(&I->ev1));
    I->d_status = dalloc(E, I, sizeof(int));
    I->d_minmax = dalloc(E, I, 2 * sizeof(float));
    if (!I->d_status || !I->d_minmax) return -1;
    CU(cudaMemset(I->d_status, 0, sizeof(int)));
    I->h_status = thb_host_alloc_pinned(sizeof(int));
    if (!I->h_status) { thb_set_error("pinned allocation failed"); return -1; }
    *I->h_status = 0;

    planner P;
    memset(&P, 0, sizeof(P));
    P.E = E; P.I = I; P.M = M;
    P.val = calloc(M->nnodes, sizeof(value));
    P.uses = calloc(M->nnodes, sizeof(int));
    P.absorbed = calloc(M->nnodes, sizeof(int));
    P.leader = calloc(M->nnodes, sizeof(int));
    for (int i = 0; i < M->nnodes; i++) {
        P.val[i].buf = -1;
        P.leader[i] = i;
        for (int k = 0; k < M->nodes[i].nin; k++) P.uses[M->nodes[i].in[k]]++;
    }
    P.uses[M->output]++;

    shape in = {slice_n, E->cur->C, E->cur->H, E->cur->W, E->cur->rank, 0, 0, 0, 0};
    {
        /* a convolution of stride 2 or 4 on very few channels as the only consumer of the input: stage the input space-to-depth,
         * so that the copy engine can load it (16 channels a pixel in padded rows, or 64) instead of a gather of 16-byte chunks
         * that are mostly padding */
        thb_node *c1 = M->nnodes > 1 ? &M->nodes[1] : 0;
        const char *off = getenv("THB200_NO_S2D"), *u8off = getenv("THB200_NO_S2D_U8");
        const int f = c1 && c1->op == OP_CONV && c1->dH == c1->dW ? c1->dH : 0;
        I->input_s2d = (f == 2 || (f == 4 && E->dtype != THB_U8)) && c1->in[0] == 0 && P.uses[0] == 1 && 4 * E->cur->C <= 16 &&
                       c1->Cin == E->cur->C && (E->cur->cp == 0 || E->cur->cp == 3) &&
                       (E->dtype == THB_F16 || E->dtype == THB_BF16 || (E->dtype == THB_U8 && !(u8off && atoi(u8off)))) &&
                       c1->padH <= c1->kH - 1 && c1->padW <= c1->kW - 1 &&
                       !(E->honour_pads && (c1->pad2H != c1->padH || c1->pad2W != c1->padW || c1->dlH > 1 || c1->dlW > 1 || c1->autopad || c1->refl_pad)) &&
                       !(off && atoi(off)) ? f : 0;
        if (I->input_s2d) { in.C = f * f * E->cur->C; in.H = (E->cur->H + f - 1) / f; in.W = (E->cur->W + f - 1) / f; }
    }
    {
        /* A stride-1 convolution with at most 64 output channels on very few input channels (VGG, the segmentation net):
         * with 32-byte pixels it is a case for the patch kernel (one copy per input patch) instead of a gather of
         * 16-byte chunks that are mostly padding. */
        thb_node *c1 = M->nnodes > 1 ? &M->nodes[1] : 0;
        const char *off = getenv("THB200_NO_PAD16");
        I->input_pad16 = !I->input_s2d && c1 && c1->op == OP_CONV && c1->in[0] == 0 && P.uses[0] == 1 && c1->dH == 1 && c1->dW == 1 &&
                         E->cur->C <= 8 && c1->Cin == E->cur->C && c1->Cout <= 64 && c1->kH <= 8 && c1->kW <= 8 && c1->kH * c1->kW > 1 &&
                         c1->padH < c1->kH && c1->padW < c1->kW && (E->dtype == THB_F16 || E->dtype == THB_BF16) &&
                         !(E->honour_pads && (c1->pad2H != c1->padH || c1->pad2W != c1->padW || c1->dlH > 1 || c1->dlW > 1 || c1->autopad || c1->refl_pad)) &&
                         !(off && atoi(off));
    }
    {
        /* uint8: a 3x3 / stride 1 / pad 1 first convolution on three planes of a float batch */
        thb_node *c1 = M->nnodes > 1 ? &M->nodes[1] : 0;
        const char *off = getenv("THB200_NO_NEIGH_U8");
        I->input_neigh = E->dtype == THB_U8 && !I->input_s2d && E->cur->cp == 0 && E->cur->C == 3 && E->cur->rank == 4 && c1 && c1->op == OP_CONV &&
                         c1->in[0] == 0 && P.uses[0] == 1 && c1->Cin == 3 && c1->kH == 3 && c1->kW == 3 && c1->dH == 1 && c1->dW == 1 &&
                         c1->padH == 1 && c1->padW == 1 &&
                         !(E->honour_pads && (c1->pad2H != c1->padH || c1->pad2W != c1->padW || c1->dlH > 1 || c1->dlW > 1 || c1->autopad || c1->refl_pad)) &&
                         !(off && atoi(off));
        if (I->input_neigh) in.C = 27;
    }
    materialise(&P, &P.val[0], in);
    if (I->input_pad16) {
        value *v = &P.val[0];
        v->ld = 16;
        I->nbufs--; /* re-create the buffer with 16 channels per pixel */
        v->buf = new_buf(&P, (size_t)in.N * in.H * in.W * v->ld * esize_of(E->dtype));
    }
    if (I->input_s2d == 4) {
        value *v = &P.val[0];
        v->ld = 64; /* one 128-byte slab a pixel */
        I->nbufs--;
        v->buf = new_buf(&P, (size_t)in.N * in.H * in.W * v->ld * esize_of(E->dtype));
    }
    if (I->input_s2d == 2) {
        /* When the rewritten convolution's kernel row fills one 128-byte K block (uint8: half of one), store the staged rows with
         * their zero padding: one copy then fetches a whole kernel row of an output pixel (thb_conv_desc.in_row_pitch). */
        thb_node *c1 = &M->nodes[1];
        const int padW = (c1->padW + 1) / 2, kW = (c1->kW - 1 - c1->padW) / 2 + padW + 1;
        const char *off = getenv("THB200_NO_PADDED_ROWS");
        value *v = &P.val[0];
        if (kW * v->ld * esize_of(E->dtype) == (E->dtype == THB_U8 ? 64 : 128) && thb_conv_padded_rows_supported(E->dtype) &&
            !(off && atoi(off))) {
            v->pad_left = padW;
            v->row_pitch = (padW + in.W + kW - 1 + 3) & ~3;
            I->nbufs--; /* re-create the buffer at its padded size */
            v->buf = new_buf(&P, (size_t)in.N * in.H * v->row_pitch * v->ld * esize_of(E->dtype));
        }
    }
    P.val[0].q_dyn = E->dtype == THB_U8;
    int rc = 0;
    for (int i = 1; i < M->nnodes && !rc; i++) {
        if (P.absorbed[i]) continue;
        rc = plan_node(&P, i);
    }
    if (!rc && P.val[M->output].buf < 0) { thb_set_error("internal: the output was not materialised"); rc = -1; }
    if (!rc) {
        I->in_val = P.val[0];
        I->out_val = P.val[M->output];
        I->out_shape = I->out_val.s;
        I->out_count = (long)I->out_shape.N * I->out_shape.C * I->out_shape.H * I->out_shape.W;
        I->head = plan_head(I);
        if (sub < 0) choose_slices(E, I);
        I->arena_bytes = pack_arena(I);
        I->arena = dalloc(E, I, I->arena_bytes);
        size_t in_bytes = (size_t)slice_n * E->cur->C * E->cur->H * E->cur->W * sizeof(float);
        I->d_in = dalloc(E, I, in_bytes);
        I->d_img = dalloc(E, I, (size_t)slice_n * E->cur->H * E->cur->W * 4);
        I->d_out = dalloc(E, I, (size_t)(I->out_count ? I->out_count : 1) * sizeof(float));
        if (!I->arena || !I->d_in || !I->d_out || !I->d_img) rc = -1;
        if (!rc && I->prefix) {
            int bad = cudaStreamCreateWithFlags(&I->copy_stream, cudaStreamNonBlocking) != cudaSuccess;
            for (int c = 0; c < I->slices; c++) bad |= cudaEventCreateWithFlags(&I->ev_slice[c], cudaEventDisableTiming) != cudaSuccess;
            if (bad) { thb_set_error("stream creation failed"); rc = -1; }
        }
        /* padded channels are never read as data, but stale NaN/Inf bit patterns would poison the
         * zero-weight products: start from a clean arena */
        if (!rc && cudaMemset(I->arena, 0, I->arena_bytes) != cudaSuccess) { thb_set_error("arena memset failed"); rc = -1; }
        /* that, and the layers' split weights, are launches on the legacy stream, for which the instance's does not wait */
        if (!rc && cudaStreamSynchronize(0) != cudaSuccess) { thb_set_error("laying the weights out failed"); rc = -1; }
    }
    free(P.val); free(P.uses); free(P.absorbed); free(P.leader);
    if (th_debug && !rc)
        fprintf(stderr, "thb200: device %d: %d launches per forward, arena %.1f MiB, %d buffers\n", device, I->nsteps,
                I->arena_bytes / 1048576.0, I->nbufs);
    return rc;
}

static void *bufptr(instance *I, int buf, int coff, int dtype)
{
    return buf < 0 ? 0 : I->arena + I->bufs[buf].offset + (size_t)coff * esize_of(dtype);
}

/* One planned launch on the instance's stream; on images [img0, img0 + cnt) only when cnt > 0 (sliceable launches). */
static int exec_step(instance *I, int t, int img0, int cnt)
{
    thb_stream st = I->stream;
    step part, *s = &I->steps[t];
    const int dt = s->dtype;
    const size_t es = esize_of(dt);
    char *x0 = bufptr(I, s->in_buf[0], s->in_coff[0], dt);
    if (x0 && s->in_off0) x0 += s->in_off0 * es;
    char *y = bufptr(I, s->out_buf, s->out_coff, dt);
    if (y && s->out_off0) y += s->out_off0 * es;
    int rc = 0;
    size_t res_off = 0, aux_off = 0, aux2_off = 0; /* bytes */
    if (cnt > 0) {
        part = *s;
        s = &part;
        thb_conv_desc *d = &s->conv;
        switch (s->kind) {
        case ST_CONV: {
            const size_t opix = (size_t)d->oH * d->oW;
            d->N = cnt;
            x0 += (size_t)img0 * d->H * (d->in_row_pitch ? d->in_row_pitch : d->W) * d->in_ld * es;
            y += (size_t)img0 * (s->pool_k ? (size_t)s->pool_oH * s->pool_oW : opix) * s->out_ld * es;
            res_off = s->dual ? (size_t)img0 * d->x2_H * d->x2_W * d->x2_ld * es : img0 * opix * d->res_ld * es;
            aux_off = sizeof(int) * (size_t)img0 * d->H * d->W;
            aux2_off = sizeof(int) * img0 * opix;
            break;
        }
        case ST_MAXPOOL:
            s->N = cnt;
            x0 += (size_t)img0 * s->H * s->W * s->in_ld[0] * es;
            y += (size_t)img0 * s->oH * s->oW * s->out_ld * es;
            aux2_off = sizeof(int) * (size_t)img0 * s->oH * s->oW;
            break;
        case ST_CSUM: {
            const long per = s->pixels / I->slice_n;
            x0 += (size_t)img0 * (s->oW ? per / s->W * s->oW : per) * s->in_ld[0] * es;
            aux_off = sizeof(int) * (size_t)img0 * per;
            s->pixels = cnt * per;
            break;
        }
        }
    }
    switch (s->kind) {
    case ST_CONV: {
        thb_conv_desc *d = &s->conv;
        if (s->dual) d->x2 = (char *)bufptr(I, s->in_buf[1], s->in_coff[1], dt) + res_off;
        else if (s->nin > 1) d->res = (char *)bufptr(I, s->in_buf[1], s->in_coff[1], dt) + res_off;
        if (s->aux_buf >= 0) d->csum = (const int *)((char *)bufptr(I, s->aux_buf, 0, THB_U8) + aux_off);
        if (s->aux2_buf >= 0) d->csum_out = (int *)((char *)bufptr(I, s->aux2_buf, 0, THB_U8) + aux2_off);
        if (s->scratch_buf >= 0) d->splitk_scratch = (float *)bufptr(I, s->scratch_buf, 0, THB_U8);
        rc = s->pool_k ? thb_conv_maxpool_fwd(d, s->pool_k, 2, s->pool_pad, s->pool_oH, s->pool_oW, x0, y, s->out_ld, st)
             : s->w_split ? thb_conv_f32_fwd(d, s->w_split, x0, y, st)
                          : thb_conv_fwd(d, x0, y, st);
        break;
    }
    case ST_GEMV:
        rc = thb_gemv_fwd(dt, x0, s->N, s->K, s->in_ld[0], s->w, s->M, s->scale, s->shift, &s->act, y, s->out_ld, st);
        break;
    case ST_MAXPOOL:
        rc = s->aux2_buf >= 0 ? thb_maxpool_sums(dt, x0, s->N, s->H, s->W, s->C, s->in_ld[0], s->kH, s->kW, s->dH, s->dW, s->padH, s->padW, s->oH, s->oW,
                                                 y, s->out_ld, (int *)((char *)bufptr(I, s->aux2_buf, 0, THB_U8) + aux2_off), st)
                              : thb_maxpool(dt, x0, s->N, s->H, s->W, s->C, s->in_ld[0], s->kH, s->kW, s->dH, s->dW, s->padH, s->padW, s->oH, s->oW,
                                            y, s->out_ld, st);
        break;
    case ST_AVGPOOL:
        rc = thb_avgpool(dt, x0, s->N, s->H, s->W, s->C, s->in_ld[0], s->kH, s->kW, s->dH, s->dW, s->padH, s->padW, s->oH,
                         s->oW, s->flag, y, s->out_ld, st);
        break;
    case ST_AFFINE:
        rc = thb_affine_act(dt, x0, s->pixels, s->C, s->in_ld[0], s->scale, s->shift, &s->act, y, s->out_ld, st);
        break;
    case ST_U8COMBINE:
        rc = thb_u8_combine(x0, s->in_ld[0], bufptr(I, s->in_buf[1], s->in_coff[1], THB_U8), s->in_ld[1], (int)s->coef[0],
                            (int)s->coef[1], s->thr, s->val, s->pixels, s->C, y, s->out_ld, st);
        break;
    case ST_U8THR:
        rc = thb_u8_threshold(x0, s->pixels, s->C, s->in_ld[0], s->thr, s->val, y, s->out_ld, st);
        break;
    case ST_COMBINE: {
        const void *xs[8];
        for (int k = 0; k < s->nin; k++) xs[k] = bufptr(I, s->in_buf[k], s->in_coff[k], dt);
        rc = thb_combine(dt, s->nin, xs, s->in_ld, s->coef, s->pixels, s->C, y, s->out_ld, st);
        break;
    }
    case ST_COPY:
        rc = thb_copy_channels(dt, x0, s->pixels, s->C, s->in_ld[0], y, s->out_ld, st);
        break;
    case ST_SOFTMAX:
        rc = thb_softmax(dt, x0, s->pixels, s->C, s->in_ld[0], y, s->out_ld, st);
        break;
    case ST_COL2IM:
        rc = thb_col2im(dt, x0, s->N, s->H, s->W, s->C, s->kH, s->kW, s->dH, s->dW, s->padH, s->padW, s->oH, s->oW,
                        s->in_ld[0], s->beta, s->bias, &s->act, y, s->out_ld, st);
        break;
    case ST_CSUM:
        rc = thb_u8_channel_sum_rows(x0, s->pixels, s->C, s->in_ld[0], s->W > 0 ? s->W : 1, s->oW, s->padW, (int *)((char *)bufptr(I, s->out_buf, 0, THB_U8) + aux_off), st);
        break;
    case ST_TO_NCHW:
        rc = thb_to_nchw(dt, x0, s->N, s->H, s->W, s->C, s->in_ld[0], y, st);
        break;
    case ST_FROM_NCHW:
        rc = thb_from_nchw(dt, x0, s->N, s->H, s->W, s->C, s->in_ld[0], y, s->out_ld, st);
        break;
    case ST_UPSAMPLE:
        rc = thb_upsample2x(dt, x0, s->N, s->H, s->W, s->C, s->in_ld[0], y, s->out_ld, st);
        break;
    case ST_ZEROPAD:
        rc = thb_zero_pad(dt, x0, s->N, s->H, s->W, s->C, s->in_ld[0], s->padW, s->kW, s->padH, s->kH, y, s->out_ld, st);
        break;
    case ST_REFLECTPAD:
        rc = thb_reflect_pad(dt, x0, s->N, s->H, s->W, s->C, s->in_ld[0], s->padW, s->kW, s->padH, s->kH, y, s->out_ld, st);
        break;
    case ST_SLICEC:
        rc = thb_slice_channels(dt, x0, s->pixels, s->flag, s->C, s->in_ld[0], y, s->out_ld, st);
        break;
    case ST_CMAX: {
        const void *xs[8];
        for (int k = 0; k < s->nin; k++) xs[k] = bufptr(I, s->in_buf[k], s->in_coff[k], dt);
        rc = thb_cmax(dt, s->nin, xs, s->in_ld, s->pixels, s->C, y, s->out_ld, st);
        break;
    }
    case ST_LOGSOFTMAX:
        rc = thb_logsoftmax(dt, x0, s->pixels, s->C, s->in_ld[0], y, s->out_ld, s->flag, st);
        break;
    case ST_NORMALIZE:
        rc = thb_l2_normalize(dt, x0, s->N, s->pixels, s->flag, (float *)bufptr(I, s->aux_buf, 0, THB_U8), y, st);
        break;
    case ST_UNPOOL:
        rc = thb_max_unpool(dt, x0, s->in_ld[0], bufptr(I, s->in_buf[1], s->in_coff[1], dt), s->in_ld[1], s->N, s->H, s->W, s->C,
                            s->kH, s->kW, s->dH, s->dW, s->padH, s->padW, s->oH, s->oW, y, s->out_ld, st);
        break;
    }
    if (rc) thb_set_error("kernel launch %d (kind %d) failed: %d %s", t, s->kind, rc, thb_last_cuda_error());
    return rc ? -1 : 0;
}

static int head_on(const instance *I) { return I->head && !th_profile && !th_minmax; }

static int run_steps_ev(thb_engine *E, instance *I, cudaEvent_t *evs, int from, int to)
{
    for (int t = from; t < to; t++) {
        step *s = &I->steps[t];
        const int dt = s->dtype;
        void *y = bufptr(I, s->out_buf, s->out_coff, dt);
        if (y && s->out_off0) y = (char *)y + s->out_off0 * esize_of(dt);
        double t0 = 0;
        if (th_profile) { cudaStreamSynchronize(I->stream); t0 = th_seconds(); }
        if (exec_step(I, t, 0, 0)) return -1;
        if (evs) cudaEventRecord(evs[t + 1], I->stream);
        if (th_minmax && y && s->out_pixels > 0 && s->out_C > 0 && s->kind != ST_CSUM) {
            /* thapi.c:141-154, :197-202: smallest and largest value of every layer's output -- how a caller picks the
             * lowp range.  A diagnostic: the tensor is read back and scanned on the host (uint8 tensors: their bytes). */
            const size_t es = esize_of(dt), bytes = (size_t)s->out_pixels * s->out_ld * es;
            unsigned char *hb = malloc(bytes ? bytes : 1);
            if (hb && cudaStreamSynchronize(I->stream) == cudaSuccess && cudaMemcpy(hb, y, bytes, cudaMemcpyDeviceToHost) == cudaSuccess) {
                float mn = INFINITY, mx = -INFINITY;
                for (long px = 0; px < s->out_pixels; px++)
                    for (int c = 0; c < s->out_C; c++) {
                        const float v = element_as_float(hb, px * s->out_ld + c, dt);
                        if (v > mx) mx = v;
                        if (v < mn) mn = v;
                    }
                printf("Layer %d output: min=%f, max=%f\n", t + 1, mn, mx);
            }
            free(hb);
        }
        if (th_profile) {
            /* thapi.c:211-233: wall clock per module, GFLOP/s for convolutions (serialises the stream) */
            cudaStreamSynchronize(I->stream);
            double dtm = th_seconds() - t0;
            if (s->kind == ST_CONV && s->flops_node >= 0) {
                thb_node *n = &E->model->nodes[s->flops_node];
                double flops = 2.0 * s->conv.N * s->conv.oH * s->conv.oW * (double)n->Cout * n->Cin * n->kH * n->kW;
                printf("%f seconds for launch %d, %f Gflops/s\n", dtm, t + 1, flops * 1e-9 / dtm);
                th_convtot += dtm; th_convflops += flops;
            } else printf("%f seconds for launch %d\n", dtm, t + 1);
        }
    }
    return 0;
}

/* The launches of one forward on the instance's stream: directly the first time, from then on as a replay of the
 * graph captured from them.  In the uint8 engine the convolutions that read the network input take kernel arguments
 * that change every forward (the input's quantisation is measured per batch, lowp_basic.c:299-321): the launches up to
 * and including the last of them are always issued directly and the graph holds the rest.  The same goes for the
 * launches of a sliced start; `from`: the first launch that has not run on the slices already.  THB200_NO_GRAPH=1 and the
 * per-module profile mode launch everything directly. */
static int run_steps(thb_engine *E, instance *I, int from)
{
    if (I->graph_state == 0 && I->runs >= 1) {
        const char *ng = getenv("THB200_NO_GRAPH");
        I->graph_state = -1;
        I->graph_from = 0;
        for (int t = 0; t < I->nsteps; t++)
            if (I->steps[t].kind == ST_CONV && I->steps[t].dyn_quant) I->graph_from = t + 1;
        if (I->graph_from < I->prefix) I->graph_from = I->prefix;
        if (I->graph_from < I->nsteps - I->head && !(ng && atoi(ng)) && !th_profile && !th_minmax) {
            cudaGraph_t g = 0;
            if (cudaStreamBeginCapture(I->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
                const int l0 = thb_kernel_launch_count();
                const int rc = run_steps_ev(E, I, 0, I->graph_from, I->nsteps - I->head);
                I->graph_launches = thb_kernel_launch_count() - l0; /* kernels in the graph (its memset nodes are not launches) */
                thb_count_launches(-I->graph_launches);             /* they have not run yet: the replay below counts them */
                const cudaError_t ce = cudaStreamEndCapture(I->stream, &g);
                if (!rc && ce == cudaSuccess && g && cudaGraphInstantiate(&I->graph, g, 0) == cudaSuccess) I->graph_state = 1;
                if (g) cudaGraphDestroy(g);
                cudaGetLastError();
            }
        }
    }
    I->runs++;
    if (I->graph_state == 1 && !th_profile && !th_minmax) {
        if (from < I->graph_from && run_steps_ev(E, I, 0, from, I->graph_from)) return -1;
        if (cudaGraphLaunch(I->graph, I->stream) == cudaSuccess) {
            thb_count_launches(I->graph_launches);
            return 0;
        }
        thb_set_error("graph launch failed: %s", cudaGetErrorString(cudaGetLastError()));
        return -1;
    }
    return run_steps_ev(E, I, 0, from, I->nsteps - head_on(I));
}

static int clear_sums(instance *I);
static int lowp_input_range(thb_engine *E, instance *set, int G, int has_x, int cp, int C, int H, int W, const float *mean,
                            const float *std, float *q_sub, float *q_mult);
static int boundary_in(thb_engine *E, instance *I, int img0, int n, int has_x, int inplace, int cp, int bgr, int C, int H, int W,
                       const float *mean, const float *std, float q_sub, float q_mult);
static int boundary_out(thb_engine *E, instance *I, float *dst, int head);

/* Per-launch device times of one forward on the first GPU from the batch staged by the last THProcess* call (events
 * around every launch on the launching stream, averaged over `iters` passes).  Entry 0 is the boundary kernel in
 * (NCHW fp32 or HWC bytes -> the engine's layout), entries 1..n the planned launches, entry n+1 the boundary kernel
 * out.  kinds: 0 tensor-core/FFMA convolution, 1 GEMV, 2 any other planned launch, 3 boundary kernel.
 * flops: algorithmic FLOPs of the launch (2 * MACs of the convolution / Linear it computes), 0 otherwise. */
int thb_engine_profile(thb_engine *E, int iters, int max_steps, int *kinds, float *ms, double *flops)
{
    if (!E || !E->cur || iters < 1 || (!E->last_has_x && !E->last_cp)) return -1;
    instance *I = &E->cur->inst[0];
    if (cudaSetDevice(I->device) != cudaSuccess) return -1;
    const int total = I->nsteps + 2;
    const int n = total < max_steps ? total : max_steps;
    cudaEvent_t *evs = calloc(total + 1, sizeof(cudaEvent_t));
    for (int t = 0; t <= total; t++) cudaEventCreate(&evs[t]);
    for (int t = 0; t < n; t++) ms[t] = 0;
    int rc = 0;
    for (int it = 0; it < iters && !rc; it++) {
        float q_sub = 0, q_mult = 0;
        rc = lowp_input_range(E, E->cur->inst, 1, E->last_has_x, E->last_cp, E->cur->C, E->cur->H, E->cur->W, E->last_mean, E->last_std, &q_sub, &q_mult);
        cudaEventRecord(evs[0], I->stream);
        if (!rc) rc = clear_sums(I);
        if (!rc) rc = boundary_in(E, I, 0, I->slice_n, E->last_has_x, 0, E->last_cp, E->last_bgr, E->cur->C, E->cur->H, E->cur->W, E->last_mean, E->last_std, q_sub, q_mult);
        cudaEventRecord(evs[1], I->stream);
        if (!rc) rc = run_steps_ev(E, I, evs + 1, 0, I->nsteps);
        if (!rc) rc = boundary_out(E, I, I->d_out, 0);
        cudaEventRecord(evs[total], I->stream);
        if (cudaStreamSynchronize(I->stream) != cudaSuccess) rc = -1;
        for (int t = 0; t < n && !rc; t++) {
            float m = 0;
            cudaEventElapsedTime(&m, evs[t], evs[t + 1]);
            ms[t] += m / iters;
        }
    }
    for (int t = 0; t < n; t++) {
        kinds[t] = 3;
        flops[t] = 0;
        if (t == 0 || t == total - 1) continue;
        step *s = &I->steps[t - 1];
        kinds[t] = s->kind == ST_CONV ? 0 : s->kind == ST_GEMV ? 1 : 2;
        if (s->flops_node >= 0) {
            thb_node *nd = &E->model->nodes[s->flops_node];
            double pix = s->kind == ST_CONV ? (double)s->conv.N * s->conv.oH * s->conv.oW : (double)s->N;
            if (nd->op == OP_DECONV) pix = (double)s->conv.N * s->conv.H * s->conv.W;
            flops[t] = 2.0 * pix * nd->Cout * nd->Cin * nd->kH * nd->kW + s->flops_extra;
        }
    }
    for (int t = 0; t <= total; t++) cudaEventDestroy(evs[t]);
    free(evs);
    return rc ? -1 : n;
}

/* Algorithmic bytes of each entry of thb_engine_profile: every tensor the launch names counted once (input, output,
 * residual, weights) at the storage type's size; 0 for launches that are neither a convolution nor a GEMV.  The
 * companion of thb_engine_profile's flops for a per-launch "slower of the two roofs" bound. */
int thb_engine_profile_bytes(thb_engine *E, int max_steps, double *bytes)
{
    if (!E || !E->cur) return -1;
    instance *I = &E->cur->inst[0];
    const int total = I->nsteps + 2;
    const int n = total < max_steps ? total : max_steps;
    for (int t = 0; t < n; t++) {
        bytes[t] = 0;
        if (t == 0 || t == total - 1) continue;
        step *s = &I->steps[t - 1];
        const double el = s->dtype == THB_F32 ? 4 : s->dtype == THB_U8 ? 1 : 2;
        if (s->kind == ST_CONV) {
            const thb_conv_desc *d = &s->conv;
            const double out = s->pool_k ? (double)d->N * s->pool_oH * s->pool_oW * d->Cout : (double)d->N * d->oH * d->oW * d->Cout;
            const double in_elems = s->dual ? (double)d->N * d->H * d->W * d->cin1 + (double)d->N * d->x2_H * d->x2_W * (d->Cin - d->cin1)
                                            : (double)d->N * d->H * d->W * d->Cin;
            bytes[t] = el * (in_elems + out * (d->res ? 2 : 1) + (double)d->Cout * d->Cin * d->kH * d->kW);
        } else if (s->kind == ST_GEMV) {
            bytes[t] = el * ((double)s->M * s->K + (double)s->N * (s->K + s->M));
        }
    }
    return n;
}

/* ================================================================================================ */
thb_engine *thb_engine_create(thb_model *model, int mode, float lowp_range, int ngpus)
{
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) {
        thb_set_error("no CUDA device: this library has no CPU engine");
        return 0;
    }
    thb_engine *E = calloc(1, sizeof(*E));
    E->model = model;
    model->refs++;
    E->mode = mode;
    E->dtype = mode == THB_MODE_F16 ? THB_F16 : mode == THB_MODE_BF16 ? THB_BF16 : mode == THB_MODE_U8 ? THB_U8 : THB_F32;
    E->range = lowp_range;
    E->ngpus = ngpus < 1 ? 1 : ngpus > ndev ? ndev : ngpus > 8 ? 8 : ngpus;
    const char *sm = getenv("THB200_STRICT_MATH");
    E->strict_math = sm && atoi(sm);
    const char *hp = getenv("THB200_HONOUR_PADS");
    E->honour_pads = hp && atoi(hp);
    /* Operators that look across the images of a batch (a slice or a join along the batch dimension, the whole-tensor
     * Normalize, the reference's LogSoftMax, which reads frame 0 for every frame) keep the batch on one GPU in one piece. */
    for (int i = 0; i < model->nnodes; i++) {
        const thb_node *nd = &model->nodes[i];
        if ((nd->op == OP_SLICE && nd->slice_axis == 0) || (nd->op == OP_CONCAT && nd->dim == 0) || nd->op == OP_NORMALIZE ||
            (nd->op == OP_LOGSOFTMAX && !E->strict_math))
            E->whole_batch = 1;
    }
    if (E->whole_batch) E->ngpus = 1;
    const char *g = getenv("THB200_GATHER");
    E->peer_gather = !(g && !strcmp(g, "host"));
    return E;
}

static void plan_drop(thb_engine *E, int slot)
{
    shape_plan *p = E->plans[slot];
    if (!p) return;
    for (int g = 0; g < 8; g++) instance_free(&p->inst[g]);
    for (int g = 0; g < 32; g++) instance_free(&p->pipe[g]);
    if (E->cur == p) E->cur = 0;
    free(p);
    E->plans[slot] = 0;
}

void thb_engine_destroy(thb_engine *E)
{
    if (!E) return;
    for (int i = 0; i < MAX_PLANS; i++) plan_drop(E, i);
    for (int i = 0; i < E->nblobs; i++)
        if (cudaSetDevice(E->blobs[i].device) == cudaSuccess) cudaFree(E->blobs[i].ptr);
    free(E->blobs);
    thb_host_free_pinned(E->h_out);
    thb_host_free_pinned(E->h_stage);
    thb_model_release(E->model);
    free(E);
}

/* contiguous batch slices, one per GPU; the remainder images go to the lowest ranks */
void thb_slice_batch(int N, int G, int g, int *offset, int *count)
{
    int base = N / G, extra = N % G;
    *count = base + (g < extra ? 1 : 0);
    *offset = g * base + (g < extra ? g : extra);
}

/* The pipelined sub-batches of one GPU's slice of n images: sub-batch c of S.  Up to four of them grow from the first to
 * the last: a small first one starts the kernels sooner, and the copy of each later one still ends before the kernels
 * ahead of it do (ResNet-50 batch 256 in two: 96 + 160 images).  Boundaries in sixteenths of the slice; slices too small
 * for that, and more than four sub-batches, are cut evenly. */
void thb_slice_sub_batches(int n, int S, int c, int *offset, int *count)
{
    static const int cut[5][5] = {{0}, {0, 16}, {0, 6, 16}, {0, 3, 8, 16}, {0, 2, 6, 11, 16}};
    if (S < 1 || S > 4 || n < 8 * S) {
        thb_slice_batch(n, S < 1 ? 1 : S, c, offset, count);
        return;
    }
    *offset = (n * cut[S][c] + 8) / 16;
    *count = (n * cut[S][c + 1] + 8) / 16 - *offset;
}

static size_t plan_bytes(const shape_plan *p)
{
    size_t b = 0;
    for (int g = 0; g < 8; g++) b += p->inst[g].device_bytes;
    for (int g = 0; g < 32; g++) b += p->pipe[g].device_bytes;
    return b;
}

/* the least recently used plan other than `keep`, -1: none */
static int plan_oldest(thb_engine *E, const shape_plan *keep)
{
    int v = -1;
    for (int i = 0; i < MAX_PLANS; i++)
        if (E->plans[i] && E->plans[i] != keep && (v < 0 || E->plans[i]->used < E->plans[v]->used)) v = i;
    return v;
}

/* After a plan that did not fit on the device: one other shape's plan makes way.  0: that was not the reason, or there is none. */
static int plans_make_way(thb_engine *E)
{
    const int v = E->out_of_memory ? plan_oldest(E, E->cur) : -1;
    if (v < 0) return 0;
    plan_drop(E, v);
    return 1;
}

/* After a plan that did not fit although no other is left: are there second copies of fp32 weights that could make way? */
static int splits_held(const thb_engine *E)
{
    int held = 0;
    for (int i = 0; i < E->nblobs; i++) held += E->blobs[i].key[1] == BL_SPLIT;
    return E->out_of_memory && held;
}
/* They go: no plan uses them any more. */
static void splits_drop(thb_engine *E)
{
    for (int i = 0; i < E->nblobs; i++)
        if (E->blobs[i].key[1] == BL_SPLIT) {
            if (cudaSetDevice(E->blobs[i].device) == cudaSuccess) cudaFree(E->blobs[i].ptr);
            E->blobs[i--] = E->blobs[--E->nblobs];
        }
}

/* Plans beyond MAX_PLAN_BYTES are dropped, the least recently used first and the current one never. */
static void plans_bound(thb_engine *E)
{
    size_t total = 0;
    for (int i = 0; i < MAX_PLANS; i++)
        if (E->plans[i]) total += plan_bytes(E->plans[i]);
    for (int v; total > MAX_PLAN_BYTES && (v = plan_oldest(E, E->cur)) >= 0;) {
        total -= plan_bytes(E->plans[v]);
        plan_drop(E, v);
    }
}

static int plan_build(thb_engine *E);

/* Make the plan of this input shape the current one, building it when it is not kept. */
static int select_plan(thb_engine *E, int N, int C, int H, int W, int rank, int cp)
{
    E->clock++;
    for (int i = 0; i < MAX_PLANS; i++) {
        shape_plan *p = E->plans[i];
        if (p && p->N == N && p->C == C && p->H == H && p->W == W && p->rank == rank && p->cp == cp) {
            p->used = E->clock;
            E->cur = p;
            return 0;
        }
    }
    int slot = -1;
    for (int i = 0; i < MAX_PLANS && slot < 0; i++)
        if (!E->plans[i]) slot = i;
    if (slot < 0) plan_drop(E, slot = plan_oldest(E, 0));
    for (int no_split = 0;;) {
        shape_plan *p = E->plans[slot] = E->cur = calloc(1, sizeof(*p));
        if (!p) { thb_set_error("out of memory"); return -1; }
        p->N = N; p->C = C; p->H = H; p->W = W; p->rank = rank; p->cp = cp;
        p->no_split = no_split;
        p->used = E->clock;
        if (!plan_build(E)) break;
        plan_drop(E, slot);
        if (plans_make_way(E)) continue;
        if (!splits_held(E)) return -1;
        splits_drop(E);
        no_split = 1;
    }
    plans_bound(E);
    return 0;
}

/* Ways to cut a batch into sub-batches, boundaries in sixteenths: growing ones where the results' way back is the longest
 * part (the first result leaves early and each later one is computed under the copy before it), shrinking ones where the
 * inputs' way in is (little is left to compute when the last input arrives), even ones between. */
static const unsigned char sub_batch_cuts[][5] = {
    {0, 16}, {0, 6, 16}, {0, 8, 16}, {0, 11, 16}, {0, 3, 8, 16}, {0, 5, 11, 16}, {0, 7, 13, 16},
    {0, 1, 3, 7, 16}, {0, 2, 6, 11, 16}, {0, 4, 8, 12, 16}, {0, 5, 10, 14, 16},
};

/* sub-batch c of a slice of n images under a cut */
static void cut_at(int n, const unsigned char *cut, int c, int *offset, int *count)
{
    *offset = (n * cut[c] + 8) / 16;
    *count = (n * cut[c + 1] + 8) / 16 - *offset;
}

/* Sub-batches per GPU of a host-input forward: the cut with the earliest last result in a model of the three stages a
 * sub-batch goes through -- its copy to the device, its kernels (model_us, and LAUNCH_US for each launch however small the
 * sub-batch is), its result's copy back -- each one at a time.  The uint8 engine needs the range of a whole float
 * batch before any kernel can start; its byte images have a static one. */
static void choose_sub_batches(thb_engine *E)
{
    shape_plan *p = E->cur;
    instance *I = &p->inst[0];
    p->chunks = 1;
    p->cut = 0;
    if ((E->dtype == THB_U8 && !p->cp) || I->slice_n < 2) return;
    const double t_in = copy_in_us(E, I), t_out = 4.0 * I->out_count / 50e3;
    double t_k = 0;
    for (int t = 0; t < I->nsteps; t++) t_k += model_us(&I->steps[t]);
    const double fixed = I->nsteps * LAUNCH_US;
    double best = 0;
    for (unsigned c = 0; c < sizeof(sub_batch_cuts) / sizeof(sub_batch_cuts[0]); c++) {
        const unsigned char *cut = sub_batch_cuts[c];
        double in = 0, k = 0, out = 0;
        int S = 0, ok = 1;
        do {
            const double f = (cut[S + 1] - cut[S]) / 16.0;
            if (cut[S + 1] < 16 && I->slice_n * (cut[S + 1] - cut[S]) < 16) ok = 0;
            /* every sub-batch at least an image, also where the boundaries are rounded and on the GPU with the fewest images */
            int off, n, n_least;
            cut_at(I->slice_n, cut, S, &off, &n);
            cut_at(p->inst[p->built - 1].slice_n, cut, S, &off, &n_least);
            if (n < 1 || n_least < 1) ok = 0;
            in += f * t_in;
            k = (in > k ? in : k) + f * t_k + fixed;
            out = (k > out ? k : out) + f * t_out;
        } while (cut[++S] < 16);
        if (!ok || S > I->slice_n) continue;
        if (c == 0 && I->slices) out -= I->hidden_us;
        if (c == 0 || out < 0.97 * best) {
            best = out;
            p->chunks = S;
            p->cut = S > 1 ? cut : 0;
        }
    }
}

static int plan_build(thb_engine *E)
{
    const int N = E->cur->N, cp = E->cur->cp;
    E->cur->peer_gather = E->peer_gather;
    E->out_of_memory = 0;
    int G = E->ngpus < N ? E->ngpus : N;
    if (G < 1) G = 1;
    int dev0 = 0;
    const char *d0 = getenv("THB200_DEVICE");
    if (d0) dev0 = atoi(d0);
    for (int g = 0; g < G; g++) {
        int off, n;
        thb_slice_batch(N, G, g, &off, &n);
        if (instance_build(E, &E->cur->inst[g], dev0 + g, off, n, -1)) return -1;
    }
    /* gather target: GPU 0 holds the whole result when peer copies are usable */
    if (G > 1 && E->cur->peer_gather) {
        for (int g = 1; g < G; g++) {
            int can = 0;
            cudaDeviceCanAccessPeer(&can, E->cur->inst[0].device, E->cur->inst[g].device);
            if (!can) E->cur->peer_gather = 0;
        }
        if (E->cur->peer_gather) {
            /* direct copies over NVLink need the access switched on from the sending GPU's side (a second request is
             * answered with cudaErrorPeerAccessAlreadyEnabled, which is fine) */
            for (int g = 1; g < G; g++) {
                cudaSetDevice(E->cur->inst[g].device);
                const cudaError_t pe = cudaDeviceEnablePeerAccess(E->cur->inst[0].device, 0);
                if (pe != cudaSuccess && pe != cudaErrorPeerAccessAlreadyEnabled) E->cur->peer_gather = 0;
                cudaGetLastError();
            }
        }
        if (E->cur->peer_gather) {
            long total = 0;
            for (int g = 0; g < G; g++) total += E->cur->inst[g].out_count;
            cudaSetDevice(E->cur->inst[0].device);
            E->cur->inst[0].d_out = dalloc(E, &E->cur->inst[0], (size_t)total * sizeof(float));
            if (!E->cur->inst[0].d_out) return -1;
        }
    }
    E->cur->built = G;
    choose_sub_batches(E);
    const char *ce = getenv("THB200_CHUNKS");
    if (ce) {
        E->cur->chunks = atoi(ce) < 1 || (E->dtype == THB_U8 && !cp) ? 1 : atoi(ce) > 4 ? 4 : atoi(ce);
        E->cur->cut = 0;
    }
    if (E->cur->chunks > N / G || E->whole_batch) E->cur->chunks = 1;
    return 0;
}

static int g_chunks_override; /* 0 = the engine's own choice */
void thb_set_pipeline_chunks(int n) { g_chunks_override = n < 0 ? 0 : n > 4 ? 4 : n; }

static void pipe_free(shape_plan *p)
{
    for (int g = 0; g < 32; g++) instance_free(&p->pipe[g]);
    p->pipe_built = 0;
}

static int pipe_instances(thb_engine *E, int S)
{
    const int G = E->cur->built;
    E->out_of_memory = 0;
    for (int g = 0; g < G; g++)
        for (int c = 0; c < S; c++) {
            int off, n;
            if (E->cur->cut && S == E->cur->chunks) cut_at(E->cur->inst[g].slice_n, E->cur->cut, c, &off, &n);
            else thb_slice_sub_batches(E->cur->inst[g].slice_n, S, c, &off, &n);
            if (instance_build(E, &E->cur->pipe[g * S + c], E->cur->inst[g].device, E->cur->inst[g].slice_off + off, n, c)) return -1;
        }
    E->cur->pipe_built = G * S;
    E->cur->pipe_chunks = S;
    return 0;
}

/* plan instances of the sub-batches (first pipelined forward of this shape with S sub-batches per GPU) */
static int pipe_build(thb_engine *E, int S)
{
    pipe_free(E->cur);
    while (pipe_instances(E, S)) {
        pipe_free(E->cur);
        if (plans_make_way(E)) continue;
        if (!splits_held(E)) return -1;
        /* the shape's own plan uses them: it is made again without */
        shape_plan *p = E->cur;
        for (int g = 0; g < 8; g++) instance_free(&p->inst[g]);
        splits_drop(E);
        p->built = 0;
        p->no_split = 1;
        if (!plan_build(E)) continue;
        for (int i = 0; i < MAX_PLANS; i++)
            if (E->plans[i] == p) plan_drop(E, i);
        return -1;
    }
    plans_bound(E);
    return 0;
}

/* per-forward parameters of a u8 convolution whose input scale is measured on the fly */
static void set_dynamic_quant(instance *I, float in_sub, float in_mult)
{
    for (int t = 0; t < I->nsteps; t++) {
        step *s = &I->steps[t];
        if (s->kind == ST_CONV && s->dyn_quant)
            thb_lowp_gemm_params(s->w_sub, s->w_mult, in_sub, in_mult, s->out_sub, s->out_mult, &s->conv.a_offset,
                                 &s->conv.b_offset, &s->conv.c_offset, &s->conv.c_mult, &s->conv.c_shift);
    }
}

/* every instance's first convolution gets the parameters that follow from the batch's extremes */
static void set_input_range(instance *set, int G, float lo, float hi, float *q_sub, float *q_mult)
{
    *q_sub = lo;
    *q_mult = hi - lo > 0 ? (float)(255.0 / (hi - lo)) : 0;
    for (int g = 0; g < G; g++) set_dynamic_quant(&set[g], *q_sub, *q_mult);
}

/* The uint8 engine's input range.  A float batch: lowp_basic.c:15-29 takes one range over the WHOLE batch tensor, so
 * the slices' extremes are reduced on the host (one 8-byte read-back per GPU) and every instance's first convolution
 * gets the parameters that follow from it.  Byte images: the loader's range is static (lowp_basic.c:82-131), nothing
 * is measured here. */
static int lowp_input_range(thb_engine *E, instance *set, int G, int has_x, int cp, int C, int H, int W, const float *mean,
                            const float *std, float *q_sub, float *q_mult)
{
    *q_sub = *q_mult = 0;
    if (E->dtype != THB_U8) return 0;
    if (!has_x) {
        if (cp != 3) { thb_set_error("the lowp image loader takes 3-plane images"); return -1; }
        return 0;
    }
    float lo = 0, hi = 0;
    for (int g = 0; g < G; g++) {
        instance *I = &set[g];
        CU(cudaSetDevice(I->device));
        if (thb_minmax_normalized(I->d_in, I->slice_n, C, H, W, mean, std, I->d_minmax, I->stream)) return -1;
        CU(cudaMemcpyAsync(I->h_minmax, I->d_minmax, 2 * sizeof(float), cudaMemcpyDeviceToHost, I->stream));
    }
    for (int g = 0; g < G; g++) {
        instance *I = &set[g];
        CU(cudaSetDevice(I->device));
        CU(cudaStreamSynchronize(I->stream));
        if (I->h_minmax[0] < lo) lo = I->h_minmax[0];
        if (I->h_minmax[1] > hi) hi = I->h_minmax[1];
    }
    set_input_range(set, G, lo, hi, q_sub, q_mult);
    return 0;
}

/* the buffers the uint8 convolutions add their channel sums into, before a forward's first launch */
static int clear_sums(instance *I)
{
    if (I->zero_bytes) CU(cudaMemsetAsync(I->arena, 0, I->zero_bytes, I->stream));
    return 0;
}

/* The boundary kernel in: images [img0, img0 + n) of the staged input (I->d_in: NCHW fp32, or I->d_img: HWC bytes) -> the
 * engine's layout and type. */
static int boundary_in(thb_engine *E, instance *I, int img0, int n, int has_x, int inplace, int cp, int bgr, int C, int H, int W,
                       const float *mean, const float *std, float q_sub, float q_mult)
{
    int rc;
    const value *iv = &I->in_val;
    const size_t stored = (size_t)iv->s.H * (iv->row_pitch ? iv->row_pitch : iv->s.W) * iv->ld; /* elements of an image */
    void *in_ptr = (char *)bufptr(I, iv->buf, 0, E->dtype) + img0 * stored * esize_of(E->dtype);
    float *d_in = I->d_in + (size_t)img0 * C * H * W;
    const unsigned char *d_img = I->d_img + (size_t)img0 * H * W * cp;
    const int f = I->input_s2d, W2 = f ? (W + f - 1) / f : 0, pitch = iv->row_pitch ? iv->row_pitch : W2;
    /* (float batches with even sides and stride 2 in the 16-bit modes have a kernel of their own) */
    if (f && (!has_x || E->dtype == THB_U8 || f != 2 || ((H | W) & 1))) {
        rc = thb_preprocess_s2d_any(has_x ? (const void *)d_in : d_img, !has_x, inplace ? d_in : 0, n, C, H, W, f, W * cp, bgr, mean, std,
                                    E->dtype, in_ptr, iv->ld, pitch, iv->pad_left, &q_sub, &q_mult, I->stream);
        if (!has_x && E->dtype == THB_U8) set_dynamic_quant(I, q_sub, q_mult);
    } else if (has_x && I->input_neigh)
        rc = thb_preprocess_neigh_u8(d_in, inplace ? d_in : 0, n, H, W, mean, std, in_ptr, I->in_val.ld, q_sub, q_mult,
                                     I->stream);
    else if (has_x && f)
        rc = thb_preprocess_s2d_padded(d_in, inplace ? d_in : 0, n, C, H, W, mean, std, E->dtype, in_ptr, iv->ld, pitch, iv->pad_left,
                                       I->stream);
    else if (has_x)
        rc = thb_preprocess(d_in, inplace ? d_in : 0, n, C, H, W, mean, std, E->dtype, in_ptr, I->in_val.ld,
                            q_sub, q_mult, I->stream);
    else if (cp == 2) /* one YUYV frame (THProcessYUYV) */
        rc = E->dtype == THB_U8 ? THB_ERR_UNSUPPORTED
                                : thb_preprocess_yuyv(d_img, H, W, mean, std, E->dtype, in_ptr, I->in_val.ld, I->stream);
    else if (E->dtype == THB_U8) {
        rc = thb_preprocess_images_lowp(d_img, n, H, W, W * cp, bgr, mean, std, in_ptr, I->in_val.ld, &q_sub,
                                        &q_mult, I->stream);
        set_dynamic_quant(I, q_sub, q_mult);
    } else
        rc = thb_preprocess_images(d_img, n, H, W, W * cp, cp, bgr, mean, std, E->dtype, in_ptr,
                                   I->in_val.ld, I->stream);
    if (rc) { thb_set_error("preprocess launch failed: %s", thb_last_cuda_error()); return -1; }
    return 0;
}

/* The boundary kernel out: the network's last tensor -> NCHW fp32 at `dst`; `head`: the network's last launch has not run yet
 * and does it itself. */
static int boundary_out(thb_engine *E, instance *I, float *dst, int head)
{
    if (head) {
        /* (directly, not from the graph: where the result goes may change from call to call) */
        step *s = &I->steps[I->nsteps - 1];
        if (s->nin > 1) s->conv.res = bufptr(I, s->in_buf[1], s->in_coff[1], s->dtype);
        if (thb_conv_nchw_fwd(&s->conv, bufptr(I, s->in_buf[0], s->in_coff[0], s->dtype), dst, I->h_status, I->stream)) {
            thb_set_error("the last convolution's launch failed: %s", thb_last_cuda_error());
            return -1;
        }
        return 0;
    }
    const value *ov = &I->out_val;
    float inv = ov->q_mult ? (float)(1.0 / ov->q_mult) : 0;
    if (thb_postprocess_status(bufptr(I, ov->buf, ov->coff, E->dtype), E->dtype, ov->s.N, ov->s.H, ov->s.W, ov->s.C, ov->ld,
                               ov->q_sub, inv, dst, I->d_status, I->h_status, I->stream)) { thb_set_error("postprocess launch failed"); return -1; }
    return 0;
}

/* The normalised values [off, off + n) of the instance's slice go back to the caller's slice on a stream of their own: the link is
 * full duplex and the forward does not wait for them (the caller does, before THProcessFloat returns). */
static int write_back(instance *I, float *slice, size_t off, size_t n)
{
    if (!I->wb_stream) {
        CU(cudaStreamCreateWithFlags(&I->wb_stream, cudaStreamNonBlocking));
        CU(cudaEventCreateWithFlags(&I->ev_wb, cudaEventDisableTiming));
    }
    CU(cudaEventRecord(I->ev_wb, I->stream));
    CU(cudaStreamWaitEvent(I->wb_stream, I->ev_wb, 0));
    CU(cudaMemcpyAsync(slice + off, I->d_in + off, n * sizeof(float), cudaMemcpyDeviceToHost, I->wb_stream));
    I->wb_pending = 1;
    return 0;
}

/* Everything one GPU does between its staged input and its NCHW fp32 result, on the instance's stream: the boundary
 * kernel in, the planned launches, the boundary kernel out.  ev0 marks the start of the planned launches.
 * `writeback`: host address the normalised input slice is copied back to (THProcessFloat's in-place side effect), or
 * NULL; `dst`: where the result goes (I->d_out, or this GPU's part of the gathered result). */
static int device_forward(thb_engine *E, instance *I, int has_x, int inplace, int cp, int bgr, int C, int H, int W,
                          const float *mean, const float *std, float q_sub, float q_mult, float *writeback, float *dst)
{
    if (clear_sums(I) || boundary_in(E, I, 0, I->slice_n, has_x, inplace, cp, bgr, C, H, W, mean, std, q_sub, q_mult)) return -1;
    if (writeback && write_back(I, writeback, 0, (size_t)I->slice_n * C * H * W)) return -1;
    CU(cudaEventRecord(I->ev0, I->stream));
    if (run_steps(E, I, 0)) return -1;
    return boundary_out(E, I, dst, head_on(I));
}

/* What the caller's batch lies in.  A copy from ordinary (pageable) memory is staged by the driver at a fraction of the link rate
 * and blocks the calling thread; only page-locked memory is known to be at hand for the host's threads too. */
enum host_memory { MEM_PAGEABLE, MEM_PINNED, MEM_OTHER };
static enum host_memory host_memory_of(const void *p)
{
    struct cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return MEM_OTHER; }
    return a.type == cudaMemoryTypeUnregistered ? MEM_PAGEABLE : a.type == cudaMemoryTypeHost ? MEM_PINNED : MEM_OTHER;
}

/* Copy into the pinned staging buffer past the caches.  The device reads the buffer next and the host never does: lines left
 * dirty in sixteen cores' caches have to be snooped out of them, at half the link's rate (38.5 MB staged and copied to the
 * device, eight pieces: 1.00 ms with memcpy, 0.83-0.88 ms with these stores; 0.71 ms is the copy alone). */
static void copy_past_caches(void *dst, const void *src, size_t n)
{
#ifdef __SSE2__
    char *d = dst;
    const char *s = src;
    const size_t head = (64 - ((size_t)d & 63)) & 63;
    if (n >= 256) {
        memcpy(d, s, head);
        d += head; s += head; n -= head;
        for (; n >= 64; n -= 64, d += 64, s += 64) {
            const __m128i a = _mm_loadu_si128((const __m128i *)s), b = _mm_loadu_si128((const __m128i *)(s + 16));
            const __m128i c = _mm_loadu_si128((const __m128i *)(s + 32)), e = _mm_loadu_si128((const __m128i *)(s + 48));
            _mm_stream_si128((__m128i *)d, a);
            _mm_stream_si128((__m128i *)(d + 16), b);
            _mm_stream_si128((__m128i *)(d + 32), c);
            _mm_stream_si128((__m128i *)(d + 48), e);
        }
        _mm_sfence();
    }
    memcpy(d, s, n);
#else
    memcpy(dst, src, n);
#endif
}

/* Threads that fill the staging buffer: eight already keep ahead of the link, and more of them disturb the thread that
 * issues the copies and launches (OMP_NUM_THREADS bounds them too). */
static int stage_threads(void)
{
    const int n = omp_get_max_threads();
    return n > 8 ? 8 : n;
}

/* host-to-host copy; from a quarter of a megabyte on by several threads */
static void parallel_copy(void *dst, const void *src, size_t bytes)
{
    const size_t blk = (size_t)128 << 10;
    const long nb = (long)((bytes + blk - 1) / blk);
#pragma omp parallel for schedule(static) if (nb > 2) num_threads(stage_threads())
    for (long b = 0; b < nb; b++) {
        const size_t o = (size_t)b * blk;
        copy_past_caches((char *)dst + o, (const char *)src + o, bytes - o < blk ? bytes - o : blk);
    }
}

/* Smallest and largest value of a float batch's planes, by what is subtracted from them: channels 0, 1 and 2, and the others.
 * Empty classes are (INFINITY, -INFINITY); NaNs do not count, as in the device's pass (thb_minmax_normalized). */
typedef struct {
    float mn[4], mx[4];
} extremes;
static const extremes NO_EXTREMES = {{INFINITY, INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY, -INFINITY}};

static void extremes_join(extremes *e, const extremes *t)
{
#pragma omp critical(thb_extremes)
    for (int k = 0; k < 4; k++) {
        if (t->mn[k] < e->mn[k]) e->mn[k] = t->mn[k];
        if (t->mx[k] > e->mx[k]) e->mx[k] = t->mx[k];
    }
}

#ifdef __SSE2__
/* four values into the running extremes (min and max with the running value as second operand keep it when the new one is a NaN) */
#define EXTREMES4(v, lo, hi) ((lo) = _mm_min_ps(v, lo), (hi) = _mm_max_ps(v, hi))
static void extremes_of4(__m128 lo, __m128 hi, float *mn, float *mx)
{
    float a[4], b[4];
    _mm_storeu_ps(a, lo);
    _mm_storeu_ps(b, hi);
    for (int q = 0; q < 4; q++) {
        if (a[q] < *mn) *mn = a[q];
        if (b[q] > *mx) *mx = b[q];
    }
}
#endif

/* The extremes of n values joined to *mn and *mx and, with `d`, the values copied there past the caches, in one pass over them. */
static void scan_values(float *d, const float *s, long n, float *mn, float *mx)
{
    float a = *mn, b = *mx;
    long i = 0;
#ifdef __SSE2__
    long head = d ? (long)((64 - ((size_t)d & 63)) & 63) / 4 : 0; /* whole lines from there on */
    if (head > n) head = n;
    for (; i < head; i++) {
        const float v = d[i] = s[i];
        if (v < a) a = v;
        if (v > b) b = v;
    }
    __m128 a0 = _mm_set1_ps(a), a1 = a0, b0 = _mm_set1_ps(b), b1 = b0;
    for (; i + 16 <= n; i += 16) {
        const __m128 t = _mm_loadu_ps(s + i), u = _mm_loadu_ps(s + i + 4), v = _mm_loadu_ps(s + i + 8), w = _mm_loadu_ps(s + i + 12);
        EXTREMES4(t, a0, b0);
        EXTREMES4(u, a1, b1);
        EXTREMES4(v, a0, b0);
        EXTREMES4(w, a1, b1);
        if (d) {
            _mm_stream_ps(d + i, t);
            _mm_stream_ps(d + i + 4, u);
            _mm_stream_ps(d + i + 8, v);
            _mm_stream_ps(d + i + 12, w);
        }
    }
    extremes_of4(a0, b0, &a, &b);
    extremes_of4(a1, b1, &a, &b);
    if (d) _mm_sfence();
#endif
    for (; i < n; i++) {
        const float v = s[i];
        if (d) d[i] = v;
        if (v < a) a = v;
        if (v > b) b = v;
    }
    *mn = a;
    *mx = b;
}

/* The same for planes [p0, p1) of an NCHW float batch (plane p = image p / C, channel p % C, HW floats), by several threads. */
static void scan_planes(float *dst, const float *x, long p0, long p1, int C, long HW, extremes *e)
{
    const long pieces = (HW + 16383) / 16384, per = ((HW + pieces - 1) / pieces + 15) & ~15L, items = (p1 - p0) * pieces;
#pragma omp parallel num_threads(stage_threads()) if (items > 4)
    {
        extremes t = NO_EXTREMES;
#pragma omp for schedule(static) nowait
        for (long q = 0; q < items; q++) {
            const long p = p0 + q / pieces, i0 = q % pieces * per, i1 = i0 + per < HW ? i0 + per : HW;
            const int k = p % C < 3 ? (int)(p % C) : 3;
            if (i0 < i1) scan_values(dst ? dst + p * HW + i0 : 0, x + p * HW + i0, i1 - i0, &t.mn[k], &t.mx[k]);
        }
        extremes_join(e, &t);
    }
}

/* Smallest and largest normalised value of the batch, both seeded with 0 (lowp_basic.c:15-29): only the extremes are normalised --
 * a subtraction and a division in fp32 are monotone. */
static void extremes_range(const extremes *e, const float *mean, const float *std, float *lo, float *hi)
{
    *lo = *hi = 0;
    for (int k = 0; k < 4; k++) {
        if (!(e->mn[k] <= e->mx[k])) continue;
        float a = e->mn[k], b = e->mx[k];
        if (k < 3) { a = (a - mean[k]) / std[k]; b = (b - mean[k]) / std[k]; }
        if (a > b) { const float t = a; a = b; b = t; }
        if (a < *lo) *lo = a;
        if (b > *hi) *hi = b;
    }
}

/* Does a pass of the host's threads over a page-locked batch, under its copy, end before the devices' pass after it?  What it can
 * save is that pass and the wait for its result: 20 to 25 us, whatever the size.  But a thread reads 6 GB/s of a batch that is in
 * no cache, several slow one another and the copy down, and the link carries 55 GB/s: from some size on, the more the longer, the
 * call waits for the host.  ResNet-18 uint8, microseconds a call with the devices' pass / the host's, batches read from memory
 * (in brackets: from the cache):
 *     threads      1               2               4               8
 *     0.6 MB   225 / 252 (208)  224 / 212 (200)  225 / 212 (200)  225 / 203 (200)
 *     1.2 MB   246 / 323 (254)  247 / 262 (218)  247 / 233 (219)  247 / 229 (218)
 *     2.4 MB   286 / 473 (317)  286 / 348 (273)  285 / 285 (259)  285 / 282 (260)
 *     4.8 MB   356 / 757 (434)  356 / 511 (365)  358 / 384 (337)  356 / 384 (345)
 *     9.6 MB   506 / 1315 (672) 506 / 829 (557)  505 / 581 (534)  507 / 579 (503) */
static int host_scan_pays(size_t bytes) { return bytes <= (size_t)stage_threads() * 300 << 10; }

/* Byte images, each wherever the caller has it, to one tightly packed array.  The threads share blocks of rows, so that
 * one large image is spread over them as well as a batch of small ones. */
static void stage_images(unsigned char *dst, unsigned char *const *images, int n, int H, size_t row, size_t stride)
{
    const int rows = row >= ((size_t)64 << 10) ? 1 : (int)(((size_t)64 << 10) / row);
    const int per = (H + rows - 1) / rows;
    const long items = (long)n * per;
#pragma omp parallel for schedule(static) if (items > 4) num_threads(stage_threads())
    for (long t = 0; t < items; t++) {
        const int i = (int)(t / per), r0 = (int)(t % per) * rows, r1 = r0 + rows < H ? r0 + rows : H;
        unsigned char *d = dst + ((size_t)i * H + r0) * row;
        const unsigned char *s = images[i] + (size_t)r0 * stride;
        if (stride == row) copy_past_caches(d, s, (size_t)(r1 - r0) * row);
        else
            for (int r = r0; r < r1; r++, d += row, s += stride) copy_past_caches(d, s, row);
    }
}

/* The copy of planes [p0, p1) of an NCHW float batch into the staging buffer, normalising the first three channels on the way
 * exactly as the boundary kernels do -- (x - mean) / std, a subtraction and a division in fp32 -- and writing the normalised
 * values back over the caller's planes: THProcessFloat's in-place side effect (thapi.c:396-403) done where the reference does
 * it, on the host, instead of a 12-bytes-per-pixel copy back from the device.  `e`: the extremes of what is staged, or NULL. */
static void stage_planes_normalised(float *dst, float *src, long p0, long p1, int C, long HW, const float *mean, const float *std,
                                    extremes *e)
{
#pragma omp parallel if ((p1 - p0) * HW > 65536) num_threads(stage_threads())
    {
        extremes t = NO_EXTREMES;
#pragma omp for schedule(static) nowait
        for (long p = p0; p < p1; p++) {
            const int c = (int)(p % C);
            float *s = src + p * HW, *d = dst + p * HW;
            if (c < 3) {
                const float m = mean[c], sd = std[c];
                float a = t.mn[c], b = t.mx[c];
                long i = 0;
#ifdef __SSE2__
                const __m128 vm = _mm_set1_ps(m), vs = _mm_set1_ps(sd);
                __m128 lo = _mm_set1_ps(a), hi = _mm_set1_ps(b);
                if (((size_t)d & 15) == 0)
                    for (; i + 4 <= HW; i += 4) {
                        const __m128 v = _mm_div_ps(_mm_sub_ps(_mm_loadu_ps(s + i), vm), vs);
                        _mm_storeu_ps(s + i, v);
                        _mm_stream_ps(d + i, v);
                        if (e) EXTREMES4(v, lo, hi);
                    }
                _mm_sfence();
                extremes_of4(lo, hi, &a, &b);
#endif
                for (; i < HW; i++) {
                    const float v = (s[i] - m) / sd;
                    s[i] = v;
                    d[i] = v;
                    if (v < a) a = v;
                    if (v > b) b = v;
                }
                t.mn[c] = a;
                t.mx[c] = b;
            } else if (e)
                scan_values(d, s, HW, &t.mn[3], &t.mx[3]);
            else
                copy_past_caches(d, s, (size_t)HW * sizeof(float));
        }
        if (e) extremes_join(e, &t);
    }
}

/* bytes staged per copy to the device, and up to which size a result is written to the host by the kernel that makes it */
static const size_t STAGE_PIECE = (size_t)4 << 20, DIRECT_RESULT_BYTES = (size_t)16 << 20;

typedef struct {
    float *x;               /* NCHW floats, or */
    unsigned char **images; /* HWC bytes */
    size_t stride;
    int cp, C, H, W;
    int staged;    /* by way of the engine's pinned buffer */
    int host_norm; /* normalised in place on the way, with these statistics */
    const float *mean, *std;
    extremes *range; /* of a staged float batch whose extremes are wanted: found on the way, or NULL */
} input_batch;

/* Images [i0, i0 + cnt) of an instance's slice to its input buffer, by copies on stream `st`. */
static int send_images(thb_engine *E, instance *I, const input_batch *in, int i0, int cnt, cudaStream_t st)
{
    const long HW = (long)in->H * in->W;
    const size_t first = (size_t)(I->slice_off + i0);
    if (in->x) {
        const long C = in->C, planes = cnt * C;
        float *dst = I->d_in + (size_t)i0 * C * HW, *xs = in->x + first * C * HW, *stage = E->h_stage + first * C * HW;
        if (!in->staged) {
            CU(cudaMemcpyAsync(dst, xs, (size_t)planes * HW * sizeof(float), cudaMemcpyHostToDevice, st));
            return 0;
        }
        /* in pieces of whole planes: the copy to the device of one piece runs while the host threads fill the next */
        long per_piece = (long)(STAGE_PIECE / sizeof(float)) / HW;
        if (per_piece < 1) per_piece = 1;
        for (long p0 = 0; p0 < planes; p0 += per_piece) {
            const long p1 = p0 + per_piece < planes ? p0 + per_piece : planes;
            const size_t o = (size_t)p0 * HW, n = (size_t)(p1 - p0) * HW;
            if (in->host_norm) stage_planes_normalised(stage, xs, p0, p1, in->C, HW, in->mean, in->std, in->range);
            else if (in->range) scan_planes(stage, xs, p0, p1, in->C, HW, in->range);
            else parallel_copy(stage + o, xs + o, n * sizeof(float));
            CU(cudaMemcpyAsync(dst + o, stage + o, n * sizeof(float), cudaMemcpyHostToDevice, st));
        }
        return 0;
    }
    const size_t row = (size_t)in->W * in->cp, img_bytes = in->H * row;
    unsigned char *dst = I->d_img + i0 * img_bytes, **images = in->images + first;
    if (in->staged) {
        unsigned char *stage = (unsigned char *)E->h_stage + first * img_bytes;
        int per_piece = (int)(STAGE_PIECE / img_bytes);
        if (per_piece < 1) per_piece = 1;
        for (int n = 0; n < cnt; n += per_piece) {
            const int k = cnt - n < per_piece ? cnt - n : per_piece;
            stage_images(stage + n * img_bytes, images + n, k, in->H, row, in->stride);
            CU(cudaMemcpyAsync(dst + n * img_bytes, stage + n * img_bytes, k * img_bytes, cudaMemcpyHostToDevice, st));
        }
    } else if (in->stride == row) {
        /* pinned, tightly packed rows: one copy per run of images that also follow one another in host memory */
        for (int n = 0; n < cnt;) {
            int run = 1;
            while (n + run < cnt && images[n + run] == images[n + run - 1] + img_bytes) run++;
            CU(cudaMemcpyAsync(dst + n * img_bytes, images[n], run * img_bytes, cudaMemcpyHostToDevice, st));
            n += run;
        }
    } else
        for (int n = 0; n < cnt; n++)
            CU(cudaMemcpy2DAsync(dst + n * img_bytes, row, images[n], in->stride, row, in->H, cudaMemcpyHostToDevice, st));
    return 0;
}

int thb_engine_forward(thb_engine *E, float *x, unsigned char **images, int stride, int bgr, int cp, int N, int C, int H,
                       int W, int rank, const float *mean, const float *std, int inplace, thb_result *res)
{
    if (N < 1 || C < 1 || H < 1 || W < 1) { thb_set_error("empty input"); return -1; }
    if (E->dtype == THB_U8 && !x) rank = 4; /* the lowp image loader always builds a 4-D tensor (lowp_basic.c:87-92) */
    if (select_plan(E, N, C, H, W, rank, cp)) return -1;
    /* host input (a float batch or byte images): run the sub-batch instances so that copies and kernels overlap */
    instance *set = E->cur->inst;
    int G = E->cur->built;
    const int peer_gather = E->cur->peer_gather;
    int S = g_chunks_override ? g_chunks_override : E->cur->chunks;
    if ((E->dtype == THB_U8 && x) || S > E->cur->inst[G - 1].slice_n || E->whole_batch) S = 1;
    if (S > 1) {
        if ((!E->cur->pipe_built || E->cur->pipe_chunks != S) && pipe_build(E, S)) return -1;
        set = E->cur->pipe;
        G = E->cur->pipe_built;
    }
    /* Peer gather: every GPU's part of the result ends up in GPU 0's result buffer (the first instance's, sized for the
     * whole batch), which goes to the host in one copy.  Instances on GPU 0 write their part there directly; the others
     * send theirs with cudaMemcpyPeerAsync on their own stream -- also when a GPU's slice runs as pipelined sub-batches. */
    float *gather = E->cur->built > 1 && peer_gather ? E->cur->inst[0].d_out : 0;
    const int dev0 = E->cur->inst[0].device;
    /* A small result is written by the boundary kernel into the pinned result buffer itself, which saves the copy that would
     * otherwise start when the kernels have ended (about 6 us for a few kilobytes as for 15 MB). */
    long total = 0;
    for (int g = 0; g < G; g++) total += set[g].out_count;
    const int direct = !gather && (size_t)total * sizeof(float) <= DIRECT_RESULT_BYTES;
    const size_t img_elems = (size_t)C * H * W;
    float q_sub = 0, q_mult = 0;

    if ((size_t)total * sizeof(float) > E->h_out_bytes) {
        thb_host_free_pinned(E->h_out);
        E->h_out_bytes = (size_t)total * sizeof(float);
        E->h_out = thb_host_alloc_pinned(E->h_out_bytes);
        if (!E->h_out) { thb_set_error("pinned result allocation failed"); return -1; }
    }
    /* A batch in pageable memory (what a caller of the reference passes) goes through a pinned buffer of the library, piece
     * by piece, filled by the host's threads: the copy of a piece to the device runs at link speed under the filling of the
     * next one, and images that lie apart in memory leave as one copy per piece.  The driver's own staging of 256 separate
     * pictures took 4.5 ms of an 8.1 ms call; small batches gain too, since the driver stages and waits for those inside the
     * call.  (THB200_NO_STAGING=1: hand the caller's pointers to the driver as they are.) */
    int staged = 0;
    const size_t in_bytes = x ? (size_t)N * img_elems * sizeof(float) : (size_t)N * H * W * cp;
    const enum host_memory mem = host_memory_of(x ? (const void *)x : images[0]);
    if (mem == MEM_PAGEABLE) {
        const char *ns = getenv("THB200_NO_STAGING");
        staged = !(ns && atoi(ns));
        if (staged && in_bytes > E->h_stage_bytes) {
            thb_host_free_pinned(E->h_stage);
            E->h_stage_bytes = in_bytes;
            E->h_stage = thb_host_alloc_pinned(E->h_stage_bytes);
            if (!E->h_stage) { E->h_stage_bytes = 0; staged = 0; }
        }
    }
    /* A staged float batch that is to be normalised in place is normalised by the host threads while they stage it: the
     * device then gets normalised values (identity statistics from here on) and copies nothing back. */
    static const float zero3[3] = {0, 0, 0}, one3[3] = {1, 1, 1};
    const float *host_mean = mean, *host_std = std;
    const int host_norm = staged && x && inplace;
    if (host_norm) { mean = zero3; std = one3; inplace = 0; }
    /* The uint8 engine needs the input range of the whole float batch before any kernel can start: it sends every slice on its
     * way, then has the range, then launches (byte images come with a static range).  The range comes from the host's threads
     * while they stage the batch, from a pass of theirs over a page-locked one while it is on its way, or from the GPUs' pass
     * over what has arrived.  The other modes launch a slice's kernels as soon as its copy is queued. */
    const int two_phase = E->dtype == THB_U8 && x;
    const int scan = two_phase && mem == MEM_PINNED && host_scan_pays(in_bytes);
    extremes range = NO_EXTREMES;
    const input_batch src = {x, images, (size_t)stride, cp, C, H, W, staged, host_norm, host_mean, host_std, two_phase && staged ? &range : 0};
    /* what the device-resident timing loop needs to repeat this forward from the staged input */
    E->last_has_x = x != 0; E->last_cp = cp; E->last_bgr = bgr;
    for (int k = 0; k < 3; k++) { E->last_mean[k] = mean[k]; E->last_std[k] = std[k]; }

    cudaEvent_t ev_call = 0;
    if (th_debug > 1 && cudaSetDevice(set[0].device) == cudaSuccess && cudaEventCreate(&ev_call) == cudaSuccess)
        cudaEventRecord(ev_call, set[0].stream);
    for (int phase = 0; phase <= two_phase; phase++) {
        if (phase == 1) {
            if (scan) scan_planes(0, x, 0, (long)N * C, C, (long)H * W, &range);
            if (scan || staged) {
                float lo, hi;
                extremes_range(&range, mean, std, &lo, &hi);
                set_input_range(set, G, lo, hi, &q_sub, &q_mult);
            } else if (lowp_input_range(E, set, G, x != 0, cp, C, H, W, mean, std, &q_sub, &q_mult)) return -1;
        }
        for (int g = 0; g < G; g++) {
            instance *I = &set[g];
            CU(cudaSetDevice(I->device));
            float *back = x && inplace ? x + (size_t)I->slice_off * img_elems : 0;
            /* (values on their way back to memory that is not page-locked would hold the calling thread up between the parts) */
            const int sliced = S == 1 && I->slices && !two_phase && (!back || mem == MEM_PINNED) && !th_profile && !th_minmax;
            for (int c = 0; sliced && c < I->slices; c++) {
                int i0, cnt;
                slice_part(I, c, &i0, &cnt);
                if (send_images(E, I, &src, i0, cnt, I->copy_stream)) return -1;
                CU(cudaEventRecord(I->ev_slice[c], I->copy_stream));
                CU(cudaStreamWaitEvent(I->stream, I->ev_slice[c], 0));
                if (c == 0 && clear_sums(I)) return -1;
                if (boundary_in(E, I, i0, cnt, x != 0, inplace, cp, bgr, C, H, W, mean, std, q_sub, q_mult)) return -1;
                if (back && write_back(I, back, i0 * img_elems, cnt * img_elems)) return -1;
                if (c == 0) CU(cudaEventRecord(I->ev0, I->stream));
                for (int t = 0; t < I->prefix; t++)
                    if (exec_step(I, t, i0, cnt)) return -1;
            }
            if (phase == 0 && !sliced && send_images(E, I, &src, 0, I->slice_n, I->stream)) return -1;
            if (phase != two_phase) continue;
            long off = 0;
            for (int k = 0; k < g; k++) off += set[k].out_count;
            float *dst = gather && I->device == dev0 ? gather + off : direct ? E->h_out + off : I->d_out;
            if (sliced) {
                if (run_steps(E, I, I->prefix) || boundary_out(E, I, dst, head_on(I))) return -1;
            } else if (device_forward(E, I, x != 0, inplace, cp, bgr, C, H, W, mean, std, q_sub, q_mult, back, dst)) return -1;
            CU(cudaEventRecord(I->ev1, I->stream));
            if (gather) {
                if (I->device != dev0)
                    CU(cudaMemcpyPeerAsync(gather + off, dev0, I->d_out, I->device, (size_t)I->out_count * sizeof(float), I->stream));
            } else if (!direct)
                CU(cudaMemcpyAsync(E->h_out + off, I->d_out, (size_t)I->out_count * sizeof(float), cudaMemcpyDeviceToHost, I->stream));
        }
    }
    float ms_max = 0;
    for (int g = G - 1; g >= 0; g--) {
        instance *I = &set[g];
        CU(cudaSetDevice(I->device));
        /* every other stream has been waited for by now: the gathered result is complete */
        if (g == 0 && gather)
            CU(cudaMemcpyAsync(E->h_out, gather, (size_t)total * sizeof(float), cudaMemcpyDeviceToHost, I->stream));
        CU(cudaStreamSynchronize(I->stream));
        if (I->wb_pending) {
            CU(cudaStreamSynchronize(I->wb_stream));
            I->wb_pending = 0;
        }
        float ms = 0;
        cudaEventElapsedTime(&ms, I->ev0, I->ev1);
        if (ev_call && I->device == set[0].device) {
            /* debug level 2: when each sub-batch's planned launches began and ended, from the start of the call */
            float a = 0, b = 0;
            cudaEventElapsedTime(&a, ev_call, I->ev0);
            cudaEventElapsedTime(&b, ev_call, I->ev1);
            fprintf(stderr, "thb200: sub-batch %d (%d images): launches from %.3f to %.3f ms\n", g, I->slice_n, a, b);
        }
        I->last_ms = ms;
        if (ms > ms_max) ms_max = ms;
        const int status = *(volatile int *)I->h_status;
        if (status) {
            *I->h_status = 0;
            cudaMemset(I->d_status, 0, sizeof(int));
            thb_set_error("a device-side wait timed out (code %d) on device %d", status, I->device);
            return -1;
        }
    }
    E->last_ms = ms_max;
    if (ev_call) cudaEventDestroy(ev_call);

    shape os = set[0].out_shape;
    res->data = E->h_out;
    res->count = total;
    int rk = os.rank;
    if (os.flat == 2) { /* a trailing View over a spatial tensor: rank from the View, data already in NCHW order */
        res->ndim = rk;
        if (rk == 2) { res->size[0] = N; res->size[1] = total / N; }
        else res->size[0] = total;
        return 0;
    }
    res->ndim = rk;
    switch (rk) {
    case 4: res->size[0] = N; res->size[1] = os.C; res->size[2] = os.H; res->size[3] = os.W; break;
    case 3: res->size[0] = os.C; res->size[1] = os.H; res->size[2] = os.W; break;
    case 2: res->size[0] = N; res->size[1] = os.C; break;
    default: res->size[0] = os.C; break;
    }
    return 0;
}

float thb_engine_last_ms(thb_engine *E) { return E ? E->last_ms : -1.f; }

/* Device-resident timing loop: the whole forward from the batch staged in device memory by the last THProcess* call
 * (NCHW fp32 or HWC bytes) to the NCHW fp32 result in device memory -- boundary kernels, the uint8 engine's input
 * range (with its 8-byte read-back) and the planned launches -- `iters` times back to back per GPU, timed with events
 * on the launching stream; max over GPUs.  No host<->device copy of the batch or the result is inside. */
float thb_engine_time_forward(thb_engine *E, int iters)
{
    if (!E || !E->cur || iters < 1 || (!E->last_has_x && !E->last_cp)) return -1.f;
    const int G = E->cur->built;
    cudaEvent_t t0[8], t1[8];
    for (int g = 0; g < G; g++) {
        if (cudaSetDevice(E->cur->inst[g].device) != cudaSuccess) return -1.f;
        cudaEventCreate(&t0[g]);
        cudaEventCreate(&t1[g]);
        cudaEventRecord(t0[g], E->cur->inst[g].stream);
    }
    int rc = 0;
    for (int it = 0; it < iters && !rc; it++) {
        float q_sub = 0, q_mult = 0;
        rc = lowp_input_range(E, E->cur->inst, G, E->last_has_x, E->last_cp, E->cur->C, E->cur->H, E->cur->W, E->last_mean, E->last_std, &q_sub, &q_mult);
        for (int g = 0; g < G && !rc; g++) {
            instance *I = &E->cur->inst[g];
            if (cudaSetDevice(I->device) != cudaSuccess) rc = -1;
            else rc = device_forward(E, I, E->last_has_x, 0, E->last_cp, E->last_bgr, E->cur->C, E->cur->H, E->cur->W, E->last_mean, E->last_std,
                                     q_sub, q_mult, 0, I->d_out);
        }
    }
    float worst = 0;
    for (int g = 0; g < G; g++) {
        instance *I = &E->cur->inst[g];
        cudaSetDevice(I->device);
        cudaEventRecord(t1[g], I->stream);
        if (cudaStreamSynchronize(I->stream) != cudaSuccess) rc = -1;
        float ms = 0;
        if (!rc) cudaEventElapsedTime(&ms, t0[g], t1[g]);
        if (ms > worst) worst = ms;
        cudaEventDestroy(t0[g]);
        cudaEventDestroy(t1[g]);
    }
    return rc ? -1.f : worst / iters;
}
