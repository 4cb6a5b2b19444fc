/* A CUDA runtime and kernel launchers that compute nothing, for testing the host library's planning and bookkeeping without a GPU:
 * device memory is address space with a budget, pinned memory is heap memory, launches are noted and succeed.  Linked with the host
 * library's sources in front of libthnets.so, whose host-side helpers (geometry, weight packing, split rules) are the real ones. */
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>
#include "thb200_kernels.h"

/* ---- what a test sets and reads ---- */
size_t fake_budget = (size_t)1 << 50, fake_live; /* device bytes */
int fake_devices = 1, fake_streams;              /* GPUs; streams alive */
int fake_minmax, fake_boundaries, fake_empty;    /* launches: of the device's range pass, of boundary kernels in, of those on nothing */
int fake_images;                                 /* that boundary kernels in were launched on */
float fake_q_sub, fake_q_mult;                   /* the input quantisation of the last boundary kernel in */
int fake_f32_tc, fake_splits, fake_tc_launches;  /* fp32 convolutions may go to the tensor cores; weights split for them; launches there */
int fake_waits;                                  /* waits for the legacy stream */

static void boundary(int n, float q_sub, float q_mult)
{
    fake_boundaries++;
    fake_images += n;
    if (n < 1) fake_empty++;
    fake_q_sub = q_sub;
    fake_q_mult = q_mult;
}

/* ---- memory ---- */
enum { MAX_BLOCKS = 1 << 16 };
static struct { char *p; size_t n; } dev[MAX_BLOCKS], host[MAX_BLOCKS];
static int ndev, nhost;
static char *next_address = (char *)0x700000000000;

cudaError_t cudaMalloc(void **p, size_t n)
{
    if (fake_live + n > fake_budget || ndev == MAX_BLOCKS) return cudaErrorMemoryAllocation;
    fake_live += n;
    dev[ndev].p = *p = next_address;
    dev[ndev++].n = n;
    next_address += (n + 511) & ~(size_t)511;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    for (int i = 0; i < ndev; i++)
        if (dev[i].p == p) {
            fake_live -= dev[i].n;
            dev[i] = dev[--ndev];
            return cudaSuccess;
        }
    return p ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned flags)
{
    (void)flags;
    if (nhost == MAX_BLOCKS || !(*p = calloc(1, n))) return cudaErrorMemoryAllocation;
    host[nhost].p = *p;
    host[nhost++].n = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p)
{
    for (int i = 0; i < nhost; i++)
        if (host[i].p == p) { host[i] = host[--nhost]; break; }
    free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p)
{
    memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    for (int i = 0; i < nhost; i++)
        if ((const char *)p >= host[i].p && (const char *)p < host[i].p + host[i].n) a->type = cudaMemoryTypeHost;
    return cudaSuccess;
}

/* ---- streams, events, devices ---- */
static cudaError_t stream_create(cudaStream_t *s) { *s = (cudaStream_t)malloc(1); fake_streams++; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; return stream_create(s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned f, int p) { (void)f; (void)p; return stream_create(s); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { fake_waits += !s; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); fake_streams--; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *ms = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = fake_devices; return cudaSuccess; }
cudaError_t cudaDeviceCanAccessPeer(int *can, int a, int b) { (void)a; (void)b; *can = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) { *lo = 0; *hi = -5; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s; (void)m; return cudaErrorNotSupported; }
const char *cudaGetErrorString(cudaError_t e) { (void)e; return "fake"; }
const char *thb_last_cuda_error(void) { return "fake"; }

/* ---- launches whose arguments are looked at ---- */
int thb_preprocess(const float *x, float *xi, int N, int C, int H, int W, const float *m, const float *s, int dt, void *y, int ld, float qs,
                   float qm, void *st)
{
    boundary(N, qs, qm);
    return 0;
}
int thb_preprocess_neigh_u8(const float *x, float *xi, int N, int H, int W, const float *m, const float *s, void *y, int ld, float qs,
                            float qm, void *st)
{
    boundary(N, qs, qm);
    return 0;
}
int thb_preprocess_s2d_any(const void *src, int bytes, float *xi, int N, int C, int H, int W, int f, int stride, int bgr, const float *m,
                           const float *s, int dt, void *y, int ld, int pitch, int pad, float *qs, float *qm, void *st)
{
    boundary(N, *qs, *qm);
    return 0;
}
int thb_preprocess_s2d_padded(const float *x, float *xi, int N, int C, int H, int W, const float *m, const float *s, int dt, void *y, int ld,
                              int pitch, int pad, void *st)
{
    boundary(N, 0, 0);
    return 0;
}
int thb_minmax_normalized(const float *x, int N, int C, int H, int W, const float *m, const float *s, float *out, void *st)
{
    fake_minmax++;
    return 0;
}

/* fp32 on the tensor cores (the host library's own rules where a test has switched them on) */
int thb_conv_f32_supported(const thb_conv_desc *d) { return fake_f32_tc && d->dtype == THB_F32 && d->kH * d->kW * d->Cin >= 64 && !d->x2 && d->Cout_pad % 64 == 0; }
int thb_conv_f32_split_weights(const thb_conv_desc *d, void *w, void *st) { fake_splits++; return 0; }
int thb_conv_f32_fwd(const thb_conv_desc *d, const void *w, const void *x, void *y, void *st) { fake_tc_launches++; return 0; }

/* ---- the rest ---- */
unsigned short thb_float_to_half_bits(float v, int bf16) { (void)v; (void)bf16; return 0; }
int thb_kernel_launch_count(void) { return 0; }
void thb_count_launches(int n) { (void)n; }
/* (under another name in C: the headers' prototypes differ) */
#define NOTHING(name) int fake_##name() __asm__(#name); int fake_##name() { return 0; }
NOTHING(cudaDeviceEnablePeerAccess) NOTHING(cudaEventRecord) NOTHING(cudaGetLastError) NOTHING(cudaGraphDestroy)
NOTHING(cudaGraphExecDestroy) NOTHING(cudaGraphInstantiate) NOTHING(cudaGraphLaunch) NOTHING(cudaMemcpy) NOTHING(cudaMemcpy2DAsync)
NOTHING(cudaMemcpyAsync) NOTHING(cudaMemcpyPeerAsync) NOTHING(cudaMemset) NOTHING(cudaMemsetAsync) NOTHING(cudaSetDevice)
NOTHING(cudaStreamEndCapture) NOTHING(cudaStreamWaitEvent)
NOTHING(thb_affine_act) NOTHING(thb_avgpool) NOTHING(thb_cmax) NOTHING(thb_col2im) NOTHING(thb_combine) NOTHING(thb_conv_fwd)
NOTHING(thb_conv_make_tmap) NOTHING(thb_conv_maxpool_fwd) NOTHING(thb_conv_nchw_fwd) NOTHING(thb_copy_channels) NOTHING(thb_from_nchw)
NOTHING(thb_gemv_fwd) NOTHING(thb_l2_normalize) NOTHING(thb_logsoftmax) NOTHING(thb_max_unpool) NOTHING(thb_maxpool)
NOTHING(thb_postprocess_status) NOTHING(thb_preprocess_images) NOTHING(thb_preprocess_images_lowp) NOTHING(thb_preprocess_yuyv)
NOTHING(thb_reflect_pad) NOTHING(thb_slice_channels) NOTHING(thb_softmax) NOTHING(thb_to_nchw) NOTHING(thb_u8_channel_sum_rows)
NOTHING(thb_maxpool_sums) NOTHING(thb_maxpool_sums_supported)
NOTHING(thb_u8_combine) NOTHING(thb_u8_threshold) NOTHING(thb_upsample2x) NOTHING(thb_zero_pad)
