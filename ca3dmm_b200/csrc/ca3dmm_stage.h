/* Page-locked staging of a device plan.  The copy engine reads the buffer when
 * the stream gets there, which may be long after the call that queued the copy
 * returned, and a copy recorded into a CUDA graph reads it at every replay. */
#ifndef CA3DMM_STAGE_H
#define CA3DMM_STAGE_H

#include <stdlib.h>
#include <cuda_runtime_api.h>
#include "ca3dmm_kernels.h"
#include "ca3dmm_util.h"

typedef struct {
    void *buf;
    size_t bytes;
    cudaEvent_t done;      /* recorded behind the last upload */
    int pending;           /* the last upload may not have run yet: 1 until `done`, 2 until the
                              call that queued it has waited for its stream */
    int in_graph;          /* a graph reads buf */
    int any_graph;         /* some graph may overwrite the device plan at any time */
    void **kept;           /* the buffers of captured uploads, held until the owner goes */
    int nkept;
} ca3dmm_stage_t;

static inline int ca3dmm_stage_create(ca3dmm_stage_t *s, size_t bytes)
{
    s->bytes = bytes;
    CA3DMM_CUDA_TRY(cudaEventCreateWithFlags(&s->done, cudaEventDisableTiming));
    if (cudaMallocHost(&s->buf, bytes) != cudaSuccess) {
        s->buf = NULL;
        cudaEventDestroy(s->done);
        return CA3DMM_ECUDA;
    }
    return CA3DMM_OK;
}

static inline void ca3dmm_stage_free(ca3dmm_stage_t *s)
{
    if (!s->buf) return;
    for (int i = 0; i < s->nkept; i++) cudaFreeHost(s->kept[i]);
    free(s->kept);
    cudaFreeHost(s->buf);
    cudaEventDestroy(s->done);
    s->buf = NULL;
}

/* Before buf is rewritten: the last upload has left it; a buffer that belongs to
 * a graph is put aside for a new one.  Also called while a stream is being
 * captured, which only the relaxed mode allows of these calls. */
static inline int ca3dmm_stage_begin(ca3dmm_stage_t *s)
{
    if (!s->pending && !s->in_graph) return CA3DMM_OK;
    enum cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    CA3DMM_CUDA_TRY(cudaThreadExchangeStreamCaptureMode(&mode));
    int rc = CA3DMM_OK;
    if (s->in_graph) {
        void *nb = NULL;
        void **k = (void **) realloc(s->kept, sizeof(void *) * (size_t) (s->nkept + 1));
        if (k) s->kept = k;
        if (!k || cudaMallocHost(&nb, s->bytes) != cudaSuccess) {
            rc = CA3DMM_ENOMEM;
        } else {
            s->kept[s->nkept++] = s->buf;
            s->buf = nb;
            s->in_graph = 0;
        }
    } else if ((s->pending == 1 ? cudaEventSynchronize(s->done) : cudaDeviceSynchronize()) !=
               cudaSuccess) {
        rc = CA3DMM_ECUDA;                /* (2: that call failed before its wait) */
    }
    if (!rc) s->pending = 0;
    cudaThreadExchangeStreamCaptureMode(&mode);
    return rc;
}

/* Queue the copy of buf; sync: the caller waits for the stream before it returns and
 * then calls ca3dmm_stage_done, which spares the event (3 us a call).  Afterwards
 * any_graph says whether the device copy can be relied on by a later call: one that
 * waits in a graph has not run yet, and each replay puts that graph's plan back. */
static inline int ca3dmm_stage_upload(ca3dmm_stage_t *s, void *dst, int sync, cudaStream_t st)
{
    enum cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (!sync && cudaStreamIsCapturing(st, &cap) != cudaSuccess) {
        cudaGetLastError();              /* the legacy stream beside another thread's capture */
        cap = cudaStreamCaptureStatusNone;
    }
    CA3DMM_CUDA_TRY(cudaMemcpyAsync(dst, s->buf, s->bytes, cudaMemcpyHostToDevice, st));
    if (cap == cudaStreamCaptureStatusActive) {
        s->in_graph = s->any_graph = 1;
    } else if (sync) {
        s->pending = 2;
    } else {
        CA3DMM_CUDA_TRY(cudaEventRecord(s->done, st));
        s->pending = 1;
    }
    return CA3DMM_OK;
}

static inline void ca3dmm_stage_done(ca3dmm_stage_t *s) { s->pending = 0; }

#endif
