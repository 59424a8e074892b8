"""The page-locked staging of a device plan (csrc/ca3dmm_stage.h) against a stand-in
of the CUDA runtime whose copies run when the test lets the stream get there: a
queued upload, and one recorded into a graph, must see the plan that its call
wrote, whatever later calls write."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#ifndef FAKE_CUDA
#define FAKE_CUDA
#include <stddef.h>
typedef int cudaError_t;
typedef void *cudaStream_t;
typedef int *cudaEvent_t;
enum { cudaSuccess = 0, cudaEventDisableTiming = 2, cudaMemcpyHostToDevice = 1 };
enum cudaStreamCaptureMode { cudaStreamCaptureModeGlobal, cudaStreamCaptureModeThreadLocal, cudaStreamCaptureModeRelaxed };
enum cudaStreamCaptureStatus { cudaStreamCaptureStatusNone, cudaStreamCaptureStatusActive, cudaStreamCaptureStatusInvalidated };
static inline const char *cudaGetErrorString(cudaError_t e) { (void) e; return "fake"; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *, unsigned);
cudaError_t cudaEventDestroy(cudaEvent_t);
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t);
cudaError_t cudaEventSynchronize(cudaEvent_t);
cudaError_t cudaMallocHost(void **, size_t);
cudaError_t cudaFreeHost(void *);
cudaError_t cudaThreadExchangeStreamCaptureMode(enum cudaStreamCaptureMode *);
cudaError_t cudaStreamIsCapturing(cudaStream_t, enum cudaStreamCaptureStatus *);
cudaError_t cudaMemcpyAsync(void *, const void *, size_t, int, cudaStream_t);
cudaError_t cudaGetLastError(void);
cudaError_t cudaDeviceSynchronize(void);
#endif
"""

MAIN = r"""
#include <stdio.h>
#include <string.h>
#include "ca3dmm_stage.h"

struct copy { int *dst; const int *src; int ran; };
static struct copy queue[64], graph[64];
static int nq, ng, capturing, live, mode;
static int ev;                        /* uploads queued when the event was recorded */

cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void) f; *e = &ev; return 0; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { (void) e; return 0; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void) s; *e = nq; return capturing; }
static void run_queue(int upto)
{
    for (int i = 0; i < upto; i++)
        if (!queue[i].ran) { *queue[i].dst = *queue[i].src; queue[i].ran = 1; }
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    if (capturing && mode != cudaStreamCaptureModeRelaxed) return 1;
    run_queue(*e);
    return 0;
}
cudaError_t cudaMallocHost(void **p, size_t n)
{
    if (capturing && mode != cudaStreamCaptureModeRelaxed) return 1;
    *p = calloc(1, n);
    live++;
    return 0;
}
cudaError_t cudaFreeHost(void *p) { free(p); live--; return 0; }
cudaError_t cudaThreadExchangeStreamCaptureMode(enum cudaStreamCaptureMode *m)
{
    enum cudaStreamCaptureMode old = mode;
    mode = *m;
    *m = old;
    return 0;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus *c)
{
    (void) s;
    *c = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return 0;
}
cudaError_t cudaMemcpyAsync(void *d, const void *src, size_t n, int k, cudaStream_t s)
{
    (void) n; (void) k; (void) s;
    struct copy c = {(int *) d, (const int *) src, 0};
    if (capturing) graph[ng++] = c; else queue[nq++] = c;
    return 0;
}
cudaError_t cudaGetLastError(void) { return 0; }

cudaError_t cudaDeviceSynchronize(void)
{
    if (capturing && mode != cudaStreamCaptureModeRelaxed) return 1;
    run_queue(nq);
    return 0;
}

static int plan_of(ca3dmm_stage_t *s, int value, int *dev, int sync)
{
    if (ca3dmm_stage_begin(s)) return 1;
    *(int *) s->buf = value;
    return ca3dmm_stage_upload(s, dev, sync, 0);
}
static int plan(ca3dmm_stage_t *s, int value, int *dev) { return plan_of(s, value, dev, 0); }
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main(void)
{
    ca3dmm_stage_t s;
    int dev[8] = {0};
    memset(&s, 0, sizeof(s));
    CHECK(ca3dmm_stage_create(&s, 64) == 0);
    /* queued uploads, none of which has run when the next plan is written */
    for (int i = 0; i < 3; i++) CHECK(plan(&s, 10 + i, &dev[i]) == 0);
    CHECK(!s.any_graph);
    run_queue(nq);
    CHECK(dev[0] == 10 && dev[1] == 11 && dev[2] == 12);
    /* two captures and a direct call between them, behind a queued upload */
    CHECK(plan(&s, 20, &dev[3]) == 0);
    capturing = 1;
    CHECK(plan(&s, 21, &dev[4]) == 0);
    capturing = 0;
    CHECK(s.any_graph);
    CHECK(plan(&s, 22, &dev[5]) == 0);
    capturing = 1;
    CHECK(plan(&s, 23, &dev[6]) == 0);
    CHECK(plan(&s, 24, &dev[7]) == 0);
    capturing = 0;
    run_queue(nq);
    for (int r = 0; r < 2; r++)
        for (int i = 0; i < ng; i++) *graph[i].dst = *graph[i].src;
    CHECK(dev[3] == 20 && dev[4] == 21 && dev[5] == 22 && dev[6] == 23 && dev[7] == 24);
    CHECK(mode == cudaStreamCaptureModeGlobal);
    /* synchronous calls: one that waited for its stream, one that failed before it did */
    CHECK(plan_of(&s, 30, &dev[0], 1) == 0);
    run_queue(nq);
    ca3dmm_stage_done(&s);
    CHECK(plan_of(&s, 31, &dev[1], 1) == 0);
    CHECK(plan(&s, 32, &dev[2]) == 0);
    run_queue(nq);
    CHECK(dev[0] == 30 && dev[1] == 31 && dev[2] == 32);
    ca3dmm_stage_free(&s);
    CHECK(live == 0);
    return 0;
}
"""


def test_uploads_keep_their_own_plan(tmp_path):
    (tmp_path / "cuda_runtime_api.h").write_text(FAKE)
    (tmp_path / "main.c").write_text(MAIN)
    exe = str(tmp_path / "stage")
    inc = ["-I", str(tmp_path), "-I", os.path.join(ROOT, "ca3dmm_b200", "csrc"),
           "-I", os.path.join(ROOT, "include")]
    subprocess.run(["gcc", "-O1", "-g", "-std=gnu11", "-Wall"] + inc + [str(tmp_path / "main.c"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
