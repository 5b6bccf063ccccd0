"""The projector's host code on a fake device layer, in which one allocation
fails: a subset projection of horizontal rays that gets no memory for the
transpose walks the columns instead, succeeds, and leaves no error text."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ufo-ir_gb300", "csrc")

FAKE = r"""
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "host.h"
struct udev { char err[512]; int allocs, fail_at; };
static int walked_columns;
void udev_set_error(udev *d, const char *fmt, ...)
{ va_list a; va_start(a, fmt); vsnprintf(d->err, sizeof d->err, fmt, a); va_end(a); }
const char *udev_error(const udev *d) { return d->err; }
int udev_create(int device, udev **out, char *err, size_t len) { *out = calloc(1, sizeof **out); return 0; }
int udev_mem_info(udev *d, size_t *f, size_t *t) { *f = *t = 1u << 30; return 0; }
int udev_try_malloc(udev *d, void **p, size_t bytes)
{ *p = NULL; if (++d->allocs == d->fail_at) return UFOIR_ERR_NOMEM; *p = malloc(bytes ? bytes : 16); return 0; }
int udev_malloc(udev *d, void **p, size_t bytes)
{ int rc = udev_try_malloc(d, p, bytes); if (rc) udev_set_error(d, "device allocation failed"); return rc; }
int udev_free(udev *d, void *p) { free(p); return 0; }
int udev_is_device_ptr(udev *d, const void *p) { return 0; }
int udev_memcpy(udev *d, void *a, const void *b, size_t n) { memcpy(a, b, n); return 0; }
int udev_memcpy_async(udev *d, void *a, const void *b, size_t n) { memcpy(a, b, n); return 0; }
int udev_take_kernel_error(udev *d) { return 0; }
int udev_sync(udev *d) { return 0; }
int udev_transpose(udev *d, const float *in, float *out, int n, int s) { return 0; }
int udev_fp(udev *d, const udev_geom *g, int a0, int na, int dir, const float *vol, const float *volT, const float *src,
            const float *w, int ws, float *out, float scale, int s) { walked_columns = volT == NULL; return 0; }
int main(int argc, char **argv)
{
    enum { N = 8, A = 4 };
    static float vol[N * N], sino[A * N];
    ufoir_ctx *ctx;
    ufoir_projector *p;
    ufoir_projector_params prm;
    ufoir_subset s = {1, 2, UFOIR_HORIZONTAL};
    size_t in[2] = {N, N}, out[2];
    ufoir_projector_params_init(&prm);
    prm.step = 0.7f;
    prm.angles_num = A;
    if (ufoir_ctx_create(0, 0, &ctx) || ufoir_projector_create(ctx, &prm, &p) || ufoir_projector_get_requisition(p, in, out))
        return 2;
    ctx->dev->allocs = 0;
    ctx->dev->fail_at = atoi(argv[1]);       /* 1 the volume, 2 the sinogram, 3 the transpose */
    int rc = ufoir_projector_subset_fp(p, vol, sino, &s);
    printf("%d %d [%s]\n", rc, walked_columns, ufoir_last_error(ctx));
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("gcc") is None, reason="no C compiler")
@pytest.mark.parametrize("fail_at,want", [(0, "0 0 []"), (3, "0 1 []"), (2, "-3 0 [device allocation failed]")])
def test_subset_projection_without_memory_for_the_transpose(tmp_path, fail_at, want):
    src, exe = tmp_path / "fake.c", tmp_path / "fake"
    src.write_text(FAKE)
    # the device functions that these calls do not reach stay unresolved
    out = subprocess.run(["gcc", "-std=c11", "-D_GNU_SOURCE", "-w", "-I", CSRC, "-I", os.path.join(ROOT, "include"), str(src),
                          os.path.join(CSRC, "projector.c"), os.path.join(CSRC, "ctx.c"), "-o", str(exe), "-lm",
                          "-Wl,--unresolved-symbols=ignore-all"], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    run = subprocess.run([str(exe), str(fail_at)], capture_output=True, text=True)
    assert run.stdout.strip() == want, (run.returncode, run.stdout, run.stderr)
