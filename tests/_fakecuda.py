"""A child python whose calls into the CUDA runtime pass through a preloaded
library that can fail one of them or count them (host code only)."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static int left, pending, mallocs;
void fake_arm(int k) { left = k; }            /* the k-th launch of the flat E kernel from now fails */
static void *real(const char *n) { return dlsym(dlopen("libcudart.so.12", RTLD_NOW | RTLD_NOLOAD), n); }
int cudaLaunchKernelExC(const void *c, const void *f, void **a)
{
    if (left > 0 && --left == 0) return pending = 701;   /* cudaErrorLaunchOutOfResources */
    return ((int (*)(const void *, const void *, void **))real("cudaLaunchKernelExC"))(c, f, a);
}
int fake_mallocs(void) { return mallocs; }    /* device allocations so far */
int cudaMalloc(void **p, size_t n)
{
    mallocs++;
    return ((int (*)(void **, size_t))real("cudaMalloc"))(p, n);
}
int cudaGetLastError(void)
{
    int e = pending;
    pending = 0;
    return e ? e : ((int (*)(void))real("cudaGetLastError"))();
}
"""


def run_child(code, tmp_path):
    """Runs `code`, which prints "agree" when all is as it should be; the fake is
    the library of LD_PRELOAD."""
    src, so = tmp_path / "fake.c", tmp_path / "fake.so"
    src.write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", code], env=env, cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "agree" in r.stdout, r.stdout + r.stderr
