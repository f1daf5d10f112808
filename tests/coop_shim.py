"""Runs a Python snippet in a process whose cooperative launches pass through a
shim in front of the CUDA runtime (LD_PRELOAD): it can hold each launch back for
a while, or let the first few through and answer the rest with the error a
device without room for the grid gives.  The GPU sees ordinary launches only."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>
#include <unistd.h>
typedef struct { unsigned x, y, z; } dim3_;
typedef int (*launch_fn)(const void*, dim3_, dim3_, void**, size_t, void*);
static int allowed = -2, delay_us;
int cudaLaunchCooperativeKernel(const void* f, dim3_ g, dim3_ b, void** a, size_t smem, void* stream) {
  if (allowed == -2) {
    const char *n = getenv("COOP_ALLOW"), *d = getenv("COOP_DELAY_US");
    delay_us = d ? atoi(d) : 0;
    allowed = n ? atoi(n) : -1;
  }
  if (delay_us) usleep(delay_us);
  if (allowed == 0) return 720; /* cudaErrorCooperativeLaunchTooLarge */
  if (allowed > 0) --allowed;
  void* rt = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
  if (!rt) return 999;
  launch_fn real = (launch_fn)dlsym(rt, "cudaLaunchCooperativeKernel");
  return real ? real(f, g, b, a, smem, stream) : 999;
}
"""


def run_under_shim(tmp_path, code, allow=None, delay_us=0, timeout=300):
    src, so = tmp_path / "coop_shim.c", tmp_path / "coop_shim.so"
    src.write_text(SOURCE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(so), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), COOP_DELAY_US=str(delay_us))
    env.pop("COOP_ALLOW", None)
    if allow is not None:
        env["COOP_ALLOW"] = str(allow)
    env["PYTHONPATH"] = os.pathsep.join([os.path.join(ROOT, "tests"), ROOT] +
                                        [p for p in [env.get("PYTHONPATH")] if p])
    out = subprocess.run([sys.executable, "-c", code], env=env, cwd=ROOT, capture_output=True, text=True,
                         timeout=timeout)
    assert out.returncode == 0, out.stdout + out.stderr
    return out.stdout
