"""Runs a Python snippet in a process whose cooperative launches pass through a
shim in front of the CUDA runtime (LD_PRELOAD): it can hold each launch back for
a while, or answer all of them, or every second one, with the error a device
without room for the grid gives.  The GPU sees ordinary launches only."""
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
static int refuse_every = -1, delay_us, count;
int cudaLaunchCooperativeKernel(const void* f, dim3_ g, dim3_ b, void** a, size_t smem, void* stream) {
  if (refuse_every < 0) {
    delay_us = atoi(getenv("COOP_DELAY_US"));
    refuse_every = atoi(getenv("COOP_REFUSE_EVERY"));
  }
  if (delay_us) usleep(delay_us);
  if (refuse_every && ++count % refuse_every == 0) return 720; /* cudaErrorCooperativeLaunchTooLarge */
  void* rt = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
  if (!rt) return 999;
  launch_fn real = (launch_fn)dlsym(rt, "cudaLaunchCooperativeKernel");
  return real ? real(f, g, b, a, smem, stream) : 999;
}
"""


def run_under_shim(tmp_path, code, refuse_every=0, delay_us=0, timeout=300):
    src, so = tmp_path / "coop_shim.c", tmp_path / "coop_shim.so"
    src.write_text(SOURCE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(so), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), COOP_DELAY_US=str(delay_us), COOP_REFUSE_EVERY=str(refuse_every))
    env["PYTHONPATH"] = os.pathsep.join([os.path.join(ROOT, "tests"), ROOT] +
                                        [p for p in [env.get("PYTHONPATH")] if p])
    out = subprocess.run([sys.executable, "-c", code], env=env, cwd=ROOT, capture_output=True, text=True,
                         timeout=timeout)
    assert out.returncode == 0, out.stdout + out.stderr
    return out.stdout
