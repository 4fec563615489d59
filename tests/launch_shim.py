"""A stand-in for the CUDA runtime's launch call, preloaded into a child
process: it notes every launch's block and whether it is cooperative, and can
refuse cooperative launches with cudaErrorNotPermitted."""
import os
import subprocess
import sys

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdio.h>
#include <stdlib.h>
#include <cuda_runtime_api.h>
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  static cudaError_t (*real)(const cudaLaunchConfig_t*, const void*, void**) = 0;
  static FILE* log = 0;
  if (!real) {
    *(void**)&real = dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), "cudaLaunchKernelExC");
    log = fopen(getenv("SHIM_LOG"), "a");
  }
  int cooperative = 0;
  for (unsigned k = 0; k < c->numAttrs; ++k)
    if (c->attrs[k].id == cudaLaunchAttributeCooperative) cooperative = c->attrs[k].val.cooperative;
  fprintf(log, "%u %d\n", c->blockDim.x, cooperative);
  fflush(log);
  if (cooperative && getenv("SHIM_REFUSE")) return cudaErrorNotPermitted;
  return real(c, f, args);
}
"""


def run(tmp_path, code, refuse=False):
    """Runs the Python code in a child process under the shim; returns the launches it noted (threads per block,
    cooperative), as one list per stretch between the child's calls of mark()."""
    src, so, log = tmp_path / "shim.c", tmp_path / "shim.so", tmp_path / "launches.log"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-I/usr/local/cuda/include", "-o", str(so), str(src), "-ldl"],
                   check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), SHIM_LOG=str(log), PYTHONPATH=ROOT)
    if refuse:
        env["SHIM_REFUSE"] = "1"
    out = subprocess.run([sys.executable, "-c", code], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    stretches = log.read_text().split("mark\n")
    return [[tuple(map(int, x.split())) for x in s.splitlines()] for s in stretches]


def mark():
    with open(os.environ["SHIM_LOG"], "a") as f:
        f.write("mark\n")
