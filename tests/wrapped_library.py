"""libpt.so linked once more from its objects with some CUDA calls wrapped, so that a test can count them or have one
refused on the host: cudaGraphInstantiate (pt_test_instantiated counts it, pt_test_refuse_instantiate refuses as many
calls as it says) and cudaLaunchKernelExC, by which programmatic launches are made (pt_test_watched_launches counts those
on the stream pt_test_watched_stream; after pt_test_accept_launches more, pt_test_refuse_launch has as many as it says
refused by the CUDA runtime, for blocks of more threads than there can be).  A script that uses it runs in a process of its own."""
import subprocess
import sys
import textwrap

from pathtracer import build

WRAPS = r"""
#include <cuda_runtime.h>
extern "C" {
int pt_test_instantiated = 0, pt_test_refuse_instantiate = 0, pt_test_accept_launches = 0, pt_test_refuse_launch = 0, pt_test_watched_launches = 0;
void* pt_test_watched_stream = nullptr;
cudaError_t __real_cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long);
cudaError_t __wrap_cudaGraphInstantiate(cudaGraphExec_t* exec, cudaGraph_t graph, unsigned long long flags) {
    if (pt_test_refuse_instantiate > 0) {
        pt_test_refuse_instantiate -= 1;
        return cudaErrorMemoryAllocation;
    }
    pt_test_instantiated += 1;
    return __real_cudaGraphInstantiate(exec, graph, flags);
}
cudaError_t __real_cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**);
cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t* config, const void* kernel, void** args) {
    pt_test_watched_launches += config->stream == pt_test_watched_stream;
    if (pt_test_refuse_launch <= 0 || pt_test_accept_launches-- > 0) return __real_cudaLaunchKernelExC(config, kernel, args);
    pt_test_accept_launches = 0;
    pt_test_refuse_launch -= 1;
    cudaLaunchConfig_t refused = *config;
    refused.blockDim.x = 4096;
    return __real_cudaLaunchKernelExC(&refused, kernel, args);
}
}
"""

PRELUDE = """
import ctypes as C, sys
sys.path[:0] = {paths!r}
from pathlib import Path
from pathtracer import abi
abi.library_path = lambda: Path({library!r})
import pathtracer as pt
from pathtracer.engine import Engine
count = lambda name: C.c_int.in_dll(pt.load(), "pt_test_" + name)
"""


def link(folder):
    (folder / "wraps.cu").write_text(WRAPS)
    library = folder / "libpt_wrapped.so"
    objects = sorted(str(o) for o in build.OUT.glob("*.o"))
    wraps = [f for name in ("cudaGraphInstantiate", "cudaLaunchKernelExC") for f in ("-Xlinker", f"--wrap={name}")]
    subprocess.run([build.NVCC, *build.ARCH, "-shared", "-Xcompiler", "-fPIC", str(folder / "wraps.cu"), *objects,
                    *wraps, "-o", str(library)], check=True, capture_output=True, timeout=300)
    return library


def run(library, script, timeout=120):
    """Runs the script with the wrapped library as `pt` and gives what it prints."""
    prelude = PRELUDE.format(paths=[str(build.PKG), str(build.ROOT), str(build.ROOT / "tests")], library=str(library))
    out = subprocess.run([sys.executable, "-c", prelude + textwrap.dedent(script)], capture_output=True, text=True,
                         timeout=timeout)
    assert out.returncode == 0, out.stdout + out.stderr
    return out.stdout
