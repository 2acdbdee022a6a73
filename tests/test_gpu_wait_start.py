"""The bounded waits of a sweep count from the end of the work it was launched behind. A kernel of the caller's may let
the next one in the stream start long before its own end (programmatic dependent launch); a sweep that starts in that
time waits for it, without its wait limit running."""
import ctypes
import subprocess

import numpy as np
import pytest

from qsv_b200 import build, compile_circuit, engine, generators as gen
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

# lets its dependents start at once, then takes `ns` nanoseconds (and ends after 2^24 turns in any case)
SOURCE = r"""
#include <cuda_runtime.h>
__global__ void early_trigger(unsigned long long ns) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (int i = 0; i < (1 << 24); i++) {
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 >= ns) break;
    }
}
extern "C" int launch_early(unsigned long long ns, void *stream) {
    early_trigger<<<1, 32, 0, (cudaStream_t)stream>>>(ns);
    return (int)cudaGetLastError();
}
"""


@pytest.mark.parametrize("mode,dtype", [("off", "c64"), ("eager", "c64"), ("off", "c128")])
def test_limit_counts_from_the_end_of_earlier_work(mode, dtype, tmp_path):
    torch = pytest.importorskip("torch")
    src, so = tmp_path / "early.cu", tmp_path / "early.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, "--shared", "-Xcompiler", "-fPIC", "-cudart", "static", "-o", str(so),
                    str(src)], check=True, timeout=300)
    launch = ctypes.CDLL(str(so)).launch_early
    launch.argtypes = [ctypes.c_ulonglong, ctypes.c_void_p]
    n = 16
    prog, _, _ = compile_circuit(gen.random_layer(n, 2, 3), n, 12, dtype=dtype)
    rng = np.random.default_rng(1)
    x = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    x = x.astype(np.complex128 if dtype == "c128" else np.complex64)
    ref = x.copy()
    old = engine.set_jit(mode)
    try:
        for _, seg in prog:
            ref = orc.run_segment(ref, seg)
            if mode == "eager":
                engine.jit_prepare(seg, n)
        for limit_us in (0, 5000):              # first with the default limit: kernels are loaded
            t = torch.from_numpy(x.copy()).cuda()
            s = torch.cuda.current_stream()
            s.synchronize()
            engine.set_wait_limit_us(limit_us)
            assert launch(30_000_000, s.cuda_stream) == 0
            for _, seg in prog:
                engine.run_segment(t, seg)
            torch.cuda.synchronize()
            assert engine.device_status() == 0
            assert np.array_equal(t.cpu().numpy(), ref)
    finally:
        engine.set_wait_limit_us(0)
        engine.set_jit(old)
