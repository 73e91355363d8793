"""The training step's two launches start under the end of the one before: the kernels may
touch nothing that the preceding launch still writes until it has completed. The library's
own step and optimiser run back to back on a stream (overlapping their starts) and with the
host waiting after every launch (nothing overlaps), from the same parameters.

Every 32 rows of the batch are the same 32, so every block and every thread group adds the same
sums to the gradient and the order in which they arrive changes nothing. Bar: the same parameters
bit for bit; a gradient of weights one step old gives others.
"""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

from pilot_b200 import beams as B
from pilot_b200.build import NVCC

pytestmark = pytest.mark.gpu
CSRC = Path(B.__file__).parent / "csrc"
KIN, PARAMS, STEPS = 112, 19777, 24


def kernels():
    L, P = B.lib(), C.c_void_p
    step = L._ZN5beams17mlp_train_step_tcEPKfPfPK13__nv_bfloat16S1_ifS2_S2_PjP11CUstream_st
    step.argtypes = [P, P, P, P, C.c_int, C.c_float, P, P, P, P]
    adam = L._ZN5beams8mlp_adamEPfS0_S0_S0_fiP11CUstream_st
    adam.argtypes = [P, P, P, P, C.c_float, C.c_int, P]
    step.restype = adam.restype = C.c_int
    return step, adam


@pytest.mark.parametrize("rows", [256, 512, 8192, 16384])
def test_overlapping_steps_read_the_finished_ones(cuda_device, rows):
    import torch
    step, adam = kernels()
    assert B.lib().beams_mlp_param_count() == PARAMS
    g = torch.Generator(device="cuda").manual_seed(rows)
    start = torch.randn(PARAMS, generator=g, device="cuda") * 0.15
    X = (torch.randn(STEPS, 32, KIN, generator=g, device="cuda") * 0.5).bfloat16().repeat(1, rows // 32, 1)
    target = torch.rand(STEPS, 32, generator=g, device="cuda").repeat(1, rows // 32)

    def train(wait, stale=False):
        P, G, m, v = start.clone(), *(torch.zeros(PARAMS, device="cuda") for _ in range(3))
        old, loss, err = P.clone(), torch.zeros(1, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        p = lambda t: C.c_void_p(t.data_ptr())
        for k in range(STEPS):
            x, y = X[k], target[k]
            assert step(p(old if stale else P), p(G), p(x), p(y), rows, 1.0 / rows, None, p(loss), p(err), st) == 0
            if wait:
                torch.cuda.synchronize()
            if stale:
                old.copy_(P)
            assert adam(p(P), p(G), p(m), p(v), 0.01, k + 1, st) == 0
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        assert int(err) == 0 and bool(torch.isfinite(P).all())
        return P

    apart = train(wait=True)
    assert not torch.equal(train(wait=True, stale=True), apart)
    for _ in range(8):
        assert torch.equal(train(wait=False), apart)


SRC = r"""
#include <cstdio>
#include "mlp_common.cuh"
__global__ void k_nothing(int) {}
int main() {
  const cudaError_t e = beams::mlp::launch_early(k_nothing, 1, 2048, 0, nullptr, 1);  // 1024 threads at most
  const cudaError_t left = cudaGetLastError();
  std::printf("%d %d", (int)(e == cudaErrorInvalidConfiguration || e == cudaErrorInvalidValue), (int)left);
  return 0;
}
"""


def test_a_refused_launch_leaves_no_error_behind(cuda_device, tmp_path):
    """The launch's own status reports it; the next call that asks for the last error has none."""
    (tmp_path / "t.cu").write_text(SRC)
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC),
                    str(tmp_path / "t.cu"), "-o", str(tmp_path / "t")], check=True)
    p = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert p.stdout == "1 0"
