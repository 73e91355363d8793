"""The training step's two launches start under the end of the one before: the kernels may
touch nothing that the preceding launch still writes until it has completed. The library's
own step and optimiser run back to back on a stream (overlapping their starts) and with the
host waiting after every launch (nothing overlaps), from the same parameters.

Every 32 rows of the batch are the same 32, so every block and every thread group adds the same
sums to the gradient and the order in which they arrive changes nothing. Bar: the same parameters
bit for bit; a gradient of weights one step old gives others.
"""
import ctypes as C

import pytest

from pilot_b200 import beams as B

pytestmark = pytest.mark.gpu
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
