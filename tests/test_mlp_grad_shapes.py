"""The closure's gradient kernel at the edges of its tiles (32 batch rows,
4 rows x 64 columns a warp, products 4 steps at a time) against the FP64
restatement of the same quantised network.

The kernel sums in FP32 over at most 64 inputs a layer and 32 rows a CTA:
relative to the largest entry of each tensor its error stays below a few
hundred roundings (2^-24), 1e-4 leaves a margin of several."""
import ctypes

import numpy as np
import pytest

import combustioncodegpu_b200 as cc
from oracle import closure_mlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 31, 32, 33, 96, 1000])
@pytest.mark.parametrize("shape", [(20, 64, 11), (64, 64, 64), (5, 7, 3), (1, 1, 1), (30, 33, 18)])
def test_gradient_matches_oracle(batch, shape):
    import torch

    n_in, h, n_out = shape
    rng = np.random.default_rng(batch + n_in)
    lib = cc.load_library()
    n = lib.cc_mlp_param_count(n_in, h, n_out)
    params = (rng.standard_normal(n) * 0.3).astype(np.float32)
    x = closure_mlp.bf16(rng.standard_normal((batch, n_in)).astype(np.float32))
    y = rng.standard_normal((batch, n_out)).astype(np.float32)
    scale = rng.uniform(0.5, 1.5, n_out).astype(np.float32)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (params, x, y, scale)]
    grad, loss = torch.empty(n, device="cuda"), torch.empty(1, device="cuda")
    work = torch.empty(lib.cc_mlp_workspace_bytes(n_in, h, n_out, batch), dtype=torch.uint8, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    got = []
    for _ in range(2):  # reproducible bit for bit, whatever the workspace holds
        work.fill_(255)
        cc._check(lib.cc_mlp_grad(n_in, h, n_out, batch, *map(ptr, dev), ptr(grad), ptr(loss), ptr(work), None))
        torch.cuda.synchronize()
        got.append((float(loss), grad.cpu().numpy().copy()))
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])
    want_loss, want = closure_mlp.loss_and_grad(params, x, y, scale, n_in, h, n_out)
    assert abs(got[0][0] - want_loss) <= 1e-5 * want_loss
    for ow, s, ob, nb in closure_mlp.layout(n_in, h, n_out)[0]:
        for a, b in ((ow, ow + s[0] * s[1]), (ob, ob + nb)):
            err = np.abs(got[0][1][a:b] - want[a:b]).max()
            assert err <= 1e-4 * np.abs(want[a:b]).max(), (a, err)
