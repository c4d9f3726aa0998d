"""The row kernels of the norms where the row's last vectors go to some lanes only, and the sum of squares at every remainder."""
import ctypes as C

import numpy as np
import pytest

from oracle import gpt_oracle as go
from tests.golden_io import global_rel_err, key_bias_indices

pytestmark = pytest.mark.gpu


# widths around each number of vectors per lane (a lane holds up to four of 4 fp32 or 8 bf16 columns), in heads of 8
@pytest.mark.parametrize("d,precision", [(8, 0), (120, 0), (136, 0), (264, 0), (392, 0), (504, 0),
                                         (8, 1), (248, 1), (264, 1), (520, 1), (776, 1), (1016, 1)])
@pytest.mark.parametrize("norm", [0, 1])
def test_training_step_of_a_width_that_leaves_lanes_empty(d, precision, norm):
    from tests.gpu_util import nnb
    cfg = go.GptConfig(64, d, d // 8, 1, 24, 9, 3, 0, norm, 0)
    params = go.init_params(cfg, 3, std=min(0.1, d ** -0.5))      # attention scores of order one: at 0.1 and width 1016 they reach 10, and so do the effects of a rounding of q or k
    r = np.random.default_rng(d)
    for i, (n, _, _) in enumerate(go.param_shapes(cfg)):
        if n.endswith("gamma") or n.endswith("beta"):
            params[i] = params[i] + (0.2 * r.standard_normal(params[i].shape)).astype(np.float32)
    tokens, labels = (r.integers(0, 64, 27).astype(np.int32) for _ in range(2))
    _, _, want = go.train(cfg, [p.copy() for p in params], [dict(tokens=tokens, labels=labels, mask=None, doc_ids=None)], steps=1, keep_first_grads=True)
    tr = nnb.GptTrainer(nnb.GptConfig(cfg.vocab, d, cfg.heads, 1, 24, 9, 3, 0, norm, 0, precision))
    tr.load_params(params)
    tr.micro_step(tokens, labels)
    got = tr.get_grads()
    # fp32: rounding of sums of up to 504 terms; bf16: about twenty tensors rounded by at most 2^-9 each on the way, partly cancelling
    assert global_rel_err(got, want, key_bias_indices(cfg)) < (1e-5 if precision == 0 else 3e-2)


@pytest.mark.parametrize("n", [1, 3, 4, 1023, 4097, 592 * 256 * 16, 592 * 256 * 16 + 4099])
@pytest.mark.parametrize("offset", [0, 1])
def test_sum_of_squares(n, offset):
    import torch
    from tests import gpu_util as g
    t = torch.randn(n + offset, device="cuda")[offset:]
    scratch = torch.zeros(int(g.call("nnb200_sumsq_scratch_floats")), device="cuda")
    out = torch.zeros(4, device="cuda")
    g.call("nnb200_grad_norm_clip", g.ptr(t), n, C.c_float(0.5), C.c_float(1.0), g.ptr(scratch), g.ptr(out), g.stream())
    # positive terms: sums of at most ~100 per thread and 600 per block, each within eps / 2
    assert np.isclose(float(out[1]), 0.5 * float(t.double().norm()), rtol=1e-5)
