"""Single-token decoding at the edges of its kernels, against the oracle's full forward pass: head sizes of every lane split
(and ones no vector load fits), more cached rows than one round of a cluster takes, rows longer than the staged norm and
than the weights a lane holds, rows no 16-byte load fits.  Weights are bf16 values, so both precisions compute the same."""
import numpy as np
import pytest

from oracle import gpt_oracle as go
from tests.golden_io import rel_err

pytestmark = pytest.mark.gpu

# (heads, head size, d_ff, vocabulary, tokens)
SHAPES = [(2, 6, 20, 33, 20), (1, 30, 36, 40, 9), (4, 24, 96, 64, 300), (2, 64, 2100, 72, 40), (9, 128, 64, 50, 12), (1, 128, 64, 64, 530), (1, 160, 72, 64, 270),
          (3, 32, 100, 4097, 3),
          # several rounds of the cluster: 1024 rows at 512 threads and one vector a lane, 512 at 256 threads or two vectors, 1024 of 64
          (1, 128, 64, 64, 2100), (9, 128, 64, 50, 1100), (1, 160, 72, 64, 1100), (1, 66, 40, 64, 2100), (1, 64, 64, 64, 2100)]


@pytest.mark.parametrize("heads,dk,ff,vocab,n", SHAPES)
@pytest.mark.parametrize("act,norm,pos", [(0, 0, 0), (1, 1, 2), (1, 1, 3)])
@pytest.mark.parametrize("precision", [0, 1])
def test_steps_equal_the_oracle(heads, dk, ff, vocab, n, act, norm, pos, precision):
    from tests import gpu_util as g
    import torch
    d = heads * dk
    cfg = go.GptConfig(vocab, d, heads, 1, ff, n, 1, act, norm, pos)
    params = [g.bf16_round(p) for p in go.init_params(cfg, 9, std=min(0.1, d ** -0.5))]
    tokens = np.random.default_rng(n).integers(0, vocab, n)
    want = go.GptOracle(cfg, [p.copy() for p in params]).forward(tokens.astype(np.float32).reshape(1, n)).T
    tr = g.nnb.GptTrainer(g.nnb.GptConfig(vocab, d, heads, 1, ff, n, 1, act, norm, pos, precision))
    tr.load_params(params)
    got = torch.stack([tr.forward_step(int(t), i, i).clone() for i, t in enumerate(tokens)]).cpu().numpy()
    plain = tr.forward_step(int(tokens[-1]), n - 1, n - 1, graph=False).cpu().numpy()
    assert rel_err(got, want) < 1e-5             # fp32 sums of up to 2100 terms in another order
    assert np.array_equal(plain, got[-1])
