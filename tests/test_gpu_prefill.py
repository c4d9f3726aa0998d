"""A prompt in one pass (nnb200_gpt_prefill) against the same tokens one at a time (nnb200_gpt_forward_step, which
test_gpu_decode.py holds against the reference): the last logits, and the logits of a token behind the cache it left."""
import numpy as np
import pytest

from oracle import gpt_oracle as go
from tests.golden_io import rel_err

pytestmark = pytest.mark.gpu


def _trainer(nnb, vocab, d, heads, layers, ff, seq, act, norm, pos, precision):
    tr = nnb.GptTrainer(nnb.GptConfig(vocab, d, heads, layers, ff, seq, 1, act, norm, pos, precision))
    tr.load_params(go.init_params(go.GptConfig(vocab, d, heads, layers, ff, seq, 1, act, norm, pos), 5, std=0.05))
    return tr


# (heads, head size, window, first part, second part): edges of the 64-row tiles, the shortest pass, a prompt longer than one
# pass takes (1024 rows), a second prompt behind a first, a head size that only the single-token kernels take
SHAPES = [(2, 32, 80, 8, 0), (3, 64, 200, 63, 65), (1, 128, 131, 129, 0), (2, 16, 1100, 1050, 0), (5, 64, 300, 1, 260), (2, 24, 40, 20, 9)]


@pytest.mark.parametrize("heads,dk,seq,n0,n1", SHAPES)
@pytest.mark.parametrize("act,norm,pos", [(0, 0, 0), (1, 1, 2), (1, 1, 3), (1, 0, 1)])
@pytest.mark.parametrize("precision", [0, 1])
def test_prefill_equals_single_steps(heads, dk, seq, n0, n1, act, norm, pos, precision):
    from tests.gpu_util import nnb
    import torch
    tr = _trainer(nnb, 72, heads * dk, heads, 2, 104, seq, act, norm, pos, precision)
    tokens = [int(t) for t in np.random.default_rng(3).integers(0, 72, n0 + n1 + 1)]
    n = n0 + n1
    for i, t in enumerate(tokens[:n]):
        want = tr.forward_step(t, i, i)
    want = want.clone()
    behind = tr.forward_step(tokens[n], n, n).clone()
    tr._decode_ws[:2 * 2 * 4 * seq * heads * dk].zero_()         # the cache of two layers
    got = tr.prefill(tokens[:n0])
    if n1:
        got = tr.prefill(tokens[n0:n], n0)
    got = got.clone()
    after = tr.forward_step(tokens[n], n, n).clone()
    torch.cuda.synchronize()
    # fp32 sums of up to 1050 terms in another order through two layers: n eps / 2 at most, their square root in practice
    assert rel_err(got.cpu().numpy(), want.cpu().numpy()) < 1e-5
    assert rel_err(after.cpu().numpy(), behind.cpu().numpy()) < 1e-5


def test_prefill_refuses_rows_outside_the_window():
    from tests.gpu_util import nnb
    tr = _trainer(nnb, 72, 32, 1, 1, 64, 16, 1, 1, 2, 0)
    for tokens, cur in (([], 0), ([1] * 17, 0), ([1] * 8, 9), ([1], -1)):
        with pytest.raises(ValueError):
            tr.prefill(tokens, cur)


@pytest.mark.parametrize("n", [8, 511, 513, 1100])
def test_prompt_in_page_locked_memory_may_be_overwritten_after_the_call(n):
    """The ids are read before nnb200_gpt_prefill returns, also from page-locked memory and behind work still queued."""
    import ctypes as C
    import torch
    from tests import gpu_util as g
    tr = _trainer(g.nnb, 72, 32, 1, 1, 64, 1104, 1, 1, 2, 0)
    ids = np.random.default_rng(n).integers(0, 72, n).astype(np.int32)
    want = tr.prefill(ids).clone()
    buf = torch.from_numpy(ids.copy()).pin_memory()
    busy = torch.randn(4096, 4096, device="cuda")
    for _ in range(20):                                          # milliseconds of work in front of the call
        busy = busy @ busy * 1e-3
    ws, logits = tr._decode_state()
    g.call("nnb200_gpt_prefill", C.byref(tr._c), g.ptr(tr.params), g.ptr(tr.shadow), g.ptr(ws), C.c_void_p(buf.data_ptr()), n, 0, g.ptr(logits), g.stream())
    buf.fill_(1)
    torch.cuda.synchronize()
    assert torch.equal(logits, want)


def test_ids_beyond_32_bits_are_what_single_steps_make_of_them():
    """A prompt of ids no 32-bit integer holds, which steps take as zero rows (or modulo 2^32), and of 0-d tensors."""
    import torch
    from tests.gpu_util import nnb
    tr = _trainer(nnb, 72, 32, 1, 1, 64, 16, 1, 1, 2, 0)
    tokens = [3, 2 ** 31 + 5, 7, 2 ** 32 + 9, -1, 70, 2 ** 40, 1, torch.tensor(5), 6]
    for i, t in enumerate(tokens):
        want = tr.forward_step(int(t), i, i)
    want = want.clone()
    assert rel_err(tr.prefill(tokens).cpu().numpy(), want.cpu().numpy()) < 1e-5
    assert len(tr.generate(tokens[:8] + [int(tokens[8])], 2, temperature=0.0)) == 2
