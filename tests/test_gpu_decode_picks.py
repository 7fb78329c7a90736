"""The blocks a decoding step selects, against picks and attention computed from the logits alone in 64 bits.  The compressed keys have
one component, so that every block's logit is given; only the selected branch has a gate, so that the picks are what the output
shows."""
import pytest
import torch

from util import assert_close_bf16, assert_close_f32

from native_sparse_attention_pytorch_b200 import ops

pytestmark = pytest.mark.gpu
DEV, NEVER = 'cuda', -200.      # a logit whose probability is zero beside any other


def step_and_picks(logits, nsel, dtype, heads=2, d=64, cpf=1, stride=4, window=3):
    cols, block = len(logits), stride * cpf
    t = cols * block + 3
    gen = torch.Generator(DEV).manual_seed(cols + nsel)
    randn = lambda *s: torch.randn(s, device=DEV, generator=gen).to(dtype)
    qr, keys, vals = randn(1, heads, d), randn(1, 1, t, d), randn(1, 1, t, d)
    q, ck = torch.zeros(1, heads, d, device=DEV, dtype=dtype), torch.zeros(1, 1, cols * cpf, d, device=DEV, dtype=dtype)
    q[..., 2] = 1.
    ck[0, 0, :, 2] = (logits * 8).repeat_interleave(cpf).to(DEV, dtype)                # 8 = sqrt(d)
    assert torch.equal(ck[0, 0, ::cpf, 2].cpu().double(), logits * 8)
    gates = torch.tensor([0., 1., 0.], device=DEV, dtype=dtype).expand(1, heads, 3).contiguous()
    mem = torch.zeros(2, 1, 1, d, device=DEV, dtype=dtype)
    got = ops.decode_step(q, qr, keys, vals, ck, randn(1, 1, cols * cpf, d), mem[0], mem[1], gates, stride=stride, block=block,
                          num_selected=nsel, window=window)
    p = torch.cat((torch.tensor([-1e3], dtype=torch.double), logits)).softmax(0)[1:]
    order = torch.sort(logits, descending=True, stable=True).indices                   # equal ones: the lower column first
    picks = [j for j in order[:nsel].tolist() if p[j] > 1e-10]
    rows = torch.cat([torch.arange(j * block, (j + 1) * block) for j in picks] + [torch.arange((t - 1) // block * block, t)]).to(DEV)
    k, v = keys[0, 0, rows].double(), vals[0, 0, rows].double()
    want = (qr[0].double() @ k.t() * d ** -0.5).softmax(-1) @ v
    return got, want.reshape(1, -1), picks


def spread(n, seed, step=0.25):
    """n different logits, `step` apart, in any order."""
    return torch.randperm(n, generator=torch.Generator().manual_seed(seed)).double() * step


def one_lane(cols, seed):
    """All that count lie 32 apart: the maxima of the other lanes bound nothing, and every column is a candidate."""
    x = torch.full((cols,), NEVER, dtype=torch.double)
    at = torch.arange(5, cols, 32)
    x[at] = spread(len(at), seed)
    return x


def tied(cols, ties, above, seed):
    """`above` columns are larger than `ties` equal ones, the rest smaller; in any order."""
    place = torch.randperm(cols, generator=torch.Generator().manual_seed(seed))
    x = spread(cols, seed) * 0.01 - 4.
    x = (x * 64).round() / 64
    x[place[:ties]] = 2.
    x[place[ties:ties + above]] = 3. + torch.arange(above).double() * 0.25
    return x


CASES = {
    'one column': lambda: (spread(1, 1), 4),
    'fewer columns than a warp': lambda: (spread(31, 2), 16),
    'as many as asked for': lambda: (spread(32, 3), 32),
    'one more than a warp': lambda: (spread(33, 4), 32),
    'more than a warp': lambda: (spread(60, 5), 16),
    'one pick': lambda: (spread(61, 6), 1),
    'one lane, fewer than asked for': lambda: (one_lane(300, 7), 16),
    'one lane, bisection': lambda: (one_lane(1300, 8), 16),
    'one lane, bisection for one more than it has': lambda: (one_lane(32 * 7, 9), 8),
    'few ties': lambda: (tied(200, 10, 5, 10), 8),
    'ties in more columns than are ranked': lambda: (tied(400, 150, 5, 11), 16),
    'nothing but ties': lambda: (torch.zeros(130, dtype=torch.double), 16),
    'ties, all below the picks': lambda: (tied(400, 150, 16, 12), 16),
    'nothing that counts': lambda: (torch.cat((torch.tensor([5.], dtype=torch.double), torch.full((99,), NEVER, dtype=torch.double))), 16),
}


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
@pytest.mark.parametrize('heads, d, cpf', [(2, 64, 1), (8, 64, 4)])
@pytest.mark.parametrize('case', CASES)
def test_picks(case, heads, d, cpf, dtype):
    logits, nsel = CASES[case]()
    if dtype == torch.bfloat16:
        logits = (logits * 8).to(dtype).double() / 8      # (what a key can hold; may tie)
    got, want, picks = step_and_picks(logits, nsel, dtype, heads, d, cpf)
    assert len(picks) <= nsel
    (assert_close_f32 if dtype == torch.float32 else assert_close_bf16)(got, want.float().cpu(), f'{case}: {picks}')
