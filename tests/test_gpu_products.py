"""The grouped matrix products of a layer step against products in 64 bits: edges of the 128 x 64 (128 x 128) tiles and of the
K steps of 64, rows that are no whole 16-byte pieces, empty sums, a second part, mask and column sums."""
import pytest
import torch

from native_sparse_attention_pytorch_b200 import _lib, ops

pytestmark = pytest.mark.gpu
F32, BF16 = torch.float32, torch.bfloat16
NT, NN, TN = 0, 1, 2


def operands(op, m, n, k, dtype, gen):
    a = torch.randn((k, m) if op == TN else (m, k), device='cuda', generator=gen).to(dtype)
    b = torch.randn((n, k) if op == NT else (k, n), device='cuda', generator=gen).to(dtype)
    return a, b


def exact(op, a, b):
    a, b = a.double(), b.double()
    return (a.t() if op == TN else a) @ (b.t() if op == NT else b)


def together(tasks, cols=0, split=0):
    out = _lib.host().products_together(tasks, ops._status_word(torch.device('cuda', 0)), cols, split)
    ops.check_device_status()
    return list(zip(out[::2], out[1::2]))


# groups of (op, m, n, k, options)
GROUPS = [
    [(NT, 62, 1024, 512, ''), (NT, 62, 24, 512, '')],
    [(NN, 129, 65, 63, ''), (TN, 127, 64, 65, ''), (NT, 1, 1, 1, ''), (NN, 128, 128, 64, '')],
    [(NN, 300, 200, 40, 'm'), (TN, 40, 200, 300, ''), (NT, 7, 33, 1000, '')],
    [(NN, 513, 96, 512, '2'), (TN, 12, 96, 513, ''), (TN, 256, 72, 513, '')],
    [(TN, 40, 72, 0, ''), (NT, 0, 16, 8, ''), (NT, 5, 9, 17, '')],
    [(NT, 2048, 1500, 1024, ''), (TN, 1024, 520, 2048, '')],
    [(TN, 136, 200, 4100, ''), (NN, 65, 130, 200, 'm')],
]


# what the launch chooses by itself, and every width of a tile and number of CTAs that share one
@pytest.mark.parametrize('dtype,cols,split', [(F32, 0, 0), (BF16, 0, 0), (F32, 64, 2), (F32, 128, 1), (F32, 128, 8), (BF16, 64, 4)])
@pytest.mark.parametrize('group', GROUPS)
def test_grouped_products(group, dtype, cols, split):
    gen = torch.Generator('cuda').manual_seed(1)
    tasks, want = [], []
    for op, m, n, k, opt in group:
        a, b = operands(op, m, n, k, dtype, gen)
        c = exact(op, a, b)
        size = exact(op, a.abs(), b.abs())
        act = a2 = b2 = None
        if '2' in opt:
            a2, b2 = operands(op, m, n, 24, dtype, gen)
            c, size = c + exact(op, a2, b2), size + exact(op, a2.abs(), b2.abs())
        if 'm' in opt:
            act = torch.randn(m, n, device='cuda', generator=gen).relu().to(dtype)
            c = c * (act > 0)
        tasks.append((op, a, b, act, a2, b2))
        want.append((c, size))
    for (got, sums), (c, size), task in zip(together(tasks, cols, split), want, tasks):
        # fp32: a few units in the last place of the sum of magnitudes; bf16: one rounding of the result on top
        err = (got.double() - c).abs()
        bound = size * 2.0 ** -21 + 1e-30 + (c.abs() * 2.0 ** -8 if dtype == BF16 else c.abs() * 2.0 ** -23)
        assert bool((err <= bound).all()), float((err - bound).max())
        if task[3] is None:
            continue
        # the sums are of the stored values, in fp32
        total, reach = got.double().sum(0), got.double().abs().sum(0)
        assert bool(((sums.double() - total).abs() <= reach * 2.0 ** -20 + 1e-30).all())


def test_values_that_do_not_split_into_bf16_terms():
    """Infinities, NaN and values that round to infinity in bf16 give what fp32 gives; the tiles beside theirs are untouched."""
    gen = torch.Generator('cuda').manual_seed(2)
    a, b = operands(NT, 200, 100, 70, F32, gen)
    a[3, 5] = float('inf')
    a[150, 60] = float('nan')
    b[90, 7] = 3.4e38
    b[91] = 0.
    b[91, 5] = 1.
    got = together([(NT, a, b, None, None, None)])[0][0]
    want = a.double() @ b.double().t()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isposinf(), want.float().isposinf())
    fine = want.float().isfinite()
    size = a.double().abs() @ b.double().abs().t()
    assert bool(((got.double() - want).abs() <= size * 2.0 ** -21)[fine].all())
