"""Grouped fp32 products with infinities and NaN: the results of fp32 arithmetic, in the time of any other product."""
import pytest
import torch

from native_sparse_attention_pytorch_b200 import _lib, ops

pytestmark = pytest.mark.gpu
NT, NN, TN = 0, 1, 2
INF, NAN = float('inf'), float('nan')


def product(op, a, b, cols=0, split=0, act=None):
    got = _lib.host().products_together([(op, a, b, act, None, None)], ops._status_word(a.device), cols, split)[0]
    ops.check_device_status()
    return got


@pytest.mark.parametrize('op, m, n, k, cols, split', [(NT, 200, 100, 70, 0, 0), (TN, 150, 130, 300, 128, 1), (NN, 130, 70, 700, 64, 8), (TN, 64, 64, 2000, 64, 4)])
def test_results_are_those_of_fp32(op, m, n, k, cols, split):
    gen = torch.Generator('cuda').manual_seed(k)
    a, b = (torch.randn(s, k, device='cuda', generator=gen) for s in (m, n))
    a[3, 5] = INF
    a[3, k // 2] = -INF                       # cancels for some columns, adds up for others
    a[4, k - 1] = NAN
    a[m - 1, 8] = -INF
    b[7, 8] = 0.                              # meets that infinity
    b[9] = -INF
    b[:, 5] = b[:, 5].abs()
    a[20:30] = torch.randn(10, k, device='cuda', generator=gen) * 1e-30
    want = a.double() @ b.double().t()
    size = a.double().abs() @ b.double().abs().t()
    ins = (a.t().contiguous() if op == TN else a, b if op == NT else b.t().contiguous())
    got = product(op, *ins, cols, split)
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.isposinf(), want.isposinf()) and torch.equal(got.isneginf(), want.isneginf())
    fine = want.isfinite()
    assert bool(((got.double() - want).abs() <= size * 2.0 ** -21 + 1e-44)[fine].all())


def test_they_take_no_longer():
    gen = torch.Generator('cuda').manual_seed(1)
    a, b = (torch.randn(1024, 1024, device='cuda', generator=gen) for _ in range(2))
    times = {}
    for name, value in (('finite', 1.), ('one infinity', INF), ('one NaN', NAN)):
        a[5, 9] = value
        marks = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        for _ in range(3):
            product(NT, a, b)
        runs = []
        for _ in range(5):
            torch.cuda._sleep(1000000)
            marks[0].record()
            for _ in range(5):
                _lib.host().products_together([(NT, a, b, None, None, None)], ops._status_word(a.device), 0, 0)
            marks[1].record()
            torch.cuda.synchronize()
            runs.append(marks[0].elapsed_time(marks[1]))
        times[name] = sorted(runs)[2]
    # (twenty times as long where they were computed apart)
    assert max(times.values()) < 2 * times['finite'], times
