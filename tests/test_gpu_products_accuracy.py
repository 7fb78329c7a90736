"""Rounding of the grouped fp32 products against 64 bits, where it adds up: sums whose terms have one sign.  The tensor cores cut
their sums towards zero, which for such sums is a bias; it must not make the products less exact than the library's."""
import pytest
import torch

from native_sparse_attention_pytorch_b200 import _lib, ops

pytestmark = pytest.mark.gpu
NT, TN = 0, 2
KINDS = {'one sign': lambda t: t.uniform_(), 'behind a ReLU': lambda t: t.normal_().relu_(), 'normal': lambda t: t.normal_()}


@pytest.mark.parametrize('kind', KINDS)
@pytest.mark.parametrize('op, m, n, k, cols, split', [
    (NT, 384, 512, 512, 0, 0), (NT, 384, 512, 2048, 128, 1), (NT, 384, 512, 4096, 64, 1), (NT, 1024, 1024, 2048, 0, 0),
    (TN, 256, 512, 4096, 0, 0), (TN, 512, 512, 15000, 0, 0), (NT, 130, 70, 64, 0, 0), (TN, 62, 200, 35840, 0, 0)])
def test_products_are_as_exact_as_the_librarys(op, m, n, k, cols, split, kind):
    a = torch.empty((k, m) if op == TN else (m, k), device='cuda')
    b = torch.empty((k, n) if op == TN else (n, k), device='cuda')
    torch.manual_seed(k + m)
    a, b = KINDS[kind](a), KINDS[kind](b)
    got = _lib.host().products_together([(op, a, b, None, None, None)], ops._status_word(a.device), cols, split)[0]
    ops.check_device_status()
    a, b = (a.t(), b) if op == TN else (a, b.t())
    want = a.double() @ b.double()
    error = lambda c: float((c.double() - want).norm() / want.norm())
    # one unit in the last place of fp32, 2^-23: below it the two differ by how the last roundings fall
    assert error(got) <= max(error(a @ b), 2.0 ** -23), (error(got), error(a @ b))
