"""The block selection of the decoding step where it can go wrong: fewer columns than a warp, several per lane, more equal
columns than the ranking holds (64), as many blocks asked for as there are."""
import pytest
import torch

import recipe
from test_gpu_decode import build, steps
from util import assert_close_bf16, assert_close_f32

pytestmark = pytest.mark.gpu


# Both sides run the decoding kernel, in the layer's one call and between the layer's modules: what is compared here is what the two
# forms of a step hand it.  Its picks are compared with picks computed apart in test_gpu_decode_picks.py.
# (cache length, selected blocks of 64, equal scores everywhere, dtype): 1, 2, 32, 33, 65 and 102 columns
@pytest.mark.parametrize('n, nsel, equal, dtype', [(66, 4, False, torch.float32), (130, 2, False, torch.bfloat16),
                                                   (2050, 16, False, torch.float32), (2114, 16, True, torch.float32),
                                                   (4162, 1, False, torch.bfloat16), (4162, 4, True, torch.bfloat16),
                                                   (6530, 16, True, torch.float32), (6530, 16, False, torch.float32)])
def test_steps_select_what_the_selection_operator_selects(n, nsel, equal, dtype):
    layer = build(dtype, 4, 2, 64, nsel=nsel, window=40)
    if equal:      # every compressed key is the bias of its network: all blocks score alike and the lowest are taken
        layer.k_compress[-1].weight.zero_()
    x = recipe.randn((2, n, 256), 5).to(dtype).to('cuda')
    tokens = recipe.randn((2, 3, 256), 6).to(dtype).to('cuda')
    with torch.no_grad():
        _, cache = layer(x, return_cache=True)
        got, _ = steps(layer, tokens, cache)
        hook = layer.combine_heads.register_forward_hook(lambda *_: None)
        want, _ = steps(layer, tokens, cache)
        hook.remove()
    (assert_close_f32 if dtype == torch.float32 else assert_close_bf16)(got, want.float().cpu(), 'outputs')
