"""The quantization of an input that several layers share, without a GPU: the quantizers and products are replaced by
functions that only keep the row counts."""
import itertools
from types import SimpleNamespace

import pytest
import torch

from bitlattice_b200 import backend, parallel


@pytest.fixture
def counted(monkeypatch):
    """Operands are the matrices they were made from; a product has an operand's rows and a weight's features."""
    made = []

    def act_operand(x2, recipe):
        made.append(tuple(x2.shape))
        return SimpleNamespace(packed=x2, global_scale=torch.ones(1))

    monkeypatch.setattr(backend, "_act_operand", act_operand)
    monkeypatch.setattr(backend, "weight_operand", lambda w: w)
    monkeypatch.setattr(backend, "fp4_mm", lambda a, w, dtype, add_to=None: torch.zeros(a.packed.shape[0], w.shape[0]))
    backend.clear_shared()
    yield made
    backend.clear_shared()


LAYERS = {
    "linear": lambda x, w, recipe: backend.nvfp4_linear(x, w, None, recipe),
    "shared input": lambda x, w, recipe: parallel.SharedInputFp4Linears.apply(x, recipe, w)[0],
    "token parallel": lambda x, w, recipe: parallel.TokenParallelFp4Linear.apply(
        x, SimpleNamespace(group=None, operand=lambda w: w), recipe, w)[0],
}


@pytest.mark.parametrize("rows", [13, 16, 32])
@pytest.mark.parametrize("first,second", list(itertools.permutations(LAYERS, 2)))
def test_layers_share_one_operand_in_any_order(counted, first, second, rows):
    """Layers with frozen weights on one input whose rows fill no multiple of 16: whichever comes first makes the
    operand, and the others take it as it is."""
    x, w = torch.randn(rows, 64), torch.randn(48, 64)
    for name in (first, second):
        assert LAYERS[name](x, w, backend.Fp4Recipe()).shape == (rows, 48)
    assert counted == [(rows, 64)]


def test_shared_input_function_takes_the_weights_after_the_recipe(counted, monkeypatch):
    """Its arguments are the input, the recipe and the weights; x^T is made when autograd records, and only then."""
    transposed = []
    monkeypatch.setattr(backend, "_input_operands", lambda x, recipe, row=True, site=None: (
        backend._act_operand(x, recipe), transposed.append(True)))
    x, ws = torch.randn(13, 64), [torch.randn(n, 64, requires_grad=True) for n in (48, 32)]
    with torch.no_grad():
        ys = parallel.SharedInputFp4Linears.apply(x, backend.Fp4Recipe(), *ws)
    assert [tuple(y.shape) for y in ys] == [(13, 48), (13, 32)] and not transposed and not ys[0].requires_grad
    ys = parallel.SharedInputFp4Linears.apply(x, backend.Fp4Recipe(), *ws)
    assert len(transposed) == 1 and all(y.requires_grad for y in ys)
