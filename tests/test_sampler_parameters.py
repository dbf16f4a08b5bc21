"""What the sampler takes as a step's parameters: lists of numbers in one conversion, any other sequence as a tensor would take
it; what is no number, is negative or does not fit is refused."""
import math
from array import array

import numpy as np
import pytest
import torch

from flexengine_b200.sampling import Sampler

LOGITS = torch.zeros(2, 8)
GOOD = ([0.5, 1.0], [0, 3], [1, 2], [3, 4])


class Seen:
    def sample(self, logits, temperature, top_k, seed, draw):
        assert (temperature.dtype, top_k.dtype, seed.dtype, draw.dtype) == (torch.float32, torch.int32, torch.int64, torch.int64)
        return [temperature.tolist(), top_k.tolist(), seed.tolist(), draw.tolist()]


def taken(*parameters):
    return Sampler(Seen()).sample_on_device(LOGITS, *parameters)


def changed(at, values):
    return GOOD[:at] + (values,) + GOOD[at + 1:]


@pytest.mark.parametrize("at,values", [(0, [None, 1.0]), (0, ["0.5", 1.0]), (0, [[0.5], [1.0]]), (1, [None, 3]), (1, ["1", 3]),
                                       (1, [[0], [1]]), (2, [None, 2]), (2, ["7", 2])])
def test_what_is_no_number_is_refused(at, values):
    with pytest.raises((TypeError, ValueError)):
        taken(*changed(at, values))


@pytest.mark.parametrize("at,values", [(0, [0.5, -1.0]), (0, [math.nan, -1.0]), (0, np.array([0.5, -1.0])), (0, torch.tensor([0.5, -1.0])),
                                       (1, [0, -1]), (1, [-0.5, 3]), (1, np.array([0, -1])), (1, (3, -2))])
def test_negative_parameters_are_refused(at, values):
    with pytest.raises(ValueError, match="must be >= 0"):
        taken(*changed(at, values))


@pytest.mark.parametrize("at,values,error", [(1, [2 ** 70, 1], ValueError), (2, [2 ** 63, 2], ValueError), (1, [math.nan, 1], RuntimeError),
                                             (1, [0, 1, 2], RuntimeError), (2, [1, 2, 3], RuntimeError)])
def test_what_does_not_fit_is_refused_as_a_tensor_refuses_it(at, values, error):
    with pytest.raises(error):
        taken(*changed(at, values))


@pytest.mark.parametrize("at,values,want", [
    (0, (0.25, 2), [0.25, 2.0]), (0, np.array([0.5, 1.0], dtype=np.float32), [0.5, 1.0]), (0, torch.tensor([0.5, 1.0], dtype=torch.bfloat16), [0.5, 1.0]),
    (0, [torch.tensor(0.5), 1.0], [0.5, 1.0]), (0, [1e39, 1.0], [math.inf, 1.0]), (0, [1e-60, 1.0], [0.0, 1.0]), (0, [True, 0.5], [1.0, 0.5]),
    (1, (2, 5), [2, 5]), (1, [1.7, 3], [1, 3]), (1, torch.tensor([4, 5]), [4, 5]), (1, [7], [7, 7]), (1, [2 ** 32 + 3, 1], [3, 1]),
    (2, range(5, 7), [5, 6]), (2, [-1, 2 ** 63 - 1], [-1, 2 ** 63 - 1]), (3, np.array([8, 9]), [8, 9]), (3, [6], [6, 6])])
def test_numbers_of_any_kind_arrive(at, values, want):
    got = taken(*changed(at, values))
    assert got[at] == want
    assert all(got[i] == GOOD[i] for i in range(4) if i != at)


def test_greedy_rows_take_whatever_stands_beside_them():
    for top_ks in ([2 ** 70, 1], [0], [1, 2, 3], (5, 5), [1, 2, None], iter([1, 2])):
        assert taken([0.0, 0], top_ks, [1], [3]) == [[0.0, 0.0], [0, 0], [0, 0], [0, 0]]
    assert Sampler(Seen()).sample_on_device(torch.zeros(0, 8), [], [], [], []) == [[], [], [], []]


@pytest.mark.parametrize("at,wrong,error", [(0, array("d", [0.5, 1.0]), TypeError), (0, [0.5, 1.0], TypeError), (1, array("q", [0, 3]), TypeError),
                                            (2, array("i", [1, 2]), TypeError), (3, array("Q", [3, 4]), TypeError), (0, array("f", [0.5]), ValueError),
                                            (1, array("i", [0]), ValueError), (2, array("q", [1, 2, 3]), ValueError), (3, array("q"), ValueError)])
def test_listed_parameters_of_another_length_or_type_are_refused_before_they_are_read(at, wrong, error, monkeypatch):
    from flexengine_b200 import ops
    taken = []
    for name, value in (("_need_cuda", lambda *t: None), ("_core", lambda: None), ("_stream", lambda: None), ("_run", lambda *args: taken.append(args))):
        monkeypatch.setattr(ops, name, value)
    good = (array("f", [0.5, 1.0]), array("i", [0, 3]), array("q", [1, 2]), array("q", [3, 4]))
    ops.sample_listed(LOGITS, *good)
    assert len(taken) == 1
    with pytest.raises(error):
        ops.sample_listed(LOGITS, *good[:at], wrong, *good[at + 1:])
    assert len(taken) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("vocab,pitch", [(32000, 32000), (4099, 4103)])
@pytest.mark.parametrize("rows", [1, 42, 43, 64, 84, 85, 168, 169])
def test_lists_give_the_tokens_of_tensors(rows, vocab, pitch):
    """Parameters as plain lists (with the launch, as far as they fit into one) and the same numbers as tensors, row for row; rows on
    16-byte boundaries and not."""
    from flexengine_b200 import ops
    dev = "cuda:0"
    gen = torch.Generator(device=dev).manual_seed(rows)
    logits = torch.empty(rows, pitch, device=dev)[:, :vocab].copy_(torch.randn(rows, vocab, device=dev, generator=gen) * 3)
    temperatures = [(0.0, 0.7, 1, 1.3)[(i + 1) % 4] for i in range(rows)]
    top_ks = [(0, 40, 1, 2000, vocab + 7)[i % 5] for i in range(rows)]
    seeds = [(i * 0x9E3779B97F4A7C15 + 77) % 2 ** 64 - 2 ** 63 for i in range(rows)]
    draws = [i * i if i % 3 else 2 ** 62 + i for i in range(rows)]
    got = Sampler().sample_on_device(logits, temperatures, top_ks, seeds, draws)
    want = ops.sample(logits, torch.tensor(temperatures, dtype=torch.float32, device=dev), torch.tensor(top_ks, dtype=torch.int32, device=dev),
                      torch.tensor(seeds, device=dev), torch.tensor(draws, device=dev))
    assert torch.equal(got, want)
    if rows > 1:          # each parameter counts: with two of them exchanged the tokens are others
        other = Sampler().sample_on_device(logits, temperatures, top_ks, draws, seeds)
        assert not torch.equal(other, want)
