"""BPTT launches where the form and its batch slices depend on more than the
number of neurons: hubs whose staged edges leave room for fewer warps, so that a
slice takes more words; degrees above 256 and nets of more neurons than the
device holds warps, in one slice of any number of words.  The same checks as the
resident launches' (spikes bit for bit, gradients, both settings of the switch)."""
import pytest

from tests import test_bptt_resident_gpu as RES

pytestmark = pytest.mark.gpu

CASES = {
    # name: (N, mean in-degree, max delay, hub in-degree, T, B, ckpt)
    "hub_two_words": (2300, 6, 3, 240, 5, 64, 2),
    "hub_four_words": (1400, 6, 4, 240, 5, 128, 3),
    "hub_no_room": (2200, 5, 2, 240, 4, 256, 2),
    "degree_above_256": (120, 10, 4, 290, 7, 100, 3),
    "degree_above_256_one_word": (120, 10, 4, 290, 7, 30, 0),
    "degree_above_256_eight_words": (90, 10, 4, 290, 6, 256, 4),
    "many_neurons": (5000, 5, 3, 0, 4, 97, 2),
    "many_neurons_six_words": (5000, 5, 3, 0, 3, 170, 2),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_forms(name, monkeypatch):
    monkeypatch.setitem(RES.CASES, name, CASES[name])
    RES.test_shapes(name)
