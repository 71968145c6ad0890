"""The ensemble's autotuner times only shapes that differ in their launches: the strip CTAs
per SM, which no launch reads, are neither timed nor adopted nor the bar that later
candidates have to clear.  Timings are scripted, on the CPU."""
import pytest
import torch

from zoomy_b200.ensemble import Ensemble

SIDES = [40, 100, 200, 300]


class Scripted(Ensemble):
    """Every timing of a shape comes from ``price(shape, nth timing of it)``."""

    price = None

    def _build_table(self):
        pass

    def init(self, t0=0.0):
        pass

    def _time_shape(self, saved_q, steps):
        key = str(self.shape()["edge_rows"] + self.shape()["interior_rows"])
        self.seen[key] = self.seen.get(key, 0) + 1
        return self.price(self.shape(), self.seen[key])


def tuned(price, dtype="float32"):
    ens = Scripted(SIDES, [0.0] * len(SIDES), dtype=dtype)
    ens.Q, ens.seen, ens.price = torch.zeros(4), {}, price
    before = ens.shape()
    return ens, before, ens.autotune(steps=2)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_a_shape_is_timed_once(dtype):
    ens, before, res = tuned(lambda shape, nth: 1.0, dtype)
    assert set(ens.seen.values()) == {1}
    assert ens.tuned_shape == before
    assert len(res) == len(ens.seen) + sum(k.startswith("ctas_per_sm=") for k in res)


def test_noise_between_equal_launches_hides_no_better_shape():
    # a second timing of the same launch comes out 30 % lower; 16 boundary rows in the first
    # class are 10 % faster than the untuned shape
    def price(shape, nth):
        ms = 0.9 if shape["edge_rows"][0] == 16 else 1.0
        return ms * (0.7 if nth > 1 else 1.0)

    ens, before, res = tuned(price)
    assert ens.tuned_shape["edge_rows"][0] == 16
    assert ens.tuned_shape["ctas_per_sm"] == before["ctas_per_sm"]
    assert ens.tuned_ms == 0.9 == min(res.values())
