"""Tuner variants: every ring shape and register bound that the tuner has taken is
still read by the kernels' sources, and a name that is not is refused instead of
being measured as if it did something."""
import pytest

from hodlrnd_gb300 import tune


def test_every_knob_is_read():
    knobs = {f"{k}_{v}" for k in "ZPSL" for v in ("STAGES", "BYTES")} | {"L_COLS", "S_MINB", "P_MINB", "L_MINB",
                                                                         "Z_ITEM_BYTES", "SMALL_ITEM_BYTES"}
    assert knobs <= tune.macros()
    for v in tune.DEFAULT_VARIANTS.values():
        assert set(v) <= tune.macros()


def test_unknown_names_are_refused():
    with pytest.raises(ValueError, match="Q_BYTES"):
        tune._variant_lib("typo", {"Q_BYTES": 1})
