"""The dense tensor falls back to one task per quartet only where the ranges are too many."""
import types

import pytest

from gaussium_gb300 import dropin, engine


def test_only_too_many_ranges_falls_back(monkeypatch):
    planned = []

    class Planned(Exception):
        pass

    def quartets(*a, **kw):
        planned.append(1)
        raise Planned
    monkeypatch.setattr(engine, "DeviceShells", lambda sb, d: types.SimpleNamespace(device="cpu"))
    monkeypatch.setattr(engine, "QuartetBatch", quartets)
    sb = types.SimpleNamespace(nbf=2, nshell=2)

    def refuse(error):
        def unique(*a, **kw):
            raise error
        monkeypatch.setattr(engine, "UniqueQuartets", unique)
    refuse(ValueError("too many primitive pairs for one PairSet"))
    with pytest.raises(ValueError, match="primitive pairs"):
        dropin.dense_eri(sb)
    assert not planned
    refuse(engine.TooManyRanges("ranges"))
    with pytest.raises(Planned):
        dropin.dense_eri(sb)
