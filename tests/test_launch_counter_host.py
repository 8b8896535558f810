"""Launches counted per library call (a library that launches nothing stands in)."""
import pytest

pytest.importorskip("torch")


class _Nothing:
    def __getattr__(self, name):
        return lambda *args: 0


@pytest.mark.parametrize("name,args,launches", [
    ("xrh_slice_grouped", (None, 3, 10, 0, None, None), 1),        # K-contiguous operands: the digits alone
    ("xrh_slice_grouped", (None, 3, 10, 4, None, None), 2),        # transposed ones: their row maxima first
    ("xrh_gemm_sliced_grouped", (None,) * 9, 2),                   # the tiles, then their marked elements
    ("xrh_coeff_digits", (None,) * 4, 2), ("xrh_coeff_rows", (None,) * 4, 1),
    ("xrh_zero", (None,) * 3, 0), ("xrh_coeff_digit_ctas", (5,), 0)])
def test_launches_of_a_call(monkeypatch, name, args, launches):
    from qodeapplications_gb300 import _lib
    monkeypatch.setattr(_lib, "lib", _Nothing)
    monkeypatch.setattr(_lib.LaunchCounter, "count", 0)
    _lib.call(name, *args)
    assert _lib.LaunchCounter.count == launches
