"""First use of the operators from several threads.  CPU only: no application is launched."""
import pytest

pytest.importorskip("torch")


def test_table_is_filled_last(monkeypatch):
    """A thread that finds the dtype table filled skips the set-up, so everything else that an
    application needs is there before the table is."""
    from summationbyparts_b200 import operators

    class Table(dict):
        def update(self, *a, **kw):
            assert callable(getattr(operators, "_raw_stream", None))
            super().update(*a, **kw)

    monkeypatch.setattr(operators, "_DTYPES", Table())
    monkeypatch.delattr(operators, "_raw_stream", raising=False)
    operators._setup()
    assert len(operators._DTYPES) == 2
