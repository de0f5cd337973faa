"""The smoke run passes on a checkout without the reference's kernel."""
import pytest

pytestmark = pytest.mark.gpu


def test_smoke_without_the_reference_kernel(engine, monkeypatch, capsys):
    import oracle.ref
    from __graft_entry__ import smoke

    def missing(*args, **kw):
        raise FileNotFoundError("not built here")

    monkeypatch.setattr(oracle.ref, "RefKernel", missing)
    smoke()
    out = capsys.readouterr().out
    assert "not built here" in out and "smoke ok" in out
