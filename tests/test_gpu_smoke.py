"""The smoke entry point, with the reference's code as its oracle where that is built and its CPU restatement elsewhere."""
import pytest

pytestmark = pytest.mark.gpu


def test_smoke(built, capsys):
    import __graft_entry__
    __graft_entry__.smoke()
    assert "smoke ok" in capsys.readouterr().out
