"""The smoke check compares a layer run with ordinary launches against one with programmatic launches, whichever mode the
process is in, and leaves that mode as it found it."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("before", [True, False])
def test_smoke_runs_both_launch_modes_and_restores_the_callers(before, monkeypatch):
    import __graft_entry__ as entry
    from tensorfold_b200 import _lib, moe

    def mode() -> bool:
        now = _lib.set_pdl(False)
        _lib.set_pdl(now)
        return now

    seen = []
    for name in ("moe", "run"):
        monkeypatch.setattr(moe, name, lambda *a, call=getattr(moe, name), name=name, **k:
                            (seen.append((name, mode())), call(*a, **k))[1])
    was = _lib.set_pdl(before)
    try:
        entry.smoke()
        assert mode() == before
    finally:
        _lib.set_pdl(was)
    assert seen[0] == ("moe", False) and ("run", True) in seen and ("run", False) not in seen
