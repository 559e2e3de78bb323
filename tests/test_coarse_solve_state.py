"""The coarsest level's inverse on demand, with the device work stubbed (CPU only)."""
import pytest


class Owner:
    """What _CoarseSolve asks of its owner."""

    def __init__(self):
        self.formed = 0
        self.build()

    def build(self):
        from loadpath_b200.mg import _CoarseSolve

        self._coarse = _CoarseSolve(self, n=3, chain=object(), v=type("V", (), {"numel": lambda s: 32})())

    def _join_coarse(self):
        pass

    def _band_buffers(self, nt):
        self._coarse["ainv"] = f"inverse {self.formed}"

    def _band_inverse(self):
        self.formed += 1


def test_inverse_is_formed_once():
    ge = Owner()
    assert ge._coarse["ainv"] == ge._coarse["ainv"] == "inverse 0" and ge.formed == 1
    with pytest.raises(KeyError):
        ge._coarse["other"]


def test_solve_of_an_earlier_hierarchy_says_so():
    """A coarse solve kept across a rebuild, or past its owner, has no band to form its inverse from; one that
    had formed it keeps it."""
    ge = Owner()
    kept, used = ge._coarse, None
    ge.build()
    with pytest.raises(RuntimeError, match="hierarchy"):
        kept["ainv"]
    assert ge.formed == 0
    used = ge._coarse
    assert used["ainv"] == "inverse 0"
    ge.build()
    late = ge._coarse
    assert used["ainv"] == "inverse 0"
    del ge
    with pytest.raises(RuntimeError):
        late["ainv"]
