"""Admission of the serving engine: the workspace of a screened call counts beside the resident trees."""
from types import SimpleNamespace

from covertreex_gb300.serving import ServingEngine, estimate_tree_bytes, screened_workspace_bytes


class _Freed:
    def free(self):
        pass


def _engine(budget, trees, dense_pair_limit=1.0e10):
    eng = ServingEngine.__new__(ServingEngine)
    eng.budget, eng.dense_pair_limit = float(budget), dense_pair_limit
    eng.trees = {i: SimpleNamespace(rid=i, n=n, m=m, nbytes=b, inflight=0, last_used=i, index=_Freed(), factor=_Freed())
                 for i, (n, m, b) in enumerate(trees)}
    eng.used_bytes, eng.reserved_bytes, eng.evicted = sum(b for _, _, b in trees), 0, set()
    return eng


def test_workspace_covers_the_passes_buffers():
    n, m = 262144, 512
    digits, lists = 10 * n * m, 4096 * (2 * 2048 * 8 + 10 * m)  # see digit_pass: b; surv and survb, a
    assert digits + lists <= screened_workspace_bytes(n, m) <= 1.01 * (digits + lists)
    assert screened_workspace_bytes(10 ** 7, m) <= (4 << 30) + 1.01 * lists  # slabs
    assert screened_workspace_bytes(n, 832) == 0


def test_admission_leaves_room_for_one_screened_call():
    n, m = 131072, 256
    est, ws = estimate_tree_bytes(n, 3, m), screened_workspace_bytes(n, m)
    full = _engine(2 * est + ws, [(n, m, est)])
    assert full._evict_for(est, set(), n, m) and not full.evicted
    short = _engine(2 * est + ws - 1, [(n, m, est)])
    assert short._evict_for(est, set(), n, m) and short.evicted == {0}
    # the protected or busy tree stays, and the build waits
    assert not _engine(2 * est + ws - 1, [(n, m, est)])._evict_for(est, {0}, n, m)
    # requests that all run dense need none; a tree alone may fill the budget
    assert _engine(2 * est, [(n, m, est)], dense_pair_limit=1e12)._evict_for(est, {0}, n, m)
    assert _engine(est, [])._evict_for(est, set(), n, m)
