"""Resident-warp tuning: a scan restores what its context had, and a context that
nobody tuned stays untuned."""
import contextlib

import pytest


class Ctx:
    warps_per_sm, tuned = 16, False

    def set_tuning(self, w):
        self.warps_per_sm, self.tuned = int(w), True

    def reset_tuning(self):
        self.warps_per_sm, self.tuned = 16, False


@pytest.mark.parametrize('set_to', [None, 16, 6])
@pytest.mark.parametrize('inside', [None, 16, 3])
@pytest.mark.parametrize('fails', [False, True])
def test_tuning_is_restored(set_to, inside, fails):
    from ufo_gb300 import drivers
    ctx = Ctx()
    if set_to is not None:
        ctx.set_tuning(set_to)
    with contextlib.suppress(RuntimeError):
        with drivers._tuned(ctx, inside):
            assert ctx.tuned == (inside is not None)
            assert ctx.warps_per_sm == (inside or 16)
            if fails:
                raise RuntimeError
    assert ctx.tuned == (set_to is not None) and ctx.warps_per_sm == (set_to or 16)


def test_resetting_needs_a_context():
    from ufo_gb300 import capi
    assert capi.load().ufo_ctx_reset_tuning(None) == -1
