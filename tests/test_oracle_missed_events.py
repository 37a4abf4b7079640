"""The oracle's skip clock after missed events (CPU): ions that were inactive
at the step of their event, or whose clock was moved past it or back to before
their wait began, go on colliding at the rate they had (counts within 5 sigma
of a run without the gap)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
from helpers import config0_ensemble, config0_ions, oracle_state


@pytest.mark.parametrize("how", ["inactive", "clock", "rewound"])
def test_collisions_go_on_after_a_gap(how):
    e = config0_ensemble()
    st = oracle_state(config0_ions(500))
    r = orc.run(e, st, 50 if how != "rewound" else 500, collision=2, seed=9)
    if how == "inactive":
        st["active"][:] = 0
        r = orc.run(e, st, 100, collision=2, seed=9, step0=50, clock=r["clock"])
        st["active"][:] = 1
    got = orc.run(e, st, 200, collision=2, seed=9, step0=150 if how != "rewound" else 0,
                  clock=r["clock"])["collisions"]
    want = orc.run(e, oracle_state(config0_ions(500)), 200, collision=2, seed=10)["collisions"]
    assert want > 1000 and abs(got - want) <= 5 * np.sqrt(2 * want)
