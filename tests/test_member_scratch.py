"""Members whose column chunks reach the shared-memory cap: few blocks for many
patches, every operator precision and instance count, single launches."""
import numpy as np
import pytest

from test_ensemble import _member, _oracle_run, _rel


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("fp32", 1e-6), ("bf16x2", 1e-6), ("fp64", 1e-9)])
@pytest.mark.parametrize("R", [1, 3, 4])
def test_members_on_few_blocks_take_the_longest_chunks(qdfn_mod, oracle_mod, precision, tol, R):
    """One geometry of ~2,000 patches on one and on five blocks: a chunk of
    columns fills its share of shared memory.  Ten steps against the oracle, at
    the mixed-precision contract's 1e-6 and FP64's 1e-9."""
    from qdfn import ensemble
    m, ref = _member(3, R, n_faults=14, patch=100.0, length=(1200.0, 1800.0))
    assert ref[5] > 1600
    runs = [_oracle_run(oracle_mod, ref, r, 10) for r in range(R)]
    for blocks in (1, 5):
        ens = ensemble.Ensemble([m], precision=precision, blocks=[blocks])
        ens.run(10, timeout_s=60)
        for r, o in enumerate(runs):
            st = ens.members[0].state(r)
            assert st["step"] == o.step == 10
            assert _rel(st["D"], o.state["D"]) < tol
        ens.close()
