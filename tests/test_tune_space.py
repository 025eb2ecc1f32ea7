"""The autotuner's search spaces: both forward kernels are in them, and no two
candidates run the same kernel in the same way."""
import itertools

import pytest


def _spaces():
    import bench
    from cbm import tune

    return {"default": tune.DEFAULT_SPACE, "batch": bench.BATCH_SPACE, "precision": bench.PREC_SPACE}


@pytest.mark.parametrize("name", ["default", "batch", "precision"])
def test_space_reaches_both_kernels_once_per_configuration(name):
    from cbm import tune

    space = _spaces()[name]
    found = tune.candidates(space)
    assert {"register", "staged"} <= {c["variant"] for c in found}
    assert "auto" not in {c["variant"] for c in found}  # one of the others, by the plan's rule
    register = [c for c in found if c["variant"] == "register"]
    assert len(register) == len(space["chunk_nnz"]) == len({c["chunk_nnz"] for c in register})
    # the staged kernel's configurations are all there
    names = [k for k in space if k != "variant"]
    staged = [c for c in found if c["variant"] == "staged"]
    assert len(staged) == len(list(itertools.product(*(space[k] for k in names))))
    assert all(set(c) == set(space) for c in found)
