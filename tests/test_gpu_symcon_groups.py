"""The symmetric contraction's group kernels where their shape changes: the last number of groups that two sets of threads
share and the first that one set takes, groups with empty slots, one atom."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["small", "medium", "large"])
@pytest.mark.parametrize("atoms", [1, 7, 592, 594])
def test_forces_with_groups_equal_those_without(model, atoms):
    """Without the list of groups the single-atom kernels run: the same polynomial in another order of operations. 592 and
    594 atoms of two species are 148 and 150 groups. Bound: 94 to 887 fp32 terms per output, 1e-5 of the norm."""
    from fastmace_b200.forcefield import B200ForceField
    from fastmace_b200.model import SPECS, init_weights
    spec = SPECS[model]
    rng = np.random.default_rng(atoms)
    edge = max(6.6, (atoms * 60.0) ** (1 / 3))
    x = torch.tensor(rng.uniform(0, edge, (atoms, 3)), device="cuda")
    numbers = np.array([11, 17] * atoms)[:atoms]
    ff = B200ForceField(spec, init_weights(spec, 2), numbers, edge * np.eye(3) if atoms > 1 else 5.0 * np.eye(3), positions=x,
                        compute_stress=True)
    assert atoms < 500 or ff.n_symcon_groups == (148 if atoms == 592 else 150)
    out = [t.clone() for t in ff(x)]
    ff.work.symcon_groups, ff.work.n_symcon_groups = None, 0
    plain = ff(x)
    for a, b in zip(out, plain):
        assert (a.double() - b.double()).norm() <= 1e-5 * b.double().norm() + 1e-9
    assert int(ff.status) == 0
