"""The benchmark's choice of the kernel that its roofline describes: the step's four kernels,
with the stages that share a launch taken together."""
import pytest

import bench

ALONE = {"pair_sr": 0.30, "pair_lr": 0.12, "bonded": 0.28, "hbond": 0.40, "shift": 0.0, "integrate": 0.45, "cells": 0.1,
         "search": 0.1}
ALG = {k: 1000.0 * (i + 1) for i, k in enumerate(ALONE)}


@pytest.mark.parametrize("in_step", [
    # as the step reports it: the force launch's time in its first stage
    {"pair_sr": 0.05, "pair_lr": 0.0, "bonded": 0.0, "hbond": 0.0, "shift": 0.0, "integrate": 0.03, "cells": 0.01, "search": 0.01},
    # the stages' times alone, which stand in where the step cannot be captured with events
    {k: v / 12 for k, v in ALONE.items()},
])
def test_roofline_names_the_force_launch(in_step):
    """No single force stage takes as long as the integrator, all of them in one launch do."""
    kernels, most = bench.step_kernels(ALG, ALONE, in_step, 12)
    assert most == "forces" and set(kernels) == {"forces", "integrate", "cells", "search"}
    f = kernels["forces"]
    assert f["alone_us_per_group"] == pytest.approx(1000 * 1.10 / 12)
    assert f["alg_bytes_per_launch"] == pytest.approx((1000 + 2000 + 3000 + 4000) / 12)
    assert kernels["integrate"]["alg_bytes_per_launch"] == pytest.approx((5000 + 6000) / 12)
    assert f["achieved_gbs"] == pytest.approx(f["alg_bytes_per_launch"] / (f["in_step_us"] * 1e-6) / 1e9)
