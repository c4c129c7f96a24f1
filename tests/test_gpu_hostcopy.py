"""Reading large fields back: the copy into pageable memory by several lanes gives the same
values as the copy into pinned memory, for whole planes a lane, planes larger than a lane's
buffer, a remainder, and fields just below and above the size where the lanes take over."""
import numpy as np
import pytest
import torch

from conftest import load_fastice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(256, 256, 256), (255, 256, 256), (1500, 1301, 9), (2000, 37, 231)])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_pageable_equals_pinned(n, dtype):
    fi = load_fastice()
    g = fi.UniformGrid(origin=(0.0,) * 3, extent=(1.0,) * 3, dims=n)
    s = fi.SBC(0.0, 0.0, 0.0)
    m = fi.IsothermalFullStokesModel(grid=g, boundary_conditions={k: (s, s) for k in "xyz"}, gravity={"x": 0.0, "y": 0.0, "z": 1.0},
                                     rheology=fi.LinearViscousRheology(1.0), solver_params=fi.pt_params(g), dtype=dtype)
    rng = np.random.default_rng(3)
    for name in ("P", "Vx", "txy"):
        want = rng.standard_normal(m.field_shape(name)).astype(np.float64 if dtype == "f64" else np.float32)
        m.set_field(name, want)
        pinned = torch.empty(want.shape, dtype=torch.float64 if dtype == "f64" else torch.float32, pin_memory=True).numpy()
        assert np.array_equal(m.get_field(name), want)
        assert np.array_equal(m.get_field(name, out=pinned), want)
    m.close()
