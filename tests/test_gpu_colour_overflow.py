"""A scene with more colours than the solver's 64 (100 spheres in one place): the
bodies beyond share the last colour, step_fixed reports AVBD_ERR_CAPACITY, and
a captured step goes on.  Its contacts between bodies of that colour get their
dual updates in every iteration, as all others do: their penalties ramp up over
the substep's iterations (by the last pass alone they would stay a tenth)."""
import numpy as np
import pytest

from ornis_gb300 import abi
from ornis_gb300.avbd import AvbdError, AvbdWorld

from test_gpu_static_capacity import crowd

pytestmark = pytest.mark.gpu


def test_duals_of_the_shared_colour():
    params = abi.default_params(gravity=(0.0, 0.0, 0.0), enable_sleep=0)
    w = AvbdWorld(params, bodies=crowd(100))
    with pytest.raises(AvbdError) as e:
        w.step_fixed(1)
    assert e.value.code == abi.AVBD_ERR_CAPACITY
    w.step_graph(1)
    st, col = w.export_state(), w.colours()
    a, b = st["pairs"]["a"], st["pairs"]["b"]
    shared = col[a] == col[b]
    assert shared.sum() > 200 and np.all(col[a][shared] == 63)
    pen = st["points"].reshape(-1, abi.MAX_POINTS)["pen"][:, 0, 0]
    print(f"median penalty: shared colour {np.median(pen[shared]):.3g}, others {np.median(pen[~shared]):.3g}")
    assert np.median(pen[shared]) > 0.3 * np.median(pen[~shared])
