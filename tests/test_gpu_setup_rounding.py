"""The set-up's quotients at the distances whose reciprocal is hard to round (GPU)."""
import numpy as np
import pytest

import mgcfd
from test_gpu_setup_tables import TABLES, table

pytestmark = pytest.mark.gpu


def test_weights_of_edges_just_below_a_power_of_two_long():
    """Edges (1, t, 0) whose length is 2 - k 2^-52 for odd k: 1 / length lies next to
    a rounding tie, and a quotient by it is one unit off when the reciprocal is.
    The device's weights and volumes are the host's, bit for bit."""
    lengths, ts = [], []
    t = np.sqrt(3.0) - np.arange(0, 400) * 2.0 ** -52
    dist = np.sqrt(1.0 + t * t)
    for k in range(1, 100, 2):
        at = np.flatnonzero(dist == 2.0 - k * 2.0 ** -52)
        assert len(at)
        ts.append(t[at[0]])
    areas = [1.0, 1.5, 0.7071067811865476, 1.0 + 2.0 ** -52, 3.0]
    ts, areas = np.repeat(ts, len(areas)), np.tile(areas, len(ts))
    m = len(ts)
    coords = np.zeros((2 * m, 3))
    coords[:, 2] = np.repeat(np.arange(m), 2)
    coords[1::2, 0] = 1.0
    coords[1::2, 1] = ts
    weights = np.zeros((m, 3))
    weights[:, 1] = areas
    level = mgcfd.Level(coords=coords, edge_to_nodes=np.arange(2 * m, dtype=np.int32).reshape(m, 2),
                        bnd_to_node=np.zeros(1, np.int32), bnd_group=np.full(1, 3, np.int32), edge_weights=weights,
                        bnd_weights=np.ones((1, 3)), node_to_mg=None)
    dev = mgcfd.Solver([level], 0.5, 2.0, increment="gather")
    host = mgcfd.Solver([level], 0.5, 2.0, increment="gather", host_setup=True)
    for k, (name, _) in TABLES.items():
        np.testing.assert_array_equal(table(dev, 0, k), table(host, 0, k), err_msg=name)
    dev.close()
    host.close()
