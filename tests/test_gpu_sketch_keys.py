"""APPROX_COUNT_DISTINCT by a key some of whose values lie outside the range that its column states: every row has its
group, as by the member lists (path 1)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
COUNT, SUM, ACD = 0, 1, 5


@pytest.mark.parametrize("zone", [(0.0, 9.0), (5.0, 24.0), (0.0, 24.0), (3.0, 3.0)])
@pytest.mark.parametrize("dtype", [np.uint32, np.int32])
def test_keys_outside_their_range(gpu, zone, dtype):
    from computeql_gb300 import ops
    rng = np.random.default_rng(int(zone[1]))
    n = 50_001
    key = rng.integers(0, 25, n).astype(dtype)
    session, value = rng.integers(0, 3000, n).astype(np.uint32), rng.integers(0, 100, n).astype(np.uint32)
    kc = ops.Column(ops.TYPE_U32 if dtype == np.uint32 else ops.TYPE_I32, n, ops.DeviceBuffer(key.nbytes, key), zone=zone, zone_map=False)
    sc, vc = ops.Column.from_numpy(session), ops.Column.from_numpy(value)

    def groups(path):
        r = ops.group_hash([kc], [COUNT, ACD, SUM], [None, sc, vc], path=path, max_groups=n)
        regs = ops.group_hash_registers()
        return {int(key[int(row)]): (r["results"][g].tolist(), regs[g].tolist()) for g, row in enumerate(r["repr_row"])}

    got, lists = groups(0), groups(1)
    assert set(got) == set(range(25)) and got == lists
    for k, (r, _) in got.items():
        assert r[0] == (key == k).sum() and r[2] == value[key == k].sum()
