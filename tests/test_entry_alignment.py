"""Entries given as a device tensor may start at any coefficient of a larger one
(a view), not only on the boundary of the encoder's 8-byte loads: set_db and
set_shards prepare the same shard from either.  Outputs are compared exactly.
"""
import numpy as np
import pytest

import dnspir_b200 as dp
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2n", [8, 11])
@pytest.mark.parametrize("offset", [1, 2, 3, 4, 7])
def test_entries_at_any_offset(log2n, offset):
    torch = pytest.importorskip("torch")
    n, l = 1 << log2n, 16
    data = np.random.default_rng(offset).integers(0, orc.T, size=(2, 8 * l, n), dtype=np.uint16)
    flat = torch.zeros(data.size + 8, dtype=torch.int16, device="cuda")
    flat[offset:offset + data.size] = torch.from_numpy(data.view(np.int16).reshape(-1)).cuda()
    view = flat[offset:offset + data.size].view(torch.uint16).view(2, 8 * l, n)
    torch.cuda.synchronize()
    assert view.data_ptr() % 8 == 2 * offset % 8
    db = dp.PIRDatabase(log2n, l)
    db.set_db(view[0])
    ref = orc.Database(log2n, l)
    ref.set_db(data[0])
    assert np.array_equal(db.get_a().astype(np.int64), ref.get_a())
    fleets = []
    for entries in (data, view):
        f = dp.Fleet.general(log2n, l, 16, 2)
        f.set_shards(0, entries)
        fleets.append(f)
    rng = orc.Rng(bytes([offset, log2n]) + bytes(30))
    args = orc.enc_double_pir(rng, log2n, l, 16, orc.gen_sk(rng, log2n), 5, 1)
    assert np.array_equal(*[f.perform_double_pir(*args) for f in fleets])
    db.close()
    for f in fleets:
        f.close()
