"""A vector that the caller changes while a call reads it: no answer is promised,
but keys that were not counted are not copied past their bucket's place, the
call reports it, and the next call is exact."""
import numpy as np
import pytest

import ggms_b200 as G
import ggms_oracle as orc
from ggms_b200 import datagen as D
from conftest import to_device

pytestmark = pytest.mark.gpu


def test_a_vector_that_changes_during_the_call():
    import torch
    ctx = G.Context(0)
    n = (1 << 24) - 3
    v = D.normal_f32(n, 8)
    ks = np.array([n // 2], np.uint32)
    exp = orc.cpu_multiselect(v, ks)
    d = to_device(v)
    # part of the vector, as it is and with every key in the answer's bucket; from
    # pinned memory: copied without an SM, beside the call's kernel
    m = 1 << 17
    spread = torch.from_numpy(v[:m].copy()).pin_memory()
    heap = torch.full_like(spread, float(exp[0])).pin_memory()
    dk, out = to_device(ks), torch.empty(1, dtype=torch.float32, device="cuda")
    o = G.default_opts(ks_on_device=1, out_on_device=1)

    def call():
        assert G.multiselect_ex(ctx, d.data_ptr(), n, dk.data_ptr(), 1, out.data_ptr(), np.float32, o) == 0
        return ctx.status()
    side = torch.cuda.Stream()
    seen = set()
    for _ in range(20):
        with torch.cuda.stream(side):
            for _ in range(100):
                d[:m].copy_(heap, non_blocking=True)
                d[:m].copy_(spread, non_blocking=True)
        for _ in range(20):
            seen.add(call())
    side.synchronize()
    assert seen <= {G.GGMS_OK, G.GGMS_E_INTERNAL} and G.GGMS_E_INTERNAL in seen, seen
    assert call() == G.GGMS_OK
    np.testing.assert_array_equal(orc.bits(out.cpu().numpy()), orc.bits(exp))
    ctx.close()
