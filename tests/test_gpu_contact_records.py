"""Contact records as they leave the device: any capacity gives the same leading records, unused bytes are zero."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from andosim_b200 import scenes

pytestmark = pytest.mark.gpu


def test_records_at_any_capacity(abi):
    sc = scenes.c4(n=23, size=0.2, spacing=0.0008)
    S = abi.Scene(sc.vertices, sc.triangles, sc.material)
    want = S.contacts(semantics="corrected")
    n = len(want)
    assert n > 1000
    size = C.sizeof(abi.Contact)
    all_bytes = np.frombuffer((abi.Contact * n)(*want), dtype=np.uint8).reshape(n, size)
    assert not all_bytes[:, abi.Contact.pad_.offset:abi.Contact.pad_.offset + 4].any()
    for cap in (1, 31, 32, n - 1, n, n + 7):
        buf = np.full((n + 8, size), 0xAB, np.uint8)
        got = C.c_int32()
        rc = abi.lib().ando_compute_contacts_corrected(S.ctx, 1e-3, None, 0, buf.ctypes.data_as(C.POINTER(abi.Contact)), cap, C.byref(got))
        assert got.value == n and rc == (abi.ANDO_OK if cap >= n else abi.ANDO_ERR_CAPACITY)
        k = min(cap, n)
        np.testing.assert_array_equal(buf[:k], all_bytes[:k])
        assert (buf[k:] == 0xAB).all()
    # the records say what the positions say: signed weights sum to zero, the witnesses are the gap apart
    c = want[0]
    for c in want[:: max(1, n // 200)]:
        assert c.vertex_count == 4 and abs(sum(c.weights)) < 1e-9
        d = np.array(c.witness_p[:]) - np.array(c.witness_q[:])
        assert abs(np.linalg.norm(d) - c.gap) < 1e-9
    S.close()
