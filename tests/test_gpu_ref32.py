"""The reference's float4 arrays through the device: upload, added accelerations, download.

Around the size that changes between the page-locked staging and copies
(24,576): every particle arrives (the FP64 download of an uploaded state is
the float4 arrays, widened), the acceleration is added to inbound particles'
xyz as (float)((double)acc + a) and nothing else changes, and the download
writes xyz and keeps w.
"""
import ctypes as C

import numpy as np
import pytest

import plume
import solveit_gpu as sv

pytestmark = pytest.mark.gpu


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("with_t", [True, False])
@pytest.mark.parametrize("n", [1, 255, 24576, 24577])
def test_round_trip(n, with_t):
    st = plume.make_plume(n, 1e-6, n)
    rng = np.random.default_rng(n)
    st["status"] = rng.choice(np.array([1, 2, 0, -1], np.int32), n, p=[0.7, 0.1, 0.1, 0.1])
    st["status"][0] = 1
    pos4, vel4, acc4, t = plume.to_ref32(st)
    with sv.ForceMethod(softening2=1e-20, method=sv.BARNES_HUT) as fm:
        for _ in range(2):  # the staging is used again
            fm.upload_ref32(pos4, vel4, acc4, t if with_t else None)
        x, v, s = fm.download()
        assert np.array_equal(x, pos4[:, :3].astype(np.float64)) and np.array_equal(v, vel4[:, :3].astype(np.float64))
        assert np.array_equal(s, st["status"])
        a = fm.accel()
        got = acc4.copy()
        got[:, :3] = rng.normal(size=(n, 3)).astype(np.float32) * 1e12
        want = got.copy()
        inb = st["status"] == 1
        want[inb, :3] = (want[inb, :3].astype(np.float64) + a[inb]).astype(np.float32)
        fm.add_accel_ref32(got)
        assert np.array_equal(got, want)
        p2, v2 = np.full((n, 4), 7.5, np.float32), np.full((n, 4), -3.25, np.float32)
        assert fm.L.sv_download_ref32(fm.h, _p(p2), _p(v2)) == 0
        assert np.array_equal(p2[:, :3], pos4[:, :3]) and np.all(p2[:, 3] == 7.5)
        assert np.array_equal(v2[:, :3], vel4[:, :3]) and np.all(v2[:, 3] == -3.25)
        p3 = np.full((n, 4), 1.0, np.float32)
        assert fm.L.sv_download_ref32(fm.h, _p(p3), None) == 0
        assert np.array_equal(p3[:, :3], pos4[:, :3])
