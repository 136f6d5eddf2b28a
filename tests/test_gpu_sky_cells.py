"""The sky distribution's cells (luminance x sin(theta), 4 x 4 sub-samples,
FP64 rounded once) against the model in extended precision on sampled rows:
the poles, the horizon and between, with the sun at the zenith, near the
horizon and between, at the smallest and largest turbidity.  The FP64 sums are
good to some 1e-13, so a cell is the FP32 value nearest to the exact one, or
its neighbour where that lies on a rounding boundary."""
import ctypes as C

import numpy as np
import pytest

from noor_b200 import _capi, scenes

pytestmark = pytest.mark.gpu

W, H = 2048, 1024
ROWS = (0, 1, 37, 255, 410, 510, 511, 512, 1023)


def _exact(sky, row):
    ld = np.longdouble
    pi = ld("3.14159265358979323846264338327950288")
    sun = [ld(x) for x in sky.solar_dir]
    acc = np.zeros(W, ld)
    for b in range(4):
        theta = (ld(row) + (ld(b) + ld(0.5)) / 4) / H * pi
        st, ct = np.sin(theta), np.cos(theta)
        if ct < 0:
            continue
        for a in range(4):
            phi = (np.arange(W).astype(ld) + (ld(a) + ld(0.5)) / 4) / W * 2 * pi
            cs = np.clip(st * np.cos(phi) * sun[0] + ct * sun[1] + st * np.sin(phi) * sun[2], -1, 1)
            gamma = np.arccos(cs)
            lum = np.zeros(W, ld)
            for k in range(3):
                c = [ld(x) for x in sky.state[k].configs[k]]
                mie = (1 + cs * cs) / (1 + c[8] * c[8] - 2 * c[8] * cs) ** ld(1.5)
                v = (1 + c[0] * np.exp(c[1] / (ct + ld(np.float32(0.01))))) * (
                    c[2] + c[3] * np.exp(c[4] * gamma) + c[5] * cs * cs + c[6] * mie + c[7] * np.sqrt(ct))
                v = v * ld(sky.state[k].radiances[k])
                q = v * ld(np.float32(0.025))
                g = np.where(q <= ld(np.float32(0.04045)), q / ld(np.float32(12.92)),
                             ((np.maximum(q, 0) + ld(np.float32(0.055))) / ld(np.float32(1.055))) ** ld(np.float32(2.4)))
                v = np.where(gamma < ld(sky.solar_radius), v * ld(sky.solar_scale), g)
                lum = lum + ld(np.float32((0.2126, 0.7152, 0.0722)[k])) * v
            acc += np.maximum(0, lum) * st
    return acc / 16


@pytest.mark.parametrize("turbidity,sun_lat", [(1.0, 0.0), (3.0, 1.047), (10.0, 1.5)])
def test_sky_cells_are_the_models(turbidity, sun_lat):
    s = scenes.sky_scene(width=16, height=16, count=2, level=1)
    s.hosek = dict(turbidity=turbidity, albedo=0.3, sun_lat=sun_lat, sun_lon=0.7, solar_scale=250.0,
                   solar_radius_scale=2.0)
    r = scenes.Renderer(s)
    try:
        func = np.zeros(W * H, np.float32)
        w, h = C.c_int(), C.c_int()
        _capi.call("noor_get_env_distribution", C.byref(w), C.byref(h), func.ctypes.data_as(_capi.pf), None, None, None,
                   None)
        assert (w.value, h.value) == (W, H)
        func = func.reshape(H, W)
        assert func[: H // 2].mean() > 0 and not func[H // 2:].any()
        for row in ROWS:
            want = _exact(r.hosek, row)
            ulp = np.spacing(np.maximum(want.astype(np.float32), np.float32(1e-30)))
            assert (np.abs(func[row].astype(np.longdouble) - want) <= 0.5000001 * ulp).all(), row
    finally:
        r.close()
