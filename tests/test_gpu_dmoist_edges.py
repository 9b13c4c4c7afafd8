"""The dmoist kernel where its classes change: values at, and up to two floats
beside, every limit of the model (humidity and temperature steps, shading,
precipitation, the slope of 30 degrees, the exposures' azimuths), zeros of
either sign, negative, infinite and NaN inputs.  Equal to the CPU restatement
bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _beside(values):
    v = np.asarray(values, np.float32)
    out = [v]
    for towards in (np.float32(np.inf), np.float32(-np.inf)):
        w = v
        for _ in range(2):
            w = np.nextafter(w, towards)
            out.append(w)
    return np.concatenate(out + [np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-42, -3.0], np.float32)])


@pytest.mark.parametrize("month,hour", [(1, 0), (3, 6), (4, 7), (6, 8), (8, 13), (10, 15), (11, 19), (12, 23)])
def test_class_limits(pp, oracle, month, hour):
    n = 60_007
    rng = np.random.default_rng(100 * month + hour)
    pick = lambda pool, shape: rng.choice(pool, shape)  # noqa: E731
    temp = _beside(list(range(-10, 55, 5)) + [9, 20, 31, 42])
    hum = _beside(list(range(0, 111, 5)))
    cloud = _beside(np.array([10, 50, 90, 100]) / 0.75)
    rain = _beside([1, 5, 15, 35])
    slope = _beside([np.tan(np.pi / 6), 0.25, 1.0, 40.0, -0.5, -1.0, -5.0])
    aspect = _beside(np.deg2rad([0, 45, 135, 225, 315, 360, 20, 180, 300]))
    x = dict(temperature=pick(temp, (24, n)), humidity=pick(hum, (24, n)), cloud_cover=pick(cloud, (24, n)),
             precipitation=pick(rain, (6, n)), slope=pick(slope, n), aspect=pick(aspect, n),
             fuel_code=rng.integers(0, 16, n).astype(np.uint8))
    g = pp.dead_fuel_moisture(hour=hour, month=month, **x)
    c = oracle.dmoist_cells(hour, month, x["temperature"], x["humidity"], x["cloud_cover"], x["slope"], x["aspect"],
                            x["fuel_code"], x["precipitation"])
    for k, ref in zip(("d1hr", "d10hr", "d100hr"), c):
        same = (g[k].view(np.uint32) == ref.view(np.uint32)) | (np.isnan(g[k]) & np.isnan(ref))
        assert same.all(), (k, int((~same).sum()))
