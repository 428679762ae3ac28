"""Which direct engine runs: lenia_info names it, the rule on the field's size and
the kernels' taps picks it, and a forced engine that cannot run says so."""
import numpy as np
import pytest

import life_simulation_b200 as lb

pytestmark = pytest.mark.gpu

BYTES = 4  # lenia_info.tc_engine of the byte form


def info(params, w, h):
    m = lb.LeniaModule(params, w, h)
    out = m.info(), m.warning
    m.close()
    return out


@pytest.mark.parametrize("w,h,radius,engine", [
    (128, 128, 5, 0), (128, 128, 32, 0), (256, 256, 13, 0), (512, 512, 5, 0), (512, 512, 13, BYTES), (1001, 703, 5, 0),
    (1001, 703, 9, BYTES), (1280, 720, 3, 0), (1280, 720, 32, BYTES), (1400, 1070, 4, 0), (1920, 1080, 3, 0),
    (1920, 1080, 13, BYTES),
])
def test_the_rule_at_measured_points(w, h, radius, engine):
    got, warning = info({"radius": radius, "kernelCore": "gaussShell"}, w, h)
    assert got["tc_engine"] == engine and not warning
    if engine == BYTES:
        assert (got["direct_tma"], got["direct_split"], got["direct_outputs_per_thread"],
                got["direct_rows_per_thread"]) == (False, 1, 16, 1)


@pytest.mark.parametrize("radius", [5, 9])
def test_larger_fields_do_not_go_back_to_fp32(radius):
    """Where the byte form is the choice for a field, it is for the same field with
    rows added up to whole rounds of tiles."""
    on = [info({"radius": radius, "kernelCore": "gaussShell"}, 1280, h)[0]["tc_engine"] for h in (384, 768, 1152, 1536)]
    assert on == sorted(on)


def test_forced_engines(monkeypatch):
    monkeypatch.setenv("LENIA_DIRECT_ENGINE", "tensor")
    got, warning = info({"radius": 5}, 64, 64)
    assert got["tc_engine"] == BYTES and not warning
    got, warning = info({"radius": 0}, 64, 64)  # a kernel without weights
    assert got["tc_engine"] == 0 and "no byte form" in warning
    monkeypatch.setenv("LENIA_DIRECT_ENGINE", "ffma")
    got, warning = info({"radius": 13}, 1920, 1080)
    assert got["tc_engine"] == 0 and not warning
    monkeypatch.delenv("LENIA_DIRECT_ENGINE")
    monkeypatch.setenv("LENIA_DIRECT_OX", "8")  # a shape of the FP32 kernels
    assert info({"radius": 13}, 1920, 1080)[0]["tc_engine"] == 0


def test_the_byte_form_steps_beside_small_growth_centres(monkeypatch):
    """|mu| < 1/64 takes the FP32 kernels whatever the engine: their bits."""
    a = np.random.default_rng(2).random((90, 120), np.float32) * np.float32(0.02)
    out = []
    for engine in ("ffma", "tensor"):
        monkeypatch.setenv("LENIA_DIRECT_ENGINE", engine)
        m = lb.LeniaModule({"radius": 9, "growthMu": 0.01, "growthSigma": 0.005}, 120, 90)
        m.reset(3)
        m.upload(a)
        m.encode(0, 2)
        out.append(m.field())
        m.close()
    np.testing.assert_array_equal(out[0], out[1])
