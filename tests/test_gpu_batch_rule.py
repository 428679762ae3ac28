"""Policy AUTO of a batch at small radii: the path whose launch is the shorter
one as measured, at sizes inside and outside the sweep's, and world counts on
both sides of the line."""
import pytest

import life_simulation_b200 as lb

pytestmark = pytest.mark.gpu

DIRECT, SPECTRAL = 0, 1


@pytest.mark.parametrize("w,h,n,radius,path", [
    (128, 64, 1, 7, DIRECT), (128, 64, 16, 7, DIRECT), (128, 64, 8, 5, DIRECT), (128, 128, 8, 6, DIRECT),
    (256, 256, 1, 8, DIRECT), (256, 256, 16, 3, DIRECT), (256, 256, 8, 9, SPECTRAL), (256, 256, 16, 6, SPECTRAL),
    (384, 216, 2, 6, DIRECT), (384, 216, 16, 8, SPECTRAL), (512, 512, 1, 7, DIRECT), (512, 512, 4, 8, SPECTRAL),
    (1024, 512, 1, 4, DIRECT), (1024, 512, 4, 6, SPECTRAL), (1920, 1080, 1, 3, DIRECT), (1920, 1080, 1, 6, SPECTRAL),
    (1920, 1080, 1, 20, SPECTRAL), (1024, 1024, 1, 13, SPECTRAL),
])
def test_auto_takes_the_measured_side(w, h, n, radius, path):
    b = lb.LeniaBatch([lb.make_world(width=w, height=h, radius=radius, mu=0.2, sigma=0.06, dt=0.1, seed=i) for i in range(n)])
    assert {b.path(i) for i in range(n)} == {path}
    b.close()


def test_auto_of_mixed_sizes_and_small_radii_repeats():
    sizes = [(128, 128), (256, 256), (1024, 512), (384, 216), (90, 70)]
    ws = [lb.make_world(width=sizes[i % 5][0], height=sizes[i % 5][1], radius=3 + i % 7, mu=0.2, sigma=0.06, dt=0.1, seed=i)
          for i in range(15)]
    paths = []
    for _ in range(2):
        b = lb.LeniaBatch(ws)
        paths.append([b.path(i) for i in range(15)])
        b.close()
    assert paths[0] == paths[1]
    assert all(p == DIRECT for p, w in zip(paths[0], ws) if w.width == 90)  # no spectral size
