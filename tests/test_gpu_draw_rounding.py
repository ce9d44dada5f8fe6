"""Path-traced pixels that a glint of the sun on a rough mirror dominates, as the
renderer has always computed them: the FP32 products of the mirror's BSDF round
in one way, whatever the code around them. One rounding more or less moves such
a pixel by 6e-8 (one ulp); the FP64 sum of its 16 samples by 1e-15."""
import math

import pytest
import torch

import pyssol as P
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("helio,width,height,elevation,azimuth,dni,key,row,col,value", [
    (122, 380, 198, 25.024479743255217, 156.2864657797519, 811.2281409631385, 469056503740,
     124, 230, 3.7847520067386746),
    (1000, 1920, 1080, 31.772008280072445, 150.70466816520863, 984.4484140925069, 596629122510,
     498, 1035, 2.4902823272355685)])
def test_glints(product, helio, width, height, elevation, azimuth, dni, key, row, col, value):
    s, _ = W.heliostat_field(product, n_helio=helio, elevation=elevation, azimuth=azimuth, dni=dni,
                             receiver_cells=64)
    ground = s.matte(0.3)
    s.instance(s.object([(s.rectangle(2000, 2000), ground, ground)]),
               P.transform_from(None, (0.0, 0.0, -0.5)), sample=0)
    cam = s.camera((0.0, -60.0, 170.0), (0.0, 280.0, 0.0), (0.0, 0.0, 1.0), fov=math.radians(75.0),
                   ratio=width / height)
    px = torch.empty((height, width, 3), dtype=torch.float64, device="cuda")
    s.draw_device("pt", cam, width, height, 16, px.data_ptr(), seed=key)
    torch.cuda.synchronize()
    assert px[row, col].tolist() == pytest.approx([value] * 3, rel=1e-12)
