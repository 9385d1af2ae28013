"""Which form of the mixed translations a plan's passes take, by order and number of boxes: the forms differ in
rounding (split TF32 against FP32), so a body's results keep their last digits only while its passes keep
their forms."""
import pytest

pytestmark = pytest.mark.gpu


def plan_info(fm, body, depth, orders):
    V, F = body
    plan = fm.Plan(V, F, k=25.0, depth=depth, p_levels=orders, rule=1, a=0.5, b=0.0, c=-1.0)
    info = plan.info
    plan.close()
    return info


def test_dense_levels(fm):
    sphere = fm.geodesic_sphere(14, 0.1)  # 56 boxes, 2,504 translations; 248 boxes, 9,744 translations
    thin = fm.ellipsoid(9, (0.025, 0.05, 0.1), lmax=8, sigma=1e-3, seed=2026)  # level 3: 76 boxes, 2,322 translations
    assert plan_info(fm, sphere, 3, {2: 14, 3: 16}).num_m2l[3] == 9744
    assert [plan_info(fm, sphere, 3, {2: 14, 3: 16}).m2l_tensor[l] for l in (2, 3)] == [1, 1]
    assert [plan_info(fm, sphere, 3, {2: 19, 3: 15}).m2l_tensor[l] for l in (2, 3)] == [0, 0]
    assert 2000 < plan_info(fm, thin, 3, {2: 14, 3: 14}).num_m2l[3] < 4000
    for p, on in ((11, 0), (12, 1), (13, 0), (14, 0)):
        assert plan_info(fm, thin, 3, {2: p, 3: p}).m2l_tensor[3] == on, p


@pytest.mark.parametrize("p2,p3,bits", [(32, 24, 0), (33, 25, 1), (34, 31, 1), (40, 30, 1), (38, 34, 5), (44, 33, 5)])
def test_three_stage_levels(fm, p2, p3, bits):
    info = plan_info(fm, fm.geodesic_sphere(8, 0.1), 3, {2: p2, 3: p3})
    assert info.num_box[3] == 248
    assert [info.pass_tc3[l] for l in (2, 3)] == [0, bits]


def test_three_stage_larger_levels(fm):
    info = plan_info(fm, fm.geodesic_sphere(16, 0.1), 4, {2: 40, 3: 30, 4: 22})
    assert info.num_box[3] == 272
    assert [info.pass_tc3[l] for l in (2, 3, 4)] == [0, 1, 0]
