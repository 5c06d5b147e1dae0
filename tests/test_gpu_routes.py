"""Which form a call takes, for the shapes with which the forms are compared elsewhere and at
the limits that the plan itself reports.

The comparisons are with the separate passes (schedules set by hand) under the bounds of
test_gpu_stream.py: 2e-7 per slice with a floor of 1e-6."""
import pytest
import torch

import test_gpu_resident as resident
import test_gpu_stream as stream
from namsa_gb300 import engine

pytestmark = pytest.mark.gpu
KMAX, BAND = 10.0, 10.0 / 3


def route(ny, nx, S, P, detector=False, plan=None):
    p = plan or engine.Plan(ny, nx)
    r = p.route(S, P, KMAX, BAND, detector)
    if plan is None:
        p.close()
    return r


def test_shapes_of_the_all_slices_tests_take_it():
    torch.cuda.set_device(0)
    for ny, nx, S, P in stream.SHAPES:
        form, size, _, _ = route(ny, nx, S, P)
        # 256^2 and 12 positions and more: never clusters; two slices are enough
        assert (form, size <= P) == ('all_slices', True), (ny, nx, S, P)
    assert route(384, 384, 3, 150)[:2] == ('all_slices', 80)      # two groups
    assert route(512, 512, 3, 9, detector=True)[0] == 'all_slices'
    assert route(512, 512, 19, 70)[:2] == ('all_slices', 40)      # uploads by eight slices, two groups
    assert route(512, 512, 1, 9)[0] == route(1024, 512, 3, 9)[0] == 'passes'


def test_shapes_of_the_cluster_tests_take_it():
    torch.cuda.set_device(0)
    seen = set()
    for ny, nx, S, P in resident.SHAPES:
        form, size, _, _ = route(ny, nx, S, P)
        assert form == 'cluster', (ny, nx, S, P)
        seen.add(size)
    assert seen == {4, 8, 16}
    assert route(128, 128, 9, 4)[0] == 'cluster' and route(128, 128, 9, 4, detector=True)[0] == 'passes'


def limit(ny, nx, S, takes, most=1024):
    """The largest P up to which takes(route) holds from 1 on."""
    plan = engine.Plan(ny, nx)
    P = 0
    while P < most and takes(route(ny, nx, S, P + 1, plan=plan)):
        P += 1
    plan.close()
    return P


def agree(ny, nx, S, P):
    a, b = stream.both(ny, nx, stream.case(ny, nx, S, P, ny + 7 * nx + P), lambda plan, x: plan.multislice(*x))
    assert stream.rel(a, b) < max(1e-6, 2e-7 * S)


@pytest.mark.parametrize('ny,nx', [(256, 256), (384, 256), (512, 256), (256, 768)])
def test_either_side_of_the_fewest_positions_of_the_all_slices_form(ny, nx):
    torch.cuda.set_device(0)
    few = limit(ny, nx, 3, lambda r: r[0] != 'all_slices', 64)
    if few:
        agree(ny, nx, 3, few)
    assert route(ny, nx, 3, few + 1)[0] == 'all_slices'
    agree(ny, nx, 3, few + 1)


@pytest.mark.parametrize('ny,nx', [(64, 64), (128, 128), (256, 128), (256, 256)])
def test_either_side_of_the_most_positions_of_the_clusters(ny, nx):
    torch.cuda.set_device(0)
    most = limit(ny, nx, 2, lambda r: r[0] == 'cluster')
    assert most >= 1
    agree(ny, nx, 2, most)
    agree(ny, nx, 2, most + 1)


@pytest.mark.parametrize('ny,nx,which', [(64, 384, 2), (64, 512, 2), (128, 768, 2), (384, 64, 3), (768, 128, 3)])
def test_either_side_of_the_most_positions_of_the_schedules_of_few_lines(ny, nx, which):
    torch.cuda.set_device(0)
    most = limit(ny, nx, 3, lambda r: r[0] == 'passes' and r[which])
    assert most >= 1
    agree(ny, nx, 3, most)
    agree(ny, nx, 3, most + 1)


def test_schedules_set_by_hand_are_the_passes():
    torch.cuda.set_device(0)
    for ny, nx, P in ((512, 512, 4), (128, 128, 2), (64, 384, 1)):
        plan = engine.Plan(ny, nx)
        assert route(ny, nx, 3, P, plan=plan) != ('passes', P, False, False)
        plan.set_schedule(*plan.schedule[:2])
        assert route(ny, nx, 3, P, plan=plan) == ('passes', P, False, False)
        plan.close()
