"""GPU tests of the quad engine (kpolaris_b200/csrc/kp_quad.cuh): the sizes
and mixes at which four lanes per ray can go wrong.

* Image sizes around the quads of a warp and the warps of a block, one to four
  frequencies: the one-launch FP64 kernel's reasons and step counts are the
  CPU oracle's, and all of its outputs the wavefront's, bit for bit (whose
  Stokes vectors tests/test_gpu_parity.py holds to the oracle's, within the
  conditioning of libm's last bits).
* Many small images of different spins and frequency counts in one batch, so
  that the quads of a warp trace different images: each is bit for bit the
  image traced alone, in either precision.
* Just as many rays as a B200's resident quads (9,472) take the FP64 far phase
  as quads, more as lanes (one ray per thread): both are the one-launch
  kernel's, bit for bit.
* The near phases and the one-launch kernel take lanes from a number of rays
  on: the smallest launches that do, of one image or several, one to four
  frequencies, every scene, are those of the quads, bit for bit.
* The mixed policy chooses quads or lanes by the image: the smallest images on
  lanes against the FP64 policy, and both kinds in one launch or one server,
  each bit for bit the image traced alone.
* The mixed policy's far field takes many steps at once and counts them: on
  rays that miss the sphere, cameras near, inside the far boundary and far
  out, and large and small step caps, its reasons are those of the FP64 policy
  and so are its step counts, up to the rays that the fused arithmetic of the
  near phases moves across a step's rounding (at most 1 in 200)."""
from __future__ import annotations

import numpy as np
import pytest

import kpolaris_b200 as kp
import oracle
from kpolaris_b200 import _abi, configs, synthetic

pytestmark = pytest.mark.gpu

ALL_FIELDS = _abi.IMAGE_FIELDS + _abi.DIAG_FIELDS + _abi.INT_FIELDS


def job(nx, ny, nf, *, spin=0.9375, inclination=50.0, adaptive=True, **camera):
    p = (configs.config2 if adaptive else configs.config1)(nx, ny)[0]
    p.spin = spin
    p.inner_radius = configs.reference_horizon(spin) * 1.05
    p.camera.inclination = configs.inclination_from_degrees(inclination)
    for k, v in camera.items():
        setattr(p.camera, k, v)
    return p, configs.riaf_model(), configs.CONFIG2_FREQS[:nf]


def assert_bitwise(a, b, what):
    for key in ALL_FIELDS:
        assert np.array_equal(a.arrays[key], b.arrays[key], equal_nan=True), (what, key)


@pytest.mark.parametrize("nx,ny,nf,adaptive", [(1, 1, 1, True), (3, 1, 2, True), (7, 1, 3, False), (8, 1, 4, True),
                                               (9, 1, 1, False), (11, 3, 4, True)])
def test_small_sizes_match_the_oracle(nx, ny, nf, adaptive):
    p, m, f = job(nx, ny, nf, adaptive=adaptive)
    got = kp.image_riaf(p, m, f)
    ref = oracle.image_riaf(p, m, f, kind="port", threads=0)
    for key in _abi.INT_FIELDS:
        assert np.array_equal(got.arrays[key], ref.arrays[key]), key
    assert_bitwise(kp.image_riaf(p, m, f, schedule=_abi.SCHEDULE_PERSISTENT), got, "wavefront")


@pytest.mark.parametrize("precision", [_abi.PRECISION_FP64, _abi.PRECISION_MIXED])
def test_mixed_warps_match_images_alone(precision):
    jobs = [job(5 + k, 3 + (k % 4), 1 + k % 4, spin=0.09 * k, inclination=15.0 + 14.0 * k, fov_y=0.16 + 0.05 * (k % 3))
            for k in range(11)]
    outs = kp.batch_riaf(jobs, precision=precision)
    for k, (p, m, f) in enumerate(jobs):
        alone = kp.image_riaf(p, m, f, precision=precision, schedule=_abi.SCHEDULE_PERSISTENT)
        assert_bitwise(outs[k], alone, k)


@pytest.mark.parametrize("nx,ny", [(97, 97), (98, 97)])
def test_far_phase_forms_agree(nx, ny):
    p, m, f = job(nx, ny, 1, inclination=17.0)
    assert_bitwise(kp.image_riaf(p, m, f, schedule=_abi.SCHEDULE_PERSISTENT), kp.image_riaf(p, m, f), (nx, ny))


@pytest.mark.parametrize("radius,fov,max_step", [(1000.0, 0.5, 2.0), (300.0, 1.2, 2.0), (121.0, 0.6, 2.0),
                                                 (1000.0, 0.3, 0.7), (5000.0, 0.1, 5.0)])
def test_far_field_runs_keep_the_step_counts(radius, fov, max_step):
    p, m, f = job(24, 20, 1, radius=radius, fov=fov, fov_y=fov)
    p.max_step = max_step
    p.max_radiation_step = max_step
    mixed = kp.image_riaf(p, m, f, precision=_abi.PRECISION_MIXED)
    fp64 = kp.image_riaf(p, m, f, schedule=_abi.SCHEDULE_PERSISTENT)
    assert np.array_equal(mixed.reason, fp64.reason)
    for key in ("pass_a_steps", "steps"):
        d = mixed.arrays[key] != fp64.arrays[key]
        assert np.mean(d) <= 0.005, (key, int(d.sum()))


def forms(image, **options):
    """An image with the launch's own choice of quads and lanes, and with
    quads in every near phase: the line is a number of rays per quad of the
    grid, which blocks_per_sm enlarges."""
    return image(**options), image(blocks_per_sm=16, **options)


# The smallest launches that take lanes on a B200 (148 SMs): 75,776 rays in
# near-A and at one frequency, 227,328 at two, 454,656 at three or four.
@pytest.mark.parametrize("sizes,nf", [([(279, 272)], 1), ([(478, 476)], 2), ([(477, 477), (97, 9), (1, 1)], 4),
                                      ([(256, 256)] * 7, 3)])
def test_near_phase_forms_agree(sizes, nf):
    jobs = [job(nx, ny, 1 + (k + nf - 1) % nf, inclination=17.0 + 9.0 * k, spin=0.9375 - 0.1 * k)
            for k, (nx, ny) in enumerate(sizes)]
    a, b = forms(lambda **o: kp.batch_riaf(jobs, precision=_abi.PRECISION_FP64, **o))
    for k in range(len(jobs)):
        assert_bitwise(a[k], b[k], k)


@pytest.fixture(scope="module")
def tori():
    grids = []
    for t in (0.0, 400.0):
        prims, model = synthetic.fm_torus(96, 48, 48, time=t)
        grids.append(kp.Grid(model, prims))
    yield grids
    for g in grids:
        g.release()


def scene_call(scene, nx, ny, tori):
    """The parameters of an image of a scene, and the call that traces it."""
    wave = dict(schedule=_abi.SCHEDULE_PERSISTENT)
    if scene in ("cks", "bl"):
        p, m, f = job(nx, ny, 1)
        if scene == "bl":
            p.coordinate_system = _abi.COORD_BOYER_LINDQUIST
        return p, lambda **o: kp.image_riaf(p, m, f, **wave, **o)
    p = synthetic.fmks_pass_a_params(tori[0].model, nx, ny)
    if scene == "fmks":
        return p, lambda **o: kp.image_grmhd(p, tori[0], [230e9], **wave, **o)
    return p, lambda **o: kp.image_grmhd_slow_light(p, tori, [0.0, 400.0], 1213.0, [230e9], **wave, **o)


@pytest.mark.parametrize("scene", ["fmks", "slow", "bl"])
def test_near_phase_forms_agree_in_other_scenes(scene, tori):
    call = scene_call(scene, 280, 271, tori)[1]
    assert_bitwise(*forms(lambda **o: call(precision=_abi.PRECISION_FP64, **o)), scene)


# One pixel above the line of the one-launch kernel (9,472 pixels of fixed
# steps, 47,360 at one frequency, 227,328 at two) against the wavefront.
@pytest.mark.parametrize("nx,ny,nf,adaptive", [(43, 221, 1, False), (43, 221, 4, False), (11, 4306, 1, True),
                                               (478, 476, 2, True)])
def test_plain_kernel_forms_agree(nx, ny, nf, adaptive):
    p, m, f = job(nx, ny, nf, adaptive=adaptive)
    assert_bitwise(kp.image_riaf(p, m, f), kp.image_riaf(p, m, f, schedule=_abi.SCHEDULE_PERSISTENT), (nx, ny))


# The smallest images of one frequency that the mixed policy traces with one
# ray per lane (above 120,000 pixels in FMKS, 80,000 in Boyer-Lindquist),
# against the FP64 policy.  A rounding moves the substeps or the end of a few rays -- some
# tens of these, on quads or lanes alike -- so reasons are held to the bar of
# the small images (99%, tests/test_gpu_grmhd.py), all but one pixel in a
# thousand to 1e-4 of the brightest, and the sums over those to the policy's
# flux and EVPA budget.
@pytest.mark.parametrize("scene,nx,ny", [("bl", 283, 283), ("fmks", 347, 346), ("slow", 347, 346)])
def test_mixed_lane_images_within_budget(scene, nx, ny, tori):
    p, call = scene_call(scene, nx, ny, tori)
    mixed, fp64 = (call(precision=x) for x in (_abi.PRECISION_MIXED, _abi.PRECISION_FP64))
    assert np.mean(mixed.reason == fp64.reason) >= 0.99
    peak = np.nanmax(fp64.arrays["image_i"])
    assert peak > 0.0
    on = np.abs(mixed.arrays["image_i"] - fp64.arrays["image_i"]) <= 1e-4 * peak
    assert np.mean(on) >= 0.999, int((~on).sum())
    i, q, u = ([r.arrays[k][on].sum() for r in (mixed, fp64)] for k in ("image_i", "image_q", "image_u"))
    assert abs(i[0] / i[1] - 1.0) <= 1e-4, i
    d = 0.5 * np.degrees(np.arctan2(u[0], q[0]) - np.arctan2(u[1], q[1]))
    assert abs((d + 90.0) % 180.0 - 90.0) <= 0.1, d


# Images on either side of that line in one launch: each kernel passes the
# other's rays over, and every image is the one traced alone.
@pytest.mark.parametrize("schedule", [_abi.SCHEDULE_PERSISTENT, _abi.SCHEDULE_GRAPH])
def test_mixed_forms_share_a_launch(schedule):
    sizes = [(31, 7, 3), (283, 283, 1), (200, 90, 2), (1, 1, 1), (320, 377, 1), (97, 61, 4)]
    jobs = [job(nx, ny, nf, inclination=20.0 + 11.0 * k, spin=0.15 * k) for k, (nx, ny, nf) in enumerate(sizes)]
    for p, _, _ in jobs:
        p.coordinate_system = _abi.COORD_BOYER_LINDQUIST
    outs = kp.batch_riaf(jobs, precision=_abi.PRECISION_MIXED, schedule=schedule)
    for k, (p, m, f) in enumerate(jobs):
        alone = kp.image_riaf(p, m, f, precision=_abi.PRECISION_MIXED, schedule=_abi.SCHEDULE_PERSISTENT)
        assert_bitwise(outs[k], alone, k)


# In a server's ticks, of a few RK jobs each, too.
@pytest.mark.parametrize("budget", [64, 0])
def test_mixed_forms_share_a_server(tori, budget):
    cfg = kp.default_server_config()
    if budget:
        cfg.tick_budget = budget
    images = [scene_call("fmks", nx, ny, tori)[0] for nx, ny in ((23, 19), (347, 346), (40, 64))]
    riaf = [job(347, 346, 1), job(50, 40, 2)]
    with kp.Server(cfg) as srv:
        tickets = [srv.submit_grmhd(p, tori[0], [230e9]) for p in images] + [srv.submit(*j) for j in riaf]
        for t in tickets:
            srv.wait(t, timeout=300.0)
        got = [srv.result(t) for t in tickets]
    for k, p in enumerate(images):
        assert_bitwise(got[k], kp.image_grmhd(p, tori[0], [230e9], precision=_abi.PRECISION_MIXED), k)
    for k, (p, m, f) in enumerate(riaf):
        assert_bitwise(got[len(images) + k], kp.image_riaf(p, m, f, precision=_abi.PRECISION_MIXED), k)
