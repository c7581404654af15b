"""Tile kernels (one launch per time step, option "tile") against the half-step kernels and the
marching ring kernels, at the sizes where a tile can go wrong: a last tile of one column or row, one
short of full, windows of uneven width, a single time step, and every row count."""
import numpy as np
import pytest

from ds2d_b200 import Elastic2D, ShotGeom, synth
from tests.helpers import rel

pytestmark = pytest.mark.gpu

# The same FP32 sums per cell in another order at most: agreement to the FP32 floor of a few
# hundred steps (1e-6), with a margin; the Born images, built from a scattered field, sit higher.
GATE, BORN_GATE = 1e-5, 3e-5


def _shots(c, uneven):
    out = []
    for k, sx in enumerate((4, c["allnx"] // 2, c["allnx"] - 3)):
        w = c["nx"] - (7 * k if uneven else 0)
        left = int(np.clip(sx - w // 2, 0, c["allnx"] - w))
        isx = c["pml"] + sx - left
        # receivers that short runs reach (the NCC source divides by each trace's norm)
        igx = np.arange(max(c["pml"], isx - 10), min(c["pml"] + w, isx + 11), 1 + k, dtype=np.int32)
        out.append(ShotGeom(left, isx, c["pml"] + 1, c["pml"] + 2, igx, w))
    return out


# (allnx, allnz, nx, pml, nt, rows): padded depths 97 (one column in the last tile), 96 (full) and
# 95, 61; padded widths 65, 64, 63, 49 (one row over, full, one short of the row blocks).
SIZES = [(60, 81, 49, 8, 60, 8), (60, 80, 48, 8, 61, 16), (60, 79, 47, 8, 60, 32),
         (40, 37, 25, 12, 1, 8), (40, 37, 25, 12, 33, 16)]


def _case(allnx, allnz, nx, pml, nt):
    c = dict(allnx=allnx, allnz=allnz, nx=nx, pml=pml, nt=nt, dx=10.0, dz=8.0, dt=0.0008)
    rng = np.random.default_rng(allnx + allnz + nt)
    vp, vs = synth.layered(allnx, allnz, seed=6)
    rho = (2000.0 + 300.0 * rng.random((allnx, allnz))).astype(np.float32)
    # a wavelet that starts at once, so short runs have signal everywhere
    w = np.sin(0.3 * np.arange(nt) + 0.5).astype(np.float32)
    return c, vp, vs, rho, w, rng


def _ctx(c, shots, **kw):
    return Elastic2D(c["allnx"], c["allnz"], c["nx"], c["pml"], c["nt"], c["dx"], c["dz"], c["dt"],
                     max_shots=len(shots), max_ntr=c["nx"], seed=9, **kw)


@pytest.mark.parametrize("uneven", [False, True])
@pytest.mark.parametrize("boundary", ["random", "pml"])
@pytest.mark.parametrize("size", SIZES)
def test_tile_elastic_matches_other_paths(cuda_device, size, boundary, uneven):
    *dims, rows = size
    c, vp, vs, rho, w, rng = _case(*dims)
    shots = _shots(c, uneven)
    ntr = sum(s.ntr for s in shots)
    obs = [rng.normal(size=(ntr, c["nt"])).astype(np.float32) for _ in range(2)]
    img = [0.05 * rng.normal(size=vp.shape).astype(np.float32) for _ in range(2)]
    got = {}
    for name, opts in (("tile", {"tile": rows}), ("half", {"fused": 0}), ("ring", {"tile": 0})):
        with _ctx(c, shots, boundary=boundary) as e:
            for k, v in opts.items():
                e.set_option(k, v)
            e.set_models(vp, vs, rho)
            e.set_wavelet(w)
            e.set_image(*img)
            out = dict(zip(("rz", "rx"), e.forward(shots)))
            e.rtm(shots, *obs)
            out.update(e.read_images(which=("pp_grad", "ps_grad", "illumination")))
            if c["nt"] > 1:  # a scattered set has no record yet after one step
                out["misfit"] = e.elsrtm(shots, *obs, 1)
                out.update({"els_" + k: v for k, v in e.read_images().items()})
            got[name] = out
    if c["nt"] > 1:  # a mean of correlations in [-1, 1] per shot: absolute error
        mis = [got[n].pop("misfit") for n in ("tile", "ring", "half")]
        assert max(mis) - min(mis) < GATE * len(shots)
    for k in got["tile"]:
        if not np.any(got["half"][k]):
            assert not np.any(got["tile"][k])
            continue
        gate = BORN_GATE if k in ("els_b_pp", "els_b_ps") else GATE
        assert rel(got["tile"][k], got["ring"][k]) < gate, k
        # the half steps leave the strips in the reconstructed state, which the Born source of the
        # first-order images reads (k_bwd_scat_ring and the tiles read the frozen band instead)
        if gate == GATE or boundary == "random":
            assert rel(got["tile"][k], got["half"][k]) < gate, k


@pytest.mark.parametrize("boundary", ["random", "pml"])
@pytest.mark.parametrize("size", SIZES)
def test_tile_acoustic_matches_half_steps(cuda_device, size, boundary):
    *dims, rows = size
    c, vp, _, rho, w, rng = _case(*dims)
    shots = _shots(c, uneven=True)
    ntr = sum(s.ntr for s in shots)
    m = 0.05 * rng.normal(size=vp.shape).astype(np.float32)
    d = [rng.normal(size=(ntr, c["nt"])).astype(np.float32) for _ in range(2)]
    got = []
    for opts in ({"tile": rows}, {"fused": 0}):
        with _ctx(c, shots, boundary=boundary) as e:
            for k, v in opts.items():
                e.set_option(k, v)
            e.set_models(vp, 0 * vp, rho)
            e.set_wavelet(w)
            got.append((*e.ac_born(shots, m), e.ac_born_adj(shots, *d)))
    for a, b in zip(*got):
        if not np.any(b):
            assert not np.any(a)
        else:
            assert rel(a, b) < GATE


def test_changed_density_is_not_replayed(cuda_device):
    """A captured batch holds the density array of its capture: models set again without one are
    modelled with the default density."""
    c, vp, vs, rho, w, _ = _case(60, 48, 48, 8, 40)
    shots = _shots(c, uneven=False)
    with _ctx(c, shots) as e, _ctx(c, shots) as f:
        e.set_wavelet(w), f.set_wavelet(w)
        e.set_models(vp, vs, rho)
        e.forward(shots)
        e.set_models(vp, vs)
        f.set_models(vp, vs)
        for a, b in zip(e.forward(shots), f.forward(shots)):
            np.testing.assert_array_equal(a, b)


def test_options_leave_the_kernel_choice_alone(cuda_device):
    """Which kernels a call runs (the names of the profile) after options that are refused, that
    shape another path, that shape this path, and after "tile" = -1."""
    from ds2d_b200._lib import DS2DError
    c, vp, vs, rho, w, _ = _case(60, 48, 48, 8, 12)
    shots = _shots(c, uneven=False)
    m = np.full(vp.shape, 0.01, np.float32)

    def tiles(e, acoustic):
        e.profile(True)
        e.ac_born(shots, m) if acoustic else e.forward(shots)
        names = set(e.profile_report())
        e.profile(False)
        return ("ac_tile" if acoustic else "fwd_tile") in names

    for boundary in ("pml", "random"):
        with _ctx(c, shots, boundary=boundary) as e:
            e.set_models(vp, vs, rho)
            e.set_wavelet(w)
            for key, value in (("no_such_option", 1), ("xr", 3), ("ac_duo", 7), ("tile", 5)):
                with pytest.raises(DS2DError):
                    e.set_option(key, value)
            assert tiles(e, False) and tiles(e, True), boundary
            e.set_option("ac_duo", 1)
            assert tiles(e, False) and tiles(e, True) == (boundary == "pml"), boundary
            e.set_option("tile", -1)
            e.set_option("bwd_cta", 128)  # random-boundary RTM steps
            assert tiles(e, False) == (boundary == "pml") and tiles(e, True), boundary
            e.set_option("xr", 64)
            assert not tiles(e, False) and tiles(e, True) == (boundary == "pml"), boundary
            e.set_option("tile", -1)
            assert tiles(e, False) and tiles(e, True), boundary


def test_stream_that_cannot_be_captured(cuda_device):
    """cudaStreamLegacy (handle 1) refuses graph capture: the calls launch directly, with the same
    results as on the context's own stream."""
    c, vp, vs, rho, w, rng = _case(60, 48, 48, 8, 40)
    shots = _shots(c, uneven=False)
    ntr = sum(s.ntr for s in shots)
    obs = [rng.normal(size=(ntr, c["nt"])).astype(np.float32) for _ in range(2)]
    m = 0.05 * rng.normal(size=vp.shape).astype(np.float32)
    out = []
    for handle in (0, 1):
        with _ctx(c, shots, boundary="pml") as e:
            e.set_stream(handle)
            e.set_models(vp, vs, rho)
            e.set_wavelet(w)
            e.set_image(m, m)
            mis = e.elsrtm(shots, *obs, 1)
            out.append([mis, *e.read_images().values(), *e.ac_born(shots, m),
                        e.ac_born_adj(shots, *obs), *e.forward(shots)])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_graph_memory_of_many_batches_is_bounded(cuda_device):
    """The normal operator over 110 single-shot batches of 2000 steps: 440 thousand launches, whose
    graphs at 4 KB a launch would hold 1.8 GB; at most 0.5 GB and the last graph are kept.  The
    image is that of direct launches."""
    import torch
    c, vp, vs, rho, w, _ = _case(60, 48, 48, 8, 2000)
    shots = [s for s in _shots(c, uneven=False)[:2] for _ in range(55)]
    m = torch.full(vp.shape, 0.01, device="cuda")
    out = []
    for graph in (1, 0):
        with Elastic2D(c["allnx"], c["allnz"], c["nx"], c["pml"], c["nt"], c["dx"], c["dz"], c["dt"],
                       boundary="pml", max_shots=1, max_ntr=c["nx"]) as e:
            e.set_option("graph", graph)
            e.set_models(vp, vs, rho)
            e.set_wavelet(w)
            img = torch.zeros_like(m)
            e.ac_normal_device(shots[:1], m.data_ptr(), img.data_ptr())  # allocates the state
            free = torch.cuda.mem_get_info()[0]
            e.ac_normal_device(shots, m.data_ptr(), img.data_ptr())
            assert free - torch.cuda.mem_get_info()[0] < 1 << 30
            out.append(img.cpu().numpy())
    np.testing.assert_array_equal(*out)


def test_elsrtm_half_steps_allocate_no_fused_state(cuda_device):
    """ELSRTM on half steps (ring 0) does not hold the fused passes' second buffers: three forward
    sets of 15 arrays, an adjoint set of 11 and a Born source of 3 (59 arrays of every slot); with
    "adjoint_born", whose backward pass is made of half steps, not the adjoint set."""
    import torch
    c, vp, vs, rho, w, rng = _case(500, 284, 500, 8, 3)
    shots = _shots(c, uneven=False)
    ntr = sum(s.ntr for s in shots)
    obs = [rng.normal(size=(ntr, c["nt"])).astype(np.float32) for _ in range(2)]
    img = 0.05 * rng.normal(size=vp.shape).astype(np.float32)
    array = 4 * len(shots) * (500 + 16) * 320
    used = {}
    for name, opts in (("fused", {}), ("half", {"ring": 0}), ("born", {"adjoint_born": 1})):
        with _ctx(c, shots, boundary="pml") as e:
            e.set_option("graph", 0)
            for k, v in opts.items():
                e.set_option(k, v)
            e.set_models(vp, vs, rho)
            e.set_wavelet(w)
            e.set_image(img, img)
            free = torch.cuda.mem_get_info()[0]
            e.elsrtm(shots, *obs, 1)
            used[name] = free - torch.cuda.mem_get_info()[0]
    assert used["half"] <= used["fused"] - 57 * array, used
    assert used["born"] <= used["fused"] - 10 * array, used


@pytest.mark.parametrize("shots_n", [13107, 13108])
def test_elsrtm_of_the_largest_batches(cuda_device, shots_n):
    """ELSRTM with a PML and the most shots that the tile launches' grid takes (five slices a shot,
    65535 in all), and one more, against the same shots in batches of 700."""
    c, vp, vs, _, w, rng = _case(16, 16, 16, 8, 24)
    igx = np.arange(8, 24, 5, dtype=np.int32)
    shots = [ShotGeom(0, 9 + k % 14, 10, 11, igx, 16) for k in range(shots_n)]
    obs = [rng.normal(size=(shots_n * len(igx), c["nt"])).astype(np.float32) for _ in range(2)]
    img = 0.05 * rng.normal(size=vp.shape).astype(np.float32)
    out = []
    for cap in (shots_n, 700):
        with Elastic2D(16, 16, 16, 8, c["nt"], c["dx"], c["dz"], c["dt"], boundary="pml",
                       max_shots=cap, max_ntr=len(igx)) as e:
            e.set_models(vp, vs)
            e.set_wavelet(w)
            e.set_image(img, img)
            mis = e.elsrtm(shots, *obs, 1)
            out.append((mis, e.read_images()))
    assert abs(out[0][0] - out[1][0]) < GATE * shots_n
    for k, v in out[1][1].items():
        if not np.any(v):  # the scattered adjoint's images
            assert not np.any(out[0][1][k]) and k not in ("pp_grad", "ps_grad", "b_pp", "b_ps")
            continue
        assert rel(out[0][1][k], v) < (BORN_GATE if k in ("b_pp", "b_ps") else GATE), k


@pytest.mark.parametrize("acoustic", [True, False])
def test_tiles_without_memory_for_their_buffers(cuda_device, acoustic):
    """With room for three of the extra arrays that the tile steps need (seven acoustic, six for
    ELSRTM), a context stays on the other kernels and gives those three back; once there is memory
    again, setting "tile" brings the tiles back."""
    import torch
    c, vp, vs, rho, w, rng = _case(592, 496, 592, 8, 12)
    shots = _shots(c, uneven=False) * 8
    ntr = sum(s.ntr for s in shots)
    obs = [rng.normal(size=(ntr, c["nt"])).astype(np.float32) for _ in range(2)]
    m = 0.05 * rng.normal(size=vp.shape).astype(np.float32)
    array = 4 * len(shots) * (592 + 16) * 512

    def run(e):
        e.profile(True)
        if acoustic:
            out = [*e.ac_born(shots, m), e.ac_born_adj(shots, *obs)]
        else:
            out = [e.elsrtm(shots, *obs, 1), *e.read_images().values()]
        tiles = any("tile" in name for name in e.profile_report())
        e.profile(False)
        return out, tiles

    with _ctx(c, shots, boundary="pml") as e:
        e.set_models(vp, vs, rho)
        e.set_wavelet(w)
        e.set_image(m, m)
        e.set_option("tile", 0)
        want, tiles = run(e)
        assert not tiles
        torch.cuda.empty_cache()
        held = [torch.empty(torch.cuda.mem_get_info()[0] - 8 * array, dtype=torch.uint8, device="cuda")]
        with pytest.raises(torch.OutOfMemoryError):
            while True:  # the rest, in blocks of one array
                held.append(torch.empty(array, dtype=torch.uint8, device="cuda"))
        del held[-3:]
        torch.cuda.empty_cache()
        left = torch.cuda.mem_get_info()[0]
        e.set_option("tile", -1)
        got, tiles = run(e)
        assert not tiles and torch.cuda.mem_get_info()[0] >= left - (16 << 20)
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
        del held
        torch.cuda.empty_cache()
        assert not run(e)[1]
        e.set_option("tile", -1)
        got, tiles = run(e)
        assert tiles
        for a, b in zip(got, want):
            assert rel(a, b) < BORN_GATE or not np.any(b)
