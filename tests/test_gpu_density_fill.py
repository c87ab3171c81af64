"""The density of solid cells after a step: each takes the density of its nearest fluid cell (first Chebyshev shell that
holds one, smallest squared distance in it, first in (dz, dy, dx) order on ties; backend-cuda.cu:1243-1290). The copy is
exact, so it is compared bit for bit with a scan written out here, over shapes whose solid count is not a multiple of the
warp, deep solids, thin domains, periodic axes and masks with one fluid cell or none."""
import numpy as np
import pytest
import torch

import scenes
import smoke_abi as abi
import smoke_b200

pytestmark = pytest.mark.gpu


def nearest_fluid(occ, z, y, x, periodic):
    n = occ.shape
    for r in range(1, max(n) + 1):
        best, cell = None, None
        for dz in range(-r, r + 1):
            for dy in range(-r, r + 1):
                step = 1 if max(abs(dz), abs(dy)) == r else 2 * r
                for dx in range(-r, r + 1, step):
                    c = [z + dz, y + dy, x + dx]
                    c = [a % b if p else a for a, b, p in zip(c, n, periodic)]
                    if any(a < 0 or a >= b for a, b in zip(c, n)) or occ[tuple(c)]:
                        continue
                    d2 = dx * dx + dy * dy + dz * dz
                    if best is None or d2 < best:
                        best, cell = d2, tuple(c)
        if cell is not None:
            return cell
    return None


PERIODIC = {"closed": (False, False, False), "plume": (True, False, True), "zout": (False, True, False)}  # (z, y, x)


def mask(kind, shape, rng):
    occ = np.ones(shape, np.uint8)
    if kind == "random":
        occ = (rng.uniform(size=shape) < 0.85).astype(np.uint8)
    elif kind == "one":
        occ[tuple(s // 3 for s in shape)] = 0
    elif kind == "ball":
        z, y, x = np.indices(shape)
        c = [(s - 1) / 2 for s in shape]
        occ = ((z - c[0]) ** 2 + (y - c[1]) ** 2 + (x - c[2]) ** 2 <= (min(shape) / 2 - 1) ** 2).astype(np.uint8)
    return occ


@pytest.mark.parametrize("shape,boundary,kind", [((13, 13, 13), "closed", "ball"), ((14, 14, 14), "plume", "ball"), ((9, 7, 11), "zout", "random"), ((5, 17, 6), "closed", "random"), ((1, 9, 8), "closed", "one"), ((6, 5, 7), "plume", "one"), ((4, 6, 5), "closed", "none")])
def test_solid_density_is_the_nearest_fluid_density(smoke_lib, cuda_stream, shape, boundary, kind):
    nz, ny, nx = shape
    cfg = scenes.make_config(nx, ny, nz, boundary=boundary)
    inp = scenes.random_inputs(cfg, seed=5, solids=False)
    occ = inp["occupancy"] = mask(kind, shape, np.random.default_rng(6))
    sim = smoke_b200.Simulation(smoke_lib, cfg, cuda_stream)
    keep = scenes.load_gpu(sim, inp)
    with torch.cuda.stream(cuda_stream):
        sim.step()
    density = sim.snapshot([abi.VIEW_DENSITY])["density"]
    sim.close()
    del keep
    assert kind == "none" or np.unique(density[occ == 0]).size > (0 if kind == "one" else 4)
    for z, y, x in zip(*np.nonzero(occ)):
        cell = nearest_fluid(occ, z, y, x, PERIODIC[boundary])
        assert density[z, y, x] == (0.0 if cell is None else density[cell]), (z, y, x, cell)


# a cell by itself up to shell 1, a warp from shell 2 on: layers of one to six solid planes, half the cells at random
@pytest.mark.parametrize("boundary", ["closed", "plume", "zout"])
@pytest.mark.parametrize("kind", ["half", "layer1", "layer3", "layer4", "layer6"])
def test_shallow_and_deep_solids(smoke_lib, cuda_stream, kind, boundary):
    nz, ny, nx = 14, 9, 35
    cfg = scenes.make_config(nx, ny, nz, boundary=boundary)
    inp = scenes.random_inputs(cfg, seed=8, solids=False)
    z = np.indices((nz, ny, nx))[0]
    occ = np.random.default_rng(9).uniform(size=(nz, ny, nx)) < 0.5 if kind == "half" else (z >= 2) & (z < 2 + int(kind[5:]))
    occ = inp["occupancy"] = occ.astype(np.uint8)
    sim = smoke_b200.Simulation(smoke_lib, cfg, cuda_stream)
    keep = scenes.load_gpu(sim, inp)
    with torch.cuda.stream(cuda_stream):
        sim.step()
    density = sim.snapshot([abi.VIEW_DENSITY])["density"]
    sim.close()
    del keep
    for c in zip(*np.nonzero(occ)):
        assert density[c] == density[nearest_fluid(occ, *c, PERIODIC[boundary])], c


def test_depth_beyond_a_32_bit_shell(smoke_lib, cuda_stream):
    """Solids up to 13 750 cells deep in a line of cells: the whole shell of that radius has more than 2^32 cells, the part of it
    inside the domain two. Ties go to the lower end (first in scan order)."""
    n, low, high = 30000, 1000, 28501  # solid [low, high)
    cfg = scenes.make_config(1, 1, n, boundary="closed")
    inp = scenes.random_inputs(cfg, seed=10, solids=False)
    occ = np.zeros((n, 1, 1), np.uint8)
    occ[low:high] = 1
    inp["occupancy"] = occ
    sim = smoke_b200.Simulation(smoke_lib, cfg, cuda_stream)
    keep = scenes.load_gpu(sim, inp)
    with torch.cuda.stream(cuda_stream):
        sim.step()
    density = sim.snapshot([abi.VIEW_DENSITY])["density"].ravel()
    sim.close()
    del keep
    z = np.arange(low, high)
    source = np.where(z - (low - 1) <= high - z, low - 1, high)
    assert density[low - 1] != density[high]
    assert np.array_equal(density[z], density[source])
