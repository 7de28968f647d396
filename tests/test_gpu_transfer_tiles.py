"""P2G and G2P over the grid sizes at which their tile shapes change, against a
plain FP64 restatement in numpy: ragged boxes (no axis a multiple of a tile),
grids just below and above each change, sparse particles (empty tiles) and
crowded cells.  h is a power of two, so pos / h is exact in FP32 and the
tolerances are those of the parity tests."""
import numpy as np
import pytest

from fluid_simulator_gb300 import native as N

from parity_util import REL_GRID, assert_close_field

pytestmark = pytest.mark.gpu

RES = 128


def particles(shape, n, seed):
    """n particles: most spread over the lower 60 % of the box, some crowded into one cell."""
    rng = np.random.default_rng(seed)
    lo, hi = np.full(3, 1.3), np.array(shape) - 1.3
    pos = lo + rng.random((n, 3)) * (hi - lo) * [1.0, 0.6, 1.0]
    pos[: n // 50] = np.array(shape) // 2 + rng.random((n // 50, 3)) * 0.99
    pos = (pos / RES).astype(np.float32)
    vel = (rng.standard_normal((n, 3))).astype(np.float32)
    c = (rng.standard_normal((n, 9)) * 20).astype(np.float32)
    return pos, vel, c


def p2g_ref(shape, pos, vel, c):
    """(u[3], weights[3], avgPNum): trilinear scatter in FP64."""
    h = 1.0 / RES
    p, g = pos.astype(np.float64), pos.astype(np.float64) * RES
    out, wts = [], []
    for a in range(4):
        off = np.array([0.0 if d == a else 0.5 for d in range(3)])
        base = np.floor(g - off)
        f = g - off - base
        num, den = np.zeros(shape), np.zeros(shape)
        for o in range(8):
            b = np.array([(o >> 2) & 1, (o >> 1) & 1, o & 1])
            w = np.where(b, f, 1.0 - f).prod(1)
            at = (base + b).astype(np.int64) - np.array([1 if d == a else 0 for d in range(3)])
            ok = ((at >= 0) & (at < shape)).all(1)
            idx = tuple(at[ok].T)
            np.add.at(den, idx, w[ok])
            if a < 3:
                val = vel[:, a].astype(np.float64)
                if c is not None:
                    val = val + (c[:, 3 * a:3 * a + 3] * ((base + b + off) * h - p)).sum(1)
                np.add.at(num, idx, (w * val)[ok])
        if a == 3:
            return out, wts, den
        out.append(np.where(den > 1e-6, num / np.maximum(den, 1e-300), 0.0))
        wts.append(den)


# P2G tiles: 7x9x5 and 23x29x30 run 4x4x4, 37x21x44 4x4x8, 48^3 and 66x70x50 4x8x8, 90x61x75
# 8x8x16, 107x90x66 (280) and the 128^3 ones 16x12x16, 208x208x200 (2197) 16x16x16
SHAPES = [(7, 9, 5), (23, 29, 30), (37, 21, 44), (48, 48, 48), (66, 70, 50), (90, 61, 75), (107, 90, 66),
          (128, 112, 128), (128, 128, 120), (208, 208, 200)]


@pytest.mark.parametrize("transfer", [N.FLIP, N.APIC])
@pytest.mark.parametrize("shape", SHAPES)
def test_p2g_matches_fp64_at_every_tile_shape(gpu, shape, transfer):
    n = min(120_000, 8 * int(np.prod(np.array(shape) - 2)))
    pos, vel, c = particles(shape, n, sum(shape))
    prm = N.default_params(transfer=transfer, resolution=RES)
    sim = N.Simulation(RES, prm, dims=[(k + 0.01) / RES for k in shape])
    assert sim.shape == shape
    sim.set_particles(pos, vel, c)
    sim.stage(N.STAGE_P2G, 0.01)
    ref, wts, avg = p2g_ref(shape, pos, vel, c if transfer == N.APIC else None)
    for a, f in enumerate((N.F_VX, N.F_VY, N.F_VZ)):
        # a face whose weight sum is within FP32 rounding of the 1e-6 threshold may go either way
        near = np.abs(wts[a] - 1e-6) < 1e-9
        assert_close_field(np.where(near, 0, sim.grid(f)), np.where(near, 0, ref[a]), REL_GRID, f"u{a}")
    assert_close_field(sim.grid(N.F_AVGPNUM), avg, REL_GRID, "avgPNum")
    cells = np.floor(pos.astype(np.float64) * RES).astype(np.int64)
    count = np.zeros(shape, np.int64)
    np.add.at(count, tuple(cells.T), 1)
    assert np.array_equal(sim.grid(N.F_COUNT), count)
    assert np.array_equal(sim.grid(N.F_FLAGS) == N.WATER, count > 0)
    sim.close()


def g2p_ref(shape, transfer, v2, u, pos, vel, fr):
    """Particle velocities (and APIC matrices) from the grid, FP64, particles in cell order."""
    g = pos.astype(np.float64) * RES
    vout, cout = np.empty(pos.shape), np.empty((len(pos), 9))
    for a in range(3):
        off = np.array([0.0 if d == a else 0.5 for d in range(3)])
        base = np.floor(g - off)
        f = g - off - base
        val, dif, grad = np.zeros(len(pos)), np.zeros(len(pos)), np.zeros((len(pos), 3))
        for o in range(8):
            b = np.array([(o >> 2) & 1, (o >> 1) & 1, o & 1])
            w = np.where(b, f, 1.0 - f)
            at = tuple(((base + b).astype(np.int64) - np.array([1 if d == a else 0 for d in range(3)])).T)
            x = v2[a][at].astype(np.float64)
            val += w.prod(1) * x
            dif += w.prod(1) * (x - u[a][at])
            for d in range(3):
                sign = np.where(f[:, d] - b[d] > 0, -1.0, 1.0)
                grad[:, d] += sign * RES * np.delete(w, d, 1).prod(1) * x
        vout[:, a] = val if transfer != N.FLIP else val * (1.0 - fr) + (dif + vel[:, a]) * fr
        cout[:, 3 * a:3 * a + 3] = grad
    return vout, cout


@pytest.mark.parametrize("transfer", [N.PIC, N.FLIP, N.APIC])
@pytest.mark.parametrize("shape", SHAPES + [(130, 200, 175)])
def test_g2p_matches_fp64_at_every_tile_shape(gpu, shape, transfer):
    n = min(150_000, 8 * int(np.prod(np.array(shape) - 2)))
    pos, vel, c = particles(shape, n, sum(shape) + 1)
    prm = N.default_params(transfer=transfer, resolution=RES)
    sim = N.Simulation(RES, prm, dims=[(k + 0.01) / RES for k in shape], track_ids=True)
    sim.set_particles(pos, vel, c)
    sim.stage(N.STAGE_P2G, 0.01)
    rng = np.random.default_rng(7)
    v2 = [rng.standard_normal(shape).astype(np.float32) for _ in range(3)]
    for a, f in enumerate((N.F_V2X, N.F_V2Y, N.F_V2Z)):
        sim.set_grid(f, v2[a])
    u = [sim.grid(f).astype(np.float64) for f in (N.F_VX, N.F_VY, N.F_VZ)]
    sim.stage(N.STAGE_G2P, 0.01)
    gp, gv, gc = sim.particles()
    rv, rc = g2p_ref(shape, transfer, v2, u, pos, vel.astype(np.float64), np.float64(np.float32(0.95)))
    assert np.array_equal(gp, pos)
    assert_close_field(gv, rv, 1e-5, "velocity")
    # APIC takes the gradient of v2; PIC and FLIP carry C along unchanged
    if transfer == N.APIC:
        assert_close_field(gc.reshape(-1, 9), rc, 1e-4, "C")
    else:
        assert np.array_equal(gc.reshape(-1, 9), c)
    sim.close()


@pytest.mark.parametrize("shape", [(6, 7, 8), (9, 10, 11), (33, 40, 12)])
@pytest.mark.parametrize("shift", [0, 1])
def test_device_exchange_at_any_alignment(gpu, shape, shift):
    """Grid fields and particle records to and from device buffers that start on a
    16-byte boundary or not, rows padded (nz not a multiple of 4) or not; particle
    counts around the block size."""
    import torch

    sim = N.Simulation(RES, N.default_params(resolution=RES), dims=[(k + 0.01) / RES for k in shape])
    cells = int(np.prod(shape))
    rng = np.random.default_rng(cells + shift)
    for f, dt in ((N.F_VX, np.float32), (N.F_FLAGS, np.uint8)):
        a = (rng.random(cells) * 3).astype(dt)
        src = torch.zeros(cells + 8, dtype=torch.from_numpy(a).dtype, device="cuda")
        dst = torch.zeros_like(src)
        src[shift:shift + cells] = torch.from_numpy(a).cuda()
        torch.cuda.synchronize()
        p = src.data_ptr() + shift * src.element_size()
        sim._check(sim.lib.fsim_set_grid(sim.ctx, f, p, N.DEVICE), "set")
        assert np.array_equal(sim.grid(f).ravel(), a)
        sim._check(sim.lib.fsim_get_grid(sim.ctx, f, dst.data_ptr() + shift * src.element_size(), N.DEVICE), "get")
        assert torch.equal(dst, src)
    for n in (1, 255, 256, 257, 1000):
        pos = rng.random((n, 3)).astype(np.float32)
        vel, c = rng.random((n, 3)).astype(np.float32), rng.random((n, 9)).astype(np.float32)
        sim.set_particles(pos, vel, c)
        gp, gv, gc = sim.particles()
        assert np.array_equal(gp, pos) and np.array_equal(gv, vel) and np.array_equal(gc.reshape(-1, 9), c)
        out = torch.zeros(n * 9 + 4, device="cuda")
        torch.cuda.synchronize()
        import ctypes
        got = ctypes.c_int64()
        sim._check(sim.lib.fsim_get_particles(sim.ctx, None, None, out.data_ptr() + 4 * shift, n, ctypes.byref(got),
                                              N.DEVICE), "particles")
        assert np.array_equal(out.cpu().numpy()[shift:shift + 9 * n].reshape(n, 9), c)
    sim.close()
