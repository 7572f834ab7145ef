"""The cube sweep of the boundary entry points at the periodic faces: floats next
to a face, whose cube can come out on the other side by rounding, boxes that do
not start at zero, positions that left the box or their cube since the sort.
The pairs are those of the oracle's FP32 predicate, bit for bit; sums within
their roundings of the FP64 oracle."""
import ctypes as C

import numpy as np
import pytest

from gpucell_gb300 import generator as gen

pytestmark = pytest.mark.gpu

U = 2.0 ** -24   # FP32 unit roundoff
F = np.float32


def _config(bbox, coor, n_b1=0, n_b2=0, mass=1.0):
    n = len(coor)
    vol = np.prod([bbox[2 * a + 1] - bbox[2 * a] for a in range(3)])
    return gen.Config(name="faces", bbox=np.array(bbox, F), pmask=7, n_b1=n_b1, n_b2=n_b2, n_fluid=n - n_b1 - n_b2,
                      coor=np.ascontiguousarray(coor, F), velhalf=np.zeros((n, 3), F), den_init=float(n / vol),
                      phys=gen.Physics(ext_force=0.0, mass=mass))


def _neighbors(ps):
    import torch
    from gpucell_gb300 import _lib
    cnt = torch.zeros(ps.n, dtype=torch.int32, device="cuda")
    h = torch.zeros(ps.n, dtype=torch.int64, device="cuda")
    _lib.call("gc_debug_neighbor_stats", ps.n, ps.p("TotalCoor"), ps.p("SortPart"), ps.p("BeginEndCube"),
              C.c_void_p(cnt.data_ptr()), C.c_void_p(h.data_ptr()))
    inv = ps.fetch()["slot_of"]
    return cnt.cpu().numpy()[inv], h.cpu().numpy().view(np.uint64)[inv]


def _against_oracle(cfg, pos, what):
    from gpucell_gb300.host import ParticleSystem
    from oracle.binding import Oracle, assert_forces_close
    vel = np.random.default_rng(5).normal(size=(cfg.n, 3)).astype(F).astype(np.float64)
    ps, o = ParticleSystem(cfg, noise=True), Oracle(cfg, noise=True)
    ps.set_state(pos=pos, vel=vel)
    ps.con_cube_list()
    o.set(pos=pos, vel=vel)
    count, ids = o.neighbor_stats()
    gc, gh = _neighbors(ps)
    assert np.array_equal(gc, count) and np.array_equal(gh, ids)
    # a lane adds at most a quarter of the terms (each good to about a dozen roundings) in sequence
    count = count.max()
    rtol = (count / 4 + 16) * U
    fluid, wall = slice(cfg.n_b1 + cfg.n_b2, None), slice(cfg.n_b1, cfg.n_b1 + cfg.n_b2)
    ps.density()
    o.call("density")
    g = ps.fetch()
    np.testing.assert_allclose(g["rho"][fluid], o.rho[fluid], rtol=rtol)
    o.set(rho=g["rho"])
    ps.bound2_vel()
    o.call("bound2_vel")
    g = ps.fetch()
    # weighted means of velocities up to 5: the weights and the products round as above
    np.testing.assert_allclose(g["vel"][wall], o.vel[wall], rtol=0, atol=2 * 5 * rtol)
    ps.eos()
    g = ps.fetch()
    o.set(vel=g["vel"], press=g["press"])
    ps.sdpd_force()
    o.call("sdpd_force")
    g = ps.fetch()
    assert_forces_close(g["force"], o.force, o.force_scale(o.SCALE_SDPD), k=16 + count / 4, what=f"{what} sdpd")
    z = np.zeros((cfg.n, 3))
    ps.set_state(force=z)
    o.set(force=z)
    ps.rep_force()
    o.call("rep_force")
    g = ps.fetch()
    assert_forces_close(g["force"], o.force, o.force_scale(o.SCALE_REP), k=64 + count / 4, what=f"{what} repulsion")


@pytest.mark.parametrize("bbox", [(-6, 6, 0, 8, -16 / 3, 16 / 3), (0, 14, -4, 4, 0, 3.1)], ids=["12", "14"])
def test_floats_next_to_the_faces(cuda_device, bbox):
    rng = np.random.default_rng(1)
    b = np.array(bbox, F)
    lo, hi = b[0::2], b[1::2]
    n = int(12 * np.prod(hi - lo))
    x = np.clip((lo + rng.uniform(0, 1, (n, 3)) * (hi - lo)).astype(F), lo, np.nextafter(hi, lo))
    wraps = 0
    for a in range(3):
        below = [hi[a]]
        for _ in range(3):
            below.append(np.nextafter(below[-1], lo[a]))
        special = np.array(below[1:] + [lo[a], np.nextafter(lo[a], hi[a])], F)
        rows = rng.choice(n, 200, replace=False)
        x[rows, a] = rng.choice(special, 200)
        m = int(np.floor(float(hi[a] - lo[a]) / (1.0 + 1e-4)))   # cubes along the axis
        wraps += int((np.floor((special - lo[a]) * F(m / float(hi[a] - lo[a]))) >= m).sum())
    assert wraps > 0   # some of them sort into the first cube
    cfg = _config(bbox, x, n_b1=n // 10, n_b2=n // 10)
    _against_oracle(cfg, x.astype(np.float64), "faces")


def test_positions_outside_the_box(cuda_device):
    rng = np.random.default_rng(2)
    bbox = (-3.1, 0, 0, 7.9, -5, 5)
    b = np.array(bbox, F)
    lo, hi = b[0::2], b[1::2]
    n = 3001
    x = np.clip((lo + rng.uniform(0, 1, (n, 3)) * (hi - lo)).astype(F), lo, np.nextafter(hi, lo))
    cfg = _config(bbox, x, n_b1=n // 10, n_b2=n // 10)
    loose = rng.random((n, 3)) < 0.3
    out = (x + (hi - lo) * (loose & (x < lo + 0.4)) - (hi - lo) * (loose & (x > hi - 0.4))).astype(F)
    assert ((out >= hi) | (out < lo)).any()
    _against_oracle(cfg, out.astype(np.float64), "outside")


@pytest.mark.parametrize("box", [(3.1, 4.2, 6.5), (9.0, 8.0, 11.0)], ids=["three", "nine"])
def test_positions_moved_since_the_sort(cuda_device, box):
    """The candidates are those of the cubes as sorted, the pairs those of the
    positions as they are, wrapped meanwhile or not."""
    from gpucell_gb300.host import ParticleSystem
    rng = np.random.default_rng(3)
    L = np.array(box, F)
    n = int(9 * np.prod(L))
    x = np.minimum((rng.uniform(0, 1, (n, 3)) * L).astype(F), np.nextafter(L, F(0)))
    ps = ParticleSystem(_config([0, box[0], 0, box[1], 0, box[2]], x), noise=False)
    m = np.floor(L.astype(np.float64) / (1.0 + 1e-4)).astype(int)
    cube = np.floor(x * (m / L.astype(np.float64)).astype(F)).astype(int) % m
    y = (x + rng.uniform(-0.3, 0.3, (n, 3))).astype(F)
    y = np.where(y >= L, y - L, np.where(y < 0, y + L, y)).astype(F)
    ps.set_state(pos=y)
    ps.density()
    rho = ps.fetch()["rho"]
    want = np.empty(n)
    for i in range(n):
        dc = np.abs(cube - cube[i])
        near = (np.minimum(dc, m - dc) <= 1).all(1)
        near[i] = False
        d = y[i] - y[near]
        d = np.where(d > L / 2, d - L, np.where(d < -L / 2, d + L, d)).astype(F).astype(np.float64)
        r = np.sqrt((d ** 2).sum(1))
        r = r[r < 1.0]
        want[i] = 21 / (2 * np.pi) * (1.0 + ((1 - r) ** 4 * (1 + 4 * r)).sum())
    np.testing.assert_allclose(rho, want, rtol=(60 / 4 + 16) * U)


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_pair_forces_cancel_next_to_a_face(cuda_device, axis):
    """Isolated pairs in the cubes next to the faces of a box that does not
    start at zero: F_ij = -F_ji to the last bit."""
    from gpucell_gb300.host import ParticleSystem
    rng = np.random.default_rng(axis)
    L = np.array([20.0, 20.0, 20.0])
    lo = np.zeros(3)
    L[axis], lo[axis] = 64.0, -64.0
    w = 64.0 / 63   # cubes along the axis
    pairs = []
    other = [a for a in range(3) if a != axis]
    for k, (p, q) in enumerate((p, q) for p in range(8) for q in range(8)):
        c = np.zeros(3)
        c[axis] = (-w, 0.0, -64.0 + w, -2 * w)[k % 4]
        c[other[0]], c[other[1]] = 1.2 + 2.4 * p, 1.2 + 2.4 * q
        e = rng.normal(size=3)
        e *= rng.uniform(0.2, 0.95) / np.linalg.norm(e)
        pairs += [c + e / 2, c - e / 2]
    x = np.array(pairs)
    x[:, axis] = np.where(x[:, axis] >= 0, x[:, axis] - 64.0, x[:, axis])
    x = x.astype(F)
    x[:, axis] = np.clip(x[:, axis], F(-64.0), np.nextafter(F(0), F(-1)))
    bbox = np.stack([lo, lo + L], 1).ravel()
    cfg = _config(bbox, x)
    vel = rng.normal(size=(cfg.n, 3)).astype(F)
    ps = ParticleSystem(cfg, noise=True)
    ps.set_state(vel=vel)
    ps.density()
    ps.eos()
    ps.sdpd_force()
    f = ps.fetch()["force"]
    assert (np.abs(f).max(1) > 0).all()
    np.testing.assert_array_equal(f[0::2], -f[1::2])
