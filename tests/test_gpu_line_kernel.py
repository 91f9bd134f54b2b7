"""The half-line stage kernel of 3-D Euler on unwarped bricks (Nq = 4..8; Kennedy-Gruber,
entropy conservative, central flux differencing and the weak form), and its curved form, against the oracle and
the generic stage kernel: grids with fewer and with more elements than its CTAs, faces on
the boundary, tendencies that set and that add, and buffers aligned to 16 bytes only.

Tolerances, those of the other pipelined kernels: max |gpu - oracle| <= 1e-12 of max |oracle|
per array in FP64 (the register after steps, a small difference of larger terms, 1e-11),
1e-6 for the state after two FP32-bulk steps.
"""

import numpy as np
import pytest

import oracle as O
from gpu_util import initial_state, oracle_law, product_scheme, rel_err, wrap_oracle_grid

pytestmark = pytest.mark.gpu

SCHEMES = ["eul_kg", "eul_ec", "eul_weak", "eul_fdc"]
# more elements than CTAs (FP64: 12, 6, 4, 3, 2 an SM at Nq = 4..8)
MANY = {4: (13, 12, 12), 5: (10, 10, 9), 6: (9, 9, 8), 7: (8, 8, 7), 8: (7, 7, 7)}


def _build(rb, nq, K, per, scheme, precision="fp64"):
    og = O.Grid(3, nq, K, [0.0] * 3, [10.0, 8.0, 9.0], per)
    law, form = product_scheme(rb, scheme, 3)
    dg = rb.DGSEM(law=law, grid=wrap_oracle_grid(og), volume_form=form, surface_numericalflux=rb.RusanovFlux(),
                  precision=precision)
    assert dg.pipelined_ctas > 0
    return og, dg, oracle_law(scheme, 3)


@pytest.mark.parametrize("nq", range(4, 9))
@pytest.mark.parametrize("scheme", SCHEMES)
def test_small_open_grid(rb, cuda_ok, scheme, nq):
    """Both tendency modes against the oracle, and two steps against the generic kernel."""
    og, dg, olaw = _build(rb, nq, (3, 2, 2), (1, 0, 1), scheme)
    q = initial_state(og, olaw, scheme, seed=3)
    ref = og.tendency(olaw, q)
    qg, dq = rb.GridArray.from_numpy(q), rb.GridArray.from_numpy(q)
    dg(dq, qg, 0.0, increment=False)
    assert rel_err(dq.numpy(), ref) <= 1e-12
    dq = rb.GridArray.from_numpy(q)
    dg(dq, qg, 0.0, increment=True)
    assert rel_err(dq.numpy(), ref + q) <= 1e-12
    out = []
    for path in ("auto", "generic"):
        dg.set_kernel_path(path)
        qs = rb.GridArray.from_numpy(q)
        rb.LSRK54(dg, qs, 1e-3).dostep(qs, 2)
        out.append(qs.numpy())
    dg.set_kernel_path("auto")
    dg.sync_status()
    assert rel_err(out[0], out[1]) <= 1e-12


@pytest.mark.parametrize("nq", range(4, 9))
@pytest.mark.parametrize("scheme", ["eul_kg", "eul_weak"])
def test_more_elements_than_ctas(rb, cuda_ok, scheme, nq):
    og, dg, olaw = _build(rb, nq, MANY[nq], (1, 1, 1), scheme)
    assert og.E > dg.pipelined_ctas
    q = initial_state(og, olaw, scheme, seed=4)
    qo, dqo = q.copy(order="F"), og.state(olaw)
    for i in range(2):
        og.lsrk54_step(olaw, qo, dqo, i * 1e-3, 1e-3)
    qg = rb.GridArray.from_numpy(q)
    s = rb.LSRK54(dg, qg, 1e-3)
    s.dostep(qg, 2)
    dg.sync_status()
    assert rel_err(qg.numpy(), qo) <= 1e-12
    assert rel_err(s.dq.numpy(), dqo) <= 1e-11
    _, dg32, _ = _build(rb, nq, MANY[nq], (1, 1, 1), scheme, "fp32_bulk")
    qg = rb.GridArray.from_numpy(q)
    rb.LSRK54(dg32, qg, 1e-3).dostep(qg, 2)
    dg32.sync_status()
    assert rel_err(qg.numpy(), qo) <= 1e-6


@pytest.mark.parametrize("nq", [5, 8])
def test_sixteen_byte_alignment(rb, cuda_ok, nq):
    """Buffers that start 16 bytes past a 32-byte boundary: the same bits as aligned ones."""
    import torch

    og, dg, olaw = _build(rb, nq, (3, 3, 2), (1, 1, 1), "eul_kg")
    q = initial_state(og, olaw, "eul_kg", seed=5)
    aligned = rb.GridArray.from_numpy(q)

    def shifted(t):
        s = torch.empty(t.numel() + 2, dtype=t.dtype, device=t.device)[2:].view(t.shape)
        assert s.data_ptr() % 32 == 16
        return rb.GridArray(s.copy_(t), aligned.ns, aligned.np, aligned.E)

    moved = shifted(aligned.data)
    a, b = rb.LSRK54(dg, aligned, 1e-3), rb.LSRK54(dg, moved, 1e-3)
    b.dq = shifted(a.dq.data)
    a.dostep(aligned, 1)
    b.dostep(moved, 1)
    dg.sync_status()
    assert torch.equal(aligned.data, moved.data) and torch.equal(a.dq.data, b.dq.data)
    assert np.isfinite(aligned.numpy()).all()


@pytest.mark.parametrize("precision", ["fp64", "fp32_bulk"])
def test_curved_sixteen_byte_alignment(rb, cuda_ok, precision):
    """The curved kernel (Nq = 8) on open faces with a state 16 bytes past a 32-byte boundary:
    the same bits as an aligned one, and the generic kernel's state to 1e-12 (FP32 bulk 1e-6)."""
    import torch

    og = O.Grid(3, 8, (2, 3, 2), [0.0] * 3, [10.0] * 3, (1, 0, 1), O.WARP_SINE, 0.1)
    law, form = product_scheme(rb, "eul_kg", 3)
    dg = rb.DGSEM(law=law, grid=wrap_oracle_grid(og), volume_form=form, surface_numericalflux=rb.RusanovFlux(),
                  precision=precision)
    assert dg.geometry == "curved" and dg.pipelined_ctas > 0
    q = initial_state(og, oracle_law("eul_kg", 3), "eul_kg", seed=6)
    a = rb.GridArray.from_numpy(q)
    t = torch.empty(a.data.numel() + 2, dtype=a.data.dtype, device=a.data.device)[2:].view(a.data.shape)
    assert t.data_ptr() % 32 == 16
    b = rb.GridArray(t.copy_(a.data), a.ns, a.np, a.E)
    for x in (a, b):
        rb.LSRK54(dg, x, 1e-3).dostep(x, 2)
    dg.sync_status()
    assert torch.equal(a.data, b.data)
    dg.set_kernel_path("generic")
    c = rb.GridArray.from_numpy(q)
    rb.LSRK54(dg, c, 1e-3).dostep(c, 2)
    assert rel_err(a.numpy(), c.numpy()) <= (1e-12 if precision == "fp64" else 1e-6)


def _continuous_state(og, seed):
    """A state whose values at a point are the same bits in every element that has it."""
    x = np.moveaxis(og.points(), 1, 2).reshape(-1, 3)  # (np * E, 3)
    key = np.round(np.mod(x / np.array([10.0, 8.0, 9.0]), 1.0) * 1e6).astype(np.int64) % 10**6
    _, point = np.unique(key, axis=0, return_inverse=True)
    r = np.random.default_rng(seed).uniform(-0.1, 0.1, (5, point.max() + 1))[:, point.ravel()]
    rho, u = 1 + r[0], [0.4 + r[1], -0.3 + r[2], 0.2 + r[3]]
    E = (0.7 + r[4]) / 0.4 + rho * sum(v * v for v in u) / 2
    return np.asfortranarray(np.stack([rho] + [rho * v for v in u] + [E]).reshape(5, og.np, og.E).transpose(1, 0, 2))


@pytest.mark.parametrize("nq", range(4, 9))
@pytest.mark.parametrize("scheme", SCHEMES)
def test_equal_traces_have_no_jump(rb, cuda_ok, scheme, nq):
    """On a state that is continuous across the faces, and at open faces, q+ - q- is exactly 0:
    Rusanov and central faces give the same bits, in tendencies and in both precisions' steps."""
    og = O.Grid(3, nq, (3, 2, 2), [0.0] * 3, [10.0, 8.0, 9.0], (1, 0, 1))
    q = _continuous_state(og, 8)
    law, form = product_scheme(rb, scheme, 3)
    for precision in ("fp64", "fp32_bulk"):
        out = []
        for flux in (rb.RusanovFlux(), rb.CentralFlux()):
            dg = rb.DGSEM(law=law, grid=wrap_oracle_grid(og), volume_form=form, surface_numericalflux=flux,
                          precision=precision)
            assert dg.pipelined_ctas > 0
            qg = rb.GridArray.from_numpy(q)
            dq = qg.similar()
            dg(dq, qg, 0.0, increment=False)
            q_out = qg.similar()
            dg.lsrk54_stage(qg, q_out, qg.similar(), 0, 0.0, 1e-3)
            out.append((dq.numpy(), q_out.numpy()))
        assert np.array_equal(out[0][0], out[1][0])
        assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("precision", ["fp64", "fp32_bulk"])
def test_curved_open_faces_have_no_jump(rb, cuda_ok, precision):
    """One element with six open faces on the curved kernel: Rusanov and central faces alike."""
    og = O.Grid(3, 8, (1, 1, 1), [0.0] * 3, [10.0] * 3, (0, 0, 0), O.WARP_SINE, 0.1)
    law, form = product_scheme(rb, "eul_kg", 3)
    q = initial_state(og, oracle_law("eul_kg", 3), "eul_kg", seed=9)
    out = []
    for flux in (rb.RusanovFlux(), rb.CentralFlux()):
        dg = rb.DGSEM(law=law, grid=wrap_oracle_grid(og), volume_form=form, surface_numericalflux=flux,
                      precision=precision)
        assert dg.geometry == "curved" and dg.pipelined_ctas > 0
        qg = rb.GridArray.from_numpy(q)
        q_out = qg.similar()
        dg.lsrk54_stage(qg, q_out, qg.similar(), 0, 0.0, 1e-3)
        out.append(q_out.numpy())
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1])


@pytest.mark.parametrize("nq", range(4, 9))
def test_fp32_scale_is_rounded_once(rb, cuda_ok, nq):
    """FP32 bulk: the factor of a line's sum, drdx / w, is formed in FP64 and rounded once.

    A gas at rest without pressure but for one interior node, p = 2 (gamma = 2: p = rho e
    exactly): along its x line the sum of a node is one product, 2 times a table entry, so
    the momentum after a stage of unit weight is known to the bit.  (Central faces: the
    wave speed of p = 0 is not taken.)"""
    H0, a = (nq + 1) // 2, 1
    f32 = np.float32
    for K, L in (((3, 1, 1), 10.0), ((7, 1, 1), 10.0), ((5, 1, 1), 0.37), ((1, 1, 1), 1.7)):
        og = O.Grid(3, nq, K, [0.0] * 3, [L, 1.0, 1.0], (1, 1, 1))
        dg = rb.DGSEM(law=rb.EulerLaw(3, 2.0), grid=wrap_oracle_grid(og), volume_form=rb.WeakForm(),
                      surface_numericalflux=rb.CentralFlux(), precision="fp32_bulk")
        assert dg.pipelined_ctas > 0
        q = np.zeros((og.np, 5, og.E), order="F")
        q[:, 0, :] = 1.0
        line = nq * (1 + nq) + np.arange(nq)  # j = k = 1
        q[line[a], 4, :] = 2.0
        qg = rb.GridArray.from_numpy(q)
        q_out = qg.similar()
        dg.lsrk_stage_range(qg, q_out, qg.similar(), 0.0, 1.0, 0, og.E, 0.0, 1.0)
        got = q_out.numpy()[line, 1, 0]
        _, w, D = og.lgl()
        S, drdx = D * w[:, None], og.volume_metrics()[0, 0, 0]
        for m in range(1, nq - 1):
            far = m >= H0  # counted from the far end, with the sign turned
            i, j = (nq - 1 - a, nq - 1 - m) if far else (a, m)
            want = f32(f32(2) * f32(S[i, j])) * f32((-drdx if far else drdx) * (1.0 / w[j]))
            if m != a:
                assert got[m] == float(want), (K, L, m)


@pytest.mark.parametrize("nq", range(4, 9))
@pytest.mark.parametrize("scheme", SCHEMES)
def test_fp32_bulk_steps(rb, cuda_ok, scheme, nq):
    """Two FP32-bulk steps of every volume form on a grid with open faces."""
    og, dg, olaw = _build(rb, nq, (3, 2, 3), (1, 0, 1), scheme, "fp32_bulk")
    q = initial_state(og, olaw, scheme, seed=12)
    qo, dqo = q.copy(order="F"), og.state(olaw)
    for i in range(2):
        og.lsrk54_step(olaw, qo, dqo, i * 1e-3, 1e-3)
    qg = rb.GridArray.from_numpy(q)
    rb.LSRK54(dg, qg, 1e-3).dostep(qg, 2)
    dg.sync_status()
    assert rel_err(qg.numpy(), qo) <= 1e-6


@pytest.mark.parametrize("ratio", [1.21, 1.23, 3.0])
@pytest.mark.parametrize("nq", range(4, 9))
def test_log_mean_branches_in_steps(rb, cuda_ok, nq, ratio):
    """One entropy-conservative step, both precisions, of a state whose density and rho/p take
    two values: on either side of the end of the logarithmic means' series (a ratio of 1.222)
    and far beyond, so that lines take their sums again with the logarithms.

    The step is short: in FP32 bulk the register's error, 5e-6 of its terms' size (some 100 here,
    see test_log_mean_branches), times 1e-4 is 1e-7 of the state; a mean that is wrong by
    1e-3 would change it by 1e-5."""
    og, dg, olaw = _build(rb, nq, (3, 2, 2), (1, 0, 1), "eul_ec")
    rng = np.random.default_rng(13)
    shape = (og.np, og.E)
    rho = np.where(rng.random(shape) < 0.5, 1.0, ratio)
    p = rho / np.where(rng.random(shape) < 0.5, 1.1, 1.1 * ratio)
    u = (0.4, -0.3, 0.2)
    E = p / 0.4 + rho * sum(v * v for v in u) / 2
    q = np.asfortranarray(np.stack([rho] + [rho * v for v in u] + [E], axis=1))
    dt = 1e-4
    qo, dqo = q.copy(order="F"), og.state(olaw)
    og.lsrk54_step(olaw, qo, dqo, 0.0, dt)
    qg = rb.GridArray.from_numpy(q)
    s = rb.LSRK54(dg, qg, dt)
    s.dostep(qg, 1)
    dg.sync_status()
    assert rel_err(qg.numpy(), qo) <= 1e-12 and rel_err(s.dq.numpy(), dqo) <= 1e-11
    _, dg32, _ = _build(rb, nq, (3, 2, 2), (1, 0, 1), "eul_ec", "fp32_bulk")
    qg = rb.GridArray.from_numpy(q)
    rb.LSRK54(dg32, qg, dt).dostep(qg, 1)
    dg32.sync_status()
    assert rel_err(qg.numpy(), qo) <= 1e-6
