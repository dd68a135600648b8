"""The planned application of the preconditioners (tables, grouped products, fused tail) against the general path of
the same optimizer on the same state: ragged and small orders, split parameters, blocks with one plain fp32
preconditioner, parameters without any, both tails, both code widths."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def run(kind, shapes, planned, bits=4, steps=3, wave_bytes=None, **hyper):
    from optimizers import _apply, _base, shampoo2
    g = torch.Generator(device="cuda").manual_seed(3)
    ps = [torch.nn.Parameter(torch.randn(s, generator=g, device="cuda") * 0.1) for s in shapes]
    cls = shampoo2.ShampooAdamW if kind == "adamw" else shampoo2.ShampooSGD
    opt = cls(ps, lr=1e-2, weight_decay=0.03, prec_maxorder=200, prec_bits=bits, stat_compute_steps=10 ** 9, prec_compute_steps=1, **hyper)
    before = _base.PLANNED_APPLY, _apply.WAVE_BYTES
    _base.PLANNED_APPLY = planned
    if wave_bytes:
        _apply.WAVE_BYTES = wave_bytes
    try:
        for k in range(steps):
            for p in ps:
                p.grad = torch.randn(p.shape, generator=g, device="cuda") * 10.0 ** (k - 2)
            opt.step()
            if k == 0:                                   # dense preconditioners from here on
                opt.param_groups[0]["prec_compute_steps"] = 10 ** 9
                for p in ps:
                    for q in opt.state[p]["preconditioner"].preconditioners:
                        n = q.var.shape[0] if q.bits >= 16 else q.var_order
                        a = torch.randn(n, n, generator=g, device="cuda") / n ** 0.5
                        q.quantize(torch.eye(n, device="cuda") + 0.3 * (a + a.T))
        plans = [pl for known in opt._apply_plans.values() for pl in known["plans"].values()]
        assert bool(plans) == planned and all(plans)
    finally:
        _base.PLANNED_APPLY, _apply.WAVE_BYTES = before
    names = ("exp_avg", "exp_avg_sq") if kind == "adamw" else ("momentum",)
    return [p.detach() for p in ps] + [opt.state[p][n] for n in names for p in ps] + [p.grad for p in ps if p.dim() < 2]


SHAPES = [(64, 64), (65, 129), (200, 72), (7,), (300, 450), (200, 200, 1, 1), (5, 96), (96, 3, 3, 3), (1, 130, 77), (128, 199), (64, 64), (1,)]


@pytest.mark.parametrize("kind,bits,hyper", [("adamw", 4, {}), ("adamw", 8, {}), ("sgd", 4, {}), ("sgd", 4, dict(nesterov=True, momentum=0.5)),
                                             ("adamw", 4, dict(start_prec_step=3))])
def test_planned_application_matches_the_general_path(kind, bits, hyper, native_lib):
    a = run(kind, SHAPES, True, bits, **hyper)
    b = run(kind, SHAPES, False, bits, **hyper)
    for x, y in zip(a, b):
        assert float((x - y).norm()) <= 3e-6 * float(y.norm()) + 1e-12
    assert native_lib.qt_device_error(1) == 0


def test_waves_give_the_same_bits(native_lib):
    a, b = run("adamw", SHAPES, True), run("adamw", SHAPES, True, wave_bytes=1 << 19)
    assert all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("width", [128, 192, 256])
def test_tile_widths_agree(width, native_lib, monkeypatch):
    """The width is chosen by size (_tile_width); only the order of a norm's partial sums depends on it."""
    from optimizers import _apply
    shapes = SHAPES + [(130, 257), (257, 130), (128, 449), (449, 64)]
    a = run("adamw", shapes, True)
    monkeypatch.setattr(_apply, "_tile_width", lambda waves, sms: width)
    for x, y in zip(a, run("adamw", shapes, True)):
        assert float((x - y).norm()) <= 1e-6 * float(y.norm())
    assert native_lib.qt_device_error(1) == 0


def test_gradients_that_move_and_graph_replay(native_lib):
    """Gradients at new addresses every step (above) and steps under cuda_graph=True give the eager results."""
    a, b = run("adamw", SHAPES, True), run("adamw", SHAPES, True, cuda_graph=True)
    for x, y in zip(a, b):
        assert float((x - y).norm()) <= 1e-6 * float(y.norm())


def test_mixed_state_falls_back(native_lib):
    """bf16 preconditioner state has no plan: the general path takes the step."""
    from optimizers import shampoo2
    p = torch.nn.Parameter(torch.randn(96, 80, device="cuda"))
    opt = shampoo2.ShampooAdamW([p], prec_bits=16, stat_compute_steps=1, prec_compute_steps=1)
    p.grad = torch.randn_like(p)
    opt.step()
    assert not opt._apply_plans and bool(torch.isfinite(p).all())


def refreshed(shapes, planned, bits, rect, graph=False):
    """State after one refresh (under graph replay: three, of which the first is eager)."""
    from optimizers import _base, shampoo2
    g = torch.Generator(device="cuda").manual_seed(5)
    ps = [torch.nn.Parameter(torch.randn(s, generator=g, device="cuda") * 0.1) for s in shapes]
    opt = shampoo2.ShampooAdamW(ps, lr=1e-3, prec_maxorder=400, prec_bits=bits, stat_compute_steps=1, prec_compute_steps=1, rect_t1=rect[0],
                                rect_t2=rect[1], cuda_graph=graph)
    before = _base.PLANNED_REFRESH
    _base.PLANNED_REFRESH = planned
    try:
        for _ in range(3 if graph else 1):
            for p in ps:
                m, k = p.shape[0], p[0].numel()
                d = torch.zeros(m, k, device="cuda")
                r = min(m, k)
                d[torch.arange(r), torch.arange(r)] = torch.linspace(0.3, 1.0, r, device="cuda")[torch.randperm(r, generator=g, device="cuda")]
                p.grad = ((d + 1e-4 * torch.randn(m, k, generator=g, device="cuda")) * 0.1).reshape(p.shape)
            opt.step()
    finally:
        _base.PLANNED_REFRESH = before
    assert any(known["refresh"] is not None for known in opt._apply_plans.values()) == planned
    out = []
    for p in ps:
        pre = opt.state[p]["preconditioner"]
        for s, q in zip(pre.statistics, pre.preconditioners):
            out.append((s.Svalue, s.max_eigenvalue, s.absmax if s.bits < 16 else s.var, q.diag if q.bits < 16 else q.var, s.var, q.var))
    return out, [p.detach() for p in ps]


@pytest.mark.parametrize("bits,rect", [(4, (1, 4)), (8, (1, 4)), (4, (0, 1)), (4, (2, 0))])
def test_planned_refresh_matches_the_general_engine(bits, rect, native_lib):
    """Orders at the edges of tiles and panels, odd and even, both sides of a block in one class, an order below 64."""
    shapes = [(64, 64), (65, 97), (128, 128), (129, 160), (96, 96), (160, 8, 20), (333, 400), (400, 333), (48, 64)]
    (a, pa), (b, pb) = refreshed(shapes, True, bits, rect), refreshed(shapes, False, bits, rect)
    for x, y in zip(a, b):
        for u, v in zip(x[:4], y[:4]):
            assert float((u - v).norm()) <= 5e-4 * float(v.norm())
        assert all(float((u != v).float().mean()) <= 2e-2 for u, v in zip(x[4:], y[4:]) if u.dtype == torch.uint8)
    for u, v in zip(pa, pb):
        assert float((u - v).norm()) <= 2e-3 * float(v.norm())       # AdamW turns a moved code into a step of lr
    assert native_lib.qt_device_error(1) == 0


def test_planned_refresh_under_graph_replay(native_lib):
    shapes = [(64, 64), (129, 160), (96, 96)]
    (a, pa), (c, pc) = refreshed(shapes, True, 4, (1, 4), graph=True), refreshed(shapes, False, 4, (1, 4), graph=True)
    for u, v in zip(pa, pc):                             # rounding moves codes, and they add up over three refreshes
        assert float((u - v).norm()) <= 2e-3 * float(v.norm())
