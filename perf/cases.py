"""The work whose speed counts: what a program that uses this package has it do.

Two kinds of calls, both through the package's public entry points:

* `quant`: the blockwise quantizer (`qtensor.functional`) on one matrix - quantize, then dequantize;
* `step`: one `optimizer.step()` of `shampoo2` / `shampoo1` on the parameters of a model, with
  gradients in place, as it follows `loss.backward()` in a training loop.

A training loop with the default intervals (statistics every 100 steps, inverse roots every 500)
runs three kinds of steps: most only apply the preconditioners ("steady"), one in a hundred also
refreshes the statistics ("stat"), one in five hundred refreshes the roots as well ("refresh").
With both intervals at 1, the benchmark's setting, every step is a "refresh".
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "low-bit-shampoo_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import qtensor.functional as F  # noqa: E402
import workloads  # noqa: E402
from optimizers import shampoo1, shampoo2  # noqa: E402
from optimizers._base import block_shapes  # noqa: E402

DEVICE = "cuda"
MAX_ORDER = 1200               # prec_maxorder of the benchmark configurations (and the default)
NEVER = 1 << 40
DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16}


# ---- the cases --------------------------------------------------------------------------
def _vit(width, depth, mlp, patch, img, classes):
    return {"model": "vit", "width": width, "depth": depth, "mlp": mlp, "patch": patch, "img": img, "classes": classes}


def _resnet(width, d1, d2, d3, d4, classes=100):
    return {"model": "resnet", "width": width, "d1": d1, "d2": d2, "d3": d3, "d4": d4, "classes": classes}


def _swin(width, d1, d2, d3, d4, classes=100):
    return {"model": "swin", "width": width, "d1": d1, "d2": d2, "d3": d3, "d4": d4, "classes": classes}


def _mlp(width, hidden, depth):
    return {"model": "mlp", "width": width, "hidden": hidden, "depth": depth}


def _step(model, optimizer="adamw", flavour="shampoo2", phase="steady", graph=False, name=None):
    case = {"kind": "step", "optimizer": optimizer, "flavour": flavour, "phase": phase, "graph": graph}
    case.update(model)
    return dict(case, name=name) if name else case


def _quant(order, bits, blocksize, dtype, diag, name=None):
    case = {"kind": "quant", "order": order, "bits": bits, "blocksize": blocksize, "dtype": dtype, "diag": diag}
    return dict(case, name=name) if name else case


def listed():
    vit_b32 = _vit(768, 12, 3072, 32, 224, 1000)
    return [
        # One statistic of the first configuration: the single-matrix round trip, a call of a few microseconds.
        _quant(1024, 4, 64, "fp32", False, name="quant_1024_4bit"),
        # 8-bit bf16 with the entry points' default block size, odd order: rows that no vector access fits.
        _quant(3001, 8, 256, "bf16", True, name="quant_3001_8bit_bf16"),
        # The largest order of the kernel sweep, diagonal kept in fp32 as for preconditioners.
        _quant(8192, 4, 64, "fp32", True, name="quant_8192_4bit_diag"),
        # The headline: ViT-B/32, every interval firing, the step replayed as a CUDA graph.
        _step(vit_b32, phase="refresh", graph=True, name="vit_b32_refresh"),
        # The same training run between two refreshes: 99 of its 100 steps.
        _step(vit_b32, phase="steady", graph=True, name="vit_b32_steady"),
        # ResNet-34 on CIFAR with its usual SGD and Swin-Tiny with AdamW (configurations 2 and 3), between two refreshes;
        # eager, as the optimizers are constructed by default.
        _step(_resnet(64, 3, 4, 6, 3), optimizer="sgd", phase="steady", name="resnet34_sgd_steady"),
        _step(_swin(96, 2, 2, 6, 2), phase="steady", name="swin_tiny_steady"),
        # A few layers of an order of the kernel sweep, or of odd ones: everything fires, or the statistics only; eager.
        _step(_mlp(512, 1000, 8), phase="refresh", name="mlp_512_refresh"),
        _step(_mlp(1189, 777, 4), phase="stat", name="mlp_odd_stat"),
        # Dense statistics with the Schur-Newton root, the other flavour a user can choose.
        _step(_mlp(768, 1200, 6), flavour="shampoo1", phase="refresh", name="mlp_dense_refresh"),
        # The smallest model of the tests and a net of its size: steps bound by launches and host work, eager and replayed.
        _step(_vit(64, 2, 192, 8, 32, 10), phase="steady", name="vit_small_steady"),
        _step(_mlp(64, 128, 4), phase="refresh", graph=True, name="mlp_small_refresh"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.3:
        bits = rng.choice((4, 4, 8))
        return _quant(_log(rng, 64, 8192), bits, rng.choice((64, 64, 128, 256)), rng.choice(("fp32", "fp32", "bf16")), rng.random() < 0.5)
    phase = rng.choice(("steady", "steady", "stat", "refresh", "refresh"))
    family = rng.choice(("vit", "resnet", "swin", "mlp")) if phase == "steady" else "mlp"
    if family == "vit":
        width = _log(rng, 48, 768)
        model = _vit(width, rng.randint(1, 12), width * rng.choice((2, 3, 4)), rng.choice((4, 8, 16, 32)), 224 if width > 192 else 32,
                     rng.choice((10, 100, 200, 1000)))
    elif family == "resnet":
        model = _resnet(_log(rng, 16, 64), *(rng.randint(1, d) for d in (3, 4, 6, 3)), classes=rng.choice((10, 100, 200)))
    elif family == "swin":
        model = _swin(_log(rng, 32, 96), *(rng.randint(1, d) for d in (2, 2, 6, 2)), classes=rng.choice((10, 100, 200)))
    else:
        width = _log(rng, 48, MAX_ORDER)
        model = _mlp(width, min(MAX_ORDER, max(48, _log(rng, width * 0.55, width * 1.8))), rng.randint(1, 12))
    flavour = rng.choice(("shampoo2", "shampoo2", "shampoo2", "shampoo1"))
    optimizer = rng.choice(("adamw", "adamw", "sgd"))
    case = _step(model, optimizer, flavour, phase, optimizer == "adamw" and rng.random() < 0.5)
    most = max(work(c)["flops"] for c in listed())
    while family == "mlp" and work(case)["flops"] > most and case["depth"] > 1:      # no costlier than the largest listed case
        case["depth"] -= 1
    return case


# ---- what a program has in hand before the call --------------------------------------------
def _thin(shape):
    """True if a gradient block of `shape` has more than twice as many rows as columns, or the other way round.

    The statistic of the long side then stays rank-deficient (half of its spectrum is dropped at every refresh and the
    gradient does not fill it), and the eigenvectors of its null space are rounding noise in every implementation.
    Steps that refresh leave such a parameter out, as one that is frozen: of ViT-B/32 that is the position embedding."""
    return any(max(m, k) > 2 * min(m, k) for m, k in block_shapes(shape, MAX_ORDER))


def _shapes(case):
    """Shapes of the parameters handed to the optimizer, in the order of model.parameters()."""
    if case["model"] == "mlp":
        a, b = case["width"], case["hidden"]
        return [s for i in range(case["depth"]) for s in (((b, a), (b,)) if i % 2 == 0 else ((a, b), (a,)))]
    with torch.device("meta"):
        if case["model"] == "vit":
            m = workloads.VisionTransformer(img=case["img"], patch=case["patch"], dim=case["width"], depth=case["depth"], heads=1,
                                            mlp=case["mlp"], classes=case["classes"])
        else:
            depths = (case["d1"], case["d2"], case["d3"], case["d4"])
            if case["model"] == "resnet":
                m = workloads.ResNetCifar(depths=depths, widths=tuple(case["width"] * k for k in (1, 2, 4, 8)), classes=case["classes"])
            else:
                heads = max(1, round(case["width"] / 32))
                m = workloads.SwinTransformer(dim=case["width"], depths=depths, heads=tuple(heads * k for k in (1, 2, 4, 8)),
                                              classes=case["classes"])
    shapes = [tuple(p.shape) for p in m.parameters()]
    return shapes if case["phase"] == "steady" else [s for s in shapes if not _thin(s)]


def _flat(shapes):
    """One buffer and its views of the given shapes, each on a 512-byte boundary."""
    offsets, total = [], 0
    for s in shapes:
        offsets.append(total)
        total += (math.prod(s) + 127) // 128 * 128
    buf = torch.zeros(total, device=DEVICE)
    return buf, [buf[o: o + math.prod(s)].view(s) for o, s in zip(offsets, shapes)]


def _prepare_quant(case, gen):
    n = case["order"]
    # a symmetric matrix as the statistics and their roots are: a dominant diagonal, values of every size beside it
    a = torch.randn(n, n, device=DEVICE, generator=gen)
    a = (a + a.T) * torch.exp(torch.randn(n, 1, device=DEVICE, generator=gen)) * 0.02
    a.diagonal().add_(torch.rand(n, device=DEVICE, generator=gen) + 0.5)
    code = F.create_linear_map(signed=True, total_bits=case["bits"], power=2).to(DEVICE)
    return {"case": case, "a": a.to(DTYPES[case["dtype"]]).contiguous(), "code": code}


def _noise(rows, cols, scale, gen):
    return torch.randn(rows, cols, device=DEVICE, generator=gen) * scale


# What a refresh makes of its inputs is fixed only as far as the 4-bit codes of the eigenbasis are: a code that flips
# moves its element by a whole step, and on dense eigenvectors a few flips grow to the size of the quantization noise
# within two steps.  The inputs of the steps that refresh therefore have eigenvectors close to the axes (the codes that
# rounding moves are those of small entries) and spectra with a gap where the kept half ends.
_SMALL = 3e-5                  # entries beside the axes, relative to those on them
_BASE = 1e-3                   # smallest singular value of a gradient block


def _singular_values(m, k, gen):
    """min(m, k) singular values, ascending, in three tiers.  A refresh keeps the smaller half of a spectrum with weight
    0.95 and takes the rest from the gradient with weight 0.05: the factors between the tiers keep the same half the
    smaller one, for the statistics of both sides."""
    m, k = min(m, k), max(m, k)
    u = 1 + 0.3 * torch.rand(m, device=DEVICE, generator=gen)
    tier = torch.ones(m, device=DEVICE)
    tier[max(0, k // 2 - (k - m)):] *= 40 ** 0.5
    tier[m // 2:] *= 6 ** 0.5
    return _BASE * tier * u


def _block_axes(m, k, gen):
    """Rows and columns on which the singular values of a gradient block lie (all steps of a run share them)."""
    r = min(m, k)
    return torch.randperm(m, device=DEVICE, generator=gen)[:r], torch.randperm(k, device=DEVICE, generator=gen)[:r]


def _cut_views(t, blocks):
    """The blocks of a gradient in the optimizer's order."""
    rows = next(d for d in t.shape if d != 1)
    t = t.view(rows, -1)
    out, r0, i = [], 0, 0
    while r0 < t.shape[0]:
        c0 = 0
        while c0 < t.shape[1]:
            m, k = blocks[i]
            out.append(t[r0: r0 + m, c0: c0 + k])
            c0 += k
            i += 1
        r0 += m
    return out


def _symmetric(n, scale, gen):
    a = _noise(n, n, scale, gen)
    return a + a.T


def _set_state(pre, grad, blocks, dense, gen):
    """Statistics and preconditioners as a run leaves them, through the holders of the reference's interface, and a
    gradient that goes on from there."""
    j = 0
    for (m, k), g in zip(blocks, _cut_views(grad, blocks)):
        sv = _singular_values(m, k, gen)
        axes = _block_axes(m, k, gen)
        g.copy_(_noise(m, k, _SMALL * _BASE, gen))
        g[axes] += sv
        for n, on in ((m, axes[0]), (k, axes[1])):
            lam = 0.5 * _BASE ** 2 * (1 + 0.3 * torch.rand(n, device=DEVICE, generator=gen))
            lam[on] = sv ** 2
            keep = max(1, n // 2)
            vals, idx = torch.sort(lam)
            stat, prec = pre.statistics[j], pre.preconditioners[j]
            j += 1
            prec.quantize(torch.diag(1 + torch.rand(n, device=DEVICE, generator=gen)) + _symmetric(n, 0.2 / math.sqrt(n), gen))
            if dense:
                stat.quantize(torch.diag(lam) + _symmetric(n, _SMALL * _BASE ** 2, gen))
                continue
            basis = torch.eye(n, device=DEVICE) + _noise(n, n, _SMALL, gen)
            if stat.bits >= 16:
                stat.var.copy_(basis)
            else:
                F.quantize_blockwise(basis, code=stat.name2qmap[stat.code], order=n, absmax=stat.absmax, out=stat.var,
                                     blocksize=stat.blocksize, bits=stat.bits)
            stat.Svalue.copy_(vals[:keep].clamp(max=1.7 * _BASE ** 2))
            stat.keep_indices.copy_(idx[:keep])
            stat.max_eigenvalue.copy_(0.05 * vals[-1])


def _prepare_step(case, gen):
    shapes = _shapes(case)
    flat, views = _flat(shapes)
    params = [torch.nn.Parameter(v) for v in views]
    gflat, grads = _flat(shapes)
    gflat.normal_(generator=gen).mul_(1e-3)
    dense = case["flavour"] == "shampoo1"
    module = shampoo1 if dense else shampoo2
    kw = dict(stat_compute_steps=NEVER, prec_compute_steps=1, prec_maxorder=MAX_ORDER, prec_bits=4, quan_blocksize=64)
    if case["optimizer"] == "adamw":
        opt = module.ShampooAdamW(params, lr=1e-3, weight_decay=0.05, **kw)
        moments = ("exp_avg", "exp_avg_sq")
    else:
        opt = module.ShampooSGD(params, lr=0.1, momentum=0.9, weight_decay=5e-4, **kw)
        moments = ("momentum",)
    for p, g in zip(params, grads):
        p.grad = g
    opt.step()                                       # creates the state; the roots of this step activate it
    # moments in one buffer each, as a program keeps them that saves or shards its optimizer state as a whole
    out = {"params": flat}
    for name in moments:
        buf, mviews = _flat(shapes)
        for p, v in zip(params, mviews):
            opt.state[p][name] = v
        out[name] = buf
    stat, root = case["phase"] != "steady", case["phase"] == "refresh"
    opt.param_groups[0]["stat_compute_steps"] = 1 if stat else NEVER
    opt.param_groups[0]["prec_compute_steps"] = 1 if root else NEVER
    opt.step()                                       # steps of the kind that follows, then the values that they start from
    if case["graph"]:
        opt.enable_cuda_graph()
        opt.step()
    flat.normal_(generator=gen).mul_(0.02)
    for name in moments:
        out[name].normal_(generator=gen).mul_(1e-3)
    if case["optimizer"] == "adamw":
        out["exp_avg_sq"].square_().add_(1e-7)
    gflat.normal_(generator=gen).mul_(1e-3)
    holders = []
    for p, g in zip(params, grads):
        blocks = block_shapes(p.shape, MAX_ORDER)
        if blocks:
            pre = opt.state[p]["preconditioner"]
            _set_state(pre, g, blocks, dense, gen)
            holders += [pre.statistics, pre.preconditioners]
    if stat:
        # spectra, codes, scales and diagonals: those of all matrices of an order lie in one buffer each
        state = [getattr(h, name, None) for hs in holders for h in hs for name in ("Svalue", "var", "absmax", "diag")]
        base = {}
        for t in state:
            if t is not None:
                b = t._base if t._base is not None else t
                base.setdefault(b.data_ptr(), b)
        out["state"] = list(base.values())
    return {"case": case, "opt": opt, "out": out, "grads": gflat}


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed))
    torch.manual_seed(int(seed))                     # start vectors of the power iterations
    return (_prepare_quant if case["kind"] == "quant" else _prepare_step)(case, gen)


def run(state):
    case = state["case"]
    if case["kind"] == "step":
        state["opt"].step()
        return state["out"]
    n, code = case["order"], state["code"]
    kw = dict(blocksize=case["blocksize"], bits=case["bits"])
    if case["diag"]:
        q, absmax, diag = F.quantize_blockwise_diagreal(state["a"], code, n, **kw)
        return q, absmax, diag, F.dequantize_blockwise_diagreal(q, code, n, absmax, diag, outdtype=DTYPES[case["dtype"]], **kw)
    q, absmax = F.quantize_blockwise(state["a"], code, n, **kw)
    return q, absmax, F.dequantize_blockwise(q, code, n, absmax, outdtype=DTYPES[case["dtype"]], **kw)


# ---- what a pass cannot do without -----------------------------------------------------------
def _state_bytes(n, diag, basis=False):
    """Stored bytes of one matrix of order n: 4-bit codes, block scales, the diagonal or the kept half of a spectrum."""
    if n * n < 4096:
        size = 4 * n * n
    else:
        size = n * n // 2 + 4 * n * ((n + 63) // 64) + (4 * n if diag else 0)
    return size + (12 * max(1, n // 2) + 4 if basis else 0)


def work(case):
    """Bytes: gradients, parameters, moments and stored state, each read and written as often as its values change hands.
    Flops: the products the algorithm names, symmetric results and one triangle of them counted once."""
    if case["kind"] == "quant":
        n, item = case["order"], 4 if case["dtype"] == "fp32" else 2
        stored = (n * n * case["bits"] + 7) // 8 + 4 * n * -(-n // case["blocksize"]) + (4 * n if case["diag"] else 0)
        return {"bytes": 2 * item * n * n + stored, "flops": 0}
    shapes = _shapes(case)
    dense = case["flavour"] == "shampoo1"
    stat, root = case["phase"] != "steady", case["phase"] == "refresh"
    size = sum(math.prod(s) for s in shapes) * (28 if case["optimizer"] == "adamw" else 20)
    flops = 0.0
    for s in shapes:
        for m, k in block_shapes(s, MAX_ORDER):
            flops += 2.0 * m * k * (m + k)                                      # P0 G P1
            for n, other in ((m, k), (k, m)):
                size += _state_bytes(n, True)                                   # preconditioner: read, or written where roots fire
                if stat:
                    size += 2 * _state_bytes(n, dense, basis=not dense)
                    flops += 1.0 * n * n * other                                # G G^T
                    if not dense:
                        # rectified basis (3), old statistic (1/2), L V^T (2), QR and Q (8/3), V^T L V's diagonal (2)
                        flops += (3 + 0.5 + 2 + 8 / 3 + 2) * n ** 3
                if root:
                    if stat is False:
                        size += _state_bytes(n, dense, basis=not dense)
                    # four rectifications of n/2 rows (3/4 each) and the root (1/2); Schur-Newton: ten iterations of four
                    # products of symmetric matrices
                    flops += 40.0 * n ** 3 if dense else (4 * 0.75 + 0.5) * n ** 3
    return {"bytes": size, "flops": flops}


def tolerance(case):
    if case["kind"] == "quant":
        return "exact"
    if case["phase"] == "steady":
        return {"rel": 1e-5}                         # fp32 products and moments
    # 4-bit state: rounding of the products moves codes of small entries (1e-4 of all codes, 1e-3 after two steps) and with
    # them single block scales; measured with the products' accumulation chains twice as long: rel 1e-3, max 0.3, differ 1e-3
    return {"rel": 5e-3, "max": 0.8, "differ": 5e-3}
