"""The workloads whose speed is followed: calls of the public operators, layers and models over the range that training,
attacking and certifying L_p-distance networks covers.

A case is a dict of plain values.  `call` says what the user's program calls:

  op       norm_dist (the autograd operator) forward, then the gradients that `need` names
  layer    NormDist / NormDistConv in training mode (distance, batch-mean shift), forward and both gradients
  certify  NormDist / NormDistConv in eval mode at p = inf without gradients: the value and both interval bounds
  bounds   bound_inf_dist (the interval-bound operator) forward and its three gradients
  model    MLPModel training step up to the gradients: logits, margins, hinge loss, every parameter's gradient

Fully connected cases have B rows of CI features; convolutions (k > 0) have B images of CI channels and side x side pixels.
Inputs are U[0, 1) images in front of a network and zero-mean activations inside it (`hidden`), weights are N(0, 1) as
the layers initialise them, upstream gradients are N(0, 1).
"""
import math

import torch

import l_inf_dist_net_v2_b200 as ldn
from l_inf_dist_net_v2_b200 import losses

EPS = 8 / 255


def listed():
    return [
        # one layer of an MNIST network, the operator called by itself: the smallest call, where launches count
        dict(name="op-mnist-p8", call="op", B=64, CI=784, CO=1024, G=1, p=8.0, need="both", hidden=False),
        # first wide layer of a CIFAR-10 network at the start of the p schedule
        dict(name="layer-cifar-p8", call="layer", B=512, CI=3072, CO=5120, G=1, p=8.0, hidden=False),
        # the same in the middle of the schedule (general exponent)
        dict(name="layer-cifar-p37.5", call="layer", B=512, CI=3072, CO=5120, G=1, p=37.5, hidden=False),
        # a hidden layer at the end of the schedule
        dict(name="layer-hidden-inf", call="layer", B=512, CI=5120, CO=5120, G=1, p="inf", hidden=True),
        # certification of a batch, one layer: value and interval bounds
        dict(name="certify-cifar", call="certify", B=512, CI=3072, CO=5120, G=1, p="inf", hidden=False),
        # the last layer: ten outputs behind 5120 features
        dict(name="op-classes-inf", call="op", B=512, CI=5120, CO=10, G=1, p="inf", need="both", hidden=True),
        # an attack on a narrow network with frozen weights: input gradient only, rows that are no multiple of 16 bytes
        dict(name="op-attack-ragged-p3", call="op", B=200, CI=1001, CO=777, G=1, p=3.0, need="input", hidden=True),
        # training through interval bounds on rows of odd length
        dict(name="bounds-ragged-train", call="bounds", B=100, CI=1023, CO=500, G=1, p="inf", hidden=True),
        # a 3 x 3 convolution of 32 x 32 images
        dict(name="conv-p8", call="layer", B=32, CI=64, CO=128, G=1, p=8.0, k=3, side=32, stride=1, pad=1, hidden=True),
        # the same operator in four groups on 16 x 16 images
        dict(name="conv-grouped-inf", call="layer", B=128, CI=64, CO=64, G=4, p="inf", k=3, side=16, stride=1, pad=1,
             hidden=True),
        # certification through a strided convolution: 7 x 7 outputs, an odd number of positions
        dict(name="certify-conv-7x7", call="certify", B=64, CI=32, CO=64, G=1, p="inf", k=3, side=14, stride=2, pad=1,
             hidden=False),
        # a whole training step of a small network at p = inf
        dict(name="mlp-step-inf", call="model", B=256, CI=3072, CO=1024, depth=4, p="inf"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _power(rng):
    """The exponents of a schedule from 8 to infinity, and the small integer ones."""
    return rng.choice([8.0, 8.0, "inf", "inf", "inf", float(rng.choice([1, 2, 3, 4, 6])), round(math.exp(rng.uniform(
        math.log(2.2), math.log(900.0))), 2)])


def draw(rng):
    call = rng.choice(["op", "op", "layer", "layer", "certify", "bounds", "model"])
    if call == "model":
        return dict(call="model", B=_log(rng, 16, 512), CI=3 * _log(rng, 14, 32) ** 2, CO=_log(rng, 100, 1500),
                    depth=rng.randint(3, 5), p=rng.choice([8.0, "inf"]))
    p = "inf" if call in ("certify", "bounds") else _power(rng)
    G = rng.choice([1, 1, 1, 2, 4])
    case = dict(call=call, B=_log(rng, 8, 512), CI=G * _log(rng, 60, 5120 // G), CO=G * _log(rng, max(1, 10 // G), 5120 // G),
                G=G, p=p, hidden=rng.random() < 0.5)
    if call in ("layer", "certify") and rng.random() < 0.4:
        case.update(B=_log(rng, 8, 128), CI=G * _log(rng, 4, 96 // G), CO=G * _log(rng, 8, 160 // G), k=rng.choice([1, 3, 3, 5]),
                    side=rng.randint(7, 32), stride=rng.choice([1, 1, 2]))
        case["pad"] = case["k"] // 2
    if call == "op":
        case["need"] = rng.choice(["both", "both", "input", "weight"])
    # no drawn case costs more than the largest listed one
    while _pairs(case) * _price(case) > 512 * 3072 * 5120 * _price(listed()[2]):
        case["B"] = max(8, case["B"] // 2)
    return case


def _price(case):
    """Operations on one (row, output, feature) triple over a pass (a logarithm or an exponential counts as 8)."""
    p, call = case["p"], case["call"]
    if call == "certify":
        return 2 + 6
    if call == "bounds":
        return 6
    if p == "inf":
        return 2
    if p == int(p) and p <= 8:
        mults = {1: 0, 2: 0, 3: 1, 4: 1, 5: 2, 6: 2, 7: 3, 8: 2}
        fwd, term = 2 + mults[int(p)], 2 + mults.get(int(p) - 1, 0)
    else:
        fwd, term = 19, 20
    return fwd + term + {"input": 1, "weight": 1}.get(case.get("need"), 2)


def _inf(case):
    return math.inf if case["p"] == "inf" else float(case["p"])


def _hw(case):
    if not case.get("k"):
        return 1
    return ((case["side"] + 2 * case["pad"] - case["k"]) // case["stride"] + 1) ** 2


def _features(case):
    return case["CI"] * (case["k"] ** 2 if case.get("k") else 1)


def _pairs(case):
    if case["call"] == "model":
        return case["B"] * (case["CI"] * case["CO"] + (case["depth"] - 2) * case["CO"] ** 2 + 10 * case["CO"])
    return case["B"] * _hw(case) * case["CO"] * _features(case) // case["G"]


def _shape(case):
    if case.get("k"):
        return (case["B"], case["CI"], case["side"], case["side"])
    return (case["B"], case["CI"], 1) if case["call"] in ("op", "bounds") else (case["B"], case["CI"])


def _out_shape(case):
    if case.get("k"):
        n = math.isqrt(_hw(case))
        return (case["B"], case["CO"], n, n)
    return (case["B"], case["CO"], 1) if case["call"] in ("op", "bounds") else (case["B"], case["CO"])


def _inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = dict(device="cuda", generator=g)
    if case["call"] == "model":
        return dict(x=torch.rand(case["B"], 1, 1, case["CI"], **f), targets=torch.randint(0, 10, (case["B"],), **f),
                    weights=[torch.randn(o, i, **f) for i, o in _sizes(case)])
    x = torch.randn(_shape(case), **f) * 0.5 if case["hidden"] else torch.rand(_shape(case), **f)
    t = dict(x=x, w=torch.randn(case["CO"], _features(case) // case["G"], **f), g=torch.randn(_out_shape(case), **f))
    if case["call"] in ("certify", "bounds"):
        lo, up = x - EPS, x + EPS
        t.update(lo=lo if case["hidden"] else lo.clamp_(0, 1), up=up if case["hidden"] else up.clamp_(0, 1))
    if case["call"] == "bounds":
        t["g2"] = torch.randn(_out_shape(case), **f)
    if case["call"] == "certify":
        t["mean"] = torch.rand(case["CO"], **f) + 3
    return t


def _sizes(case):
    widths = [case["CI"]] + [case["CO"]] * (case["depth"] - 1) + [10]
    return list(zip(widths[:-1], widths[1:]))


def prepare(case, seed):
    t = _inputs(case, seed)
    p = _inf(case)
    if case["call"] == "model":
        net = ldn.MLPModel(depth=case["depth"], width=case["CO"], input_dim=[1, 1, case["CI"]])
        with torch.no_grad():
            for layer, w in zip(net.fc_dist, t["weights"]):
                layer.weight.copy_(w)
        net = net.cuda().train()
        ldn.set_p_norm(net, p)
        return dict(case=case, net=net, loss=losses.hinge(mix=0.25), x=t["x"], targets=t["targets"], params=list(net.parameters()))
    state = dict(case=case, p=p, **t)
    if case["call"] in ("layer", "certify"):
        if case.get("k"):
            layer = ldn.NormDistConv(case["CI"], case["CO"], case["k"], stride=case["stride"], padding=case["pad"],
                                     groups=case["G"], bias=False, p=p)
        else:
            layer = ldn.NormDist(case["CI"], case["CO"], groups=case["G"], bias=False, p=p)
        layer = layer.cuda()
        with torch.no_grad():
            layer.weight.copy_(t["w"])
        if case["call"] == "certify":
            layer.mean_shift.running_mean.copy_(t["mean"])
            layer.eval()
        else:
            layer.train()
        state["layer"] = layer
        state["x"].requires_grad_(case["call"] == "layer")
    if case["call"] == "op":
        state["x"].requires_grad_(case["need"] != "weight")
        state["w"].requires_grad_(case["need"] != "input")
    if case["call"] == "bounds":
        for k in ("lo", "up", "w"):
            state[k].requires_grad_()
    return state


def run(s):
    call = s["case"]["call"]
    if call == "op":
        y = ldn.norm_dist(s["x"], s["w"], s["p"], s["case"]["G"])
        return y, torch.autograd.grad(y, [t for t in (s["x"], s["w"]) if t.requires_grad], s["g"])
    if call == "layer":
        y, _, _ = s["layer"](s["x"])
        return y, torch.autograd.grad(y, [s["x"], s["layer"].weight], s["g"])
    if call == "certify":
        with torch.no_grad():
            return s["layer"](s["x"], s["lo"], s["up"])
    if call == "bounds":
        lo, up = ldn.bound_inf_dist(s["lo"], s["up"], s["w"], s["case"]["G"])
        return lo, up, torch.autograd.grad([lo, up], [s["lo"], s["up"], s["w"]], [s["g"], s["g2"]])
    logits, margins = s["net"](s["x"], targets=s["targets"], eps=EPS)
    loss = s["loss"](logits, margins, s["targets"])
    return logits, margins, loss, torch.autograd.grad(loss, s["params"])


def work(case):
    call, pairs = case["call"], _pairs(case)
    if call == "model":
        # input, and per layer: weight read and its gradient written, activation written and its gradient written
        floats = case["B"] * case["CI"] + sum(2 * i * o + 2 * case["B"] * o for i, o in _sizes(case))
        return dict(bytes=4 * floats, flops=pairs * _price(case))
    x, w, y = math.prod(_shape(case)), case["CO"] * _features(case) // case["G"], math.prod(_out_shape(case))
    if call == "certify":
        floats = 3 * x + w + 3 * y
    elif call == "bounds":
        floats = 4 * x + 2 * w + 4 * y
    else:
        need = case.get("need", "both")
        floats = x + w + 2 * y + (x if need != "weight" else 0) + (w if need != "input" else 0)
    return dict(bytes=4 * floats, flops=pairs * _price(case))


def tolerance(case):
    p = case["p"]
    if case["call"] == "model":
        # the batch means' order of summation moves activations by an ulp, which moves an arg-max now and then; one
        # moved arg-max is a few entries of a gradient of thousands
        return dict(rel=1e-2, max=0.99)
    # measured against 64 bits: 2e-6 (p = inf, behind the mean shift; two runs of its gradients differ as much), 1e-5
    # (p = 8 behind the mean shift, which takes most of the value away), 6e-6 (p = 37.5) and 1e-4 (p near 1000)
    if p == "inf":
        return dict(rel=1e-5, max=2e-4)
    if p <= 100:
        return dict(rel=4e-5, max=2e-3)
    return dict(rel=4e-4, max=2e-2)


# ---- the same results in 64 bits, with plain torch -----------------------------------------------------------------


def _chunks(case, rows, w):
    """Row ranges whose (rows, outputs, features) differences take about 2 GB in 64 bits."""
    step = max(1, (1 << 28) // (w.shape[0] * w.shape[1]))
    return [slice(i, min(rows, i + step)) for i in range(0, rows, step)]


def _rows(case, t):
    """(B, C, ...) inputs as (groups, rows, features of a group): unfolded, one row per position."""
    if case.get("k"):
        t = torch.nn.functional.unfold(t, case["k"], 1, case["pad"], case["stride"])
    else:
        t = t.reshape(t.shape[0], -1, 1)
    B, C, HW = t.shape
    return t.reshape(B, case["G"], C // case["G"], HW).permute(1, 0, 3, 2).reshape(case["G"], B * HW, C // case["G"])


def _out_rows(case, t):
    t = t.reshape(t.shape[0], case["CO"], -1)
    B, C, HW = t.shape
    return t.reshape(B, case["G"], C // case["G"], HW).permute(1, 0, 3, 2).reshape(case["G"], B * HW, C // case["G"])


def _from_out_rows(case, t):
    G, M, n = t.shape
    return t.reshape(G, case["B"], M // case["B"], n).permute(1, 0, 3, 2).reshape(_out_shape(case))


def _distance(a, w, p):
    """(rows, features) x (outputs, features) -> (rows, outputs) in 64 bits, and at p = inf where the maximum of the 32-bit
    differences stands first, with its sign."""
    out, pos, neg = [], [], []
    for r in _chunks(None, a.shape[0], w):
        if math.isinf(p):
            d = a[r].unsqueeze(1) - w.unsqueeze(0)
            v, i = d.abs().max(dim=-1)
            first = torch.where(d.abs() == v.unsqueeze(-1), torch.arange(d.shape[-1], device=d.device), d.shape[-1]).amin(-1)
            out.append(v.double())
            pos.append(first)
            neg.append(torch.gather(d, -1, first.unsqueeze(-1)).squeeze(-1) < 0)
        else:
            d = (a[r].double().unsqueeze(1) - w.double().unsqueeze(0)).abs_()
            top = d.amax(-1, keepdim=True).clamp_min(1e-10)
            out.append(top.squeeze(-1) * d.div_(top).pow_(p).sum(-1).pow_(1 / p))
    return torch.cat(out), (torch.cat(pos), torch.cat(neg)) if pos else None


def _gradients(a, w, y, where, g, p):
    """Gradients of sum(g * distance) with respect to the rows and the weights."""
    a64, w64 = a.double(), w.double()
    if where is not None:
        pos, neg = where
        v = torch.where(neg, -g, g)
        ga = torch.zeros_like(a64).scatter_add_(1, pos, v)
        gw = torch.zeros_like(w64).scatter_add_(1, pos.t().contiguous(), -v.t().contiguous())
        return ga, gw
    ga, gw = torch.empty_like(a64), torch.zeros_like(w64)
    for r in _chunks(None, a.shape[0], w):
        d = a64[r].unsqueeze(1) - w64.unsqueeze(0)
        sign = torch.where(d >= 0, 1.0, -1.0).double()
        term = d.abs_().div_(y[r].unsqueeze(-1)).pow_(p - 1).mul_(sign).mul_(g[r].unsqueeze(-1))
        ga[r] = term.sum(1)
        gw -= term.sum(0)
    return ga, gw


def exact(case, seed):
    if case["call"] == "model":
        return None
    t = _inputs(case, seed)
    G, p = case["G"], _inf(case)
    w = t["w"].reshape(G, case["CO"] // G, -1)
    if case["call"] in ("certify", "bounds"):
        lo, up = _rows(case, t["lo"]), _rows(case, t["up"])
        low, high = [], []
        for g in range(G):
            l, u = [], []
            for r in _chunks(case, lo.shape[1], w[g]):
                t1 = w[g].double().unsqueeze(0) - lo[g][r].double().unsqueeze(1)
                t2 = up[g][r].double().unsqueeze(1) - w[g].double().unsqueeze(0)
                l.append(-torch.minimum(t1, t2).amin(-1).clamp_max(-1e-10))
                u.append(torch.maximum(t1, t2).amax(-1).clamp_min(1e-10))
            low.append(torch.cat(l))
            high.append(torch.cat(u))
        low, high = (_from_out_rows(case, torch.stack(v)) for v in (low, high))
        if case["call"] == "bounds":
            return low, high, [None, None, None]
        shift = t["mean"].double().view((1, -1) + (1,) * (low.dim() - 2))
        x = _rows(case, t["x"])
        y = _from_out_rows(case, torch.stack([_distance(x[g], w[g], p)[0] for g in range(G)]))
        return y - shift, low - shift, high - shift
    rows = _rows(case, t["x"])
    up = t["g"].double()
    if case["call"] == "layer":
        dims = [0] + list(range(2, up.dim()))
        up = up - up.mean(dims, keepdim=True)
    g = _out_rows(case, up)
    y, ga, gw = [], [], []
    for k in range(G):
        yk, where = _distance(rows[k], w[k], p)
        gak, gwk = _gradients(rows[k], w[k], yk, where, g[k], p)
        y.append(yk)
        ga.append(gak)
        gw.append(gwk)
    y, gw = _from_out_rows(case, torch.stack(y)), torch.cat(gw)
    ga = torch.stack(ga).reshape(G, case["B"], _hw(case), -1).permute(1, 0, 3, 2).reshape(case["B"], _features(case), _hw(case))
    if case.get("k"):
        ga = torch.nn.functional.fold(ga, (case["side"],) * 2, case["k"], 1, case["pad"], case["stride"])
    ga = ga.reshape(_shape(case))
    if case["call"] == "layer":
        return y - y.mean([0] + list(range(2, y.dim())), keepdim=True), [ga, gw]
    return y, [v for v, n in ((ga, "weight"), (gw, "input")) if case["need"] != n]
