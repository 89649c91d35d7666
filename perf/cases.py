"""The work that a user of this library has it do, as cases to be timed.

Every case goes through the public Python entry points over the C ABI.  Two
net families are used, the two that the tests and the benchmark use: the
reference's own shapes ("reference": 32 planes, ELU, 3x3 head; the value net
64 wide) and the benchmark nets ("benchmark": 24 planes, 128 wide, ReLU, 1x1
head).  Weights are He-normal, as the trained ones are not public; planes are
0/1 with about the share of ones that the feature gather gives.
"""
import math

import numpy as np
import torch

import leela_gb300 as lg
from leela_gb300 import distill

POINTS = 361
CHUNK = 256  # positions per chunk of the serving contexts (the benchmark's batch)


def listed():
    return [
        # One leaf of the engine's search, as the drop-in backend evaluates it:
        # host planes in, probabilities and a value out, FP32.
        dict(name="leaf-reference-1", kind="nets", nets="reference", precision="fp32", where="host", B=1, max_batch=8,
             temperature=1.0),
        # The engine's nets over the leaves that its threads gathered, FP32, an odd size.
        dict(name="batch-reference-77", kind="nets", nets="reference", precision="fp32", where="host", B=77,
             max_batch=CHUNK, temperature=1.0),
        # A handful of leaves on the GPU already, FP32.
        dict(name="fp32-pair-5", kind="nets", nets="benchmark", precision="fp32", where="device", B=5, max_batch=CHUNK,
             temperature=1.0),
        # Labels of the full FP32 net for the distillation (its batch there is 1024).
        dict(name="fp32-pair-1024", kind="nets", nets="benchmark", precision="fp32", where="device", B=1024,
             max_batch=1024, temperature=1.0),
        # One leaf in BF16: latency.
        dict(name="bf16-pair-1", kind="nets", nets="benchmark", precision="bf16", where="device", B=1, max_batch=CHUNK,
             temperature=1.0),
        # The leaves of a few search threads, BF16.
        dict(name="bf16-pair-24", kind="nets", nets="benchmark", precision="bf16", where="device", B=24,
             max_batch=CHUNK, temperature=1.0),
        # The benchmark's step: 8,192 positions through both nets.
        dict(name="bf16-pair-8192", kind="nets", nets="benchmark", precision="bf16", where="device", B=8192,
             max_batch=CHUNK, temperature=1.0),
        # Boards in, probabilities and values out, the gather on the GPU: a
        # ragged batch end to end from host memory, FP16.
        dict(name="fp16-boards-2100", kind="boards", precision="fp16", B=2100, max_batch=CHUNK, temperature=1.0),
        # The root of a search: all 8 symmetries of one position, averaged.
        dict(name="bf16-ensemble-1", kind="ensemble", precision="bf16", B=1, max_batch=CHUNK, temperature=1.0),
        # All 32 input planes of both sets, ladders included.
        dict(name="gather-1000", kind="gather", B=1000, nplanes=32),
        # A training pass of the student at the distillation's batch: forward,
        # loss and gradients.
        dict(name="student-grads-512", kind="grads", B=512, c_in=24, width=64, n3x3=5, fc_hidden=64),
        # The student serving leaves.
        dict(name="student-serve-8192", kind="student", B=8192, n3x3=5, fc_hidden=64, temperature=1.0),
    ]


def _size(rng, lo, hi):
    """A size between lo and hi, even over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["nets", "nets", "nets", "nets", "nets", "boards", "ensemble", "gather", "grads", "student"])
    temperature = rng.choice([1.0, 1.0, 0.7])
    if kind == "nets":
        precision = rng.choice(["fp32", "fp32", "bf16", "bf16", "fp16", "fp8w"])
        nets = rng.choice(["reference", "benchmark"]) if precision == "fp32" else "benchmark"
        where = rng.choice(["device", "host"])
        if precision == "fp32":
            max_batch = rng.choice([8, CHUNK, 1024])
            B = _size(rng, 1, max_batch)
        else:
            max_batch = CHUNK
            B = _size(rng, 1, 8192 if where == "device" else 2048)
        return dict(kind=kind, nets=nets, precision=precision, where=where, B=B, max_batch=max_batch,
                    temperature=temperature)
    if kind == "boards":
        return dict(kind=kind, precision=rng.choice(["bf16", "fp16"]), B=_size(rng, 1, 4000), max_batch=CHUNK,
                    temperature=temperature)
    if kind == "ensemble":
        return dict(kind=kind, precision=rng.choice(["bf16", "fp16", "fp32"]), B=_size(rng, 1, 32), max_batch=CHUNK,
                    temperature=temperature)
    if kind == "gather":
        return dict(kind=kind, B=_size(rng, 1, 8192), nplanes=rng.choice([24, 32]))
    if kind == "grads":
        return dict(kind=kind, B=_size(rng, 16, 512), c_in=24, width=64, n3x3=rng.choice([3, 5]), fc_hidden=64)
    return dict(kind=kind, B=_size(rng, 1, 8192), n3x3=5, fc_hidden=64, temperature=temperature)


# ------------------------------------------------------------------ shapes

FAMILIES = {  # c_in, width1, width, n3x3, head_k, elu, act_head, fc_hidden, value map (1 + tanh) / 2
    ("reference", 0): (32, 96, 128, 11, 3, True, True, 0, False),
    ("reference", 1): (32, 64, 64, 10, 3, True, True, 256, True),
    ("benchmark", 0): (24, 128, 128, 11, 1, False, False, 0, False),
    ("benchmark", 1): (24, 128, 128, 11, 1, False, False, 256, False),
}


def _convs(nets, value):
    c_in, width1, width, n3x3, head_k = FAMILIES[nets, value][:5]
    sizes = [(5, c_in, width1)]
    for i in range(n3x3):
        sizes.append((3, width1 if i == 0 else width, width))
    return sizes + [(head_k, width, 1)]


def _he(convs, fcs, gen):
    """He-normal weights, zero biases, flat: per conv W[O][C][k][k] then b[O], per FC W[O][I] then b[O]."""
    parts = []
    for k, c, o in convs:
        parts += [torch.randn(o * c * k * k, generator=gen) * math.sqrt(2.0 / (c * k * k)), torch.zeros(o)]
    for i, o in fcs:
        parts += [torch.randn(o * i, generator=gen) * math.sqrt(2.0 / i), torch.zeros(o)]
    return torch.cat(parts)


def _net_weights(nets, value, gen):
    hidden = FAMILIES[nets, value][7]
    return _he(_convs(nets, value), [(POINTS, hidden), (hidden, 1)] if hidden else [], gen)


def _student_weights(c_in, width, n3x3, hidden, gen):
    convs = [(5, c_in, width)] + [(3, width, width)] * n3x3 + [(1, width, 1), (1, width, 1)]
    return _he(convs, [(POINTS, hidden), (hidden, 1)], gen)


def _generator(seed, device="cpu"):
    return torch.Generator(device).manual_seed(seed)


def _planes(B, c_in, seed):
    """[B][c_in][361] bytes, 0 or 1, on the GPU: groups of planes that share
    out the points between them as the gather's do (own stones / opponent's /
    empty, then liberty counts of what is there)."""
    gen = _generator(seed, "cuda")
    fill = torch.rand((B, 1), generator=gen, device="cuda") * 0.6
    u = torch.rand((B, POINTS), generator=gen, device="cuda")
    stone = torch.where(u < fill / 2, 0, torch.where(u < fill, 1, 2))
    planes = torch.zeros((B, c_in, POINTS), dtype=torch.uint8, device="cuda")
    for s in range(3):
        planes[:, s] = stone == s
    # groups of up to five planes for each kind of point
    rest = list(range(3, c_in))
    for g in range(0, len(rest), 5):
        group = rest[g:g + 5]
        level = torch.randint(0, len(group), (B, POINTS), generator=gen, device="cuda")
        here = stone == (g // 5) % 3
        for i, c in enumerate(group):
            planes[:, c] = here & (level == i)
    return planes


def _boards(B, seed):
    """Legal positions on the GPU: stones at random over a random share of the
    points, strings without a liberty taken off; whose move it is; last two
    moves, ko point and komi flag."""
    gen = _generator(seed, "cuda")
    fill = torch.rand((B, 1), generator=gen, device="cuda") * 0.7
    u = torch.rand((B, POINTS), generator=gen, device="cuda")
    sq = torch.where(u < fill / 2, 0, torch.where(u < fill, 1, 2)).reshape(B, 19, 19)

    def near(mask):
        out = torch.zeros_like(mask)
        out[:, 1:] |= mask[:, :-1]
        out[:, :-1] |= mask[:, 1:]
        out[:, :, 1:] |= mask[:, :, :-1]
        out[:, :, :-1] |= mask[:, :, 1:]
        return out

    free = near(sq == 2)
    alive = [(sq == s) & free for s in (0, 1)]
    for _ in range(64):
        alive = [a | (near(a) & (sq == s)) for s, a in enumerate(alive)]
    sq = torch.where(alive[0], 0, torch.where(alive[1], 1, 2)).reshape(B, POINTS).to(torch.int8)
    to_move = torch.randint(0, 2, (B,), generator=gen, device="cuda").to(torch.int8)
    moves = torch.randint(0, POINTS, (B, 4), generator=gen, device="cuda").to(torch.int32)
    moves[:, 2] = -1
    moves[:, 3] &= 1
    return sq, to_move, moves


def _desc(nets, value, precision, seed):
    w = _net_weights(nets, value, _generator(1000 + 2 * seed + value)).numpy()
    make = {("reference", 0): lg.NetDesc.reference_policy, ("reference", 1): lg.NetDesc.reference_value,
            ("benchmark", 0): lg.NetDesc.config1_policy, ("benchmark", 1): lg.NetDesc.config1_value}
    return make[nets, value](w, precision)


def _context(nets, precision, max_batch, seed):
    return lg.Context(policy=_desc(nets, 0, precision, seed), value=_desc(nets, 1, precision, seed),
                      max_batch=max_batch)


def _net_planes(case, seed):
    c_in = FAMILIES[case.get("nets", "benchmark"), 0][0]
    return _planes(case["B"], c_in, 2 * seed), _planes(case["B"], c_in, 2 * seed + 1)


def _student_inputs(case, seed):
    """Planes, target probabilities (a sharpened random policy) and target
    values in [-1, 1] of a training batch."""
    B = case["B"]
    gen = _generator(seed, "cuda")
    target = torch.softmax(3.0 * torch.randn((B, POINTS), generator=gen, device="cuda"), dim=1)
    value = torch.tanh(torch.randn(B, generator=gen, device="cuda"))
    return _planes(B, case["c_in"], seed), target, value


# ------------------------------------------------------------------ passes

def prepare(case, seed):
    kind, B = case["kind"], case["B"]
    st = dict(case=case)
    if kind in ("nets", "ensemble"):
        st["ctx"] = _context(case.get("nets", "benchmark"), case["precision"], case["max_batch"], seed)
        planes = _net_planes(case, seed)
        if case.get("where") == "host":
            st["planes"] = [p.cpu().numpy() for p in planes]
        else:
            st["planes"] = planes
            st["probs"], st["logits"] = torch.empty((2, B, POINTS), device="cuda")
            st["value"] = torch.empty(B, device="cuda")
    elif kind == "boards":
        st["ctx"] = _context("benchmark", case["precision"], case["max_batch"], seed)
        sq, tm, _ = _boards(B, seed)
        st["boards"] = sq.cpu().numpy(), tm.cpu().numpy()
    elif kind == "gather":
        st["boards"] = _boards(B, seed)
        st["out"] = torch.empty((2, B, case["nplanes"], POINTS), dtype=torch.uint8, device="cuda")
    elif kind == "grads":
        st["net"] = distill.Student(case["c_in"], case["width"], case["n3x3"], case["fc_hidden"], max_batch=B)
        st["net"].set_params(_student_weights(case["c_in"], case["width"], case["n3x3"], case["fc_hidden"],
                                              _generator(seed)).numpy())
        st["batch"] = _student_inputs(case, seed)
    else:
        w = _student_weights(24, 64, case["n3x3"], case["fc_hidden"], _generator(seed)).numpy()
        st["net"] = distill.FastNet(w, 24, case["n3x3"], case["fc_hidden"], max_batch=B)
        st["planes"] = _planes(B, 24, seed)
        st["probs"], st["logits"] = torch.empty((2, B, POINTS), device="cuda")
        st["value"], st["entropy"] = torch.empty((2, B), device="cuda")
    # the calls run on whatever stream is current then, so the inputs are done first
    torch.cuda.synchronize()
    return st


def run(state):
    case = state["case"]
    kind, B, T = case["kind"], case["B"], case.get("temperature", 1.0)
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "nets" and case["where"] == "host":
        pp, pv = state["planes"]
        probs, logits = state["ctx"].policy(pp, T, return_logits=True)
        return [probs, logits, state["ctx"].value(pv)]
    if kind == "nets":
        pp, pv = state["planes"]
        state["ctx"].policy_device(pp.data_ptr(), B, state["probs"].data_ptr(), T, state["logits"].data_ptr(), stream)
        state["ctx"].value_device(pv.data_ptr(), B, state["value"].data_ptr(), stream)
        return [state["probs"], state["logits"], state["value"]]
    if kind == "ensemble":
        pp, pv = state["planes"]
        state["ctx"].policy_avg8_device(pp.data_ptr(), B, state["probs"].data_ptr(), T, stream)
        state["ctx"].value_avg8_device(pv.data_ptr(), B, state["value"].data_ptr(), stream)
        return [state["probs"], state["value"]]
    if kind == "boards":
        sq, tm = state["boards"]
        probs, logits = state["ctx"].policy_boards(sq, tm, T, return_logits=True)
        return [probs, logits, state["ctx"].value_boards(sq, tm)]
    if kind == "gather":
        sq, tm, mv = state["boards"]
        for which in (0, 1):
            lg.gather_device(sq.data_ptr(), tm.data_ptr(), B, which, case["nplanes"], state["out"][which].data_ptr(),
                             stream, mv.data_ptr())
        return [state["out"]]
    if kind == "grads":
        planes, target, value = state["batch"]
        (kl, mse), grads = state["net"].grads(planes.data_ptr(), B, target.data_ptr(), value.data_ptr(), 1.0)
        return [np.array([kl, mse], dtype=np.float32), grads]
    state["net"].device(state["planes"].data_ptr(), B, state["probs"].data_ptr(), state["value"].data_ptr(), T,
                        state["logits"].data_ptr(), state["entropy"].data_ptr(), stream)
    return [state["probs"], state["logits"], state["value"], state["entropy"]]


# ------------------------------------------------------------------ work

def _conv_work(convs):
    """(multiply-adds x 2 of one position, weights) of a list of convs."""
    return (sum(2 * POINTS * k * k * c * o for k, c, o in convs), sum(k * k * c * o + o for k, c, o in convs))


def work(case):
    kind, B = case["kind"], case["B"]
    if kind == "gather":
        return {"bytes": B * (POINTS + 17) + 2 * B * case["nplanes"] * POINTS, "flops": 0}
    if kind in ("grads", "student"):
        c_in, width, hidden = case.get("c_in", 24), case.get("width", 64), case["fc_hidden"]
        convs = [(5, c_in, width)] + [(3, width, width)] * case["n3x3"] + [(1, width, 1)] * 2
        flops, weights = _conv_work(convs)
        flops += 2 * (POINTS + 1) * hidden
        weights += (POINTS + 2) * hidden + 1
        if kind == "grads":
            # the input gradient of the first layer is not needed
            total = 3 * flops - 2 * POINTS * 25 * c_in * width
            return {"bytes": B * (c_in * POINTS + 4 * POINTS + 4) + 8 * weights, "flops": B * total}
        return {"bytes": B * (c_in * POINTS + 8 * POINTS + 8) + 2 * weights, "flops": B * flops}
    nets = case.get("nets", "benchmark")
    fp32 = case["precision"] == "fp32"
    flops = weights = 0
    for value in (0, 1):
        f, w = _conv_work(_convs(nets, value))
        hidden = FAMILIES[nets, value][7]
        flops += f + 2 * (POINTS + 1) * hidden
        weights += w + (POINTS + 2) * hidden
    c_in = FAMILIES[nets, 0][0]
    times = 8 if kind == "ensemble" else 1
    per_in = POINTS + 1 if kind == "boards" else 2 * c_in * POINTS
    per_out = 4 * POINTS + 4 if kind == "ensemble" else 8 * POINTS + 4
    return {"bytes": B * (per_in + per_out) + weights * (4 if fp32 else 2), "flops": times * B * flops}


# ------------------------------------------------------------------ 64 bits

def _conv64(x, w, b, k):
    """x [B][C][361] -> [B][O][361], zero padding, as one matrix product."""
    B, C = x.shape[:2]
    if k > 1:
        x = torch.nn.functional.unfold(x.reshape(B, C, 19, 19), k, padding=k // 2)
    return torch.matmul(w.reshape(w.shape[0], -1), x) + b[:, None]


def _take(flat, shapes):
    out, at = [], 0
    for s in shapes:
        n = math.prod(s)
        out.append(flat[at:at + n].reshape(s))
        at += n
    return out


def _forward64(nets, value, flat, planes, temperature):
    """Logits and probabilities, or values, of the net in 64 bits."""
    elu, act_head, hidden, half_map = FAMILIES[nets, value][5:]
    act = torch.nn.functional.elu if elu else torch.relu
    convs = _convs(nets, value)
    shapes = [s for k, c, o in convs for s in ((o, c, k, k), (o,))]
    if hidden:
        shapes += [(hidden, POINTS), (hidden,), (1, hidden), (1,)]
    p = _take(flat.to(planes.device, torch.float64), shapes)
    x = planes.to(torch.float64)
    for i, (k, _, _) in enumerate(convs):
        x = _conv64(x, p[2 * i], p[2 * i + 1], k)
        if i + 1 < len(convs) or act_head:
            x = act(x)
    x = x[:, 0]
    if not hidden:
        return x, torch.softmax(x / temperature, dim=1)
    w1, b1, w2, b2 = p[2 * len(convs):]
    t = torch.tanh(act(x @ w1.T + b1) @ w2.T + b2)[:, 0]
    return (1 + t) / 2 if half_map else t


def _rotations():
    """Index tables of the 8 symmetries: out[i] = in[table[s][i]]."""
    idx = torch.arange(POINTS).reshape(19, 19)
    out = []
    for s in range(8):
        t = idx
        if s & 1:
            t = t.flip(0)
        if s & 2:
            t = t.flip(1)
        if s >= 4:
            t = t.T
        out.append(t.reshape(-1))
    return out


def _exact_nets(case, seed):
    nets, T, times = case.get("nets", "benchmark"), case["temperature"], 8 if case["kind"] == "ensemble" else 1
    if case["B"] * times > 1100:
        return None  # too long in 64 bits
    pp, pv = _net_planes(case, seed)
    wp, wv = (_net_weights(nets, v, _generator(1000 + 2 * seed + v)) for v in (0, 1))
    tables = [t.to(pp.device) for t in _rotations()] if times == 8 else [None]
    probs = logits = value = 0
    for t in tables:
        for_p, for_v = (pp, pv) if t is None else (pp[..., t], pv[..., t])
        parts = [_forward64(nets, 0, wp, for_p[i:i + 128], T) for i in range(0, len(pp), 128)]
        lg_, pr = (torch.cat(x) for x in zip(*parts))
        if t is not None:
            pr = torch.empty_like(pr).index_copy_(1, t, pr)
        logits = lg_
        probs = probs + pr / len(tables)
        value = value + torch.cat([_forward64(nets, 1, wv, for_v[i:i + 128], T)
                                   for i in range(0, len(pv), 128)]) / len(tables)
    return [probs, value] if times == 8 else [probs, logits, value]


def _student64(flat, case, planes):
    """Head outputs of the student in 64 bits: logits and values."""
    c_in, width, n, hidden = case.get("c_in", 24), case.get("width", 64), case["n3x3"], case["fc_hidden"]
    convs = [(5, c_in, width)] + [(3, width, width)] * n + [(1, width, 1)] * 2
    shapes = [s for k, c, o in convs for s in ((o, c, k, k), (o,))]
    p = _take(flat, shapes + [(hidden, POINTS), (hidden,), (1, hidden), (1,)])
    x = planes.to(torch.float64)
    for i in range(n + 1):
        x = torch.relu(_conv64(x, p[2 * i], p[2 * i + 1], convs[i][0]))
    logits = _conv64(x, p[2 * n + 2], p[2 * n + 3], 1)[:, 0]
    v = _conv64(x, p[2 * n + 4], p[2 * n + 5], 1)[:, 0]
    w1, b1, w2, b2 = p[2 * n + 6:]
    return logits, torch.tanh(torch.relu(v @ w1.T + b1) @ w2.T + b2)[:, 0]


def _exact_grads(case, seed):
    planes, target, value = _student_inputs(case, seed)
    flat = _student_weights(case["c_in"], case["width"], case["n3x3"], case["fc_hidden"], _generator(seed))
    flat = flat.to("cuda", torch.float64).requires_grad_()
    B = case["B"]
    loss = np.zeros(2)
    for i in range(0, B, 64):
        logits, v = _student64(flat, case, planes[i:i + 64])
        t = target[i:i + 64].to(torch.float64)
        kl = (t * (torch.log(t.clamp_min(1e-300)) - torch.log_softmax(logits, dim=1))).sum() / B
        mse = ((v - value[i:i + 64].to(torch.float64)) ** 2).sum() / B
        (kl + mse).backward()
        loss += np.array([kl.item(), mse.item()])
    return [loss, flat.grad.cpu().numpy()]


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind in ("nets", "ensemble"):
            return _exact_nets(case, seed)
        if kind == "student":
            flat = _student_weights(24, 64, case["n3x3"], case["fc_hidden"], _generator(seed))
            flat = flat.to("cuda", torch.float64)
            planes = _planes(case["B"], 24, seed)
            parts = [_student64(flat, case, planes[i:i + 256]) for i in range(0, case["B"], 256)]
            logits, v = (torch.cat(x) for x in zip(*parts))
            probs = torch.softmax(logits / case["temperature"], dim=1)
            return [probs, logits, v, -(probs * torch.log(probs)).sum(dim=1)]
    if kind == "grads":
        return _exact_grads(case, seed)
    return None  # gathered planes are bytes; from boards the planes are the library's own
