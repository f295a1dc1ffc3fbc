"""The work that a user of this library has it do, as timed cases: the scan layer in training, stacks of layers at
inference, one large scene, the whole ISSM block, and the steps around the scan (gated norm, point reordering with its
convolution, generation of dt / B / C).  Values follow BASELINE.json's distributions: x, z ~ N(0, 1), B and C scaled by
1 / sqrt(states), softplus(dt) of N(0, 1) - 4 clamped to [1e-3, 1e-1], A = -exp(U(log 1, log 16)) per head."""
import math

import torch

from dest3d_b200 import ISSM_chunk_scan_combined, PointLiteConv, issm_bidirectional_scan, reorder_points, rmsnorm_fn
from dest3d_b200.adaptive_params import adaptive_dt_bc
from dest3d_b200.issm_block import MultiHeadISSMScan

DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
DT_LIMIT = (1e-3, 1e-1)


def listed():
    detector = dict(H=8, P=36, N=256, Q=256, G=1)           # 8 heads x 36 channels, 256 object queries as states
    return [
        # one scene through one ISSM block at inference: the smallest call, launches and host work count
        dict(name="block_infer_b1_L1024", kind="block", b=1, L=1024, K=256, d_model=144, M=16, H=8, train=False),
        # one decoder block in training at the detector's batch size, under bf16 autocast
        dict(name="block_train_b8_L1024", kind="block", b=8, L=1024, K=256, d_model=144, M=16, H=8, train=True),
        # the scan of that block and its gated norm alone (the scan takes no z: the norm applies the gate)
        dict(name="layer_norm_b8_L1024", kind="layer", b=8, L=1024, dtype="bf16", gate="norm", **detector),
        # dense indoor scans, 40000 points each: the largest training step
        dict(name="layer_b16_L40000", kind="layer", b=16, L=40000, dtype="bf16", gate="z", **detector),
        # training in full precision
        dict(name="layer_f32_b2_L1024", kind="layer", b=2, L=1024, dtype="f32", gate="z", **detector),
        # another model width (64 channels per head, 64 states, two groups) and a ragged sequence
        dict(name="layer_b4_L2047_P64_N64", kind="layer", b=4, L=2047, dtype="bf16", gate="z", H=4, P=64, N=64, Q=64, G=2),
        # six stacked layers at inference, 512 queries
        dict(name="stack_b16_L4096_N512", kind="stack", b=16, L=4096, dtype="bf16", layers=6, H=8, P=36, N=512, Q=128, G=1),
        # the same in full precision
        dict(name="stack_f32_b16_L4096_N512", kind="stack", b=16, L=4096, dtype="f32", layers=2, H=8, P=36, N=512, Q=128, G=1),
        # ONE large scene in training: few streams, the library cuts the sequence into slices
        dict(name="scene_b1_L40000", kind="scene", b=1, L=40000, dtype="bf16", **detector),
        # the gated RMSNorm over the detector's 288 features, many points
        dict(name="norm_262144x288", kind="norm", rows=262144, hidden=288, dtype="bf16"),
        # serialisation of the points and the depthwise convolution that follows it, training
        dict(name="points_b64_L16384_C290", kind="points", b=64, L=16384, C=290, dtype="bf16"),
        # dt, B and C of both directions from the point-to-query features, training
        dict(name="params_b16_L4096_K256", kind="params", b=16, L=4096, K=256, M=16, H=8, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "layer", "layer", "layer_wide", "stack", "scene", "norm", "points", "params"])
    if kind == "block":
        train = rng.random() < 0.5
        return dict(kind="block", b=rng.randint(1, 8), L=_log(rng, 200, 4096), K=rng.choice([128, 256, 256]), d_model=144, M=16, H=8, train=train)
    if kind in ("layer", "layer_wide"):
        dtype = rng.choice(["bf16", "bf16", "f32"]) if kind == "layer" else "bf16"
        if kind == "layer_wide":
            shape = dict(H=rng.choice([2, 4, 8]), P=rng.choice([48, 64, 80]), N=rng.choice([32, 64, 100, 192]), G=rng.choice([1, 2]))
        else:
            shape = dict(H=8, P=rng.choice([32, 36, 36, 40]), N=rng.choice([128, 256, 256]), G=1)
        L = _log(rng, 100, 40000 if kind == "layer" and dtype == "bf16" else 4096)
        b = rng.randint(1, 16)
        cap = 6.0e8 if kind == "layer" and dtype == "bf16" else 2.0e7    # states x points x heads
        while b > 1 and b * L * shape["H"] * shape["N"] > cap:
            b -= 1
        return dict(kind="layer", b=b, L=L, dtype=dtype, gate=rng.choice(["norm", "z"]), Q=rng.choice([64, 128, 256]), **shape)
    if kind == "stack":
        dtype = rng.choice(["bf16", "f32"])
        return dict(kind="stack", b=rng.randint(1, 16), L=_log(rng, 256, 4096 if dtype == "bf16" else 1024), dtype=dtype, layers=rng.choice([2, 6]) if dtype == "bf16" else 2,
                    H=8, P=36, N=rng.choice([256, 512, 512]), Q=rng.choice([64, 128]), G=1)
    if kind == "scene":
        return dict(kind="scene", b=rng.choice([1, 1, 2]), L=_log(rng, 4000, 60000), dtype="bf16", H=8, P=36, N=256, Q=256, G=1)
    dtype = rng.choice(["bf16", "bf16", "f32"])
    if kind == "norm":
        return dict(kind="norm", rows=_log(rng, 1000, 262144), hidden=rng.choice([128, 256, 288, 288, 300, 512]), dtype=dtype)
    if kind == "points":
        return dict(kind="points", b=rng.randint(1, 32), L=_log(rng, 500, 16384), C=rng.choice([64, 145, 288, 290, 290]), dtype=dtype)
    return dict(kind="params", b=rng.randint(1, 8), L=_log(rng, 100, 4096), K=rng.choice([100, 128, 256, 256]), M=rng.choice([8, 16, 16]), H=8, dtype=dtype)


class _Rand:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def n(self, *shape, dtype=torch.float32, scale=1.0, shift=0.0):
        t = torch.randn(*shape, device="cuda", generator=self.g, dtype=dtype)
        return (t * scale if scale != 1.0 else t) + shift if shift != 0.0 else (t * scale if scale != 1.0 else t)

    def u(self, *shape):
        return torch.rand(*shape, device="cuda", generator=self.g)


def _scan_inputs(r, c, layers=1):
    b, L, H, P, N, G, dt = c["b"], c["L"], c["H"], c["P"], c["N"], c["G"], DTYPES[c["dtype"]]
    s = dict(x=r.n(b, L, H, P, dtype=dt), x_back=r.n(b, L, H, P, dtype=dt), dt=r.n(b, L, H, N, dtype=dt),
             init=r.n(b, H, P, N, dtype=dt, scale=1 / 16))
    for k in ("B", "C", "B_back", "C_back"):
        s[k] = r.n(b, L, G, N, dtype=dt, scale=N ** -0.5)
    s["A"] = [(-torch.exp(r.u(H) * math.log(16.0)))[:, None].repeat(1, N) for _ in range(layers)]
    s["D"] = [r.n(H) for _ in range(layers)]
    s["dt_bias"] = torch.full((H, N), -4.0, device="cuda")
    return s


def _grad(*ts):
    return [t.requires_grad_() for t in ts]


def prepare(case, seed):
    c, r = case, _Rand(seed)
    kind = c["kind"]
    if kind == "block":
        torch.manual_seed(int(seed))
        mod = MultiHeadISSMScan(d_model=c["d_model"], d_state=c["K"], d_dist=c["M"], chunk_size=256, nheads=c["H"], expand=2, use_biscan=True).cuda()
        s = dict(mod=mod, ins=[r.n(c["b"], c["L"], c["d_model"]), r.n(c["b"], c["K"], c["d_model"], scale=0.25),
                               r.n(c["b"], c["L"], c["K"], c["M"])], xyz=r.n(c["b"], c["L"], 3),
                 mask=(r.u(c["b"], c["L"], c["K"]) > 0.1).float(), train=c["train"])
        s["leaves"] = []
        if c["train"]:
            s["leaves"] = _grad(*s["ins"]) + list(mod.parameters())
            s["douts"] = [r.n(c["b"], c["L"], c["d_model"]).bfloat16(), r.n(c["b"], c["K"], c["d_model"]).bfloat16()]
        else:
            mod.requires_grad_(False)
    elif kind in ("layer", "scene"):
        s = _scan_inputs(r, c)
        dt = DTYPES[c["dtype"]]
        s["gate"], s["Q"] = c.get("gate"), c["Q"]
        s["z"] = r.n(c["b"], c["L"], c["H"], c["P"], dtype=dt) if s["gate"] else None
        s["w"] = r.n(c["H"] * c["P"], scale=0.02, shift=1.0) if s["gate"] == "norm" else None
        names = ["x", "x_back", "dt", "B", "C", "B_back", "C_back", "dt_bias", "init"] + [k for k in ("z", "w") if s[k] is not None]
        s["leaves"] = _grad(*[s[k] for k in names], s["A"][0], s["D"][0])
        s["douts"] = [r.n(c["b"], c["L"], c["H"], c["P"], dtype=dt), r.n(c["b"], c["H"], c["P"], c["N"], scale=1 / 16)]
    elif kind == "stack":
        s = _scan_inputs(r, c, c["layers"])
        s["Q"] = c["Q"]
    else:
        dt = DTYPES[c["dtype"]]
        if kind == "norm":
            s = dict(x=r.n(c["rows"], c["hidden"], dtype=dt), z=r.n(c["rows"], c["hidden"], dtype=dt), w=r.n(c["hidden"], scale=0.02, shift=1.0),
                     douts=[r.n(c["rows"], c["hidden"], dtype=dt)])
            s["leaves"] = _grad(s["x"], s["z"], s["w"])
        elif kind == "points":
            torch.manual_seed(int(seed))
            mod = PointLiteConv(c["C"], c["C"]).cuda()
            x = r.n(c["b"], c["L"], c["C"], dtype=dt)
            order = torch.argsort(r.u(c["b"], c["L"]), dim=1)
            s = dict(mod=mod, x=x, order=order, inverse=torch.argsort(order, dim=1), douts=[r.n(c["b"], c["L"], c["C"], dtype=dt)])
            s["leaves"] = _grad(x) + list(mod.parameters())
        else:
            b, L, K, M, H = c["b"], c["L"], c["K"], c["M"], c["H"]
            s = dict(dist=r.n(b, L, K, M, dtype=dt), w_dt=r.n(H, M, scale=0.3), w_bc=r.n(2, M, scale=0.3), tok=r.n(b, L, H, dtype=dt),
                     toks=[r.n(b, L, 1, dtype=dt) for _ in range(4)], bias=r.n(H, shift=-2.0), mask=(r.u(b, L, K) > 0.3).float(),
                     douts=[r.n(b, L, H, K, dtype=dt)] + [r.n(b, L, 1, K, dtype=dt) for _ in range(4)])
            s["leaves"] = _grad(s["dist"], s["w_dt"], s["w_bc"], s["tok"], *s["toks"], s["bias"])
    s["kind"] = kind
    return s


def run(s):
    kind = s["kind"]
    if kind == "block":
        if not s["train"]:
            with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
                return s["mod"](*s["ins"], s["xyz"], s["mask"])
        with torch.autocast("cuda", dtype=torch.bfloat16):
            outs = s["mod"](*s["ins"], s["xyz"], s["mask"])
    elif kind == "layer":
        key, states = issm_bidirectional_scan(s["x"], s["x_back"], s["dt"], s["A"][0], s["B"], s["C"], s["B_back"], s["C_back"], s["Q"], D=s["D"][0],
                                              z=s["z"] if s["gate"] == "z" else None, dt_bias=s["dt_bias"], initial_states=s["init"],
                                              dt_softplus=True, dt_limit=DT_LIMIT)
        if s["gate"] == "norm":
            b, L, H, P = key.shape
            key = rmsnorm_fn(key.reshape(b, L, H * P), s["w"], None, s["z"].reshape(b, L, H * P), eps=1e-5, norm_before_gate=False).reshape(b, L, H, P)
        outs = (key, states)
    elif kind == "stack":
        with torch.no_grad():
            states = s["init"]
            for A, D in zip(s["A"], s["D"]):
                out, states = issm_bidirectional_scan(s["x"], s["x_back"], s["dt"], A, s["B"], s["C"], s["B_back"], s["C_back"], s["Q"], D=D,
                                                      dt_bias=s["dt_bias"], initial_states=states, dt_softplus=True, dt_limit=DT_LIMIT)
        return out, states
    elif kind == "scene":
        outs = []
        for x, B, C, rev in ((s["x"], s["B"], s["C"], False), (s["x_back"], s["B_back"], s["C_back"], True)):
            outs += ISSM_chunk_scan_combined(x, s["dt"], s["A"][0], B, C, s["Q"], D=s["D"][0], dt_bias=s["dt_bias"], initial_states=s["init"],
                                             dt_softplus=True, dt_limit=DT_LIMIT, return_final_states=True, reverse=rev, slices="auto")
        grads = torch.autograd.grad(outs, s["leaves"], [s["douts"][0], s["douts"][1]] * 2)
        return [o.detach() for o in outs] + list(grads)
    elif kind == "norm":
        outs = (rmsnorm_fn(s["x"], s["w"], None, s["z"], eps=1e-5, norm_before_gate=False),)
    elif kind == "points":
        outs = (s["mod"](None, reorder_points(s["x"], s["order"], s["inverse"])),)
    else:
        outs = adaptive_dt_bc(s["dist"], s["w_dt"], s["w_bc"], s["tok"], s["bias"], *s["toks"], s["mask"])
    grads = torch.autograd.grad(outs, s["leaves"], s["douts"])
    return [o.detach() for o in outs] + list(grads)


def _scan_work(c, backward):
    """Both directions: every input once (dt is shared by the directions), every output once, the states that enter and
    leave; operations of the recurrence itself: decay, update and output of every (point, state, channel), twice that
    again in the backward."""
    e = 2 if c["dtype"] == "bf16" else 4
    b, L, H, P, N, G = (c[k] for k in ("b", "L", "H", "P", "N", "G"))
    gates = 1 if c.get("gate") else 0
    n = L * H * N * e + (3 + gates) * L * H * P * e + 4 * L * G * N * e + H * P * N * (e + 4)
    f = 2 * 5 * L * H * P * N
    if backward:
        n += L * H * N * e + (3 + gates) * L * H * P * e + 4 * L * G * N * e + H * P * N * (e + 4)
        f *= 3
    return b * n, b * f


def work(case):
    c, kind = case, case["kind"]
    if kind in ("layer", "scene"):
        n, f = _scan_work(c, True)
        return {"bytes": n, "flops": f}
    if kind == "stack":
        n, f = _scan_work(c, False)
        return {"bytes": c["layers"] * n, "flops": c["layers"] * f}
    if kind == "block":
        b, L, K, D, M, H = (c[k] for k in ("b", "L", "K", "d_model", "M", "H"))
        inner = 2 * D
        gemm = 2 * b * (L * D * (2 * inner + 2 + H) + L * inner * D + 2 * K * D * inner + L * K * M * (H + 2))
        n = b * 4 * (2 * L * D + 2 * K * D + L * K * M + L * K)
        f = gemm + 2 * 5 * b * L * inner * K
        if c["train"]:
            n, f = n + b * 4 * (2 * L * D + 2 * K * D + L * K * M), 3 * f
        return {"bytes": n, "flops": f}
    e = 2 if c["dtype"] == "bf16" else 4
    if kind == "norm":
        return {"bytes": 6 * c["rows"] * c["hidden"] * e, "flops": 30 * c["rows"] * c["hidden"]}   # x, z, dy in; y, dx, dz out
    if kind == "points":
        n = c["b"] * c["L"]
        return {"bytes": 4 * n * c["C"] * e + 16 * n, "flops": 3 * 14 * n * c["C"]}                # x, dy in; y, dx out; two index lists
    n = c["b"] * c["L"] * c["K"]
    # dist, mask and the five output gradients in; dt, four B / C rows and ddist out
    return {"bytes": n * (2 * c["M"] * e + 2 * (c["H"] + 4) * e + 4), "flops": 3 * 2 * n * c["M"] * (c["H"] + 2)}


def tolerance(case):
    """bf16 operands and results: 2^-9 per rounding, a few of them in a row; float32: the tolerance to which this
    repository holds its float32 scans, and 32-bit sums elsewhere."""
    if case["kind"] == "block" or case["dtype"] == "bf16":
        return {"rel": 1e-2}
    return {"rel": 1e-4 if case["kind"] in ("layer", "stack") else 1e-5}
