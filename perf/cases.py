"""The work that a user of this library has it do, as measurable cases.

Every case is a dict of plain values.  ``prepare`` makes what a program holds before the call
(an engine with weights, G-buffers, resident env maps, SH transport), ``run`` makes one pass
through the public entry points of ``neural_wavelet_prt_demo_b200.engine``, ``work`` states the
bytes and operations the pass cannot do without, and ``exact`` evaluates the same pass in
64 bits with plain torch.  Sizes come from the repository's configurations, tests and bench.

Kinds:

* ``relight``  one frame: ``TCNNPass_p1`` + ``TCNNPass_p2`` (the frame loop of a viewer);
* ``ranges``   one quantum of the serving loop: ``relightRanges`` over resident frames;
* ``request``  one serving request with a rotated env map: rotate, register (Haar + top-K),
               relight a resident frame, release the env map;
* ``wavelets`` env maps -> their wavelet tables (Haar + top-K), one map after a rotation or a
               whole set at once;
* ``project``  SH projection of a cubemap;
* ``shdot``    per-pixel SH transport vectors times the env SH;
* ``shmesh``   the per-vertex SH path: vertex radiance, then the pixels' interpolation;
* ``tonemap``  the final-colour pass of a relit frame.
"""
import math

import numpy as np
import torch

from neural_wavelet_prt_demo_b200 import engine, netconfig, synth

DEV = "cuda:0"
NETS = {"small": netconfig.CONFIG_SMALL, "large": netconfig.CONFIG_LARGE}


def listed():
    return [
        # the parity network's frame at its full size: the smallest relight call
        {"name": "relight_bf16_128_k64_small", "kind": "relight", "net": "small", "precision": "bf16",
         "width": 128, "height": 128, "K": 64, "hit": 1.0},
        # the reference's default window and wavelet count, on the 1080p network
        {"name": "relight_bf16_512_k64", "kind": "relight", "net": "large", "precision": "bf16",
         "width": 512, "height": 512, "K": 64, "hit": 0.9},
        # the headline frame
        {"name": "relight_bf16_1080p_k300", "kind": "relight", "net": "large", "precision": "bf16",
         "width": 1920, "height": 1080, "K": 300, "hit": 1.0},
        # the engine's default arithmetic (the FP32 drop-in) at the parity configuration
        {"name": "relight_fp32_128_k64_small", "kind": "relight", "net": "small", "precision": "fp32",
         "width": 128, "height": 128, "K": 64, "hit": 1.0},
        # the FP32 drop-in on the 1080p network, a ragged window
        {"name": "relight_fp32_611x407_k64", "kind": "relight", "net": "large", "precision": "fp32",
         "width": 611, "height": 407, "K": 64, "hit": 0.9},
        # a packed quantum of the serving stream: whole small frames and a part of a large one
        {"name": "serve_quantum", "kind": "ranges", "net": "large",
         "jobs": "512x512:128:0-0 256x256:300:0-0 1280x720:64:0-0 1920x1080:300:131072-196608"},
        # one serving request for a rotated env map
        {"name": "serve_request_256_k64", "kind": "request", "net": "large", "width": 256, "height": 256, "K": 64},
        # one map rotated and transformed: the latency a new env map adds
        {"name": "rotate_wavelets_64_k300", "kind": "wavelets", "S": 64, "K": 300, "maps": 1},
        # a set of env maps transformed at once (offline preparation of a rotation set)
        {"name": "wavelets_1024maps_k300", "kind": "wavelets", "S": 64, "K": 300, "maps": 1024},
        # the env SH of a cubemap
        {"name": "sh_project_128", "kind": "project", "S": 128},
        # the per-vertex SH path on a mesh, seen at 1080p
        {"name": "sh_mesh_40k_1080p", "kind": "shmesh", "vertices": 40000, "n": 81, "pixels": 1920 * 1080},
        # the final colours of a ragged frame just under 1440p
        {"name": "tonemap_2559x1439", "kind": "tonemap", "width": 2559, "height": 1439},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["relight", "relight", "relight", "ranges", "request", "wavelets", "wavelets", "project",
                       "shdot", "shmesh", "tonemap"])
    if kind == "relight":
        net = rng.choice(["small", "large"])
        precision = rng.choice(["bf16", "bf16", "fp32"])
        w, h = _log_int(rng, 64, 1920), _log_int(rng, 48, 1080)
        K = _log_int(rng, 16, 512)
        most = 5.5e8 if precision == "bf16" else 1.4e7
        K = max(1, min(K, int(most / (w * h))))
        return {"kind": kind, "net": net, "precision": precision, "width": w, "height": h, "K": K,
                "hit": rng.choice([1.0, 0.9])}
    if kind == "ranges":
        jobs = []
        for _ in range(rng.randint(2, 6)):
            w, h = rng.choice([(256, 256), (512, 512), (1280, 720), (1920, 1080), (800, 600)])
            K = rng.choice([64, 128, 300])
            n = w * h
            begin = 128 * rng.randrange(0, n // 256)
            end = min(n, begin + _log_int(rng, 2000, 200000))
            jobs.append("%dx%d:%d:%d-%d" % (w, h, K, begin, end))
        return {"kind": kind, "net": rng.choice(["small", "large"]), "jobs": " ".join(jobs)}
    if kind == "request":
        w, h = rng.choice([(256, 256), (512, 512), (1280, 720), (333, 251)])
        return {"kind": kind, "net": rng.choice(["small", "large"]), "width": w, "height": h,
                "K": rng.choice([64, 128, 300, 77])}
    if kind == "wavelets":
        return {"kind": kind, "S": rng.choice([16, 32, 64, 64]), "K": _log_int(rng, 16, 1024),
                "maps": rng.choice([1, _log_int(rng, 1, 1024)])}
    if kind == "project":
        return {"kind": kind, "S": _log_int(rng, 16, 256)}
    if kind == "shdot":
        return {"kind": kind, "pixels": _log_int(rng, 1000, 1920 * 1080), "n": rng.choice([9, 25, 49, 81, 81])}
    if kind == "shmesh":
        return {"kind": kind, "vertices": _log_int(rng, 500, 40000), "n": rng.choice([25, 49, 64, 81, 81]),
                "pixels": _log_int(rng, 10000, 1920 * 1080)}
    return {"kind": "tonemap", "width": _log_int(rng, 100, 2560), "height": _log_int(rng, 100, 1440)}


# ------------------------------------------------------------------ inputs
def _gen(seed, stream):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + stream) % (1 << 62))


def _uniform(seed, stream, shape, lo, hi):
    return torch.rand(shape, generator=_gen(seed, stream), device=DEV) * (hi - lo) + lo


def _normal(seed, stream, shape):
    return torch.randn(shape, generator=_gen(seed, stream), device=DEV)


def _level_layout(cfg):
    ve = cfg["vtx_enc"]
    res, size, off, o = [], [], [], 0
    for lvl in range(ve["n_levels"]):
        n = int(math.floor(ve["base_resolution"] * math.pow(ve["per_level_scale"], lvl)))
        s = min(1 << ve["log2_hashmap_size"], (n + 1) ** 3)
        res.append(n)
        size.append(s)
        off.append(o)
        o += s
    return res, size, off, o


def _shapes(cfg):
    ve, op, cn = cfg["vtx_enc"], cfg["out_prd"], cfg["cmp_net"]

    def mlp(n_in, width, hidden, n_out):
        dims = [n_in] + [width] * hidden + [n_out]
        return list(zip(dims[:-1], dims[1:]))

    D = ve["n_levels"] * ve["n_features_per_level"]
    aux = cfg["cmp_enc"]["n_padded_dims"]
    return (D, mlp(D, op["n_neurons"], op["n_hidden_layers"], op["n_output_dims"]),
            mlp(op["n_output_dims"] + aux, cn["n_neurons"], cn["n_hidden_layers"], 3))


def _weights(net, seed):
    """Hash features of a trained grid's size, Xavier-uniform MLPs, all rounded to FP16 values
    as a checkpoint trained in half precision holds them."""
    cfg = NETS[net]
    D, op, cn = _shapes(cfg)
    r = lambda t: t.half().float()  # noqa: E731
    hp = r(_uniform(seed, 1, _level_layout(cfg)[3] * cfg["vtx_enc"]["n_features_per_level"], -0.5, 0.5))
    mats = []
    for li, (i, o) in enumerate(op + cn):
        a = math.sqrt(6.0 / (i + o))
        mats.append(r(_uniform(seed, 10 + li, (o, i), -a, a)))
    emb = r(_normal(seed, 2, (D, 6 * cfg["wve_enc"]["face_size"] ** 2)) * 0.1)
    return hp, mats[:len(op)], mats[len(op):], emb


def _gbuffer(n, seed, hit):
    """A G-buffer with the reference's encodings (synth.make_gbuffer's distributions)."""
    unit = lambda v: v / v.norm(dim=1, keepdim=True)  # noqa: E731
    f4 = lambda v: torch.cat([v, torch.ones((v.shape[0], 1), device=DEV)], 1).contiguous()  # noqa: E731
    nrm = unit(_normal(seed, 31, (n, 3)))
    d = -unit(_normal(seed, 32, (n, 3)))
    refl = unit(d - 2.0 * (d * nrm).sum(1, keepdim=True) * nrm)
    flag = torch.ones(n, dtype=torch.uint8, device=DEV)
    if hit < 1.0:
        flag = (_uniform(seed, 38, n, 0.0, 1.0) < hit).to(torch.uint8)
    return dict(pos=f4(_uniform(seed, 30, (n, 3), 0.0, 1.0)), normal=f4(nrm / 2 + 0.5), reflect=f4(refl / 2 + 0.5),
                rough=_uniform(seed, 33, n, 0.05, 1.0), kd=f4(_uniform(seed, 34, (n, 3), 0.0, 1.0)),
                ks=f4(_uniform(seed, 35, (n, 3), 0.0, 1.0)), direct=f4(_uniform(seed, 36, (n, 3), 0.0, 0.5)), flag=flag)


def _frame(g, w, h):
    z = lambda: torch.zeros((w * h, 4), dtype=torch.float32, device=DEV)  # noqa: E731
    return engine.FullFrame(w, h, g["pos"], g["normal"], g["reflect"], g["rough"], g["kd"], g["ks"], g["direct"],
                            g["flag"], z(), z())


def _faces(S, seed, maps=1):
    f = torch.exp(_normal(seed, 50, (maps, 6, S, S, 3)) * 1.5)  # log-normal radiance
    return f


def _rotation(seed):
    q, r = np.linalg.qr(np.random.default_rng(seed).normal(size=(3, 3)))
    q = q * np.sign(np.diag(r))
    if np.linalg.det(q) < 0:
        q[:, 0] = -q[:, 0]
    return q.astype(np.float32)


def _haar(x):
    """Mallat-layout non-standard Haar transform of [..., S, S, 3], in x's own type."""
    x = x.clone()
    n = x.shape[-3]
    while n > 1:
        a, b = x[..., 0:n:2, 0:n:2, :], x[..., 0:n:2, 1:n:2, :]
        c, d = x[..., 1:n:2, 0:n:2, :], x[..., 1:n:2, 1:n:2, :]
        s0, d0, s1, d1 = a + b, a - b, c + d, c - d
        h = n // 2
        x[..., :n, :n, :] = torch.cat([torch.cat([(s0 + s1) * 0.5, (d0 + d1) * 0.5], -2),
                                       torch.cat([(s0 - s1) * 0.5, (d0 - d1) * 0.5], -2)], -3)
        n = h
    return x


def _select(faces, K):
    """Indices of the K largest |luminance| coefficients (ties: the smaller index) of [E,6,S,S,3]."""
    c = _haar(faces).reshape(faces.shape[0], -1, 3)
    key = (c[..., 0] * 0.212671 + c[..., 1] * 0.715160 + c[..., 2] * 0.072169).abs()
    return torch.sort(key, dim=1, descending=True, stable=True)[1][:, :K]


def _table(faces, K):
    """(idx [K], strength [K, 3] in faces' type) of one map [6, S, S, 3]; selected in 32 bits."""
    idx = _select(faces.float().unsqueeze(0), K)[0]
    return idx, _haar(faces).reshape(-1, 3)[idx]


def _engine(net, seed):
    hp, op, cn, emb = _weights(net, seed)
    cat = lambda ms: torch.cat([m.reshape(-1) for m in ms]).cpu().numpy()  # noqa: E731
    e = engine.RenderEngine(NETS[net])
    e.loadWeights(synth.Weights(hp.cpu().numpy(), cat(op), cat(cn), emb.cpu().numpy()))
    return e


def _jobs(case):
    out = []
    for j in case["jobs"].split():
        size, K, span = j.split(":")
        w, h = (int(v) for v in size.split("x"))
        b, e = (int(v) for v in span.split("-"))
        out.append((w, h, int(K), b, e or w * h))
    return out


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind in ("relight", "ranges", "request"):
        e = st["engine"] = _engine(case["net"], seed)
        S = NETS[case["net"]]["wve_enc"]["face_size"]
    if kind == "relight":
        idx, strength = _table(_faces(S, seed)[0], case["K"])
        env = engine.EnvironmentMap(top_coefficients=idx.cpu().numpy(), top_strength=strength.cpu().numpy())
        st["env"] = e.addEnvironmentMap(env)
        st["frame"] = _frame(_gbuffer(case["width"] * case["height"], seed, case["hit"]), case["width"], case["height"])
        e.setFrame(0, st["frame"])
        st["cfg"] = engine.RenderConfig(precision=case["precision"])
    elif kind == "ranges":
        st["ranges"], st["out"] = [], []
        for i, (w, h, K, b, end) in enumerate(_jobs(case)):
            idx, strength = _table(_faces(S, seed + 100 * i)[0], K)
            env = e.addEnvironmentMap(engine.EnvironmentMap(top_coefficients=idx.cpu().numpy(),
                                                            top_strength=strength.cpu().numpy()))
            fr = _frame(_gbuffer(w * h, seed + 100 * i, 1.0), w, h)
            e.setFrame(i, fr)
            e.TCNNPass_p1(i)
            st["ranges"].append((env, i, fr.fbPredictedIndirect, fr.fbPredictedIndirectWithDirect, b, end))
            st["out"].append((fr.fbPredictedIndirect, fr.fbPredictedIndirectWithDirect))
        st["cfg"] = engine.RenderConfig(precision="bf16")
    elif kind == "request":
        st["faces"] = _faces(S, seed)[0].contiguous()
        st["R"] = _rotation(seed)
        st["K"] = case["K"]
        st["frame"] = _frame(_gbuffer(case["width"] * case["height"], seed, 1.0), case["width"], case["height"])
        e.setFrame(0, st["frame"])
        e.TCNNPass_p1(0)
        st["cfg"] = engine.RenderConfig(precision="bf16")
    elif kind == "wavelets":
        f = _faces(case["S"], seed, case["maps"])
        st["faces"] = (f[0] if case["maps"] == 1 else f).contiguous()
        st["R"] = _rotation(seed) if case["maps"] == 1 else None
        st["K"] = min(case["K"], 6 * case["S"] ** 2)
    elif kind == "project":
        st["faces"] = _faces(case["S"], seed)[0].contiguous()
    elif kind == "shdot":
        st["T"], st["L"] = _sh_transport(case, seed)
    elif kind == "shmesh":
        st.update(_sh_mesh(case, seed))
        st["engine"] = engine.RenderEngine(netconfig.CONFIG_SMALL)
    elif kind == "tonemap":
        st["src"] = _radiance(case, seed)
    return st


def _bands(n):
    l = torch.floor(torch.sqrt(torch.arange(n, device=DEV, dtype=torch.float32)))  # noqa: E741
    return 1.0 / l.clamp_min(1.0)


def _sh_transport(case, seed):
    n = case["n"]
    inv = _bands(n)
    return (_normal(seed, 60, (case["pixels"], n)) * (inv * inv)).contiguous(), _normal(seed, 61, (n, 3)).contiguous()


def _sh_mesh(case, seed):
    V, n, P = case["vertices"], case["n"], case["pixels"]
    inv = _bands(n)
    T = _normal(seed, 70, (V, n, n))
    T *= inv.view(1, n, 1)
    T *= inv.view(1, 1, n)
    brdf = _normal(seed, 71, (V, n, 3)) * (inv * inv).view(1, n, 1) * _uniform(seed, 72, (V, 1, 1), 0.0, 1.0)
    uv = _uniform(seed, 73, (P, 2), 0.0, 1.0)
    uv = torch.where(uv.sum(1, keepdim=True) > 1.0, 1.0 - uv, uv)
    # neighbouring pixels see neighbouring triangles, whose vertices lie near one another
    base = (torch.arange(P, device=DEV) * V // P + torch.randint(0, 64, (P,), generator=_gen(seed, 74), device=DEV)) % V
    tri = (base.view(P, 1) + torch.randint(0, 8, (P, 3), generator=_gen(seed, 75), device=DEV)) % V
    return {"T": T.contiguous(), "brdf": brdf.contiguous(), "L": _normal(seed, 76, (n, 3)).contiguous(),
            "uv": uv.contiguous(), "tri": tri.to(torch.int32).contiguous()}


def _radiance(case, seed):
    n = case["width"] * case["height"]
    x = torch.cat([torch.exp(_normal(seed, 80, (n, 3)) * 1.2 - 1.5), torch.ones((n, 1), device=DEV)], 1)
    return x.contiguous()


def run(st):
    kind = st["kind"]
    if kind == "relight":
        e, fr = st["engine"], st["frame"]
        e.TCNNPass_p1(0)
        e.TCNNPass_p2(st["env"], 0, st["cfg"])
        return fr.fbPredictedIndirect, fr.fbPredictedIndirectWithDirect
    if kind == "ranges":
        st["engine"].relightRanges(st["ranges"], st["cfg"])
        return st["out"]
    if kind == "request":
        e, fr = st["engine"], st["frame"]
        faces = engine.env_rotate(st["faces"], st["R"])
        env = e.addEnvironmentFaces(faces, st["K"])
        e.relightRanges([(env, 0, fr.fbPredictedIndirect, fr.fbPredictedIndirectWithDirect, 0, 0)], st["cfg"])
        e.releaseEnvironmentMap(env)
        return fr.fbPredictedIndirect, fr.fbPredictedIndirectWithDirect
    if kind == "wavelets":
        if st["R"] is None:
            idx, strength = engine.haar_topk(st["faces"], st["K"])
            return {"idx": idx, "strength": strength}
        faces = engine.env_rotate(st["faces"], st["R"])
        idx, strength = engine.haar_topk(faces, st["K"])
        return {"faces": faces, "idx": idx, "strength": strength}
    if kind == "project":
        return engine.sh_project(st["faces"])
    if kind == "shdot":
        return engine.sh_dot(st["T"], st["L"])
    if kind == "shmesh":
        vc = engine.sh_vertex_radiance(st["T"], st["brdf"], st["L"])
        return vc, st["engine"].shInterpolate(vc, st["tri"], st["uv"])
    return engine.tonemap_srgb(st["src"])


# ------------------------------------------------------------------ what a pass cannot do without
def _net_cost(net):
    """(flops per evaluation, flops per pixel, weight bytes)."""
    cfg = NETS[net]
    D, op, cn = _shapes(cfg)
    aux = cfg["cmp_enc"]["n_padded_dims"]
    per_eval = sum(2 * i * o for i, o in op + cn) - 2 * aux * cn[0][1]
    grid = _level_layout(cfg)[3] * cfg["vtx_enc"]["n_features_per_level"]
    return per_eval, 2 * aux * cn[0][1], 4 * (grid + sum(i * o for i, o in op + cn)), D


def _relight_work(net, jobs, with_g):
    """jobs: (pixels, K).  Bytes: what the pass reads of each pixel (the G-buffer with p1, else
    its 16-float row, direct light and flag), both outputs, the tables and the weights."""
    per_eval, per_px, wbytes, D = _net_cost(net)
    b, f = wbytes, 0.0
    for n, K in jobs:
        b += n * ((5 * 16 + 4 + 16 + 1 if with_g else 64 + 16 + 1) + 32) + K * (4 * D + 16)
        f += n * (K * per_eval + per_px)
    return {"bytes": float(b), "flops": float(f)}


def work(case):
    kind = case["kind"]
    if kind == "relight":
        return _relight_work(case["net"], [(case["width"] * case["height"], case["K"])], True)
    if kind == "ranges":
        return _relight_work(case["net"], [(e - b, K) for _, _, K, b, e in _jobs(case)], False)
    if kind == "request":
        S = NETS[case["net"]]["wve_enc"]["face_size"]
        w = _relight_work(case["net"], [(case["width"] * case["height"], case["K"])], False)
        return {"bytes": w["bytes"] + 2.0 * 72 * S * S, "flops": w["flops"]}
    if kind == "wavelets":
        S, E = case["S"], case["maps"]
        K = min(case["K"], 6 * S * S)
        return {"bytes": float(E * (72 * S * S * (2 if E == 1 else 1) + 16 * K)), "flops": float(E * 6 * S * S * 3 * 4)}
    if kind == "project":
        S = case["S"]
        return {"bytes": float(72 * S * S + 81 * 12), "flops": float(6 * S * S * 81 * 3 * 2)}
    if kind == "shdot":
        return {"bytes": float(case["pixels"] * (4 * case["n"] + 16)), "flops": float(case["pixels"] * case["n"] * 6)}
    if kind == "shmesh":
        V, n, P = case["vertices"], case["n"], case["pixels"]
        return {"bytes": float(V * (4 * n * n + 12 * n + 12) + P * (12 + 8 + 16)), "flops": float(V * 6 * (n * n + n))}
    return {"bytes": float(case["width"] * case["height"] * 20), "flops": 0.0}


# ------------------------------------------------------------------ the same passes in 64 bits
def _hash_encode(cfg, hp, pos):
    F = cfg["vtx_enc"]["n_features_per_level"]
    res, size, off, _ = _level_layout(cfg)
    tab = hp.view(-1, F).double()
    p = pos.double().clamp(0.0, 1.0)
    out = []
    for N, T, o in zip(res, size, off):
        x = p * N
        i0 = torch.minimum(torch.floor(x).long(), torch.full((), N - 1, device=DEV))
        w = x - i0
        acc = 0.0
        for c in range(8):
            b = [c & 1, (c >> 1) & 1, (c >> 2) & 1]
            wc = 1.0
            for d in range(3):
                wc = wc * (w[:, d] if b[d] else 1.0 - w[:, d])
            X, Y, Z = (i0[:, d] + b[d] for d in range(3))
            if (N + 1) ** 3 <= T:
                e = X + Y * (N + 1) + Z * (N + 1) ** 2
            else:
                e = (X ^ ((Y * 2654435761) & 0xFFFFFFFF) ^ ((Z * 805459861) & 0xFFFFFFFF)) & (T - 1)
            acc = acc + wc.view(-1, 1) * tab[o + e]
        out.append(acc)
    return torch.cat(out, 1)


def _relight64(net, weights, g, idx, strength, begin=0, end=None):
    """(indirect, with_direct) [n, 4] in 64 bits; pixels outside [begin, end) stay 0."""
    cfg = NETS[net]
    hp, op, cn, emb = weights
    op, cn = [m.double() for m in op], [m.double() for m in cn]
    E = emb[:, idx].double().t().contiguous()  # [K, D]
    L = strength.double()
    K, m = E.shape[0], op[-1].shape[0]
    n = g["flag"].shape[0]
    end = n if end is None else end
    ind = torch.zeros((n, 4), dtype=torch.float64, device=DEV)
    wd = torch.zeros((n, 4), dtype=torch.float64, device=DEV)
    step = max(128, 600000 // K)
    for s in range(begin, end, step):
        sl = slice(s, min(end, s + step))
        q = sl.stop - sl.start
        enc = _hash_encode(cfg, hp, g["pos"][sl, :3])
        rough = torch.log(25.0 * g["rough"][sl].double() + 1.0) / math.log(26.0)
        aux = torch.cat([g["normal"][sl, :3].double(), g["reflect"][sl, :3].double(), rough.view(-1, 1),
                         2.0 * g["kd"][sl, :3].double() - 1.0, 2.0 * g["ks"][sl, :3].double() - 1.0,
                         torch.ones((q, cn[0].shape[1] - m - 13), dtype=torch.float64, device=DEV)], 1)
        h = (enc.view(q, 1, -1) * E.view(1, K, -1)).view(q * K, -1)
        for i, W in enumerate(op):
            h = h @ W.t()
            if i + 1 < len(op):
                h.relu_()
        pre = (aux @ cn[0][:, m:].t()).view(q, 1, -1)
        h = ((h @ cn[0][:, :m].t()).view(q, K, -1) + pre).view(q * K, -1).relu_()
        for i, W in enumerate(cn[1:]):
            h = h @ W.t()
            if i + 2 < len(cn):
                h.relu_()
        rgb = (h.view(q, K, 3) * L.view(1, K, 3)).clamp_min_(0.0).sum(1) * g["flag"][sl].double().view(-1, 1)
        ind[sl, :3] = rgb
        wd[sl, :3] = rgb + g["direct"][sl, :3].double()
        ind[sl, 3] = wd[sl, 3] = 1.0
    return ind, wd


def _rotate(faces, R):
    """Point-sampled rotation of a cubemap [6, S, S, 3] (the texel choice in 32 bits)."""
    S = faces.shape[1]
    R = torch.from_numpy(R).to(DEV)
    t = torch.arange(6 * S * S, device=DEV)
    f, r, c = t // (S * S), (t // S) % S, t % S
    uc = 2.0 * ((c.float() + 0.5) / S) - 1.0
    vc = 2.0 * ((r.float() + 0.5) / S) - 1.0
    one = torch.ones_like(uc)
    x = torch.stack([one, -one, uc, uc, uc, -uc])[f, t]
    y = torch.stack([vc, vc, one, -one, vc, vc])[f, t]
    z = torch.stack([uc, -uc, vc, -vc, -one, one])[f, t]
    sx, sy, sz = ((R[0, k] * x + R[1, k] * y) + R[2, k] * z for k in range(3))
    ax, ay, az = sx.abs(), sy.abs(), sz.abs()
    maxa, su, sv, sf = torch.ones_like(x), torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(f)
    mx, my, mz = (ax >= ay) & (ax >= az), (ay >= ax) & (ay >= az), (az >= ax) & (az >= ay)
    for cond, a, u, v, face in ((mx & (sx > 0), ax, sz, sy, 0), (mx & ~(sx > 0), ax, -sz, sy, 1),
                                (my & (sy > 0), ay, sx, sz, 2), (my & ~(sy > 0), ay, sx, -sz, 3),
                                (mz & ~(sz > 0), az, sx, sy, 4), (mz & (sz > 0), az, -sx, sy, 5)):
        maxa, su, sv = torch.where(cond, a, maxa), torch.where(cond, u, su), torch.where(cond, v, sv)
        sf = torch.where(cond, torch.full_like(sf, face), sf)
    col = torch.floor((0.5 * (su / maxa + 1.0)) * S).long() % S
    row = torch.floor((0.5 * (sv / maxa + 1.0)) * S).long() % S
    return faces[sf, row, col].view(6, S, S, 3)


def _sh_project64(faces):
    S = faces.shape[1]
    t = torch.arange(6 * S * S, device=DEV)
    f, r, c = t // (S * S), (t // S) % S, t % S
    uc = 2.0 * (c.double() + 0.5) / S - 1.0
    vc = 2.0 * (r.double() + 0.5) / S - 1.0
    one = torch.ones_like(uc)
    q = uc * uc + vc * vc + 1.0
    inv = q.rsqrt()
    x = torch.stack([one, -one, uc, uc, uc, -uc])[f, t] * inv
    y = torch.stack([vc, vc, one, -one, vc, vc])[f, t] * inv
    z = torch.stack([uc, -uc, vc, -vc, -one, one])[f, t] * inv
    s = (1.0 - z * z).clamp_min(0.0).sqrt()
    phi = torch.atan2(y, x)
    P = {}
    for m in range(9):
        pmm = torch.ones_like(z)
        for i in range(1, m + 1):
            pmm = pmm * (-(2.0 * i - 1.0)) * s
        P[m, m] = pmm
        if m < 8:
            P[m + 1, m] = z * (2.0 * m + 1.0) * pmm
        for l in range(m + 2, 9):  # noqa: E741
            P[l, m] = ((2.0 * l - 1.0) * z * P[l - 1, m] - (l + m - 1.0) * P[l - 2, m]) / (l - m)
    wf = faces.reshape(-1, 3).double() * (inv ** 3 * 4.0 / (S * S)).view(-1, 1)
    out = torch.zeros((81, 3), dtype=torch.float64, device=DEV)
    for l in range(9):  # noqa: E741
        for m in range(l + 1):
            k = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
            if m == 0:
                out[l * l + l] = ((k * P[l, 0]).view(-1, 1) * wf).sum(0)
            else:
                kp = math.sqrt(2.0) * k * P[l, m]
                out[l * l + l + m] = ((kp * torch.cos(m * phi)).view(-1, 1) * wf).sum(0)
                out[l * l + l - m] = ((kp * torch.sin(m * phi)).view(-1, 1) * wf).sum(0)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "relight":
        S = NETS[case["net"]]["wve_enc"]["face_size"]
        idx, strength = _table(_faces(S, seed)[0], case["K"])
        g = _gbuffer(case["width"] * case["height"], seed, case["hit"])
        return _relight64(case["net"], _weights(case["net"], seed), g, idx, strength)
    if kind == "ranges":
        S = NETS[case["net"]]["wve_enc"]["face_size"]
        weights, out = _weights(case["net"], seed), []
        for i, (w, h, K, b, end) in enumerate(_jobs(case)):
            idx, strength = _table(_faces(S, seed + 100 * i)[0], K)
            out.append(_relight64(case["net"], weights, _gbuffer(w * h, seed + 100 * i, 1.0), idx, strength, b, end))
        return out
    if kind == "request":
        S = NETS[case["net"]]["wve_enc"]["face_size"]
        idx, strength = _table(_rotate(_faces(S, seed)[0], _rotation(seed)), case["K"])
        g = _gbuffer(case["width"] * case["height"], seed, 1.0)
        return _relight64(case["net"], _weights(case["net"], seed), g, idx, strength)
    if kind == "wavelets":
        K = min(case["K"], 6 * case["S"] ** 2)
        f = _faces(case["S"], seed, case["maps"])
        if case["maps"] == 1:
            rot = _rotate(f[0], _rotation(seed))
            idx = _select(rot.unsqueeze(0), K)[0]
            return {"faces": rot.double(), "idx": None, "strength": _haar(rot.double()).reshape(-1, 3)[idx]}
        idx = _select(f, K)
        c = _haar(f.double()).reshape(f.shape[0], -1, 3)
        return {"idx": None, "strength": torch.gather(c, 1, idx.unsqueeze(-1).expand(-1, -1, 3))}
    if kind == "project":
        return _sh_project64(_faces(case["S"], seed)[0])
    if kind == "shdot":
        T, L = _sh_transport(case, seed)
        out = torch.ones((T.shape[0], 4), dtype=torch.float64, device=DEV)
        out[:, :3] = (T.double() @ L.double()).abs()
        return out
    if kind == "shmesh":
        s = _sh_mesh(case, seed)
        L, V = s["L"].double(), case["vertices"]
        vc = torch.empty((V, 3), dtype=torch.float64, device=DEV)
        for b in range(0, V, 8192):
            light = torch.matmul(s["T"][b:b + 8192].double(), L)
            vc[b:b + 8192] = (light * s["brdf"][b:b + 8192].double()).sum(1).abs()
        tri, u, v = s["tri"].long(), s["uv"][:, :1].double(), s["uv"][:, 1:].double()
        out = torch.ones((tri.shape[0], 4), dtype=torch.float64, device=DEV)
        out[:, :3] = (1.0 - u - v) * vc[tri[:, 0]] + u * vc[tri[:, 1]] + v * vc[tri[:, 2]]
        return vc, out
    return None
