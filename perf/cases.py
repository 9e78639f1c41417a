"""Performance cases: the calls a program that trains or serves a cross-layer transcoder spends its time in.

``listed()`` names twelve of them, ``draw(rng)`` gives more of the same ranges.  Every case goes through one of three
entry points:

* ``train``  ``FusedBatchTopKEngine.train_step``: one optimisation step in the middle of a run (warm AdamW moments); returns
  the loss terms, every updated parameter and its moments;
* ``infer``  ``SparseForward.forward_dict`` (serving) or, with ``"eval"``, ``SparseForward.reconstruct`` with targets (what the
  evaluator runs); returns the reconstructions (and the per-layer squared errors);
* ``theta``  ``accumulate_theta_batch_sparse``: one batch of the BatchTopK -> JumpReLU threshold statistics.

Inputs are sums of about 32 random dictionary directions with exponential magnitudes plus noise, standardised per layer: what
the synthetic stores hand over.  Weights have the distribution of the initialisation.
"""
import math

import torch

DEV = "cuda"
LR = 1e-4
ADAM = (0.9, 0.999, 1e-8, 0.01)  # beta1, beta2, eps, weight decay of the default optimizer (AdamW)
WARM_STEPS = 100                 # optimizer steps behind the warm moments
LOSS_SCALE = 256.0               # fp16: a scale that has settled
AUX_FACTOR = 1.0 / 32.0
DEAD_WINDOW = 1000


def _case(name, kind, fn, tying, dtype, L, d, F, B, k, **more):
    return dict(name=name, kind=kind, fn=fn, tying=tying, dtype=dtype, L=L, d=d, F=F, B=B, k=k, **more)


def listed():
    return [
        # the headline training step: GPT-2-small shape, 32x features, BatchTopK k = 200
        _case("train-gpt2", "train", "batchtopk", "none", "bf16", 12, 768, 24576, 4096, 200),
        # one rank's share of the same job on eight GPUs (features and k divided by eight)
        _case("train-gpt2-shard", "train", "batchtopk", "none", "bf16", 12, 768, 3072, 4096, 25),
        # Pythia-70m shape with tied decoders and half-precision weights (dynamic loss scale)
        _case("train-pythia-per-source", "train", "batchtopk", "per_source", "fp16", 6, 512, 32768, 8192, 200),
        # the other tied layout: one decoder per target layer
        _case("train-pythia-per-target", "train", "batchtopk", "per_target", "bf16", 6, 512, 16384, 4096, 64),
        # thresholds trained natively: JumpReLU with the tanh sparsity penalty
        _case("train-jumprelu", "train", "jumprelu", "none", "bf16", 12, 768, 4096, 4096, 33, lam=1e-4),
        # a small run with ragged sizes, per-token top-k, dead features (auxiliary loss) and gradient clipping
        _case("train-topk-ragged", "train", "topk", "none", "bf16", 5, 520, 2056, 776, 24, dead=0.05, clip=1.0),
        # serving a converted model on a handful of tokens: latency
        _case("serve-16", "infer", "jumprelu", "none", "bf16", 12, 768, 24576, 16, 200),
        # feature extraction on medium batches with few active features
        _case("infer-512", "infer", "batchtopk", "none", "bf16", 12, 768, 24576, 512, 32),
        # evaluation of the headline model on one training-size batch
        _case("eval-gpt2", "infer", "batchtopk", "none", "bf16", 12, 768, 24576, 4096, 200, eval=True),
        # tied decoders, per-token top-k
        _case("infer-per-source", "infer", "topk", "per_source", "bf16", 6, 512, 32768, 2048, 64),
        # Llama-3.2-1B layer count and width, a ragged batch
        _case("infer-llama-ragged", "infer", "jumprelu", "none", "bf16", 16, 2048, 8200, 1000, 100),
        # one batch of threshold estimation
        _case("theta-gpt2", "theta", "batchtopk", "none", "bf16", 12, 768, 24576, 1024, 200),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        kind = rng.choice(("train", "train", "infer", "infer", "theta"))
        fn = "batchtopk" if kind == "theta" else rng.choice(("batchtopk", "batchtopk", "jumprelu", "topk"))
        c = dict(kind=kind, fn=fn, tying=rng.choice(("none", "none", "per_source", "per_target")),
                 dtype=rng.choice(("bf16", "fp16")) if kind == "train" else "bf16",
                 L=rng.randint(2, 16), d=8 * _log_int(rng, 16, 256), F=8 * _log_int(rng, 128, 4096), B=_log_int(rng, 16, 4096),
                 k=_log_int(rng, 12, 256))
        if kind == "train":
            c["B"] = _log_int(rng, 256, 8192)
            if fn == "jumprelu":
                c["lam"] = 1e-4
            elif c["tying"] == "none" and rng.random() < 0.3:
                c["dead"] = 0.05
                c["B"] -= c["B"] % 8  # the auxiliary term's gradient products contract over the tokens in 16-byte steps
            if rng.random() < 0.3:
                c["clip"] = 1.0
        elif kind == "infer" and rng.random() < 0.5:
            c["eval"] = True
        # not larger than the largest listed case, sparse enough for the entry lists, a step below the headline step's state
        params = c["L"] * c["F"] * c["d"] + _dec_params(c)
        if c["k"] * 128 > c["L"] * c["F"] or c["B"] * c["L"] * c["F"] > 4096 * 12 * 24576:
            continue
        if params > (6e8 if kind == "train" else 1.7e9):
            continue
        if fn == "jumprelu" and kind == "train" and c["B"] * c["F"] * c["d"] * c["L"] ** 2 > 4096 * 4096 * 768 * 144:
            continue
        return c


def _rows(c):
    return [c["L"] - s if c["tying"] == "none" else 1 for s in range(c["L"])]


def _dec_params(c):
    return sum(_rows(c)) * c["F"] * c["d"]


def _t16(c):
    return torch.float16 if c["dtype"] == "fp16" else torch.bfloat16


# ------------------------------------------------------------------------------------------------ inputs
def _tokens(c, g):
    """Inputs and targets ``[L, B, d]``, standardised per layer and element."""
    L, B, d, t16 = c["L"], c["B"], c["d"], _t16(c)
    nd, per_tok = 4 * d, 32
    X = torch.empty(L, B, d, device=DEV, dtype=t16)
    Y = torch.empty_like(X)
    acc = torch.zeros(B, d, device=DEV)
    for l in range(L):
        words = torch.randn(nd, d, device=DEV, generator=g)
        pick = torch.randint(0, nd, (B, per_tok), device=DEV, generator=g)
        mag = -torch.log1p(-torch.rand(B, per_tok, device=DEV, generator=g).clamp_(max=1 - 1e-6))
        coef = torch.zeros(B, nd, device=DEV).scatter_add_(1, pick, mag)
        x = coef @ words + 0.8 * torch.randn(B, d, device=DEV, generator=g)
        x = (x - x.mean(0)) / (x.std(0) + 1e-6)
        acc = acc + x @ (torch.randn(d, d, device=DEV, generator=g) / math.sqrt(d))
        y = acc / math.sqrt(l + 1.0) + 0.05 * torch.randn(B, d, device=DEV, generator=g)
        X[l], Y[l] = x.to(t16), y.to(t16)
    return X, Y


def _gradient_scales(c):
    """Typical size of one feature's weight gradient, of a decoder bias' and of an encoder bias' in the middle of a run."""
    unit = 2.0 / (c["B"] * c["d"])
    return {"w": 0.3 * unit, "dec_bias": unit * math.sqrt(c["B"]), "enc_bias": unit, "log_threshold": unit}


def _plain(c, seed):
    """Every tensor a case starts from, as plain torch."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    L, d, F, t16 = c["L"], c["d"], c["F"], _t16(c)
    n_bias = L * (L + 1) // 2 if c["tying"] == "none" else L
    X, Y = _tokens(c, g)
    bound_e, bound_d = 1.0 / math.sqrt(F), 1.0 / math.sqrt(L * d)
    p = {
        "enc_weight": torch.empty(L, F, d, device=DEV, dtype=t16).uniform_(-bound_e, bound_e, generator=g),
        "enc_bias": torch.empty(L, F, device=DEV, dtype=t16).uniform_(-0.1 * bound_e, 0.1 * bound_e, generator=g),
        "dec_weight": [torch.empty(F, r, d, device=DEV, dtype=t16).uniform_(-bound_d, bound_d, generator=g) for r in _rows(c)],
        "dec_bias": torch.empty(n_bias, d, device=DEV, dtype=t16).uniform_(-0.02, 0.02, generator=g),
    }
    if c["fn"] == "jumprelu":
        # the threshold that leaves about k of a token's L * F pre-activations active, spread by a few per cent per feature
        z = -math.sqrt(2.0) * float(torch.erfinv(torch.tensor(2.0 * c["k"] / (L * F) - 1.0, dtype=torch.float64)))
        theta = math.log(z * math.sqrt(d / 3.0) * bound_e)
        p["log_threshold"] = theta + 0.02 * torch.randn(L, F, device=DEV, generator=g)
    s = {"X": X, "Y": Y, "params": p, "sigma": 0.5 + torch.rand(L, d, device=DEV, generator=g)}
    if c["kind"] == "train":
        sizes = _gradient_scales(c)

        def moments(t, size):
            m = torch.empty(t.shape, device=DEV).normal_(0.0, size, generator=g)
            v = torch.empty(t.shape, device=DEV).uniform_(0.5 * size * size, 1.5 * size * size, generator=g)
            return m, v

        s["moments"] = {n: ([moments(w, sizes["w"]) for w in t] if n == "dec_weight" else moments(t, sizes.get(n, sizes["w"])))
                        for n, t in p.items()}
        if c.get("dead"):
            s["dead"] = torch.rand(L, F, device=DEV, generator=g) < c["dead"]
    return s


def prepare(case, seed):
    from crosslayer_coding_b200 import CLTConfig, CrossLayerTranscoder, TrainingConfig

    c = case
    s = _plain(c, seed)
    p = s.pop("params")
    cfg = CLTConfig(num_features=c["F"], num_layers=c["L"], d_model=c["d"], activation_fn=c["fn"], batchtopk_k=c["k"], topk_k=c["k"],
                    clt_dtype="float16" if c["dtype"] == "fp16" else "bfloat16", decoder_tying=c["tying"])
    model = CrossLayerTranscoder(cfg, device=DEV)
    with torch.no_grad():
        for n, t in p.items():
            if n == "dec_weight":
                for w, src in zip(model.dec_weight, t):
                    w.copy_(src)
            else:
                getattr(model, n).copy_(t)
    del p
    state = {"case": c, "model": model, "X": s["X"], "Y": s["Y"], "sigma": s["sigma"]}
    if c["kind"] == "train":
        from crosslayer_coding_b200.training.fused_engine import FusedBatchTopKEngine

        tc = TrainingConfig(learning_rate=LR, training_steps=100000, activation_path="unused", precision=c["dtype"],
                            sparsity_lambda=c.get("lam", 0.0), preactivation_coef=0.0, loss_scale_init=LOSS_SCALE,
                            gradient_clip_val=c.get("clip"), aux_loss_factor=AUX_FACTOR if c.get("dead") else None,
                            dead_feature_window=DEAD_WINDOW)
        eng = FusedBatchTopKEngine(model, tc, c["B"], sigma_tg=s["sigma"])
        eng.opt_step = WARM_STEPS
        mom = s.pop("moments")
        for n, of in (("enc", "enc_weight"), ("encb", "enc_bias"), ("decb", "dec_bias"), ("theta", "log_threshold")):
            if of not in mom:
                continue
            m, v = mom[of]
            getattr(eng, n + "_m").copy_(m)
            getattr(eng, n + "_v").copy_(v)
        for i, (m, v) in enumerate(mom["dec_weight"]):
            eng.dec_m[i].copy_(m)
            eng.dec_v[i].copy_(v)
        if c.get("dead"):
            eng.dead_counter.view(c["L"], c["F"]).masked_fill_(s["dead"], DEAD_WINDOW + 1)
            eng.set_dead_count_hint(int(s["dead"].sum(dim=1).max()))
        state["engine"] = eng
    else:
        from crosslayer_coding_b200.models.sparse_forward import SparseForward

        model.eval()
        state["forward"] = SparseForward(model, c["B"])
        state["inputs"] = {l: s["X"][l] for l in range(c["L"])}
        if c["kind"] == "theta":
            state["stats"] = {n: torch.zeros(c["L"], c["F"], device=DEV) for n in ("sum_min", "cnt_min", "mean", "std")}
            state["stats"]["batches"] = torch.zeros(c["L"], device=DEV)
    return state


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    c = state["case"]
    if c["kind"] == "infer":
        if not c.get("eval"):
            return state["forward"].forward_dict(state["inputs"])
        yhat = state["forward"].reconstruct(state["X"], state["Y"], state["sigma"])
        return {"yhat": yhat, "sq_err": state["forward"].sq_err}
    if c["kind"] == "theta":
        from crosslayer_coding_b200.models.theta import accumulate_theta_batch_sparse

        accumulate_theta_batch_sparse(state["forward"], state["X"], state["stats"])
        return state["stats"]
    eng, m = state["engine"], state["model"]
    out = eng.train_step(state["X"], state["Y"], WARM_STEPS, LR, sparsity_lambda=c.get("lam", 0.0),
                         aux_factor=AUX_FACTOR if c.get("dead") else 0.0, dead_window=DEAD_WINDOW if c.get("dead") else None)
    r = {"losses": out.vector[:5], "enc_weight": m.enc_weight, "enc_bias": m.enc_bias, "dec_weight": list(m.dec_weight), "dec_bias": m.dec_bias,
         "enc_m": eng.enc_m, "enc_v": eng.enc_v, "encb_m": eng.encb_m, "decb_m": eng.decb_m, "dec_m": eng.dec_m, "dec_v": eng.dec_v}
    if c["fn"] == "jumprelu":
        r["log_threshold"], r["theta_m"] = m.log_threshold, eng.theta_m
    return r


# ------------------------------------------------------------------------------------------------ floors
def work(case):
    c = case
    L, d, F, B = c["L"], c["d"], c["F"], c["B"]
    n_ent = B * c["k"]
    rows = {"none": (L + 1) / 2.0, "per_source": 1.0, "per_target": (L + 1) / 2.0}[c["tying"]]  # decoder rows behind an entry
    touched = L * F * (1.0 - math.exp(-n_ent / (L * F)))                                        # features with an entry
    gemm = 2.0 * L * B * d * F
    targets = (L + 1) / 2.0
    if c["kind"] == "theta":
        return {"bytes": 2.0 * L * F * d + 2.0 * L * B * d + 32.0 * L * F, "flops": gemm}
    dec_rows = touched * rows if c["tying"] != "per_target" else min(touched * rows, 1.0 * L * F)
    if c["kind"] == "infer":
        ev = 1 if c.get("eval") else 0
        return {"bytes": 2.0 * L * F * d + 2.0 * dec_rows * d + (2.0 + 4.0 + 2.0 * ev) * L * B * d, "flops": gemm + 2.0 * n_ent * targets * d}
    params = L * F * d + _dec_params(c)
    # weights and both moments in and out, inputs and targets in
    flops = gemm + 2.0 * 3.0 * n_ent * targets * d + 2.0 * n_ent * d + 12.0 * params
    if c["fn"] == "jumprelu":  # the window of the threshold gradient covers most positions: dL/da is needed at all of them
        flops += 2.0 * B * F * d * targets * L
    if c.get("dead"):
        flops += 8.0 * L * B * d * F * c["dead"]
    return {"bytes": 20.0 * params + 4.0 * L * B * d, "flops": flops}


def tolerance(case):
    return {"rel": 0.02, "max": 0.99}


# ------------------------------------------------------------------------------------------------ 64-bit restatement
def _select(c, pre):
    """0/1 mask of the kept entries of ``pre [L, B, F]`` (float64 values of the stored 16-bit pre-activations)."""
    L, B, F = pre.shape
    z = (pre - pre.mean(1, keepdim=True)) / (pre.std(1, keepdim=True) + 1e-6)
    rank = z.permute(1, 0, 2).reshape(B, L * F)
    del z
    mask = torch.zeros(B, L * F, device=DEV, dtype=torch.bool)
    if c["fn"] == "batchtopk":
        mask.view(-1)[torch.topk(rank.reshape(-1), c["k"] * B, sorted=False).indices] = True
    else:
        mask.scatter_(1, torch.topk(rank, c["k"], dim=1, sorted=False).indices, True)
    return mask.view(B, L, F).permute(1, 0, 2)


def _preact(c, s):
    """Pre-activations in 64 bits, rounded to the 16-bit type they are stored in."""
    p = s["params"]
    return torch.stack([(s["X"][l].double() @ p["enc_weight"][l].double().t() + p["enc_bias"][l].double()).to(_t16(c)).double()
                        for l in range(c["L"])])


def _pair(s, t, L):
    return s * L - (s * (s - 1)) // 2 + (t - s)


def _dec_of(c, dec, s, t):
    return dec[s][:, t - s] if c["tying"] == "none" else dec[s if c["tying"] == "per_source" else t][:, 0]


def _decode(c, acts, dec, bias, t):
    out = 0
    for s in range(t + 1):
        out = out + acts[s] @ _dec_of(c, dec, s, t)
        if c["tying"] != "per_target":
            out = out + bias[_pair(s, t, c["L"]) if c["tying"] == "none" else s]
    return out + bias[t] if c["tying"] == "per_target" else out


def exact(case, seed):
    c = case
    L, B, F, d = c["L"], c["B"], c["F"], c["d"]
    if c["kind"] == "train" and (B * L * F > 4e8 or _dec_params(c) > 6e8):
        return None  # the dense 64-bit step does not fit the time
    s = _plain(c, seed)
    p = s["params"]
    pre = _preact(c, s)
    if c["fn"] == "jumprelu":
        theta = p["log_threshold"].double().exp()
        mask = pre >= theta[:, None, :]
    else:
        mask = _select(c, pre)
    if c["kind"] == "theta":
        mean, std = pre.mean(1), pre.std(1)
        low = torch.where(mask & (pre > 0), (pre - mean[:, None]) / (std[:, None] + 1e-6), math.inf).amin(1)
        hit = torch.isfinite(low)
        return {"sum_min": torch.where(hit, low, 0.0), "cnt_min": hit.double(), "mean": mean, "std": std,
                "batches": torch.ones(L, device=DEV, dtype=torch.float64)}
    acts = pre * mask
    if c["kind"] == "infer":
        del pre, mask
        dec, bias = p["dec_weight"], p["dec_bias"].double()
        yhat = []
        for t in range(L):
            out = torch.zeros(B, d, device=DEV, dtype=torch.float64)
            for q in range(t + 1):
                out += acts[q] @ _dec_of(c, dec, q, t).double()
                if c["tying"] != "per_target":
                    out += bias[_pair(q, t, L) if c["tying"] == "none" else q]
            yhat.append(out + bias[t] if c["tying"] == "per_target" else out)
        if not c.get("eval"):
            return dict(enumerate(yhat))
        yhat = torch.stack(yhat)
        return {"yhat": yhat, "sq_err": ((yhat - s["Y"].double()) * s["sigma"].double()[:, None]).square().sum((1, 2))}
    return _exact_step(c, s, pre, mask, acts)


def _exact_step(c, s, pre, mask, acts):
    L, B, F, d = c["L"], c["B"], c["F"], c["d"]
    p, mom = s["params"], s["moments"]
    sg, Y, X = s["sigma"].double(), s["Y"].double(), s["X"].double()
    dec = [w.double().requires_grad_() for w in p["dec_weight"]]
    dec_b = p["dec_bias"].double().requires_grad_()
    acts = acts.requires_grad_()
    yhat = [_decode(c, acts, dec, dec_b, t) for t in range(L)]
    recon = sum((((yhat[t] - Y[t]) * sg[t]).square().mean() for t in range(L)), torch.zeros((), device=DEV, dtype=torch.float64))
    zero = torch.zeros((), device=DEV, dtype=torch.float64)
    penalty, aux = zero, zero
    if c.get("lam"):
        for l in range(L):
            if c["tying"] == "per_target":
                norm = sum(dec[t].square().sum((1, 2)) for t in range(l, L)).sqrt()
            else:
                norm = dec[l].square().sum((1, 2)).sqrt()
            penalty = penalty + torch.tanh(acts[l] * norm).sum()
        penalty = c["lam"] * penalty
    aux_in = None
    if c.get("dead"):
        aux_in = pre.clone().requires_grad_()
        for l in range(L):
            n_dead = int(s["dead"][l].sum())
            if n_dead == 0:
                continue
            kk = min(512, n_dead)
            keep = torch.zeros(B, F, device=DEV, dtype=torch.bool)
            keep.scatter_(1, torch.topk(torch.where(s["dead"][l], pre[l], -math.inf), kk, dim=1, sorted=False).indices, True)
            rec = (aux_in[l] * keep) @ _dec_of(c, dec, l, l) + dec_b[_pair(l, l, L) if c["tying"] == "none" else l]
            aux = aux + min(n_dead / kk, 1.0) * (rec - (Y[l] - yhat[l]) * sg[l]).square().mean()
        aux = AUX_FACTOR * aux
    total = recon + penalty + aux
    total.backward()
    g_pre = acts.grad * mask
    if aux_in is not None:
        g_pre = g_pre + aux_in.grad
    grads = {
        "enc_weight": torch.stack([g_pre[l].t() @ X[l] for l in range(L)]), "enc_bias": g_pre.sum(1),
        "dec_weight": [w.grad for w in dec], "dec_bias": dec_b.grad,
    }
    if c["fn"] == "jumprelu":
        theta = p["log_threshold"].double().exp()
        window = (pre - theta[:, None]).abs() <= 0.5
        grads["log_threshold"] = -(acts.grad * pre * window).sum(1) * theta
    clip = 1.0
    if c.get("clip"):
        flat = [t for v in grads.values() for t in (v if isinstance(v, list) else [v])]
        clip = min(1.0, c["clip"] / (math.sqrt(sum(float(t.square().sum()) for t in flat)) + 1e-6))
    b1, b2, eps, wd = ADAM
    n = WARM_STEPS + 1

    def adam(w, g, m, v):
        m = b1 * m.double() + (1 - b1) * g * clip
        v = b2 * v.double() + (1 - b2) * (g * clip).square()
        return w.detach().double() * (1 - LR * wd) - LR / (1 - b1 ** n) * m / ((v / (1 - b2 ** n)).sqrt() + eps), m, v

    new = {k: ([adam(w, g, *mv) for w, g, mv in zip(p[k], grads[k], mom[k])] if k == "dec_weight" else adam(p[k], grads[k], *mom[k])) for k in grads}
    r = {"losses": torch.stack([total, recon, penalty, zero, aux]).detach(), "enc_weight": new["enc_weight"][0], "enc_bias": new["enc_bias"][0],
         "dec_weight": [t[0] for t in new["dec_weight"]], "dec_bias": new["dec_bias"][0],
         "enc_m": new["enc_weight"][1], "enc_v": new["enc_weight"][2], "encb_m": new["enc_bias"][1], "decb_m": new["dec_bias"][1],
         "dec_m": [t[1] for t in new["dec_weight"]], "dec_v": [t[2] for t in new["dec_weight"]]}
    if c["fn"] == "jumprelu":
        r["log_threshold"], r["theta_m"] = new["log_threshold"][0], new["log_threshold"][1]
    return r
