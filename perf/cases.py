"""The work that programs have this framework do, as a list of timed cases.

A case is one call of a training program: an optimizer step between two refreshes of its
preconditioners, a step that refreshes them, a GPA-AdamW step, the fused LM head + loss, or a whole
training step of a small decoder.  ``prepare`` builds what such a program holds before the call
(parameters, gradients, the optimizer with its state some steps into a run), ``run`` makes the call
through the public classes and returns every tensor it updates.

Gradients are what layers produce: rows and columns whose scales differ by decades (log-normal), a few
dominant directions on top of full-rank noise.
"""

import math
import random

import torch

import optimizers_b200 as ob

# Steps between two refreshes in the cases that time an ordinary step: no refresh falls inside a timing run.
_PERIOD = 100_000


def _weights(*shapes):
    return ";".join("x".join(str(n) for n in s) for s in shapes)


def _shapes(text):
    return [tuple(int(n) for n in s.split("x")) for s in text.split(";")]


def _decoder_layer(d, mlp, bias=True):
    """Parameters of one pre-LN decoder layer: fused QKV, attention output, MLP in and out, two norms."""
    mats = [(3 * d, d), (d, d), (mlp, d), (d, mlp)]
    if not bias:
        return mats
    out = []
    for rows, cols in mats:
        out += [(rows, cols), (rows,)]
    return out + [(d,)] * 4


def listed():
    return [
        # Latency: the 784-512-10 perceptron on which the optimizer is introduced, blocks of 256, Adam grafting.
        dict(name="mlp_step", kind="step", weights=_weights((512, 784), (512,), (10, 512), (10,)), block=256,
             optimizer="shampoo", graft="adam", averaging="none", weight_decay=0.0, ema=0.999),
        # Convolutions (order-3 blocks), batch-norm vectors, momentum: a slice of the CIFAR ResNet-18 configuration.
        dict(name="resnet_step", kind="step",
             weights=_weights((64, 3, 3, 3), (64,), (64, 64, 3, 3), (64,), (128, 64, 3, 3), (128,), (256, 128, 3, 3), (256,),
                              (256, 128, 1, 1), (10, 512)),
             block=1024, optimizer="shampoo", graft="adam", averaging="momentum", weight_decay=0.0, ema=0.999),
        # Two layers of the GPT-2 124M decoder with biases and norms, blocks of 2048, AdaGrad grafting, summed factors.
        dict(name="gpt2_step", kind="step", weights=_weights(*(_decoder_layer(768, 3072) * 2)), block=2048,
             optimizer="shampoo", graft="adagrad", averaging="none", weight_decay=0.0, ema=1.0),
        # Odd and ragged widths, unaligned rows, decoupled weight decay, primal averaging; KL statistics.
        dict(name="ragged_kl_step", kind="step", weights=_weights((1000, 1337), (333, 1000), (77, 333), (1337,), (333,)), block=512,
             optimizer="kl", graft="rmsprop", averaging="gpa", weight_decay=0.01, ema=0.99),
        # The largest root-inverse step: one 8192 x 8192 weight, sixteen blocks of 2048.
        dict(name="wide_step", kind="step", weights=_weights((8192, 8192)), block=2048,
             optimizer="shampoo", graft="sgd", averaging="none", weight_decay=0.0, ema=0.999),
        # Eigenvalue-corrected (SOAP) step over the matrices of one 2048-wide SwiGLU decoder layer, blocks of 4096.
        dict(name="llama_soap_step", kind="step",
             weights=_weights(*([(2048, 2048)] * 4), (8192, 2048), (8192, 2048), (2048, 8192), (2048,), (2048,)), block=4096,
             optimizer="soap", graft="none", averaging="none", weight_decay=0.0, ema=0.999),
        # Refresh by eigendecomposition: every factor (256 to 2048) of one GPT-2 124M layer.
        dict(name="gpt2_eigh_refresh", kind="refresh", weights=_weights(*_decoder_layer(768, 3072, bias=False)), block=2048,
             optimizer="shampoo", graft="adagrad", averaging="none", weight_decay=0.0, ema=1.0),
        # Refresh by the coupled Newton iteration, factors of 1024 and below.
        dict(name="newton_refresh", kind="refresh", weights=_weights((1024, 4096), (1024, 1024), (600, 1024)), block=1024,
             optimizer="newton", graft="adam", averaging="none", weight_decay=0.0, ema=0.999),
        # Refresh of the SOAP eigenbases by one warm-started QR iteration.
        dict(name="soap_qr_refresh", kind="refresh", weights=_weights((1024, 1024), (1024, 1024), (1024, 768), (700, 300)), block=1024,
             optimizer="soap", graft="none", averaging="none", weight_decay=0.0, ema=0.999),
        # GPA-AdamW over a 124M-parameter decoder's matrices, fp32.
        dict(name="gpa_step", kind="gpa", weights=_weights(*(_decoder_layer(768, 3072, bias=False) * 4), (50257, 768)), dtype="float32",
             weight_decay=0.01),
        # LM head + cross-entropy, forward and backward: 16 sequences of 1024 tokens, the GPT-2 vocabulary.
        dict(name="lm_head_loss", kind="head", tokens=16384, width=768, vocab=50257),
        # A training step of a small GPT-2 style decoder: forward, backward and optimizer step, bf16 autocast.
        dict(name="gpt2_train", kind="train", layers=2, width=768, heads=12, vocab=8192, batch=8, seq=1024, block=2048),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dim(rng, lo, hi):
    """A width: a multiple of 64, or of 8, or any number."""
    n = _log_int(rng, lo, hi)
    step = rng.choice([64, 64, 8, 1])
    return max(lo, n // step * step) if n >= step else n


def draw(rng: random.Random):
    kind = rng.choice(["step", "step", "step", "step", "step", "refresh", "refresh", "gpa", "head", "train"])
    while kind in ("step", "refresh"):
        if kind == "step":
            optimizer = rng.choice(["shampoo", "shampoo", "shampoo", "soap", "kl"])
            shapes = []
            for _ in range(rng.randint(1, 6)):
                shapes.append((_dim(rng, 24, 4096), _dim(rng, 24, 4096)))
                if rng.random() < 0.4:
                    shapes.append(shapes[-1][:1])
            case = dict(
                kind="step", weights=_weights(*shapes), block=rng.choice([256, 512, 1024, 2048]), optimizer=optimizer,
                graft=rng.choice(["adam", "adagrad", "rmsprop", "sgd"]), averaging=rng.choice(["none", "none", "momentum", "gpa"]),
                weight_decay=rng.choice([0.0, 0.01]), ema=rng.choice([0.99, 0.999, 1.0]),
            )
        else:
            optimizer = rng.choice(["shampoo", "shampoo", "newton", "soap"])
            shapes = [(_dim(rng, 48, 1536), _dim(rng, 48, 1536)) for _ in range(rng.randint(1, 4))]
            case = dict(
                kind="refresh", weights=_weights(*shapes), block=rng.choice([256, 512, 1024, 2048]), optimizer=optimizer,
                graft="none" if optimizer == "soap" else "adam", averaging="none", weight_decay=0.0, ema=0.999,
            )
        # No larger than the largest listed case, and few enough tensors to hand back whole.
        if work(case)["flops"] < (2.5e12 if kind == "step" else 3e11) and _tensors(case) <= 63:
            return case
    if kind == "gpa":
        shapes = [(_dim(rng, 32, 4096), _dim(rng, 32, 4096)) for _ in range(rng.randint(1, 12))]
        shapes += [s[:1] for s in shapes if rng.random() < 0.5][: 20 - len(shapes)]
        return dict(kind="gpa", weights=_weights(*shapes), dtype=rng.choice(["float32", "float32", "bfloat16"]), weight_decay=0.01)
    if kind == "head":
        return dict(kind="head", tokens=_log_int(rng, 512, 16384), width=8 * _log_int(rng, 16, 128), vocab=_log_int(rng, 1000, 50257))
    width = 64 * rng.choice([4, 8, 12])
    return dict(kind="train", layers=rng.randint(1, 2), width=width, heads=width // 64, vocab=_log_int(rng, 1000, 8192),
                batch=rng.randint(1, 8), seq=64 * rng.randint(2, 16), block=rng.choice([512, 1024, 2048]))


# ----------------------------------------------------------------------------------------------
# What a program holds before the call
# ----------------------------------------------------------------------------------------------
def _gradient(shape, gen, scales):
    """A layer gradient of the given shape; ``scales`` are its row and column scales (fixed over a run)."""
    if len(shape) == 1:
        return torch.randn(shape, device="cuda", generator=gen) * 1e-4
    rows, cols = shape[0], math.prod(shape[1:])
    r_scale, c_scale = scales
    rank = min(rows, cols, 8)
    # dominant singular values of 7 / sqrt(k) times the edge of the noise's spectrum
    strength = torch.arange(1, rank + 1, device="cuda").rsqrt() * (7.0 / math.sqrt(rows) + 7.0 / math.sqrt(cols))
    g = torch.randn(rows, cols, device="cuda", generator=gen)
    g += (torch.randn(rows, rank, device="cuda", generator=gen) * strength) @ torch.randn(rank, cols, device="cuda", generator=gen)
    return (g * (r_scale * c_scale * 1e-4)).view(shape)


def _scales(shape, gen):
    if len(shape) == 1:
        return None
    rows, cols = shape[0], math.prod(shape[1:])
    decades = lambda n: torch.pow(10.0, 0.25 * torch.randn(n, device="cuda", generator=gen))  # noqa: E731
    return decades(rows).unsqueeze(1), decades(cols).unsqueeze(0)


def _parameters(shapes, gen, dtype=torch.float32):
    """One buffer, and the parameters as aligned views of it (the way flat-parameter wrappers keep them)."""
    sizes = [(math.prod(s) + 127) // 128 * 128 for s in shapes]
    flat = (torch.randn(sum(sizes), device="cuda", generator=gen) * 0.02).to(dtype)
    return flat, [torch.nn.Parameter(part[: math.prod(s)].view(s)) for part, s in zip(flat.split(sizes), shapes)]


def _shampoo(params, case, period):
    """The optimizer a program constructs for ``case``; refreshes every ``period`` steps from step ``period`` on."""
    graft = {
        "none": None, "sgd": ob.SGDPreconditionerConfig(), "adagrad": ob.AdaGradPreconditionerConfig(epsilon=1e-10),
        "rmsprop": ob.RMSpropPreconditionerConfig(beta2=0.99, epsilon=1e-8),
        "adam": ob.AdamPreconditionerConfig(beta2=0.999, epsilon=1e-8),
    }[case["graft"]]
    preconditioner = {
        "shampoo": ob.RootInvShampooPreconditionerConfig(),
        "newton": ob.RootInvShampooPreconditionerConfig(amortized_computation_config=ob.CoupledNewtonConfig()),
        "kl": ob.RootInvKLShampooPreconditionerConfig(),
        "soap": ob.EigenvalueCorrectedShampooPreconditionerConfig(amortized_computation_config=ob.QREigendecompositionConfig()),
    }[case["optimizer"]]
    averaging = {
        "none": None, "momentum": ob.ClassicMomentumConfig(momentum=0.9),
        "gpa": ob.GeneralizedPrimalAveragingConfig(eval_interp_coeff=0.9, train_interp_coeff=0.7),
    }[case["averaging"]]
    opt = ob.DistributedShampoo(
        params, lr=1e-3, betas=(0.9, case["ema"]), epsilon=1e-7, weight_decay=case["weight_decay"],
        max_preconditioner_dim=case["block"], precondition_frequency=period[0], start_preconditioning_step=period[1],
        grafting_config=graft, preconditioner_config=preconditioner, iterate_averaging_config=averaging,
    )
    opt.train()
    return opt


def _accumulate(opt, params, shapes, gen, steps):
    """``steps`` optimizer steps on fresh gradients; the gradients of one more step are left in place."""
    scales = [_scales(s, gen) for s in shapes]
    for k in range(steps + 1):
        for p, s, sc in zip(params, shapes, scales):
            p.grad = _gradient(s, gen, sc)
        if k < steps:
            opt.step()


def _set_step(opt, value):
    """The run is resumed at step ``value`` (the step counter of a group is one tensor under all its parameters)."""
    for state in opt.state.values():
        if "step" in state:
            state["step"].fill_(value)


def _load_eigenbases(opt, gen):
    """The run is resumed from a checkpoint that holds eigenbases (orthonormal, of no special relation to the
    gradients that follow) and no second moments yet."""
    state = opt.state_dict()
    for of_param in state["state"].values():
        for key in of_param:
            if not str(key).startswith("block_"):
                continue
            factors = of_param[key]["shampoo"]
            factors["corrected_eigenvalues"].zero_()
            for basis in factors["factor_matrices_eigenvectors"].values():
                basis.copy_(torch.linalg.qr(torch.randn(basis.shape, device="cuda", generator=gen))[0])
    opt.load_state_dict(state)


def prepare(case, seed):
    kind = case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind in ("step", "refresh"):
        shapes = _shapes(case["weights"])
        flat, params = _parameters(shapes, gen)
        if kind == "step":
            # Four steps that collect statistics, one refresh (or loaded eigenbases), one ordinary step behind it.
            opt = _shampoo(params, case, (_PERIOD, _PERIOD))
            if case["optimizer"] == "soap":
                _load_eigenbases(opt, gen)
                _set_step(opt, _PERIOD + 1)
            else:
                _set_step(opt, _PERIOD - 5)
            _accumulate(opt, params, shapes, gen, 6)
        else:
            # Four steps that collect statistics; from the next one on every step refreshes.
            opt = _shampoo(params, case, (1, 5))
            if case["optimizer"] == "soap":
                _load_eigenbases(opt, gen)
            _accumulate(opt, params, shapes, gen, 4)
        return dict(kind=kind, opt=opt, params=params, flat=flat)
    if kind == "gpa":
        shapes = _shapes(case["weights"])
        flat, params = _parameters(shapes, gen, getattr(torch, case["dtype"]))
        opt = ob.GPAAdamW(params, lr=1e-3, weight_decay=case["weight_decay"])
        opt.train()
        for k in range(2):
            for p in params:
                p.grad = (torch.randn(p.shape, device="cuda", generator=gen) * 1e-3).to(p.dtype)
            if k == 0:
                opt.step()
        return dict(kind=kind, opt=opt, params=params, flat=flat)
    if kind == "head":
        x = torch.randn(case["tokens"], case["width"], device="cuda", generator=gen).to(torch.bfloat16).requires_grad_(True)
        w = (torch.randn(case["vocab"], case["width"], device="cuda", generator=gen) * 0.02).requires_grad_(True)
        targets = torch.randint(0, case["vocab"], (case["tokens"],), device="cuda", generator=gen)
        return dict(kind=kind, x=x, w=w, targets=targets)
    from optimizers_b200.models import GPT2, GPT2Config

    devices = [torch.cuda.current_device()]
    with torch.random.fork_rng(devices=devices):
        torch.manual_seed(seed)
        model = GPT2(GPT2Config(vocab_size=case["vocab"], n_ctx=case["seq"], n_layer=case["layers"], n_head=case["heads"],
                                d_model=case["width"], d_mlp=4 * case["width"])).cuda()
    params = list(model.parameters())
    flat, views = _parameters([tuple(p.shape) for p in params], gen)
    for p, v in zip(params, views):
        v.data.copy_(p.data)
        p.data = v.data
    opt = _shampoo(params, dict(case, optimizer="shampoo", graft="adagrad", averaging="none", weight_decay=0.0, ema=1.0),
                   (_PERIOD, _PERIOD))
    _set_step(opt, _PERIOD - 3)
    tokens = torch.randint(0, case["vocab"], (4, case["batch"], case["seq"] + 1), device="cuda", generator=gen)
    for k in range(3):
        _train_step(model, opt, tokens[k])
    return dict(kind=kind, opt=opt, params=params, flat=flat, model=model, tokens=tokens[3])


# ----------------------------------------------------------------------------------------------
# One call, and all that it updates
# ----------------------------------------------------------------------------------------------
def _train_step(model, opt, tokens):
    with torch.autocast("cuda", dtype=torch.bfloat16):
        loss = model(tokens[:, :-1], tokens[:, 1:])
    loss.backward()
    opt.step()
    opt.zero_grad(set_to_none=True)
    return loss


def _statistics(opt, params, fields):
    """The tensors of the optimizer's state named ``fields``, block by block.  Eigenvectors are left out (where
    eigenvalues nearly coincide their order is arbitrary): they show in the parameters, as moments and averages
    do in those of the following call."""
    out = []
    for p in params:
        state = opt.state[p]
        for key in state:
            if not str(key).startswith("block_"):
                continue
            for field in fields:
                value = getattr(state[key]["shampoo"], field, None)
                if value is not None:
                    out += list(value) if isinstance(value, (tuple, list)) else [value]
    return out


def run(state):
    kind = state["kind"]
    if kind == "head":
        from optimizers_b200.models.fused_ops import lm_head_cross_entropy

        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = lm_head_cross_entropy(state["x"], state["w"], state["targets"])
        dx, dw = torch.autograd.grad(loss, (state["x"], state["w"]))
        return [loss, dx, dw]
    params, opt = state["params"], state["opt"]
    if kind == "train":
        return [_train_step(state["model"], opt, state["tokens"]).detach(), state["flat"]]
    opt.step()
    if kind == "gpa":
        return [state["flat"], *(opt.state[p][k] for p in params for k in ("exp_avg", "exp_avg_sq", "z"))]
    # An ordinary step leaves roots and bases as they are; a refresh replaces them, and with a basis the order of
    # the second moments in it.
    fields = ("factor_matrices", "inv_factor_matrices" if kind == "refresh" else "corrected_eigenvalues")
    return [state["flat"], *_statistics(opt, params, fields)]


# ----------------------------------------------------------------------------------------------
# What the path cannot do without
# ----------------------------------------------------------------------------------------------
def _blocks(shape, block):
    """Sizes of the blocks a parameter is cut into (small neighbouring dims merge up to ``block``)."""
    dims = []
    for n in shape:
        if dims and dims[-1] * n <= block:
            dims[-1] *= n
        else:
            dims.append(n)
    if len(dims) > 1 and dims[0] == 1:
        dims = dims[1:]
    cuts = [[min(block, n - i) for i in range(0, n, block)] for n in dims]
    out = [()]
    for c in cuts:
        out = [o + (k,) for o in out for k in c]
    return out


def _tensors(case):
    """Tensors that ``run`` hands back for a step or refresh: factors (and roots, or second moments) of every block."""
    count = 1
    for s in _shapes(case["weights"]):
        for b in _blocks(s, case["block"]):
            count += len(b) * (2 if case["kind"] == "refresh" and case["optimizer"] != "soap" else 1) + (case["optimizer"] == "soap")
    return count


def _step_work(shapes, block, optimizer, graft, averaging):
    """One step: gradient, weight and moments read, weight and moments written; triangular factors read and
    written, roots (or eigenvectors) read; the Gram products (one triangle) and the preconditioning products."""
    nbytes = flops = 0.0
    elementwise = 4 * (1 + 2 + 2 + (2 if graft in ("adam", "adagrad", "rmsprop") else 0) + (2 if averaging != "none" else 0))
    for s in shapes:
        for b in _blocks(s, block):
            n = math.prod(b)
            nbytes += elementwise * n
            for d in b:
                nbytes += 4 * (d * (d + 1) + (d * (d + 1) / 2 if optimizer != "soap" else d * d))
                flops += n * d  # half of the Gram product
                flops += 2 * n * d  # preconditioning
                if optimizer == "kl" and len(b) > 1:
                    flops += 2 * n * d
                if optimizer == "soap":
                    flops += 4 * n * d  # projection of two gradients and one way back
            if optimizer == "soap":
                nbytes += 8 * n
    return nbytes, flops


def work(case):
    kind = case["kind"]
    if kind in ("step", "refresh"):
        shapes = _shapes(case["weights"])
        nbytes, flops = _step_work(shapes, case["block"], case["optimizer"], case["graft"], case["averaging"])
        if kind == "refresh":
            for s in shapes:
                for b in _blocks(s, case["block"]):
                    for d in b:
                        # 4/3 d^3 to tridiagonal form, 3 d^3 for the vectors, d^3 for the root; Newton: ten
                        # iterations of four products; QR: two congruences, a factorisation, the new basis
                        flops += {"shampoo": 16 / 3, "newton": 40, "soap": 26 / 3}[case["optimizer"]] * d**3
                        nbytes += 4 * d * d
        return dict(bytes=nbytes, flops=flops)
    if kind == "gpa":
        n = sum(math.prod(s) for s in _shapes(case["weights"]))
        size = 4 if case["dtype"] == "float32" else 2
        return dict(bytes=(3 * size + 24) * n, flops=20 * n)
    if kind == "head":
        t, c, v = case["tokens"], case["width"], case["vocab"]
        return dict(bytes=4 * t * c + 8 * v * c, flops=6.0 * t * c * v)
    c, v, t, layers = case["width"], case["vocab"], case["batch"] * case["seq"], case["layers"]
    shapes = [(v, c), (case["seq"], c), (c,), (c,)] + _decoder_layer(c, 4 * c) * layers
    nbytes, flops = _step_work(shapes, case["block"], "shampoo", "adagrad", "none")
    flops += 6.0 * t * (12 * c * c * layers + c * v) + 7.0 * layers * t * case["seq"] * c
    nbytes += 8 * sum(math.prod(s) for s in shapes) + layers * t * c * 60
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    """About four times the difference between the path and the same mathematics through plain PyTorch (fp32
    library products and eigensolver, fp32 loss of bf16 logits), the largest over these ranges."""
    kind = case["kind"]
    if kind == "gpa":
        return {"rel": 5e-5} if case["dtype"] == "float32" else {"rel": 4e-3}
    if kind == "head":
        return {"rel": 1e-2, "max": 0.1}
    if kind == "train":
        return {"rel": 2e-3, "max": 0.1}
    if kind == "refresh":
        # The new SOAP basis orders its columns by their Rayleigh quotients, and neighbours that agree to rounding swap.
        return {"rel": 2.5e-2, "max": 0.3} if case["optimizer"] == "soap" else {"rel": 5e-3, "max": 0.9}
    return {"rel": 1e-3, "max": 0.05}
