"""The work that users of this framework have it do on one GPU, as cases to be timed.

Kinds, each through the entry points that a user's program calls:

step       one denoising step of a whole model (ShapedDiT.forward_graphed), weights resident
request    a text-to-image request: all steps with classifier-free guidance (SD3ShapedPipeline.diffusion_stage)
attention  one long-context attention layer (the hetuDiT*LongContextAttention operators), joint text rows as a
           segment of their own
ring       what one rank of a ring does in a layer: its own K/V block, then the other ranks' blocks merged into it
           (kernels.attn_fwd in its partial and merge modes)
patch      what a PipeFusion stage does in a layer for one patch: fresh K/V rows into the stale buffer
           (kernels.kv_scatter), then the patch's queries against the whole buffer (kernels.attn_fwd)
guidance   guidance + scheduler step of a patch of latents (kernels.cfg_euler_step)
migration  the byte moves of a tensor-parallel re-slice of a block's linear layers (kernels.copy_pieces)

Weights are N(0, 0.02) and inputs N(0, 1), made from the seed: there are no checkpoints here.
"""
import torch

import hetu_dit_b200.model_executor.models.shaped_dit as shapes
from hetu_dit_b200 import _C, kernels
from hetu_dit_b200.config import EngineConfig
from hetu_dit_b200.core.distributed import parallel_state as ps
from hetu_dit_b200.core.distributed.runtime_state import ModelGeometry, initialize_runtime_state
from hetu_dit_b200.core.parallel import (hetuDiTFluxLongContextAttention, hetuDiTJointLongContextAttention,
                                         hetuDiTLongContextAttention)
from hetu_dit_b200.model_executor.models.shaped_dit import ShapedDiT
from hetu_dit_b200.model_executor.pipelines.pipeline_sd3_shaped import SD3ShapedPipeline

DEV = "cuda:0"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
# heads, head size of the models' attention layers
LAYERS = {"FLUX_DEV": (24, 128), "SD3_MEDIUM": (24, 64), "COGVIDEOX_5B": (48, 64), "HUNYUAN_VIDEO": (24, 128)}


def listed():
    return [
        # the benchmark's step: a 1024 x 1024 image, full prompt
        {"name": "flux_step_1024", "kind": "step", "model": "FLUX_DEV", "frames": 1, "rows": 64, "cols": 64,
         "text": 512, "batch": 1, "dtype": "bf16"},
        # a small image of an odd aspect ratio with a short prompt: ragged row counts everywhere
        {"name": "flux_step_ragged", "kind": "step", "model": "FLUX_DEV", "frames": 1, "rows": 37, "cols": 53,
         "text": 231, "batch": 1, "dtype": "bf16"},
        # 1024 x 1024 with both guidance halves in one batch, as the pipelines run it
        {"name": "sd3_step_1024", "kind": "step", "model": "SD3_MEDIUM", "frames": 1, "rows": 64, "cols": 64,
         "text": 333, "batch": 2, "dtype": "bf16"},
        # a short video clip; the whole clip of the benchmark (11 frames) takes the attention of the "ring" case below
        {"name": "cogvideox_step_clip", "kind": "step", "model": "COGVIDEOX_5B", "frames": 3, "rows": 48, "cols": 85,
         "text": 224, "batch": 1, "dtype": "bf16"},
        # a short clip of the other video model (all 33 frames take longer than a pass may)
        {"name": "hunyuan_step_clip", "kind": "step", "model": "HUNYUAN_VIDEO", "frames": 3, "rows": 45, "cols": 80,
         "text": 256, "batch": 1, "dtype": "bf16"},
        # a whole request at the smallest resolution of the serving trace, fewer steps than its 20
        {"name": "sd3_request_512", "kind": "request", "model": "SD3_MEDIUM", "rows": 32, "cols": 32, "text": 77,
         "steps": 8, "dtype": "fp16"},
        # attention of one layer over a whole video (33 latent frames of 45 x 80 tokens)
        {"name": "attention_video", "kind": "attention", "model": "HUNYUAN_VIDEO", "heads": 24, "tokens": 118800,
         "text": 256, "batch": 1, "joint": "rear", "dtype": "bf16"},
        # one rank of a Ulysses degree of 8 on the benchmark's step: 3 of 24 heads over all rows
        {"name": "attention_3_heads", "kind": "attention", "model": "FLUX_DEV", "heads": 3, "tokens": 4096,
         "text": 512, "batch": 1, "joint": "front", "dtype": "bf16"},
        # one rank of a ring of 4 on the benchmark's video: 11 frames x 12 rows x 85 columns, text rows in front
        {"name": "ring_rank_video", "kind": "ring", "model": "COGVIDEOX_5B", "heads": 48, "tokens": 11220,
         "text": 224, "ring": 4, "dtype": "bf16"},
        # a quarter of a 1024 x 1024 image, both guidance halves, against the stale K/V of the whole image
        {"name": "pipefusion_patch", "kind": "patch", "model": "SD3_MEDIUM", "tokens": 4096, "patches": 4,
         "text": 154, "batch": 2, "dtype": "fp16"},
        # the last stage's work on a patch: the smallest call there is, launch latency
        {"name": "guidance_patch", "kind": "guidance", "tokens": 1024, "batch": 1, "dtype": "bf16"},
        # a plan switch re-slices the linear layers of a double block over two tensor-parallel ranks
        {"name": "migration_block", "kind": "migration", "model": "FLUX_DEV", "blocks": 1, "degree": 2,
         "dtype": "bf16"},
    ]


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))

    kind = rng.choice(["step", "step", "step", "request", "attention", "attention", "ring", "patch", "guidance",
                       "migration"])
    if kind == "step":
        model = rng.choice(["FLUX_DEV", "SD3_MEDIUM", "COGVIDEOX_5B", "HUNYUAN_VIDEO"])
        video = model in ("COGVIDEOX_5B", "HUNYUAN_VIDEO")
        return {"kind": kind, "model": model, "frames": rng.randint(1, 3) if video else 1, "rows": rng.randint(16, 45 if video else 64),
                "cols": rng.randint(16, 80 if video else 64), "text": rng.randint(77, 256 if video else 512),
                "batch": rng.randint(1, 2) if model == "SD3_MEDIUM" else 1, "dtype": "bf16"}
    if kind == "request":
        return {"kind": kind, "model": "SD3_MEDIUM", "rows": rng.randint(16, 64), "cols": rng.randint(16, 64),
                "text": rng.randint(77, 333), "steps": rng.randint(4, 8), "dtype": rng.choice(["bf16", "fp16"])}
    if kind == "attention":
        model = rng.choice(sorted(LAYERS))
        heads = LAYERS[model][0]
        return {"kind": kind, "model": model, "heads": rng.choice([heads, heads // 2, heads // 4, heads // 8]),
                "tokens": log_int(256, 60000), "text": rng.randint(33, 512), "batch": 1,
                "joint": rng.choice(["none", "front", "rear"]), "dtype": rng.choice(["bf16", "bf16", "fp16"])}
    if kind == "ring":
        model = rng.choice(sorted(LAYERS))
        return {"kind": kind, "model": model, "heads": LAYERS[model][0] // rng.choice([1, 2]), "tokens": log_int(512, 12000),
                "text": rng.randint(77, 256), "ring": rng.choice([2, 4, 8]), "dtype": rng.choice(["bf16", "bf16", "fp16"])}
    if kind == "patch":
        patches = rng.choice([2, 4])
        return {"kind": kind, "model": rng.choice(["SD3_MEDIUM", "FLUX_DEV"]), "tokens": patches * rng.randint(96, 2304),
                "patches": patches, "text": rng.randint(77, 333), "batch": rng.randint(1, 2),
                "dtype": rng.choice(["bf16", "fp16"])}
    if kind == "guidance":
        return {"kind": kind, "tokens": log_int(96, 9216), "batch": 1, "dtype": rng.choice(["bf16", "fp16"])}
    return {"kind": "migration", "model": rng.choice(["FLUX_DEV", "SD3_MEDIUM"]), "blocks": rng.randint(1, 3),
            "degree": rng.choice([2, 4]), "dtype": rng.choice(["bf16", "fp16"])}


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(gen, *shape, dtype):
    return torch.randn(*shape, generator=gen, device=DEV, dtype=torch.float32).to(dtype)


def _model(case, seed):
    if not ps.model_parallel_is_initialized():
        ps.init_distributed_environment(0, 1, None)
        ps.get_parallel_groups().activate_plan([0])
    before = torch.get_default_dtype()
    torch.set_default_dtype(DTYPES[case["dtype"]])
    try:
        with torch.device(DEV):
            model = ShapedDiT(getattr(shapes, case["model"]))
    finally:
        torch.set_default_dtype(before)
    return model.init_weights(seed=seed, std=0.02)


def prepare(case, seed):
    torch.cuda.set_device(torch.device(DEV))
    kind, gen = case["kind"], _gen(seed)
    dtype = DTYPES[case["dtype"]]
    state = {"case": case}
    if kind in ("step", "request"):
        model = _model(case, seed)
        shape = model.shape
        n = case.get("frames", 1) * case["rows"] * case["cols"]
        batch = case.get("batch", 1)
        halves = batch if kind == "step" else 2  # a request brings the negative and the positive prompt
        state["latents"] = _randn(gen, batch, n, shape.token_in, dtype=dtype)
        state["text"] = _randn(gen, halves, case["text"], shape.text_dim, dtype=dtype)
        state["pooled"] = _randn(gen, halves, shape.pooled_dim, dtype=dtype) if shape.pooled_dim else None
        if kind == "step":
            state["model"] = model
            state["grid"] = (case["rows"], case["cols"]) if case["frames"] == 1 and shape.block_kind == "mmdit" and \
                shape.stale_kv else (case["frames"], case["rows"], case["cols"])
            state["t"] = torch.full((batch,), 0.75, device=DEV)
            state["g"] = torch.full((batch,), 3.5, device=DEV)
            if state["pooled"] is None:
                state["pooled"] = torch.zeros((batch, 1), dtype=dtype, device=DEV)  # not read by this model
        else:
            cfg = EngineConfig()
            cfg.runtime_config.dtype = dtype
            rt = initialize_runtime_state(ModelGeometry(shape.heads, shape.head_dim), cfg)
            rt.set_input_parameters(height=case["rows"] * 16, width=case["cols"] * 16, batch_size=1,
                                    num_inference_steps=case["steps"])
            state["pipeline"] = SD3ShapedPipeline(model, guidance_scale=5.0, grid=(case["rows"], case["cols"]))
        # a serving process has seen the resolution before: its step is captured by now
        for _ in range(2):
            run(state)
        return state
    if kind in ("attention", "ring", "patch"):
        D = LAYERS[case["model"]][1]
        H = case.get("heads", LAYERS[case["model"]][0])
        B, T, S = case.get("batch", 1), case["text"], case["tokens"]

        def rows(n):
            return _randn(gen, B, n, H, D, dtype=dtype)

        if kind == "attention":
            if not ps.model_parallel_is_initialized():
                ps.init_distributed_environment(0, 1, None)
                ps.get_parallel_groups().activate_plan([0])
            state["q"], state["k"], state["v"] = rows(S), rows(S), rows(S)
            if case["joint"] == "none":
                state["op"] = hetuDiTLongContextAttention()
            else:
                state["op"] = hetuDiTFluxLongContextAttention() if case["joint"] == "front" else hetuDiTJointLongContextAttention()
                state["tq"], state["tk"], state["tv"] = rows(T), rows(T), rows(T)
        elif kind == "ring":
            state["q"], state["tq"], state["tk"], state["tv"] = rows(S), rows(T), rows(T), rows(T)
            state["k"] = [rows(S) for _ in range(case["ring"])]
            state["v"] = [rows(S) for _ in range(case["ring"])]
        else:
            n = S // case["patches"]
            state["q"], state["k"], state["v"] = rows(n), rows(n), rows(n)
            state["tq"], state["tk"], state["tv"] = rows(T), rows(T), rows(T)
            state["stale"] = _randn(gen, B, S, 2 * H * D, dtype=dtype)
            state["start"] = n * (case["patches"] // 2)
        return state
    if kind == "guidance":
        B, n = case["batch"], case["tokens"]
        state["noise"] = _randn(gen, 2 * B, n, 64, dtype=dtype)
        state["sample"] = _randn(gen, B, n, 64, dtype=dtype)
        state["sigmas"] = torch.linspace(1.0, 0.0, 21, device=DEV)
        return state
    # migration: rank 0 of `degree` takes its slices of every linear layer out of the whole weights. Layers that
    # produce the hidden size's products are cut by rows (outputs), layers that consume them by columns (inputs).
    d = getattr(shapes, case["model"]).hidden
    layers = []
    for _ in range(case["blocks"]):
        for _ in range(2):  # image and text stream
            layers += [(d, d, "rows")] * 3 + [(d, d, "cols"), (4 * d, d, "rows"), (d, 4 * d, "cols")]
    state["full"], state["part"], pieces = [], [], []
    es = torch.empty((), dtype=dtype).element_size()
    for out_f, in_f, how in layers:
        w = _randn(gen, out_f, in_f, dtype=dtype)
        if how == "rows":
            part = torch.zeros((out_f // case["degree"], in_f), dtype=dtype, device=DEV)
            pieces.append((w.data_ptr(), part.data_ptr(), 1, 0, 0, 1, 0, 0, part.numel() * es))
        else:
            part = torch.zeros((out_f, in_f // case["degree"]), dtype=dtype, device=DEV)
            pieces.append((w.data_ptr(), part.data_ptr(), 1, 0, 0, out_f, in_f * es, part.shape[1] * es, part.shape[1] * es))
        state["full"].append(w)
        state["part"].append(part)
    state["pieces"] = pieces
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    with torch.no_grad():
        if kind == "step":
            return state["model"].forward_graphed(state["latents"], state["text"], state["pooled"], state["t"], state["g"],
                                                  grid=state["grid"])
        if kind == "request":
            return state["pipeline"].diffusion_stage(state["latents"], state["text"], state["pooled"], case["steps"])
        if kind == "attention":
            if case["joint"] == "none":
                return state["op"](None, state["q"], state["k"], state["v"])
            return state["op"](None, state["q"], state["k"], state["v"], joint_tensor_query=state["tq"],
                               joint_tensor_key=state["tk"], joint_tensor_value=state["tv"], joint_strategy=case["joint"])
        if kind == "ring":
            q = [state["tq"], state["q"]]
            B, _, H, D = state["q"].shape
            sq = state["q"].shape[1] + state["tq"].shape[1]
            acc = torch.empty((B, sq, H, D), dtype=torch.float32, device=DEV)
            acc_lse = torch.empty((B, H, sq), dtype=torch.float32, device=DEV)
            kernels.attn_fwd(q, [state["tk"], state["k"][0]], [state["tv"], state["v"][0]], mode=_C.ATTN_PARTIAL_FIRST,
                             acc_out=acc, acc_lse=acc_lse)
            return kernels.attn_fwd(q, state["k"][1:], state["v"][1:], mode=_C.ATTN_MERGE_FINAL, acc_out=acc,
                                    acc_lse=acc_lse, return_lse=True)
        if kind == "patch":
            stale, (B, n, H, D) = state["stale"], state["q"].shape
            kernels.kv_scatter(stale, state["k"].view(B, n, H * D), state["v"].view(B, n, H * D), state["start"])
            k, v = (t.view(B, -1, H, D) for t in stale.chunk(2, dim=-1))
            return kernels.attn_fwd([state["q"], state["tq"]], [k, state["tk"]], [v, state["tv"]]), stale
        if kind == "guidance":
            return kernels.cfg_euler_step(state["noise"], state["sample"], state["sigmas"], 7, 5.0)
        kernels.copy_pieces(state["pieces"], torch.device(DEV))
        return state["part"]


def _step_work(case, halves):
    """Every weight read once, inputs read and outputs written once; linear layers and attention of every block."""
    shape = getattr(shapes, case["model"])
    d, L = shape.hidden, case["text"]
    n = case.get("frames", 1) * case["rows"] * case["cols"]
    S = n + L
    flops = halves * shape.n_blocks * (24.0 * d * d * S + 4.0 * S * S * d)
    flops += halves * 2.0 * (2 * n * shape.token_in * d + L * shape.text_dim * d)
    if shape.block_kind == "cogvideox":
        mats, adaln = 12.0 * shape.n_blocks, 12.0 * shape.n_blocks * shape.temb_dim
    else:
        mats = 24.0 * shape.n_double + 12.0 * shape.n_single
        adaln = (12.0 * shape.n_double + 3.0 * shape.n_single) * d
    weights = mats * d * d + adaln * d + (2 * shape.token_in + shape.text_dim) * d
    flops += halves * 2.0 * adaln * d
    return 2.0 * (weights + halves * (2 * n * shape.token_in + L * shape.text_dim)), flops


def work(case):
    kind = case["kind"]
    if kind in ("step", "request"):
        steps = case.get("steps", 1)
        nbytes, flops = _step_work(case, case["batch"] if kind == "step" else 2)
        return {"bytes": steps * nbytes, "flops": steps * flops}
    if kind in ("attention", "ring", "patch"):
        D = LAYERS[case["model"]][1]
        H = case.get("heads", LAYERS[case["model"]][0])
        B, S = case.get("batch", 1), case["tokens"]
        T = 0 if case.get("joint") == "none" else case["text"]
        row = 2.0 * B * H * D
        if kind == "attention":
            sq, skv, extra = S + T, S + T, 0.0
        elif kind == "ring":
            sq, skv, extra = S + T, case["ring"] * S + T, 4.0 * B * H * (S + T)  # the log-sum-exp is returned
        else:
            n = S // case["patches"]
            sq, skv, extra = n + T, S + T, 2 * 2 * row * n  # fresh K and V read and stored into the stale buffer
        return {"bytes": row * (2 * sq + 2 * skv) + extra, "flops": 4.0 * B * H * D * sq * skv}
    if kind == "guidance":
        n = case["batch"] * case["tokens"] * 64
        return {"bytes": 4 * 2.0 * n, "flops": 9.0 * n}
    d = getattr(shapes, case["model"]).hidden
    return {"bytes": 2 * 2.0 * case["blocks"] * 2 * 12 * d * d / case["degree"], "flops": 0.0}


def tolerance(case):
    """Measured once: attention against 64-bit arithmetic (bf16 2.3e-3, largest 1.0e-2; fp16 2.9e-4, 1.4e-3), a step
    against the same weights with the linear layers' and attention's sums in another order (1.6e-2, largest 7.6e-2,
    after 57 to 60 blocks in bf16; the request in fp16 1.0e-3, 4.3e-3). About four times that, a step at most 3e-2."""
    kind, fp16 = case["kind"], case["dtype"] == "fp16"
    if kind in ("migration", "guidance"):
        return "exact"
    if kind in ("step", "request"):
        return {"rel": 4e-3, "max": 2e-2} if fp16 else {"rel": 3e-2, "max": 0.3}
    return {"rel": 1.2e-3, "max": 6e-3} if fp16 else {"rel": 1e-2, "max": 4e-2}
