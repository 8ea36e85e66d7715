"""The sampling work that a user of this library has it do, as cases to be measured.

Every case is one pass of a decode loop's sampling stage through the public entry points, over seeded synthetic
logits: the operator slot and the sampler.h surface (one row, the caller waits for its token), a session batcher's
step and verify calls, and prepared batch descriptors launched again as a serving loop does. Sizes and
distributions are those of the repository's configurations and benchmark (vocabularies of 128256, 151936 and
262144 columns, N(0, sigma^2) and heavy-tailed Gumbel rows) or generic ones; one vocabulary is odd, so that rows
leave the 16-byte grid.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from geistlib_b200 import api

#: Logits per launch that a drawn case may have: a quarter of the largest listed case, less where rows are summed.
MOST_VALUES = 1 << 27


# ---- cases -----------------------------------------------------------------------------------------------------

def _case(call, seqs, vocab, mode, **more):
    """call: slot, host_row, probs, batch, step or verify. mode: greedy, top_k, top_p, temperature, or mixed."""
    c = {"call": call, "seqs": seqs, "rows_per_seq": 1, "vocab": vocab, "mode": mode, "temperature": 0.8, "top_k": 40, "top_p": 0.95,
         "logits": "normal", "sigma": 2.5, "boosted": 8, "history": 0, "rep": 1.0, "freq": 0.0, "pres": 0.0, "softcap": 0.0,
         "masked": 0, "hint": True}
    c.update(more)
    return c


def listed():
    named = {
        # the engine's argmax operator on one device row: the smallest call, the caller waits for four bytes
        "slot_argmax_1x151936": _case("slot", 1, 151936, "greedy"),
        # the sampler.h surface on a host row, as a single-session engine on the CPU side calls it
        "host_row_top_k_1x128256": _case("host_row", 1, 128256, "top_k"),
        # one session's row with a penalty history: the token and the post-filter probability vector
        "probs_1x128256": _case("probs", 1, 128256, "top_k", history=64, rep=1.1),
        # a decode step of a few chat sessions: nucleus sampling with a repetition penalty, the host waits for the tokens
        "step_top_p_8x151936": _case("step", 8, 151936, "top_p", temperature=0.7, top_p=0.9, logits="gumbel", sigma=4.0, boosted=0, history=200, rep=1.1),
        # batched greedy decoding with frequency and presence penalties
        "greedy_penalties_64x151936": _case("batch", 64, 151936, "greedy", sigma=3.0, boosted=0, history=256, freq=0.2, pres=0.3),
        # a constrained decode step: sessions of a soft-capped model with a large vocabulary, half of them under a column mask
        "step_softcap_mask_48x262144": _case("step", 48, 262144, "top_k", temperature=1.0, top_k=64, softcap=30.0, masked=24),
        # a serving batch of sessions with different settings, no hint, on an odd vocabulary (rows off the 16-byte grid)
        "mixed_96x100003": _case("batch", 96, 100003, "mixed", history=48, rep=1.1, hint=False),
        # verify rows of speculative decoding: 6 proposals and the bonus row per sequence, plain temperature, prefix-accept
        "verify_32x7x128256": _case("verify", 32, 128256, "temperature", rows_per_seq=7, temperature=1.0),
        # the benchmark's headline batch: top-k with a repetition penalty over 64-id histories
        "top_k_penalties_256x128256": _case("batch", 256, 128256, "top_k", history=64, rep=1.1),
        # the same rows under nucleus sampling: many of them are flat, their nuclei run to tens of thousands of ids
        "top_p_flat_256x128256": _case("batch", 256, 128256, "top_p"),
        # nucleus sampling over heavy-tailed rows of a large vocabulary
        "top_p_256x262144": _case("batch", 256, 262144, "top_p", temperature=0.85, top_p=0.9, logits="gumbel", sigma=4.0, boosted=0),
        # box-scale batch: top-k with a repetition penalty over 1024-id histories
        "top_k_penalties_4096x128256": _case("batch", 4096, 128256, "top_k", temperature=0.7, top_k=50, boosted=0, history=1024, rep=1.15),
    }
    return [dict(c, name=n) for n, c in named.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: vocabularies from 4096 to 262144 (a third of them odd), 1 to 4096 sequences."""
    call = rng.choice(["batch", "batch", "batch", "batch", "step", "step", "verify", "slot", "host_row", "probs"])
    mode = rng.choice(["greedy", "top_k", "top_k", "top_p", "temperature", "mixed"])
    vocab = rng.choice([128256, 151936, 262144]) if rng.random() < 0.4 else _log_int(rng, 4096, 262144)
    if vocab % 2 == 0 and rng.random() < 0.33:
        vocab -= 1
    rows_per_seq = 1
    if call in ("slot", "host_row", "probs"):
        seqs = 1
        mode = {"slot": "greedy", "probs": "top_k"}.get(call, "top_k" if mode == "greedy" else mode)
        if mode == "mixed":
            mode = "temperature"
    elif call == "verify":
        rows_per_seq = rng.randint(2, 12)
        seqs = _log_int(rng, 1, 48)
    else:
        seqs = _log_int(rng, 1, 256 if call == "step" else 4096)
    most = MOST_VALUES if mode in ("greedy", "top_k") else MOST_VALUES // 8
    seqs = max(1, min(seqs, most // (vocab * rows_per_seq)))
    more = {"rows_per_seq": rows_per_seq, "temperature": round(rng.uniform(0.5, 1.2), 3), "top_k": _log_int(rng, 2, 256),
            "top_p": round(rng.uniform(0.8, 0.98), 3)}
    if rng.random() < 0.4:
        more.update(logits="gumbel", sigma=4.0, boosted=0)
    else:
        more.update(sigma=round(rng.uniform(2.0, 4.0), 2), boosted=rng.choice([0, 8, 8]))
    if call in ("batch", "step", "verify", "probs") and rng.random() < 0.6:
        more["history"] = _log_int(rng, 16, 1024)
        more[rng.choice(["rep", "rep", "freq"])] = round(rng.uniform(1.05, 1.2), 3)
        more["pres"] = rng.choice([0.0, 0.3])
    if call in ("step", "batch") and rng.random() < 0.2:
        more["softcap"] = 30.0
    if call == "step" and rng.random() < 0.2:
        more["masked"] = (seqs + 1) // 2
    if call == "batch":
        more["hint"] = mode != "mixed" and rng.random() < 0.7
    return _case(call, seqs, vocab, mode, **more)


# ---- inputs ----------------------------------------------------------------------------------------------------

_context = None


def _ctx():
    """The process's sampling context, as a program keeps one."""
    global _context
    if _context is None:
        _context = api.Context(torch.cuda.current_device())
    return _context


def _logits(c, rows, gen):
    """fp32 rows: N(0, sigma^2) with a few ids raised by 12 (what a confident model's row looks like), or Gumbel * sigma."""
    V = c["vocab"]
    if c["logits"] == "gumbel":
        x = torch.rand(rows, V, generator=gen, device="cuda").clamp_(1e-30, 1.0 - 2.0 ** -24)
        x.log_().neg_().log_().mul_(-c["sigma"])
    else:
        x = torch.randn(rows, V, generator=gen, device="cuda").mul_(c["sigma"])
    if c["boosted"]:
        idx = torch.randint(V, (rows, c["boosted"]), generator=gen, device="cuda")
        x.scatter_add_(1, idx, torch.full(idx.shape, 12.0, device="cuda"))
    return x


def _settings(c):
    """(T, top_k, top_p) of every sequence; a mixed batch cycles through the four modes."""
    greedy, top_k = (0.0, 0, 1.0), (c["temperature"], c["top_k"], 1.0)
    top_p, plain = (c["temperature"], 0, c["top_p"]), (c["temperature"], 0, 1.0)
    of = {"greedy": [greedy], "top_k": [top_k], "top_p": [top_p], "temperature": [plain], "mixed": [greedy, top_k, top_p, plain]}[c["mode"]]
    return [of[i % len(of)] for i in range(c["seqs"])]


def _states(n, gen):
    return torch.randint(1, 2 ** 62, (n,), generator=gen, device="cuda", dtype=torch.int64)


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rows, V = c["seqs"] * c["rows_per_seq"], c["vocab"]
    s = {"case": c}
    if c["call"] == "slot":
        s["row"] = _logits(c, 1, gen)[0].contiguous()
        _ctx()
        return s
    if c["call"] == "host_row":
        s["row"] = _logits(c, 1, gen)[0].cpu().numpy()
        s["rng"] = api.rng_seed(1 + seed)
        s["ws"] = api.SamplerWorkspace(V)
        return s
    x = _logits(c, rows, gen)
    hist = torch.randint(V, (c["seqs"], max(c["history"], 1)), generator=gen, device="cuda", dtype=torch.int32)
    if c["call"] in ("step", "verify"):
        if c["call"] == "verify":
            # proposals drawn from draft rows that differ from the target's by a little noise
            d = (x + torch.randn(x.shape, generator=gen, device="cuda") * 0.5) / c["temperature"]
            d -= torch.rand(d.shape, generator=gen, device="cuda").clamp_(1e-30, 1.0 - 2.0 ** -24).log_().neg_().log_()
            d = d.argmax(dim=1).view(c["seqs"], c["rows_per_seq"])
            fed = torch.randint(V, d.shape, generator=gen, device="cuda")
            fed[:, 1:] = d[:, :-1]
            s["fed"] = fed.to(torch.int32).cpu().numpy()
        b = api.Batcher(_ctx(), V, c["seqs"], max_history=c["history"] + 64)
        h = hist.cpu().numpy()
        mask = None
        if c["masked"]:
            mask = torch.randint(-2 ** 31, 2 ** 31, (c["masked"], (V + 31) // 32), generator=gen, device="cuda").to(torch.int32).cpu().numpy()
        s["sessions"] = []
        for i, (T, k, p) in enumerate(_settings(c)):
            sid = b.open(temperature=T, top_p=p, top_k=k, seed=seed + 1 + i, rep=c["rep"], freq=c["freq"], pres=c["pres"])
            if c["history"]:
                b.push_history(sid, h[i])
            if c["softcap"]:
                b.set_softcap(sid, c["softcap"])
            if i < c["masked"]:
                b.set_logit_mask(sid, mask[i])
            s["sessions"].append(sid)
        s["sessions"] = np.asarray(s["sessions"], np.int32)
        s["batcher"], s["x"] = b, x
        return s
    T, k, p = (torch.tensor(v, device="cuda") for v in zip(*_settings(c)))
    kw = {}
    if c["history"]:
        n = c["seqs"]
        kw = {"history": hist, "history_len": torch.full((n,), c["history"], dtype=torch.int32, device="cuda"),
              **{name: torch.full((n,), c[name], device="cuda") for name in ("rep", "freq", "pres")}}
    if c["softcap"]:
        kw["softcap"] = torch.full((c["seqs"],), c["softcap"], device="cuda")
    hint = api.FINISH_AUTO
    if c["hint"]:
        hint = {"greedy": api.FINISH_GREEDY, "top_k": api.FINISH_GREEDY_TOPK, "mixed": api.FINISH_AUTO}.get(c["mode"], api.FINISH_GENERAL)
    args = (x, T.float(), k.to(torch.int32), p.float(), _states(c["seqs"], gen))
    s["out"] = _ctx().sample_batch(*args, kept_cap=c["top_k"] if c["call"] == "probs" else 0, launch=False,
                                   finish_hint=api.FINISH_AUTO if c["call"] == "probs" else hint, **kw)
    s["inputs"] = (args, kw)  # the descriptor holds pointers into these
    return s


# ---- one pass --------------------------------------------------------------------------------------------------

def run(state):
    c = state["case"]
    if c["call"] == "slot":
        return _ctx().argmax_f32(state["row"])
    if c["call"] == "host_row":
        ws, row, rng = state["ws"], state["row"], state["rng"]
        if c["mode"] == "top_k":
            tok = ws.top_k(row, c["top_k"], c["temperature"], rng)
        elif c["mode"] == "top_p":
            tok = ws.top_p(row, c["top_p"], c["temperature"], rng)
        else:
            tok = api.sampler_temperature(row, c["temperature"], rng)
        return {"token": tok, "rng": np.array([rng.state], np.uint64).view(np.int64)}
    if c["call"] == "step":
        return {"tokens": state["batcher"].step(state["sessions"], state["x"])}
    if c["call"] == "verify":
        accepted, n_out, tokens = state["batcher"].verify(state["sessions"], state["fed"], state["x"])
        return {"accepted": accepted, "n_out": n_out, "tokens": tokens}
    out = state["out"]
    _ctx().relaunch(out, torch.cuda.current_stream().cuda_stream)
    if c["call"] == "probs":
        dense = _ctx().scatter_kept(out, c["vocab"])
        return {"tokens": out["tokens"], "rng": out["rng_state"], "kept_idx": out["kept_idx"], "kept_prob": out["kept_prob"], "dense": dense}
    return {"tokens": out["tokens"], "rng": out["rng_state"]}


# ---- what a pass cannot do without, and how far two correct ones can be apart ------------------------------------

def work(case):
    c = case
    rows = c["seqs"] * c["rows_per_seq"]
    values = rows * c["vocab"]
    per_seq = 16 + 12 + 4 * (c["history"] if c["call"] not in ("slot", "host_row") else 0)  # generator word in and out, settings, ids
    b = 4 * values + 4 * rows + per_seq * c["seqs"] + c["masked"] * ((c["vocab"] + 31) // 32) * 4
    if c["call"] == "probs":
        b += 4 * c["vocab"] + 8 * c["top_k"]
    # a comparison each; where the whole row is summed, subtract, scale, exponential and add as well
    return {"bytes": b, "flops": values * (1 if c["mode"] in ("greedy", "top_k") else 5)}


def tolerance(case):
    c = case
    if c["call"] == "probs":
        return {"rel": 1e-6, "max": 1e-5, "differ": 0.0}  # probabilities are correctly rounded quotients; ids are exact
    if c["mode"] in ("greedy", "top_k") and not c["softcap"]:
        return "exact"
    # A draw over a whole row turns on sums of 10^5 terms: another order moves them by about 1e-8, and a draw that
    # lies that close to a step takes the neighbouring id (measured against sequential sums on the CPU: 2 of 1536 rows;
    # two of 256 are let through).
    return {"rel": 0.0, "differ": 0.008}
