"""Lefatar configurations drawn at random from fixed seeds: other sizes, head counts, orders of layers, constants
and rotated parts than any other test has (rows of the latent cache that the tensor-core kernels take and rows
they refuse, matrix memories in both forms of their kernels, feed-forward widths that are no multiple of 8,
routers with and without groups).  Each runs a prompt whole, the same prompt in portions, and its last tokens one
by one, in both precisions, against the plain implementation."""
import functools

import numpy as np
import pytest

import lefatar_tiny as lt
import plain_lefatar as plain
from helpers import check_logits

pytestmark = pytest.mark.gpu

SEEDS = list(range(10))


def draw(seed):
    rng = np.random.default_rng(1000 + seed)
    pick = lambda xs: xs[int(rng.integers(len(xs)))]          # noqa: E731
    width = pick([40, 56, 64, 72, 96])
    layers = []
    for _ in range(int(rng.integers(2, 6))):
        if rng.random() < 0.5:
            mixer = {"heads": pick([1, 2, 3, 4]), "dim": pick([8, 16, 24, 32, 48, 64]),
                     "vdim": 4 * int(rng.integers(2, 19)), "gate_cap": float(pick([5.0, 8.0, 16.0, 30.0]))}
            kind = "mlstm"
        else:
            rot_dim = pick([4, 8, 12, 16])
            mixer = {"heads": pick([1, 2, 3, 5, 6]), "dim": pick([8, 16, 24, 32]), "rot_dim": rot_dim,
                     "vdim": 4 * int(rng.integers(2, 13)), "q_rank": pick([16, 24, 40, 64]),
                     "kv_rank": pick([8, 20, 36, 48, 52, 64]), "scale": float(rng.uniform(0.1, 0.3)),
                     "rot": {"base": float(pick([100.0, 10000.0, 500000.0])), "dims": 2 * int(rng.integers(1, rot_dim // 2 + 1))}}
            kind = "latent_attention"
        r = rng.random()
        if r < 0.2:
            mlp = None
        elif r < 0.55:
            mlp = {"kind": "dense", "ff": int(pick([24, 36, 50, 64, 100]))}
        else:
            per, count = pick([1, 2, 3]), pick([1, 2, 4])
            keep = int(rng.integers(1, count + 1))
            mlp = {"kind": "moe", "expert": {"ff": int(pick([8, 20, 33, 48]))},
                   "router": {"experts": per * count, "top": int(rng.integers(1, keep * per + 1)),
                              "scale": float(pick([1.0, 2.0, 2.5])), "groups": {"count": count, "keep": keep}}}
        layers.append({"type": kind, "mixer": mixer, "mlp": mlp})
    return {"architecture": "Lefatar", "vocab": pick([97, 130, 251]), "width": width,
            "norm": {"eps": float(pick([1e-6, 1e-5]))}, "layers": layers}


@functools.lru_cache(maxsize=None)
def model_of(seed):
    cfg = draw(seed)
    return cfg, lt.make_weights(cfg, 77 + seed)


@functools.lru_cache(maxsize=None)
def plain_of(seed, tokens, flips=frozenset()):
    """(logits, every token's distance from another choice of experts, the undecided (layer, head) pairs)."""
    cfg, w = model_of(seed)
    margins, first = [], []
    logits = plain.forward(cfg, w, list(tokens), margins=margins, first=first, flips=flips)
    margin = np.min(np.stack(margins), axis=0) if margins else np.full(len(tokens), np.inf)
    return logits, margin, [(i, a) for i, ratios in first for a, r in enumerate(ratios) if r <= UNDECIDED]


# The read-out of a sequence's first token in a matrix memory is v times the SIGN of k . q, whatever its size.  A bfloat16
# run knows k . q to about |k| |q| 2^-8 only: the rows that k and q are products of are rounded to 8 bits of mantissa, and
# each part before them adds an error of 0.002 to 0.004 of its output (2^-8 = 0.0039).  Below that either sign is right.
UNDECIDED = 2.0 ** -8


def plain_runs(seed, tokens):
    """The plain run first, then those that differ from it in the sign of undecided first read-outs."""
    todo, seen = [frozenset()], set()
    while todo:
        flips = todo.pop(0)
        if flips in seen:
            continue
        seen.add(flips)
        logits, margin, undecided = plain_of(seed, tokens, flips)
        assert len(undecided) <= 2, "a configuration that a bfloat16 run cannot be held to"
        todo += [flips | {pair} for pair in undecided]
        yield logits, margin


def compare(got, seed, tokens, dtype, what):
    """float32 runs: against the plain run.  bfloat16 runs: against the plain run with one choice of the signs that
    bfloat16 leaves undecided, the same choice for all positions (the one that the run is closest to)."""
    got = np.asarray(got)
    runs = list(plain_runs(seed, tuple(tokens)))
    if dtype == "bfloat16":
        # a router's choice closer than 0.08 logits may fall the other way in bfloat16 and changes the positions
        # after it too: the run is compared up to the first such position
        assert np.isfinite(got).all(), what
        close_calls = [np.nonzero(margin <= 0.08)[0] for _, margin in runs]
        uptos = [int(c[0]) if len(c) else len(got) for c in close_calls]
        best = min((i for i in range(len(runs)) if uptos[i] >= uptos[0]),      # (none that compares fewer positions)
                   key=lambda i: np.abs(got[:uptos[i]] - runs[i][0][:uptos[i]]).max(initial=0.0))
        if uptos[best]:
            check_logits(got[:uptos[best]], runs[best][0][:uptos[best]], dtype, what)
        return
    diff = np.abs(got.astype(np.float64) - runs[0][0])
    assert np.isfinite(got).all() and diff.max() <= 2e-4 and diff.mean() <= 1e-5, \
        f"{what}: max |diff| {diff.max():.3e}, mean {diff.mean():.3e}"


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("seed", SEEDS)
def test_random_configuration(seed, dtype, tmp_path):
    from alpacca_b200.engine.engine import Engine
    from alpacca_b200.engine.loading import load_model_dir
    from alpacca_b200.engine.step import StepEntry
    cfg, w = model_of(seed)
    d = lt.write_model_dir(tmp_path / "m", cfg, w)
    eng = Engine(load_model_dir(d, dtype, "cuda", max_positions=256), max_tokens=512, max_slots=3)
    toks = np.random.default_rng(seed).integers(0, cfg["vocab"], 70).tolist()

    def run(slot, part):
        out = eng.step([StepEntry(slot, part, list(range(len(part))))]).cpu().numpy()
        eng.wait()
        return out
    for cuts in ((70,), (33, 2, 35), (64, 1, 1, 1, 1, 1, 1)):
        s = eng.alloc_slot()
        got, at = [], 0
        for n in cuts:
            got.append(run(s, toks[at:at + n]))
            at += n
        eng.free_slot(s)
        compare(np.concatenate(got), seed, toks, dtype, f"random lefatar {seed} {cuts}")
    eng.cache.check()
