"""Helpers of the layer-stack tests: tokens, portions, row-wise errors against a plain implementation."""
import ctypes

import torch

TOL = {"fp32": 2e-4, "bf16": 4e-2}


def tokens(cfg, n, seed=5):
    return torch.randint(0, cfg["vocab"], (n,), generator=torch.Generator().manual_seed(seed)).tolist()


def error(got, want):
    """Per row: root mean square of the centred difference over that of the centred reference."""
    d = got.double().cpu() - want
    d, w = d - d.mean(-1, keepdim=True), want - want.mean(-1, keepdim=True)
    return d.pow(2).mean(-1).sqrt() / w.pow(2).mean().sqrt()


def feed(eng, toks, sizes):
    """Logits of every token, fed in portions of the given sizes (the last size repeats)."""
    eng.reset()
    out, at, i = [], 0, 0
    while at < len(toks):
        n = min(sizes[min(i, len(sizes) - 1)], len(toks) - at)
        out.append(eng.extend(toks[at:at + n], list(range(n))))
        at, i = at + n, i + 1
    return torch.cat(out)


SET_EVERY_TIME = {"StackGemmArgs": ("rows", "item_rows", "max_items"), "EpArgs": ("tokens", "max_items", "item_rows"),
                  "LatentAttnArgs": ("rows", "kv0", "kv_rows", "first", "last", "v_ld")}


def watch_kept_blocks(pf):
    """From now on every argument block that a prompt takes from the kept ones is compared with one built anew, but for what is set every
    time; returns the counts of blocks made and compared."""
    met, keep = {"made": 0, "checked": 0}, pf.kept

    def parts(a):
        if isinstance(a, dict):
            return [(k, None if t is None else (t.data_ptr(), t.shape, t.dtype)) for k, t in a.items()]
        out = []
        for s in a if isinstance(a, tuple) else (a,):
            if isinstance(s, ctypes.Structure):
                raw, free = bytes(s), SET_EVERY_TIME.get(type(s).__name__, ("rows",))
                out += [(f[0], raw[getattr(type(s), f[0]).offset:][:getattr(type(s), f[0]).size]) for f in s._fields_ if f[0] not in free]
        return out

    def kept(key, build):
        met["made"] += key not in pf._kept
        a, fresh = keep(key, build), build()
        met["checked"] += 1
        assert parts(a) == parts(fresh) and parts(a), key
        return a

    pf.kept = kept
    return met
