"""The work that users of this framework have it do, as measurable cases.

A case is one call sequence through the public entry points (the Python
binding of the C ABI in include/cubff_gb300.h), on inputs made from a seed:

  tape     one 128-byte pair tape evaluated: a single program tried against a
           partner (the CLI's --run, RunSingleProgram)
  soup     a checkpoint's bytes loaded into a device-resident soup, a number of
           epochs run, the soup read back
  batch    many soups advanced together, each loaded and read back (parameter
           sweeps, the server's rounds)
  kernel   pairings and pipelined epochs on caller-owned device buffers
  epoch    one epoch launch on caller-owned device buffers and pairings
  selfrep  the self-replication score of every program of a soup

Soups start either from uniform random bytes (epoch 0) or, as most of a long
run does, from an evolved state: `evolve` epochs after a random start, with
`planted` copies of a self-replicator among the programs where a random start
would need thousands of epochs to find one.
"""
import ctypes
import math

import numpy as np
import torch

from cubff_gb300 import abi, workloads

RATE = 1 << 18  # 2^-12 per byte, the reference's default mutation rate

# A bff self-replicator: heads at 64 and 0, then "[,>}]" copies the first
# program over the second.
REPLICATOR = bytes([64, 0]) + b"[,>}]"


def listed():
    return [
        # The smallest call: one program tried once.  Latency and launches.
        {"name": "one tape", "kind": "tape", "lang": "bff"},
        # A short job of the serving stream: few programs, many epochs.
        {"name": "small soup", "kind": "soup", "lang": "bff_noheads", "n": 1022, "epochs": 64,
         "evolve": 0, "planted": 0},
        # The benchmark's soup and epochs: random start, 20 epochs.
        {"name": "headline soup", "kind": "soup", "lang": "bff_noheads", "n": 1 << 17,
         "epochs": 20, "evolve": 0, "planted": 0},
        # After self-replicators have taken over: what most of a long run is.
        {"name": "replicators", "kind": "soup", "lang": "bff", "n": 1 << 17, "epochs": 16,
         "evolve": 192, "planted": 256},
        # The other language families, past their first epochs.
        {"name": "forth soup", "kind": "soup", "lang": "forth", "n": 1 << 17, "epochs": 16,
         "evolve": 256, "planted": 0},
        {"name": "subleq soup", "kind": "soup", "lang": "subleq", "n": 1 << 17, "epochs": 64,
         "evolve": 128, "planted": 0},
        {"name": "rsubleq4 odd soup", "kind": "soup", "lang": "rsubleq4", "n": 40962, "epochs": 64,
         "evolve": 64, "planted": 0},
        # 2-D pairing on the benchmark's grid.
        {"name": "grid soup", "kind": "soup", "lang": "bff_noheads", "n": 512 * 256, "epochs": 32,
         "evolve": 0, "planted": 0, "width": 512, "radius": 2},
        # Many soups of the benchmark mix's languages and rates, at the sizes
        # of served jobs.
        {"name": "batch of 32", "kind": "batch", "soups": 32, "lo": 10.0, "hi": 15.0,
         "epochs": 64},
        # A program of its own driving the engine's kernels on torch buffers.
        {"name": "device epochs", "kind": "kernel", "lang": "bff", "n": 1 << 15, "epochs": 64},
        {"name": "one epoch", "kind": "epoch", "lang": "bff_noheads", "n": 1 << 17},
        # Scores at a callback, on a soup in which replicators are about.
        {"name": "selfrep scores", "kind": "selfrep", "lang": "bff", "n": 1 << 14, "evolve": 128,
         "planted": 64},
    ]


def _even(rng, lo, hi):
    """An even number of programs, log-uniform in [lo, hi]."""
    return 2 * round(2.0 ** rng.uniform(math.log2(lo), math.log2(hi)) / 2)


def draw(rng):
    kind = rng.choice(["tape", "soup", "soup", "soup", "batch", "kernel", "epoch", "selfrep"])
    bffs = ["bff", "bff_noheads", "bff_noheads_4bit", "bff_perm", "bff8", "bff_selfmove"]
    forths = ["forth", "forthcopy", "forthtrivial", "forthtrivial_reset"]
    others = ["subleq", "rsubleq4"]
    if kind == "tape":
        return {"kind": kind, "lang": rng.choice(bffs + forths + others), "fill": rng.random()}
    if kind == "batch":
        lo = rng.uniform(10.0, 13.0)
        return {"kind": kind, "soups": rng.randint(3, 32), "lo": lo, "hi": rng.uniform(lo, 15.0),
                "epochs": rng.randint(8, 64)}
    if kind == "kernel":
        return {"kind": kind, "lang": rng.choice(bffs + forths + others),
                "n": _even(rng, 512, 1 << 16), "epochs": rng.randint(4, 64)}
    if kind == "epoch":
        return {"kind": kind, "lang": rng.choice(bffs + forths + others),
                "n": _even(rng, 256, 1 << 17)}
    if kind == "selfrep":
        return {"kind": kind, "lang": "bff", "n": _even(rng, 256, 1 << 14),
                "evolve": rng.randint(0, 96), "planted": rng.choice([0, 64])}
    family = rng.choice(["random", "evolved", "grid"])
    if family == "grid":
        width, height = rng.randint(16, 512), rng.randint(8, 128) * 2
        return {"kind": kind, "lang": rng.choice(["bff", "bff_noheads"]), "n": width * height,
                "epochs": rng.randint(4, 32), "evolve": 0, "planted": 0, "width": width,
                "radius": rng.randint(1, 3)}
    if family == "random":
        return {"kind": kind, "lang": rng.choice(bffs + forths + others),
                "n": _even(rng, 256, 1 << 17), "epochs": rng.randint(4, 64), "evolve": 0,
                "planted": 0}
    lang = rng.choice(["bff"] + forths + others)
    return {"kind": kind, "lang": lang, "n": _even(rng, 2048, 1 << 16),
            "epochs": rng.randint(4, 16), "evolve": rng.randint(64, 192),
            "planted": 128 if lang == "bff" else 0}


_engine = None


def _the_engine():
    global _engine
    if _engine is None:
        _engine = abi.Engine(0)
    return _engine


def _start(soup, n, planted, evolve, seed):
    """The bytes of a soup `evolve` epochs after its start, with `planted`
    self-replicators among the random programs of the start."""
    if planted:
        data = soup.read().reshape(n, 64)
        rng = np.random.default_rng(seed)
        where = rng.choice(n, size=min(planted, n), replace=False)
        data[where, :len(REPLICATOR)] = np.frombuffer(REPLICATOR, dtype=np.uint8)
        soup.write(data.tobytes())
    if evolve:
        soup.run(evolve)
    return soup.read().tobytes()


def _soup(case, seed):
    n, grid = case["n"], case.get("width")
    soup = abi.Soup(_the_engine(), case["lang"], n, seed, RATE,
                    abi.PAIR_PATTERN if grid else abi.PAIR_SHUFFLE)
    if grid:
        soup.set_pattern(*workloads.grid_pattern(grid, n // grid, case["radius"]))
    return soup, _start(soup, n, case.get("planted", 0), case.get("evolve", 0), seed)


def _batch_sizes(case):
    """Even program counts, log-uniform in [2^lo, 2^hi], the case's own."""
    rng = np.random.default_rng(case["soups"])
    return [2 * round(2.0 ** rng.uniform(case["lo"], case["hi"]) / 2)
            for _ in range(case["soups"])]


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "tape":
        rng = np.random.default_rng(seed)
        tape = rng.integers(0, 256, 128, dtype=np.uint8)
        if case.get("fill", 0.0) > 0.5:  # mostly commands of the Forth and perm tables
            tape[:] = rng.integers(0, 14, 128, dtype=np.uint8)
        else:
            tape[:len(REPLICATOR)] = np.frombuffer(REPLICATOR, dtype=np.uint8)
        state |= {"lang": abi.language_id(case["lang"]), "tape": tape}
    elif kind in ("soup", "selfrep"):
        state["soup"], state["bytes"] = _soup(case, seed)
    elif kind == "batch":
        soups, data = [], []
        for s, n in enumerate(_batch_sizes(case)):
            soup = abi.Soup(_the_engine(), workloads.MIX_LANGS[s % len(workloads.MIX_LANGS)], n,
                            seed + s, workloads.MIX_RATES[s % len(workloads.MIX_RATES)])
            soups.append(soup)
            data.append(soup.read().tobytes())
        state |= {"soups": soups, "bytes": data}
    else:
        n, epochs = case["n"], case.get("epochs", 1)
        lib, dev = abi.lib(), torch.device("cuda")
        stream = torch.cuda.current_stream().cuda_stream
        first = torch.empty(n * 64, dtype=torch.uint8, device=dev)
        abi.check(lib.cubff_init_programs(workloads.seed_of(seed, 0), n, first.data_ptr(), 0, n,
                                          stream))
        state |= {"first": first, "programs": torch.empty_like(first), "seed": seed,
                  "lang": abi.language_id(case["lang"]),
                  "pairs": torch.empty(epochs * n, dtype=torch.int32, device=dev),
                  "counts": torch.zeros(2 * epochs, dtype=torch.int64, device=dev),
                  "scratch": torch.empty(lib.cubff_shuffle_scratch_bytes(n, epochs),
                                         dtype=torch.uint8, device=dev)}
        if kind == "kernel":
            state["work"] = torch.empty(lib.cubff_run_epochs_workspace_bytes(n, epochs),
                                        dtype=torch.uint8, device=dev)
        else:  # an epoch on pairings of the caller's own
            abi.check(lib.cubff_shuffle_indices(seed, 0, 1, n, state["pairs"].data_ptr(),
                                                state["scratch"].data_ptr(),
                                                state["scratch"].numel(), stream))
    return state


def run(state):
    case = state["case"]
    kind, epochs = case["kind"], case.get("epochs", 1)
    if kind == "tape":
        tape = state["tape"].copy()
        ops, raw = ctypes.c_uint64(0), ctypes.c_uint64(0)
        abi.check(abi.lib().cubff_eval_pair(state["lang"], tape.ctypes.data, ctypes.byref(ops),
                                            ctypes.byref(raw)))
        return {"tape": tape, "ops": ops.value, "raw": raw.value}
    if kind == "soup":
        soup = state["soup"]
        soup.write(state["bytes"])
        soup.set_epoch(case["evolve"])
        ops, raw = soup.run(epochs)
        return {"soup": soup.read(), "ops": ops.view(np.int64), "raw": raw.view(np.int64)}
    if kind == "batch":
        for soup, data in zip(state["soups"], state["bytes"]):
            soup.write(data)
            soup.set_epoch(0)
        ops = abi.batch_run(_the_engine(), state["soups"], epochs)
        return {"soups": np.concatenate([s.read() for s in state["soups"]]),
                "ops": ops.view(np.int64)}
    if kind == "selfrep":
        return {"scores": state["soup"].selfrep(case["evolve"]).view(np.int64)}
    lib, n, seed = abi.lib(), case["n"], state["seed"]
    stream = torch.cuda.current_stream().cuda_stream
    programs, pairs, counts = state["programs"], state["pairs"], state["counts"]
    programs.copy_(state["first"])
    counts.zero_()
    if kind == "epoch":
        abi.check(lib.cubff_mutate_and_run(state["lang"], programs.data_ptr(), pairs.data_ptr(),
                                           workloads.seed_of(seed, 0), RATE, counts.data_ptr(),
                                           counts.data_ptr() + 8, n, n // 2, stream))
    else:
        scratch, work = state["scratch"], state["work"]
        abi.check(lib.cubff_shuffle_indices(seed, 0, epochs, n, pairs.data_ptr(),
                                            scratch.data_ptr(), scratch.numel(), stream))
        abi.check(lib.cubff_run_epochs(state["lang"], programs.data_ptr(), pairs.data_ptr(), None,
                                       seed, 0, epochs, RATE, n, counts.data_ptr(),
                                       work.data_ptr(), work.numel(), stream))
    return {"programs": programs, "counts": counts}


def work(case):
    """Bytes: the programs read and written once.  Operations: the SplitMix64
    draws that every pair needs (128 of 21 integer operations each).  How many
    interpreter steps follow depends on the programs; they are not counted."""
    kind = case["kind"]
    if kind == "tape":
        return {"bytes": 2 * 128, "flops": 0}
    if kind == "batch":
        n = sum(_batch_sizes(case))
    else:
        n = case["n"]
    if kind == "selfrep":  # 13 x 5 evaluations, each against a 64-byte random partner
        return {"bytes": n * (64 + 8), "flops": n * 13 * 64 * 42}
    return {"bytes": 2 * 64 * n, "flops": case.get("epochs", 1) * n / 2 * 128 * 21}
