"""Performance cases: what programs built on pentago_b200 have it do.

A case is a dict of plain values with a "kind":

  lines    end-engine block lines: one line through ``end.compute_lines`` (the
           reference's schedule_compute_line, one call per line) or a batch
           of the four lines through many blocks as a prepared ``end.Plan``
  sweep    one slice of a backward sweep: every line of every section of a
           slice, then the sections' win counts
  mid      a batch of midsolve boards with the caller's scratch
  rans_enc, rans_dec    solved blocks to format-2 streams, and back
  lm_enc, lm_dec        solved blocks to learned-model streams, and back
  train    one training step of the learned model
  store    blocks of a solved slice coded for HBM, packed, and decoded again
           (what a compressed sweep does with every section)
  shard    a slice's entries scattered into training shards

``listed`` gives the fixed cases, ``draw`` others of the same ranges,
``prepare`` what a program holds before the call, ``run`` one pass, ``work``
the bytes and operations of a pass that any implementation has to spend, and
``exact`` the training step in 64 bits (every other output is whole numbers).
"""
import functools
import math

import numpy as np
import torch

from pentago_b200 import capi, end, learned, mid, rans, shard, slice_store, supertensor, sweep

# The 30-stone section of the line benchmark (shape 160 x 160 x 318 x 318), the
# 30-stone root of the learned coder's slice, and a 33-stone section whose
# solved slice stands for the data the coders meet.
LINE_SECTION = "4,4,4,4,4,3,3,4"
TRAIN_SECTION = "4,4,4,5,4,3,3,3"
SOLVED_ROOTS = ("4,4,5,4,4,5,4,3", "4,5,4,4,5,4,4,3", "4,4,4,5,5,4,4,3", "4,3,5,4,4,4,4,5")
# (root, slice) of the drawn sweeps: slices of 2.7 to 11.8 GB in 1 to 10 sections
SWEEPS = tuple((r, s) for r in SOLVED_ROOTS for s in (33, 34)) + (
    ("5,4,4,5,4,4,3,3", 32), ("5,4,4,5,4,4,3,3", 33), ("5,4,4,5,4,4,3,3", 34), ("5,4,5,4,3,3,3,4", 33),
    ("5,4,5,4,3,3,3,4", 34), ("5,4,4,4,3,4,4,4", 34), ("4,4,4,5,4,3,3,3", 34))


def listed():
    return [
        # One line per call, as the message-passing driver of the reference makes
        # them when a line's inputs have arrived: planning and launch count.
        {"name": "line_one", "kind": "lines", "section": LINE_SECTION, "blocks": 1, "dims": 1, "plan": False,
         "accumulate": False},
        # The benchmark's step: the four full lines through each of 16 blocks.
        {"name": "lines_batch", "kind": "lines", "section": LINE_SECTION, "blocks": 16, "dims": 4, "plan": True,
         "accumulate": False},
        # A slice of an in-core sweep below the 33-stone root, with its counts.
        {"name": "sweep_slice", "kind": "sweep", "root": SOLVED_ROOTS[0], "slice": 33},
        # The web backend's positions: a batch of 26-stone boards, and one board
        # with the fewest stones midsolve takes.
        {"name": "mid_64", "kind": "mid", "boards": 64, "stones": 26, "spread": 0},
        {"name": "mid_18", "kind": "mid", "boards": 1, "stones": 18, "spread": 0},
        # The reference's coder on blocks of a solved slice, both directions.
        {"name": "rans_encode", "kind": "rans_enc", "streams": 1024, "symbols": 1 << 20},
        {"name": "rans_decode", "kind": "rans_dec", "streams": 1024, "symbols": 1 << 20},
        # The learned coder on the same blocks, in one call of the size the
        # slice coder makes, and its training step at the default batch on 1%
        # of the 30-stone slice's blocks.
        {"name": "learned_encode", "kind": "lm_enc", "blocks": 2048},
        {"name": "learned_decode", "kind": "lm_dec", "blocks": 2048},
        {"name": "train_step", "kind": "train", "blocks": 2120, "batch": 32768},
        # Part of a section of a compressed sweep, coded and decoded.
        {"name": "store_section", "kind": "store", "blocks": 6000},
        # A whole slice into 1,024 training shards.
        {"name": "shard_slice", "kind": "shard", "slice": 9, "shards": 1024, "lo": 0, "hi": 1024},
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _random_section(rng, stones):
    """Counts of a section of `stones` stones (black has the extra one), at most nine to a quadrant."""
    while True:
        cells = [1] * ((stones + 1) // 2) + [2] * (stones // 2) + [0] * (36 - stones)
        rng.shuffle(cells)
        c = [[cells[9 * q:9 * q + 9].count(k) for k in (1, 2)] for q in range(4)]
        if any(sum(x) < 9 for x in c):
            return ",".join(str(v) for x in c for v in x)


def draw(rng):
    kind = rng.choice(["lines", "lines", "sweep", "mid", "mid", "rans_enc", "rans_dec", "lm_enc", "lm_dec", "train",
                       "store", "shard"])
    if kind == "lines":
        # (a line of a 35-stone section has no input: what it meets in the output makes its data)
        stones = rng.randint(20, 35)
        return {"kind": kind, "section": _random_section(rng, stones), "blocks": _log_int(rng, 1, 16),
                "dims": rng.randint(1, 4), "plan": rng.random() < 0.5,
                "accumulate": stones == 35 or rng.random() < 0.3}
    if kind == "sweep":
        root, slice_ = rng.choice(SWEEPS)
        return {"kind": kind, "root": root, "slice": slice_}
    if kind == "mid":
        stones = rng.randint(18, 33)
        most = 256 if stones >= 26 else 24 if stones >= 22 else 4
        return {"kind": kind, "boards": _log_int(rng, 1, most), "stones": stones,
                "spread": rng.randint(0, min(4, 34 - stones))}
    if kind in ("rans_enc", "rans_dec"):
        symbols = _log_int(rng, 1 << 8, 1 << 23)
        return {"kind": kind, "streams": _log_int(rng, 1, min(4096, (1 << 30) // symbols)), "symbols": symbols}
    if kind in ("lm_enc", "lm_dec"):
        return {"kind": kind, "blocks": _log_int(rng, 1, 2000)}
    if kind == "train":
        return {"kind": kind, "blocks": _log_int(rng, 8, 2120), "batch": _log_int(rng, 1000, 32768)}
    if kind == "store":
        return {"kind": kind, "blocks": _log_int(rng, 1, 6000)}
    shards = 1 << rng.randint(0, 16)
    lo = rng.choice((0, rng.randrange(shards)))
    return {"kind": kind, "slice": rng.randint(3, 9), "shards": shards, "lo": lo,
            "hi": rng.choice((shards, rng.randint(lo + 1, shards)))}


def _counts(text):
    v = [int(x) for x in text.split(",")]
    return [v[0:2], v[2:4], v[4:6], v[6:8]]


def _sig(text):
    return end.section_sig(_counts(text))


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _case_rng(case):
    """What a case's sizes are drawn from: the same for every seed."""
    return np.random.default_rng(sum(ord(c) * 7**(k % 9) for k, c in enumerate(str(sorted(case.items())))))


def _random_nodes(n, g):
    """n nodes [win, not lost], about 3% of the bits lost and 6% tied: a parent is won where one of its moves (eight
    rotations of each of one to nine placements) reaches a lost child, so denser losses would leave nothing to decide."""
    r = lambda: torch.randint(-2**63, 2**63 - 1, (n, 4), dtype=torch.int64, device="cuda", generator=g)
    x = r() & r() & r()
    lost = x & r() & r()
    return torch.cat([~(lost | x & r()), ~lost], 1)


def _open_dims(section):
    return [d for d, c in enumerate(_counts(section)) if sum(c) < 9]


# ---------------------------------------------------------------------------
# What a program holds before the call


def _prepare_lines(case, seed):
    rng, g = _case_rng(case), _generator(seed)
    sig = _sig(case["section"])
    blocks = [(s + 7) // 8 for s in end.section_shape(sig)]
    dims = _open_dims(case["section"])
    lines = []
    for _ in range(case["blocks"]):
        b = [int(rng.integers(0, n)) for n in blocks]
        first = int(rng.integers(0, len(dims)))
        for k in range(min(case["dims"], len(dims))):
            d = dims[(first + k) % len(dims)]
            line = end.Line(sig, d, [b[q] for q in range(4) if q != d],
                            flags=capi.PG_LINE_OR if case["accumulate"] else capi.PG_LINE_STORE)
            info = end.line_info(line)
            line.input = _random_nodes(info.input_nodes, g) if info.input_nodes else None
            line.output = (_random_nodes(info.output_nodes, g) if case["accumulate"] else
                           torch.zeros((info.output_nodes, 8), dtype=torch.int64, device="cuda"))
            lines.append(line)
    return {"lines": lines, "plan": end.Plan(lines) if case["plan"] else None}


def _prepare_sweep(case, seed):
    root = _sig(case["root"])
    sigs = sweep.descendent_sections(root, case["slice"])
    child_sigs = sweep.descendent_sections(root, case["slice"] + 1)
    child = _random_nodes(int(sweep.slice_layout(child_sigs)[-1]), _generator(seed))
    parent = torch.zeros((int(sweep.slice_layout(sigs)[-1]), 8), dtype=torch.int64, device="cuda")
    counts = torch.zeros((len(sigs), 3), dtype=torch.int64, device="cuda")
    return {"sigs": sigs, "child_sigs": child_sigs, "child": child, "parent": parent, "counts": counts}


def _prepare_mid(case, seed):
    rng = np.random.default_rng(seed)
    stones = case["stones"] + _case_rng(case).integers(0, case["spread"] + 1, case["boards"])
    raws = np.concatenate([mid.random_boards(int(rng.integers(1 << 40)), 1, int(n)) for n in stones])
    # some queries come from the middle of a turn: a stone placed, the rotation to come
    raws |= rng.integers(0, 2, len(raws)).astype(np.uint64) << np.uint64(63)
    scratch = torch.empty(mid.scratch_bytes(raws), dtype=torch.uint8, device="cuda")
    out = torch.zeros((len(raws), mid.RECORD_BYTES), dtype=torch.uint8, device="cuda")
    return {"raws": raws, "scratch": scratch, "out": out}


def _solved(case, seed, blocks):
    """Blocks of a solved 33-stone slice: their references, nodes (back to back) and node counts.  The case alone
    says how large each block is, the seed which block of that size it is."""
    rng = np.random.default_rng(seed)
    root = _sig(SOLVED_ROOTS[seed % len(SOLVED_ROOTS)])
    _, nodes, sigs = sweep.sweep(root, keep_last=True)
    refs, first, count = learned.slice_blocks(sigs, sweep.slice_layout(sigs))
    want = _case_rng(case).permutation(np.sort(count))[:blocks]
    pick = np.zeros(blocks, np.int64)
    for n in np.unique(want):
        pick[want == n] = rng.permutation(np.nonzero(count == n)[0])[:(want == n).sum()]
    start = np.zeros(blocks + 1, np.int64)
    start[1:] = np.cumsum(count[pick])
    at = torch.arange(int(start[-1]), device="cuda")
    at += torch.repeat_interleave(torch.from_numpy(first[pick] - start[:-1]).cuda(),
                                  torch.from_numpy(count[pick]).cuda())
    return learned.subset(refs, pick), nodes[at], count[pick]


def _symbol_streams(case, seed):
    """Nodes of solved blocks and the bounds of the streams their symbols are cut into (odd lengths)."""
    rng = _case_rng(case)
    lens = rng.integers(case["symbols"] - case["symbols"] // 8, case["symbols"] + 1, case["streams"])
    offsets = np.zeros(len(lens) + 1, np.int64)
    offsets[1:] = np.cumsum(lens)
    need = (int(offsets[-1]) + 255) // 256
    blocks = min(20000, max(1, 2 * ((need + 4095) // 4096) + 20))
    _, nodes, _ = _solved(case, seed, blocks)
    return nodes[torch.arange(need, device="cuda") % len(nodes)], offsets


def _model(seed):
    """A model that predicts a symbol from its neighbours and the previous node's, with noise in every weight."""
    rng = np.random.default_rng(seed)
    p = np.zeros(learned.N_PARAMS, np.float32)
    w1 = rng.standard_normal((124, 64)).astype(np.float32) * 0.05
    w2 = rng.standard_normal((64, 64)).astype(np.float32) * 0.05
    w3 = rng.standard_normal((64, 3)).astype(np.float32) * 0.05
    for v in range(3):
        w1[88 + v:120:4, v] += 0.5
        w1[120 + v, v] += 1.5
        w2[v, v] += 1
        w3[v, v] += 1
    p[learned.P_W1:learned.P_B1] = w1.reshape(-1)
    p[learned.P_W2:learned.P_B2] = w2.reshape(-1)
    p[learned.P_W3:learned.P_B3] = w3.reshape(-1)
    return learned.export(torch.from_numpy(p))


def _prepare_learned(case, seed, decode):
    refs, nodes, count = _solved(case, seed, case["blocks"])
    offsets = np.zeros(len(count) + 1, np.int64)
    offsets[1:] = np.cumsum(256 * count)
    s = {"refs": refs, "count": count, "model": _model(seed)}
    data = _store_for(len(nodes), len(count))
    if not decode:
        return dict(s, nodes=nodes, offsets=torch.from_numpy(offsets).cuda(), data=data)
    s["data"], s["offsets"], s["sizes"] = _pack(data, *learned.encode(
        s["model"], refs, rans.node_symbols(nodes, 1), torch.from_numpy(offsets).cuda(), count))
    return s


def _train_inputs(case, seed):
    """Training blocks of the 30-stone section, their symbols (a value per node with noise), and the state of the
    optimizer some way into a training run."""
    rng, g = np.random.default_rng(seed), _generator(seed)
    shape = np.array([len(_rmin_quadrants()[tuple(c)]) for c in _counts(TRAIN_SECTION)])
    grid = (shape + 7) // 8
    pick = np.sort(rng.choice(int(np.prod(grid)), case["blocks"], replace=False))
    block = np.stack(np.unravel_index(pick, grid), 1)
    count = np.minimum(8, shape - 8 * block).prod(1)
    n = int(count.sum())
    value = torch.randint(0, 3, (n, 1), dtype=torch.uint8, device="cuda", generator=g)
    noise = torch.randint(0, 12, (n, 256), dtype=torch.uint8, device="cuda", generator=g)
    symbols = torch.where(noise < 3, noise, value).reshape(-1)
    params = rng.standard_normal(learned.N_PARAMS) * 0.15
    params[learned.P_W2:learned.P_B2] *= math.sqrt(2 / 64) / 0.15
    return {"block": block, "count": count, "shape": shape, "symbols": symbols, "seed": seed,
            "params": params.astype(np.float32),
            "m": (rng.standard_normal(learned.N_PARAMS) * 1e-3).astype(np.float32),
            "v": (rng.uniform(0.5, 2, learned.N_PARAMS) * 1e-6).astype(np.float32), "step": 100}


def _prepare_train(case, seed):
    t = _train_inputs(case, seed)
    refs = (capi.pg_block_ref_t * len(t["block"]))()
    for k, b in enumerate(t["block"]):
        refs[k].section = _sig(TRAIN_SECTION)
        for q in range(4):
            refs[k].block[q] = int(b[q])
    offsets = np.zeros(len(t["count"]) + 1, np.int64)
    offsets[1:] = np.cumsum(256 * t["count"])
    trainer = learned.Trainer(refs, t["symbols"], torch.from_numpy(offsets).cuda(), t["count"], seed=t["seed"],
                              params=torch.from_numpy(t["params"]).cuda())
    at = {k: torch.from_numpy(t[k]).cuda() for k in ("params", "m", "v")}
    return {"trainer": trainer, "at": at, "step": t["step"], "batch": case["batch"]}


def _prepare_store(case, seed):
    _, nodes, count = _solved(case, seed, case["blocks"])
    first = np.zeros(len(count) + 1, np.int64)
    first[1:] = np.cumsum(count)
    caps = (slice_store.store_bound(count) + 15) // 16 * 16
    offsets = np.zeros(len(count) + 1, np.int64)
    offsets[1:] = np.cumsum(caps)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return {"nodes": nodes, "first": dev(first[:-1]), "count": dev(count.astype(np.int32)), "bound": int(offsets[-1]),
            "offsets": dev(offsets[:-1]), "data": _store_for(len(nodes), len(count))}


def _prepare_shard(case, seed):
    m, blocks, nodes = shard.synthetic_slice(case["slice"], seed)
    loc = shard.shard_locator_t(case["shards"])
    n = sum(loc.shard_size(m.total(), s) for s in range(case["lo"], case["hi"]))
    return {"blocks": blocks, "nodes": nodes, "symbols": torch.zeros(max(n, 1), dtype=torch.uint8, device="cuda")}


def prepare(case, seed):
    capi.check(capi.lib().pg_init())
    kind = case["kind"]
    if kind == "rans_enc":
        nodes, offsets = _symbol_streams(case, seed)
        s = {"nodes": nodes, "offsets": offsets, "data": _store_for(len(nodes), case["streams"])}
    elif kind == "rans_dec":
        nodes, offsets = _symbol_streams(case, seed)
        data, at, sizes = _pack(_store_for(len(nodes), case["streams"]),
                                *rans.encode_device(rans.node_symbols(nodes, 1), offsets))
        s = {"data": data, "at": at.cpu().numpy(), "sizes": sizes.cpu().numpy(), "offsets": offsets}
    elif kind in ("lm_enc", "lm_dec"):
        s = _prepare_learned(case, seed, kind == "lm_dec")
    else:
        s = {"lines": _prepare_lines, "sweep": _prepare_sweep, "mid": _prepare_mid, "train": _prepare_train,
             "store": _prepare_store, "shard": _prepare_shard}[kind](case, seed)
    return dict(s, case=case)


# ---------------------------------------------------------------------------
# One pass


def _store_for(nodes, streams):
    """Room for the packed streams of a batch: any of the coders' streams fits the raw nodes and some headers."""
    return torch.zeros(64 * nodes + 4096 * streams, dtype=torch.uint8, device="cuda")


def _pack(data, out, offsets, sizes):
    """The coded streams of a batch into `data`, each starting on a 16-byte boundary: (data, starts, sizes)."""
    dev = out.device
    host = sizes if isinstance(sizes, np.ndarray) else sizes.cpu().numpy()
    starts = np.zeros(len(host) + 1, np.int64)
    starts[1:] = np.cumsum((host + 15) // 16 * 16)
    if starts[-1] > data.numel():
        raise ValueError("the coded streams do not fit")
    d = [x if isinstance(x, torch.Tensor) else torch.from_numpy(np.ascontiguousarray(x)).to(dev)
         for x in (offsets, sizes, starts)]
    capi.check(capi.lib().pg_pack_streams(out.data_ptr(), d[0].data_ptr(), d[1].data_ptr(), len(host), data.data_ptr(),
                                          d[2].data_ptr(), capi.stream_handle()))
    return data, d[2], d[1]


def _run_lines(s):
    if s["plan"] is not None:
        s["plan"].run()
    else:
        end.compute_lines(s["lines"])
    return [line.output for line in s["lines"]]


def _run_sweep(s):
    L, st = capi.lib(), capi.stream_handle()
    capi.check(L.pg_end_sweep_slice(capi.ptr(s["sigs"]), len(s["sigs"]), s["parent"].data_ptr(),
                                    capi.ptr(s["child_sigs"]), len(s["child_sigs"]), s["child"].data_ptr(), st))
    capi.check(L.pg_section_counts(capi.ptr(s["sigs"]), len(s["sigs"]), s["parent"].data_ptr(),
                                   s["counts"].data_ptr(), st))
    return s["parent"], s["counts"]


def _run_train(s):
    t = s["trainer"]
    for k, v in s["at"].items():
        getattr(t, k).copy_(v)
    t.step = s["step"]
    t.run(1, s["batch"])
    return {"params": t.params, "m": t.m, "v": t.v, "grad": t.grad, "loss": t.loss}


def _run_store(s):
    L, st = capi.lib(), capi.stream_handle()
    k, nodes = len(s["count"]), s["nodes"]
    table = torch.empty(3 * 1024, dtype=torch.int16, device="cuda")
    capi.check(L.pg_store_table(nodes.data_ptr(), s["first"].data_ptr(), s["count"].data_ptr(), k, 1,
                                table.data_ptr(), st))
    out = torch.empty(s["bound"], dtype=torch.uint8, device="cuda")
    sizes = torch.zeros(k, dtype=torch.int64, device="cuda")
    capi.check(L.pg_store_encode(nodes.data_ptr(), s["first"].data_ptr(), s["count"].data_ptr(), k, 1,
                                 table.data_ptr(), out.data_ptr(), s["offsets"].data_ptr(), sizes.data_ptr(), st))
    data, at, sizes = _pack(s["data"], out, s["offsets"], sizes)
    back = torch.empty_like(nodes)
    status = torch.zeros(k, dtype=torch.int64, device="cuda")
    capi.check(L.pg_store_decode(data.data_ptr(), at.data_ptr(), sizes.data_ptr(), s["count"].data_ptr(),
                                 s["first"].data_ptr(), k, 1, table.data_ptr(), back.data_ptr(), status.data_ptr(), st))
    return table, data, sizes, back, status


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "lines":
        return _run_lines(s)
    if kind == "sweep":
        return _run_sweep(s)
    if kind == "mid":
        return mid.values_device(s["raws"], out=s["out"], scratch=s["scratch"])
    if kind == "rans_enc":
        data, _, sizes = _pack(s["data"], *rans.encode_device(rans.node_symbols(s["nodes"], 1), s["offsets"]))
        return data, sizes
    if kind == "rans_dec":
        return rans.decode_device(s["data"], s["at"], s["sizes"], s["offsets"])
    if kind == "lm_enc":
        data, _, sizes = _pack(s["data"], *learned.encode(s["model"], s["refs"], rans.node_symbols(s["nodes"], 1),
                                                          s["offsets"], s["count"]))
        return data, sizes
    if kind == "lm_dec":
        symbols, _, status = learned.decode(s["model"], s["refs"], s["data"], s["offsets"], s["sizes"], s["count"])
        return symbols, status
    if kind == "train":
        return _run_train(s)
    if kind == "store":
        return _run_store(s)
    capi.check(capi.lib().pg_shard_scatter(case["slice"], case["shards"], case["lo"], case["hi"], s["blocks"],
                                           len(s["blocks"]), s["nodes"].data_ptr(), supertensor.RAW,
                                           s["symbols"].data_ptr(), None, capi.stream_handle()))
    return s["symbols"]


# ---------------------------------------------------------------------------
# What a pass cannot do without


@functools.lru_cache(maxsize=None)
def _rmin_quadrants():
    """Rotation-minimal quadrant states by (black, white) count, in the order of the database's sections: as (black
    mask, white mask), states that a reflection moves first, each beside its reflection."""
    def turn(v):
        return sum(1 << (3 * (2 - y) + x) for x in range(3) for y in range(3) if v >> (3 * x + y) & 1)

    def mirror(v):
        return sum(1 << (3 * (2 - y) + 2 - x) for x in range(3) for y in range(3) if v >> (3 * x + y) & 1)

    turned, mirrored = [turn(v) for v in range(512)], [mirror(v) for v in range(512)]
    pack = [sum(3**i for i in range(9) if v >> i & 1) for v in range(512)]
    least, unpack = {}, {}
    for b in range(512):
        for w in range(512):
            if b & w:
                continue
            q = pack[b] + 2 * pack[w]
            unpack[q] = (b, w)
            x, y, m = b, w, q
            for _ in range(3):
                x, y = turned[x], turned[y]
                m = min(m, pack[x] + 2 * pack[y])
            least[q] = m

    def key(q):
        b, w = unpack[q]
        r = least[pack[mirrored[b]] + 2 * pack[mirrored[w]]]
        return min(q, r) + 19683 * (q == r), q

    out = {}
    for q in sorted((q for q in least if least[q] == q), key=key):
        b, w = unpack[q]
        out.setdefault((bin(b).count("1"), bin(w).count("1")), []).append((b, w))
    return out


def _section_nodes(sig):
    return math.prod(end.section_shape(int(sig)))


def work(case):
    """Bytes: every input read once and every output written once.  Operations: the network's multiply-adds."""
    kind = case["kind"]
    flops = 0
    if kind == "lines":
        c = _counts(case["section"])
        dims = _open_dims(case["section"])
        shape = end.section_shape(_sig(case["section"]))
        nodes = 0.0
        for d in dims:  # a line of average extent: the child quadrant's states and the parent's, times the cross-section
            child = [list(x) for x in c]
            child[d][sum(map(sum, c)) & 1] += 1
            cross = math.prod(shape[q] / ((shape[q] + 7) // 8) for q in range(4) if q != d)
            inputs = end.section_shape(end.section_sig(child))[d] if sum(map(sum, c)) < 35 else 0
            nodes += cross * (shape[d] + inputs) / len(dims)
        nbytes = 64 * nodes * case["blocks"] * min(case["dims"], len(dims))
    elif kind == "sweep":
        root = _sig(case["root"])
        nbytes = 64 * sum(_section_nodes(x) for s in (case["slice"], case["slice"] + 1)
                          for x in sweep.descendent_sections(root, s))
    elif kind == "mid":
        # levels of 16-byte halfsupers, each written once and read once by the level below
        items = lambda spots: sum(math.comb(spots, n >> 1) * math.comb(spots - (n >> 1), n - (n >> 1))
                                  for n in range(spots + 1))
        nbytes = case["boards"] * (2 * 32 * items(36 - case["stones"] - case["spread"] // 2) + mid.RECORD_BYTES)
    elif kind in ("rans_enc", "rans_dec"):
        symbols = case["streams"] * case["symbols"] * 15 / 16
        nbytes = symbols * (0.25 + 0.12 if kind == "rans_enc" else 1 + 0.12)
    elif kind in ("lm_enc", "lm_dec"):
        symbols = case["blocks"] * 256 * 2940
        nbytes = symbols * (0.25 + 0.1 if kind == "lm_enc" else 1 + 0.1)
        flops = symbols * 2 * (64 * 13 + 64 * 64 + 64 * 3)
    elif kind == "train":
        nbytes = case["batch"] * (8 + 14) + 4 * learned.N_PARAMS * 7
        flops = case["batch"] * 2 * (2 * 64 * 43 + 3 * 64 * 64 + 3 * 64 * 3)
    elif kind == "store":
        nodes = case["blocks"] * 2940
        nbytes = nodes * (64 + 16 + 16 + 64)
    else:
        total = int(capi.check(capi.lib().pg_shard_total(case["slice"])))
        nbytes = total * (0.25 + (case["hi"] - case["lo"]) / case["shards"])
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# The training step in 64 bits


def _splitmix(z):
    with np.errstate(over="ignore"):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


def _bf16(x):
    return torch.from_numpy(np.ascontiguousarray(x)).to(torch.bfloat16).double()


def _grid(w):
    """Columns as integers of magnitude at most 127 times a power of two."""
    e = 7 - np.frexp(np.abs(w).max(0))[1]
    return torch.from_numpy(np.ldexp(np.clip(np.rint(np.ldexp(w.astype(np.float64), e)), -127, 127), -e))


def exact(case, seed):
    if case["kind"] != "train":
        return None
    t = _train_inputs(case, seed)
    batch, step = case["batch"], t["step"] + 1
    # The step's samples: (block, node, rotation) drawn by a hash of the seed, the step and the index
    with np.errstate(over="ignore"):
        h = _splitmix(np.uint64(t["seed"]) ^ _splitmix(np.uint64(step) * np.uint64(0x100000001B3) +
                                                       np.arange(batch, dtype=np.uint64)))
    first = np.zeros(len(t["count"]) + 1, np.int64)
    first[1:] = np.cumsum(t["count"])
    c = ((h & np.uint64(0xFFFFFFFFFF)) % np.uint64(first[-1])).astype(np.int64)
    s = np.searchsorted(first, c, side="right") - 1
    i, r = c - first[s], (h >> np.uint64(56)).astype(np.int64)
    # Features: stones, rotation, the neighbouring rotations coded before, the previous node of the coder's run
    F = np.zeros((batch, 124))
    extent = np.minimum(8, t["shape"] - 8 * t["block"])[s]
    rest = i.copy()
    quadrants = [np.array(_rmin_quadrants()[tuple(x)]) for x in _counts(TRAIN_SECTION)]
    for q in (3, 2, 1, 0):
        masks = quadrants[q][8 * t["block"][s, q] + rest % extent[:, q]]
        rest = rest // extent[:, q]
        for cell in range(9):
            for side in range(2):
                F[:, 18 * q + 2 * cell + side] = masks[:, side] >> cell & 1
    symbol = lambda node, rot: t["symbols"][torch.from_numpy(256 * (first[s] + node) + rot).cuda()].cpu().numpy()
    rows = np.arange(batch)
    for q in range(4):
        digit = r >> (2 * q) & 3
        F[rows, 72 + 4 * q + digit] = 1
        for k, d in ((0, 1), (1, 3)):
            n = r + ((((digit + d) & 3) - digit) << (2 * q))
            F[rows, 88 + 4 * (2 * q + k) + np.where((n & 127) < (r & 127), symbol(i, n), 3)] = 1
    inside = i % ((t["count"][s] + 31) // 32) != 0
    F[rows, 120 + np.where(inside, symbol(np.maximum(i - 1, 0), r), 3)] = 1
    F, y = torch.from_numpy(F), torch.from_numpy(symbol(i, r)).long()
    # The network with its coding weights: bf16 stone rows and biases, gridded context rows and layer 2
    p = t["params"]
    a, b = learned.P_W1, learned.P_B1
    w1 = p[a:b].reshape(124, 64)
    w1 = torch.cat([_bf16(w1[:72]), _grid(w1[72:])])
    b1, b2 = _bf16(p[learned.P_B1:learned.P_W2]), _bf16(p[learned.P_B2:learned.P_W3])
    w2 = _grid(p[learned.P_W2:learned.P_B2].reshape(64, 64))
    w3, b3 = _bf16(p[learned.P_W3:learned.P_B3]).reshape(64, 3), _bf16(p[learned.P_B3:])
    act = torch.clamp(torch.round(16 * (b1 + F @ w1)), 0, 255) / 16
    a2 = b2 + act @ w2
    h2 = torch.relu(a2)
    z = b3 + h2 @ w3
    logp = torch.log_softmax(z, 1)
    loss = -logp.gather(1, y[:, None]).sum() * 1.44269504
    dz = torch.exp(logp)
    dz[torch.arange(batch), y] -= 1
    d2 = (dz @ w3.T) * (a2 > 0)
    d1 = (d2 @ w2.T) * ((act > 0) & (act < 255 / 16))
    grad = torch.cat([(F.T @ d1).reshape(-1), d1.sum(0), (act.T @ d2).reshape(-1), d2.sum(0),
                      (h2.T @ dz).reshape(-1), dz.sum(0)])
    g = grad / batch
    m = 0.9 * torch.from_numpy(t["m"]).double() + 0.1 * g
    v = 0.999 * torch.from_numpy(t["v"]).double() + 0.001 * g * g
    params = torch.from_numpy(p).double() - 3e-3 * (m / (1 - 0.9**step)) / (torch.sqrt(v / (1 - 0.999**step)) + 1e-8)
    return {"params": params, "m": m, "v": v, "grad": grad, "loss": loss.reshape(1)}
