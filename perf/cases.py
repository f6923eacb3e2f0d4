"""The work that users of this framework have it do, as cases to time.

A case is one call (or one drain of queued calls) through the public entry
points: a block of reads to its streams (`block_run`, `block_run_device`),
several blocks through the batched path, packing alone (`pack_device`), and
training and running the learned mismatch coder (`Learner`).  Reads are drawn
on the GPU by the rules of `curc_b200.synth` (uniform or GC-biased genomes
with diverged repeats, substitutions, N bases, normal insert sizes).
"""
import ctypes
import math

import numpy as np
import torch

from curc_b200 import Context, Learner, lib

# One context per process, as a program that compresses one block after
# another keeps it; streams only, no stage intermediates.
_CTX = None


def _context():
    global _CTX
    if _CTX is None:
        _CTX = Context(0)
        _CTX.keep_intermediates(False)
        _CTX.batch_workers(4)
    return _CTX


# ------------------------------------------------------------------- cases

def listed():
    return [
        # the smallest blocks: a tail block, an amplicon or a test file, where launches and latency count
        _block("se100_2k", 2_000, 100, 20_000),
        # the smallest block of the batched workload: 75 bp single end
        _block("se75_50k", 50_000, 75, 250_000, err=0.003),
        # 100k x 100 bp single end from host memory, the basic configuration of the tests
        _block("se100_100k_host", 100_000, 100, 1_000_000, host=True),
        # a small paired-end block with preserved order
        _block("pe150_100k_pairs_po", 200_000, 150, 2_000_000, err=0.002, paired=True, po=True, gc=0.4, repeats=0.05),
        # odd counts and length, errors rising along the read, more N: a block of long reads
        _block("se251_700k_po", 700_003, 251, 3_600_000, err=0.001, err_end=0.015, n_rate=0.0002, po=True, gc=0.45,
               repeats=0.08),
        # an ordinary paired-end block, order not preserved (the default mode of the command line)
        _block("pe151_1M_pairs", 2_000_000, 151, 10_000_000, err=0.002, paired=True, gc=0.4, repeats=0.05),
        # the benchmark's block: 10M pairs x 150 bp, preserved order
        _block("pe150_10M_pairs_po", 20_000_000, 150, 50_000_000, err=0.002, paired=True, po=True, gc=0.4,
               repeats=0.05),
        # a large block of long reads (the 250 bp workload at a fifth of its size)
        _block("se250_8M_po", 8_000_000, 250, 40_000_000, err=0.001, err_end=0.015, n_rate=0.0002, po=True, gc=0.45,
               repeats=0.08),
        # many small blocks of different genomes queued from host memory and drained on four pipelines
        {"name": "batch_12_mixed", "kind": "batch", "blocks": 12, "most": 400_000},
        # packing alone, for a program that keeps its reads on the device
        {"name": "pack_20M_x150", "kind": "pack", "n": 20_000_000, "L": 150, "n_rate": 0.0001},
        # the learned mismatch coder: coding the mismatches of a block, and training on one
        {"name": "learn_encode_500k_pairs", "kind": "encode", "n": 1_000_000, "genome": 5_000_000},
        {"name": "learn_train_100k_pairs", "kind": "train", "n": 200_000, "genome": 1_000_000, "epochs": 2},
    ]


def _block(name, n, L, genome, err=0.001, err_end=None, n_rate=0.0001, paired=False, po=False, gc=0.5, repeats=0.0,
           host=False):
    c = {"kind": "block", "n": n, "L": L, "genome": genome, "err": err, "err_end": err if err_end is None else err_end,
         "n_rate": n_rate, "paired": paired, "po": po, "gc": gc, "repeats": repeats, "host": host}
    return dict(c, name=name) if name else c


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["block", "pack", "batch", "encode", "train"], [14, 2, 2, 1, 1])[0]
    if kind == "pack":
        L = rng.randint(36, 300)
        return {"kind": kind, "n": _log_uniform(rng, 1_000, 3_000_000_000 // max(L, 150)), "L": L,
                "n_rate": rng.choice([0.0, 0.0001, 0.002])}
    if kind == "batch":
        return {"kind": kind, "blocks": rng.randint(3, 12), "most": _log_uniform(rng, 60_000, 400_000)}
    if kind == "encode":
        n = 2 * _log_uniform(rng, 20_000, 500_000)
        return {"kind": kind, "n": n, "genome": n * 150 // rng.randint(20, 60)}
    if kind == "train":
        n = 2 * _log_uniform(rng, 20_000, 100_000)
        return {"kind": kind, "n": n, "genome": n * 150 // rng.randint(20, 60), "epochs": rng.randint(1, 2)}
    L = rng.choice([75, 100, 101, 125, 150, 151, 250, rng.randint(60, 300)])
    paired = rng.random() < 0.5
    n = _log_uniform(rng, 1_000, 1_000_000_000 // L)
    n += n % 2 if paired else 0
    genome = max(2_000, int(n * L / math.exp(rng.uniform(math.log(10), math.log(100)))))
    err = rng.uniform(0.001, 0.005)
    return _block(None, n, L, genome, err=err, err_end=err * rng.choice([1, 1, 3]),
                  n_rate=rng.choice([0.0, 0.0001, 0.0002]), paired=paired, po=rng.random() < 0.5,
                  gc=rng.choice([0.5, 0.45, 0.4]), repeats=rng.choice([0.0, 0.05, 0.08]),
                  host=n <= 200_000 and rng.random() < 0.4)


# ------------------------------------------------------------------ inputs

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _substitute(base, shift):
    """Another base: `shift` (1..3) steps further in A C G T."""
    acgt = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")
    code = ((base >> 1) ^ (base >> 2)) & 3
    return acgt[((code + shift) & 3).long()]


def _genome(g, length, gc, repeats):
    acgt = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")
    u = torch.rand(length, generator=g, device="cuda")
    at = (1 - gc) / 2
    seq = acgt[(u >= at).long() + (u >= 0.5 - at + gc / 2) + (u >= 1 - at)]
    count = int(repeats * length / 3000)
    if count and length > 20_000:
        r = torch.rand(count, 3, generator=g, device="cuda").cpu().numpy()
        for a, b, c in r:
            ln = 1000 + int(a * 4000)
            src, dst = int(b * (length - ln)), int(c * (length - ln))
            seg = seq[src:src + ln].clone()
            m = torch.rand(ln, generator=g, device="cuda") < 0.01
            shift = torch.randint(1, 4, (ln,), generator=g, device="cuda", dtype=torch.uint8)
            seq[dst:dst + ln] = torch.where(m, _substitute(seg, shift), seg)
    return seq


def _reads(g, n, L, genome, err, err_end, n_rate, paired, gc, repeats):
    """(n, L) ASCII reads on the device in block order (mates interleaved)."""
    comp = torch.zeros(256, dtype=torch.uint8, device="cuda")
    for a, b in zip(b"ACGTN", b"TGCAN"):
        comp[a] = b
    seq = _genome(g, max(genome, 4 * L), gc, repeats)
    rate = torch.linspace(err, err_end, L, device="cuda")
    out = torch.empty(n, L, dtype=torch.uint8, device="cuda")
    cols = torch.arange(L, device="cuda")
    step = max(2, 200_000_000 // L // 2 * 2)
    for a in range(0, n, step):
        k = min(step, n - a)
        if paired:
            ins = (torch.randn(k // 2, generator=g, device="cuda") * 50 + 400).round().long()
            ins = ins.clamp(min=L, max=seq.numel() // 2)
            # whole numbers and 64-bit products: a float32 genome length would round past the end
            first = (torch.rand(k // 2, generator=g, device="cuda", dtype=torch.float64)
                     * (seq.numel() - ins + 1)).long()
            first = torch.minimum(first, seq.numel() - ins)
            start = torch.stack([first, first + ins - L], 1)
            flip = torch.rand(k // 2, 1, generator=g, device="cuda") < 0.5  # fragment from the reverse strand
            start = torch.where(flip, start.flip(1), start).reshape(-1)
            rc = torch.cat([flip, ~flip], 1).reshape(-1)
        else:
            start = (torch.rand(k, generator=g, device="cuda", dtype=torch.float64) * (seq.numel() - L + 1)).long()
            start = start.clamp(max=seq.numel() - L)
            rc = torch.rand(k, generator=g, device="cuda") < 0.5
        # a reverse-complemented read walks its window backwards
        at = torch.where(rc, start + L - 1, start)[:, None] + torch.where(rc, -1, 1)[:, None] * cols
        rd = seq[at]
        del at
        rd = torch.where(rc[:, None], comp[rd.long()], rd)
        m = torch.rand(k, L, generator=g, device="cuda") < rate
        r, c = m.nonzero(as_tuple=True)
        shift = torch.randint(1, 4, (r.numel(),), generator=g, device="cuda", dtype=torch.uint8)
        rd[r, c] = _substitute(rd[r, c], shift)
        if n_rate:
            rd[torch.rand(k, L, generator=g, device="cuda") < n_rate] = ord("N")
        out[a:a + k] = rd
    return out


def _learn_reads(g, case):
    """Paired 150 bp reads with errors rising from 0.1% to 1% (curc_b200.learned's workload)."""
    return _reads(g, case["n"], 150, case["genome"], 0.001, 0.010, 0.0001, True, 0.4, 0.05)


def _batch_blocks(case):
    """(reads, length, genome) of each block: sizes over the whole range, 10x to 50x coverage."""
    lo, hi = math.log(5_000), math.log(case["most"])
    for b in range(case["blocks"]):
        n = int(math.exp(lo + (hi - lo) * b / (case["blocks"] - 1)))
        L = (75, 100, 150, 250)[b % 4]
        yield n, L, max(2_000, n * L // (10, 25, 50)[b % 3])


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "block":
        reads = _reads(g, *(case[k] for k in ("n", "L", "genome", "err", "err_end", "n_rate", "paired", "gc", "repeats")))
        if case["host"]:
            reads = reads.cpu().numpy()
        body = _body(case["n"], case["L"], case["genome"], (case["err"] + case["err_end"]) / 2 + case["n_rate"],
                     case["paired"], case["po"])
        return {"case": case, "ctx": _context(), "reads": reads, "body": body}
    if kind == "batch":
        rng = np.random.default_rng(seed)
        blocks, bodies = [], []
        for n, L, genome in _batch_blocks(case):
            blocks.append(_reads(g, n, L, genome, float(rng.uniform(0.001, 0.005)), 0.005, 0.0001, False, 0.5,
                                 0.0).cpu().numpy())
            bodies.append(_body(n, L, genome, 0.005, False, False))
        return {"case": case, "ctx": _context(), "blocks": blocks, "bodies": bodies}
    if kind == "pack":
        n, L = case["n"], case["L"]
        reads = _reads(g, n, L, 2_000_000, 0.002, 0.002, case["n_rate"], False, 0.4, 0.0)
        return {"case": case, "ctx": _context(), "reads": reads,
                "packed": torch.empty(n, (L + 31) // 32, dtype=torch.int64, device="cuda"),
                "has_n": torch.empty(n, dtype=torch.uint8, device="cuda")}
    # a context of its own: the learner works on its context's last block
    ctx = Context(0)
    ctx.keep_intermediates(False)
    lrn = Learner(0)
    if kind == "encode":
        small = _reads(g, 20_000, 150, 100_000, 0.001, 0.010, 0.0001, True, 0.4, 0.05)
        ctx.block_run_device(small.data_ptr(), 20_000, 150, True, True)
        lrn.add_block(ctx)
        lrn.train(epochs=2, batch=1024, seed=1)
    reads = _learn_reads(g, case)
    torch.cuda.synchronize()
    ctx.block_run_device(reads.data_ptr(), case["n"], 150, True, True)
    if kind == "train":
        lrn.add_block(ctx)
    most = int(12 * _anchors(case)) + 200_000
    return {"case": case, "ctx": ctx, "lrn": lrn, "reads": reads,
            "body": {"bytes": torch.zeros(most, dtype=torch.uint8), "sizes": torch.zeros(1, dtype=torch.int64),
                     "filled": 0}}


# -------------------------------------------------------------------- runs

_NAMES = ["strand", "mis_cnt", "mis_base", "decoder_table", "read_off", "unmap_read_off", "unmap_n_read_off",
          "pe_order", "id_to_pos", "ref", "unmap_ref", "unmap_n_ref", "ref_off", "ref_len_map", "unmap_ref_off",
          "unmap_ref_len", "unmap_n_ref_off", "unmap_n_ref_len", "sizes"]


def _view(ctx, name):
    """A result of the last block run where it lies (curc_block_get)."""
    p, nb = ctypes.c_void_p(), ctypes.c_uint64()
    if lib().curc_block_get(ctx.handle, name.encode(), ctypes.byref(p), ctypes.byref(nb)) != 0:
        raise KeyError(name)
    return p.value, nb.value


def _body(n, L, genome, err, paired, po):
    """What a program keeps of a block before it runs the next one: a buffer
    for the streams one after another, and their sizes."""
    # the pseudogenomes stay near the genome's size where the reads cover it well
    ref = min(1.3 * n * L, genome * (7 if n * L >= 30 * genome else 14))
    most = int(n * (3 + (8 if po else 6 if paired else 2)) + 8 * n * L * err + ref) + 200_000
    return {"bytes": torch.zeros(most, dtype=torch.uint8), "sizes": torch.zeros(len(_NAMES) + L // 5, dtype=torch.int64),
            "filled": 0}


def _keep(body, parts):
    at, sizes = 0, []
    for p, nb in parts:
        if nb:
            src = torch.from_numpy(np.frombuffer((ctypes.c_uint8 * nb).from_address(p), dtype=np.uint8))
            body["bytes"][at:at + nb].copy_(src)
        at += nb
        sizes.append(nb)
    if at < body["filled"]:
        body["bytes"][at:body["filled"]].zero_()
    body["filled"] = at
    body["sizes"].copy_(torch.tensor(sizes))
    return {"bytes": body["bytes"], "sizes": body["sizes"]}


def _streams(ctx, L, body):
    return _keep(body, [_view(ctx, name) for name in _NAMES + ["mis_off_%d" % m for m in range(1, L // 5 + 1)]])


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "block":
        if case["host"]:
            ctx.block_run(state["reads"], case["po"], case["paired"])
        else:
            ctx.block_run_device(state["reads"].data_ptr(), case["n"], case["L"], case["po"], case["paired"])
        return _streams(ctx, case["L"], state["body"])
    if kind == "batch":
        tickets, out = {}, {}
        for k, reads in enumerate(state["blocks"]):
            tickets[ctx.batch_submit(reads)] = k

        def on_block(ticket):
            k = tickets[ticket]
            out[k] = _streams(ctx, state["blocks"][k].shape[1], state["bodies"][k])

        ctx.batch_drain(on_block)
        return [out[k] for k in range(len(out))]
    if kind == "pack":
        ctx.pack_device(state["reads"].data_ptr(), case["n"], case["L"], state["packed"].data_ptr(),
                        state["has_n"].data_ptr())
        return {"packed": state["packed"], "has_n": state["has_n"]}
    if kind == "encode":
        stream = state["lrn"].encode(ctx)
        return _keep(state["body"], [(ctypes.cast(stream, ctypes.c_void_p).value, len(stream))])
    loss = state["lrn"].train(epochs=case["epochs"], batch=4096, seed=1)
    return {"loss": loss, "model": np.frombuffer(state["lrn"].model(), dtype=np.uint8)}


# -------------------------------------------------------------------- work

def _streams_bytes(n, L, genome, err, paired, po):
    """Bytes of a block's streams: strand, mismatch count and position or
    order per read, base and offset per mismatch, the pseudogenome (about
    twice the genome, since both strands are assembled)."""
    return n * (2 + (8 if po else 6 if paired else 2)) + 3 * n * L * err + 2 * genome


def _anchors(case):
    """Gaps coded by the learned coder: one per mismatch of the reads (150 bp, 0.55% on average)."""
    return case["n"] * 150 * 0.0055


def work(case):
    kind = case["kind"]
    if kind == "block":
        err = (case["err"] + case["err_end"]) / 2
        return {"bytes": case["n"] * case["L"] + _streams_bytes(case["n"], case["L"], case["genome"], err,
                                                                 case["paired"], case["po"]), "flops": 0}
    if kind == "batch":
        total = 0
        for n, L, genome in _batch_blocks(case):
            total += n * L + _streams_bytes(n, L, genome, 0.004, False, False)
        return {"bytes": total, "flops": 0}
    if kind == "pack":
        return {"bytes": case["n"] * (case["L"] + 8 * ((case["L"] + 31) // 32) + 1), "flops": 0}
    layer = 2 * (128 * 128 + 20 * 128)  # the first layer's inputs are one-hot
    if kind == "encode":
        # records, packed reads and pseudogenome read once, the stream written
        return {"bytes": case["n"] * (16 + 40) + case["genome"] / 2 + 2 * _anchors(case), "flops": layer * _anchors(case)}
    return {"bytes": 24 * _anchors(case) * case["epochs"], "flops": 6 * (2 * 128 * 128 + 20 * 128) * _anchors(case) * case["epochs"]}


def exact(case, seed):
    """Streams, packed words and model bytes are whole numbers; the training
    loss follows from FP32 updates over hundreds of steps and has no value of
    its own in 64 bits."""
    return None
