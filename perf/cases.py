"""Performance cases: what programs on this library do, from one read against a
few references to batches that fill the GPU.

A case is a dict of plain values.  ``call`` names the public entry point it goes
through, ``shape`` the pairs' length distribution (``SHAPES``), ``pairs`` how
many there are; the rest are that entry's options.  All inputs come from the
package's seeded workload generator.  Outputs are whole numbers (scores,
positions, path operations).
"""
import importlib

import numpy as np
import torch

gbsw = importlib.import_module("gpu-bsw_gb300")
workloads = importlib.import_module("gpu-bsw_gb300.workloads")

DNA_SCORES = gbsw.scoring.DNA_SCORES_BENCH
AA_GAPS = gbsw.scoring.AA_GAPS

# name: (kind, maker(pairs, seed), longest sequence, mean symbols per pair, mean cells per pair)
SHAPES = {
    # reads of 100-150 against 200-500 bp references, 5% substitutions, 1% indels
    "plain_dna": (gbsw.DNA, workloads.plain_dna, 500, 475, 43_750),
    # reads of 150-300 against 400-1,024 bp references, one in five unrelated
    "dna_throughput": (gbsw.DNA, workloads.dna_throughput, 1024, 937, 160_200),
    # 70% short reads against 300 bp, 30% contigs of 1,000-2,048 against 1,500-4,096 bp
    "mixed_dna": (gbsw.DNA, workloads.mixed_dna, 4096, 1_690, 1_300_000),
    # long reads of 3,000-12,000 against 4,000-16,000 bp
    "long_dna": (gbsw.DNA, workloads.long_dna, 16000, 17_500, 72_000_000),
    # protein pairs, log-normal lengths of median 300 within 50-1,000
    "protein": (gbsw.PROTEIN, workloads.protein, 1000, 680, 135_600),
    # long protein chains
    "protein_long": (gbsw.PROTEIN, lambda n, seed: workloads.custom_protein(n, seed, 512, 1200), 1200, 1_712,
                     733_000),
}
# most pairs a case of the shape holds (memory, time and the time it takes to make them)
MOST_PAIRS = {"plain_dna": 200_000, "dna_throughput": 120_000, "mixed_dna": 200_000, "long_dna": 1_000,
              "protein": 60_000, "protein_long": 20_000}

# path operations a pair has at most on average over a batch of the shape
OPS_PER_PAIR = {"plain_dna": 40, "dna_throughput": 60, "mixed_dna": 200, "long_dna": 2_000, "protein": 220,
                "protein_long": 600}


def listed():
    return [
        # an interactive query: sixteen reads as Python strings through the drop-in
        # function, where launches, waits and the host's own work are the time
        {"name": "dropin_16_reads", "call": "dropin", "shape": "plain_dna", "pairs": 16},
        # one small batch inside a GPU pipeline: inputs and results stay on the device
        {"name": "plain_dna_1k_device", "call": "device", "shape": "plain_dna", "pairs": 1_000},
        # a sequencing chunk as raw bytes in page-locked memory; 3% of the reads hold an
        # N, so their pairs take the byte-compare path beside the A/C/G/T ones
        {"name": "dna_reads_20k_host", "call": "host16", "shape": "dna_throughput", "pairs": 20_000, "n_share": 0.03},
        # the headline batch, device-resident
        {"name": "dna_100k_device", "call": "device", "shape": "dna_throughput", "pairs": 100_000},
        # the same batch end to end: packed in pinned host memory, results back
        {"name": "dna_100k_packed", "call": "packed16", "shape": "dna_throughput", "pairs": 100_000},
        # an assembly's mix of reads and contigs, most cells in the long pairs: the largest
        {"name": "mixed_dna_200k_device", "call": "device", "shape": "mixed_dna", "pairs": 200_000},
        # a handful of long reads, too few to fill the GPU one pair per group
        {"name": "long_dna_61_device", "call": "device", "shape": "long_dna", "pairs": 61},
        # a small protein search from host buffers, int32 results
        {"name": "protein_500_host", "call": "host32", "shape": "protein", "pairs": 500},
        # the protein batch, device-resident
        {"name": "protein_30k_device", "call": "device", "shape": "protein", "pairs": 30_000},
        # CIGAR paths of an aligned DNA batch, host buffers in and out
        {"name": "traceback_dna_100k", "call": "traceback", "shape": "dna_throughput", "pairs": 100_000},
        # the same for proteins
        {"name": "traceback_protein_7k", "call": "traceback", "shape": "protein", "pairs": 7_001},
        # an alignment service under a burst: DNA and protein jobs of 1-5,000 pairs each
        {"name": "server_24_jobs", "call": "server", "shape": "serving", "pairs": 5_000, "jobs": 24},
    ]


def _log_uniform(rng, low, high):
    return int(round(low * (high / low) ** rng.random()))


def draw(rng):
    """One more case: an entry point, a shape it is used with, and a size spread
    over the logarithm of the shape's range."""
    call = rng.choice(["dropin", "device", "device", "device", "host16", "host32", "packed16", "traceback", "server"])
    if call == "server":
        return {"call": call, "shape": "serving", "pairs": _log_uniform(rng, 100, 5_000), "jobs": rng.randint(2, 24)}
    if call == "dropin":
        shape = rng.choice(["plain_dna", "dna_throughput", "protein"])
        return {"call": call, "shape": shape, "pairs": _log_uniform(rng, 1, 5_000)}
    shape = rng.choice(sorted(SHAPES))
    # a path's direction memory grows with its cells: fewer pairs of the long shapes
    most = MOST_PAIRS[shape] // (10 if call == "traceback" and shape in ("mixed_dna", "long_dna") else 1)
    case = {"call": call, "shape": shape, "pairs": _log_uniform(rng, 1, most)}
    if call in ("host16", "host32") and SHAPES[shape][0] == gbsw.DNA:
        case["n_share"] = round(rng.choice([0.0, 0.01, 0.05]), 3)
    return case


def _scoring(kind):
    if kind == gbsw.DNA:
        return gbsw.make_scoring(gbsw.DNA, scores=DNA_SCORES)
    return gbsw.make_scoring(gbsw.PROTEIN, matrix=gbsw.scoring.BLOSUM62, gaps=AA_GAPS)


_handles = {}


def _aligner():
    """The program's one context, kept from batch to batch."""
    if "aligner" not in _handles:
        _handles["aligner"] = gbsw.Aligner(0)
    return _handles["aligner"]


def _server():
    """The service's one server, up before the jobs come."""
    if "server" not in _handles:
        _handles["server"] = gbsw.Server(0)
    return _handles["server"]


def _pinned(array):
    return torch.from_numpy(array).pin_memory().numpy()


def _with_n(batch, share, seed):
    """`share` of the queries with one base read as N."""
    rng = np.random.default_rng(seed)
    hit = np.nonzero(rng.random(batch.n) < share)[0]
    at = batch.query_off[hit] + (rng.random(len(hit)) * batch.query_lengths()[hit]).astype(np.int64)
    batch.query[at] = ord("N")
    return batch


def _jobs(case, seed):
    """Six jobs in ten of reads, the others of proteins, of 1 to ``pairs`` pairs
    each: the case says how many of what, the seed which."""
    sizes = np.random.default_rng([case["jobs"], case["pairs"]])
    jobs = []
    for k in range(case["jobs"]):
        pairs = int(sizes.integers(1, case["pairs"] + 1))
        kind, make = SHAPES["dna_throughput" if sizes.random() < 0.6 else "protein"][:2]
        jobs.append((_scoring(kind), make(pairs, seed * 1_000_003 + k)))
    return jobs


def _leave_out_pathless(aligner, batch, scoring, results, pairs):
    """Zeroes the score of the pairs whose reported begin and end belong to different,
    equally good alignments (one pair in some 100,000): no path joins the two, and
    the traceback refuses the call."""
    part = batch if len(pairs) == batch.n else batch.subset(pairs)
    try:
        aligner.traceback_batch(part, scoring, results[pairs])
    except gbsw.GbswError as error:
        if error.status != -1:
            raise
        if len(pairs) == 1:
            results[pairs[0], 0] = 0
            return
        for half in np.array_split(pairs, 2):
            _leave_out_pathless(aligner, batch, scoring, results, half)


def prepare(case, seed):
    call = case["call"]
    if call == "server":
        return {"call": call, "server": _server(), "jobs": _jobs(case, seed)}
    kind, make, longest, _, _ = SHAPES[case["shape"]]
    batch = make(case["pairs"], seed)
    state = {"call": call, "kind": kind, "scoring": _scoring(kind)}
    if call == "dropin":
        pairs = [batch.strings(k) for k in range(batch.n)]
        state.update(reads=[q.decode() for _, q in pairs], contigs=[r.decode() for r, _ in pairs])
        return state
    state["aligner"] = _aligner()
    if call == "device":
        state["inputs"] = [torch.from_numpy(x).cuda() for x in (batch.ref, batch.ref_off, batch.query, batch.query_off)]
        state["results"] = [torch.empty(batch.n, dtype=torch.int32, device="cuda") for _ in range(5)]
        state.update(pairs=batch.n, longest=longest)
        return state
    if case.get("n_share"):
        batch = _with_n(batch, case["n_share"], seed)
    if call == "traceback":
        state["results"] = np.array(state["aligner"].align_batch(batch, state["scoring"]))
        _leave_out_pathless(state["aligner"], batch, state["scoring"], state["results"], np.arange(batch.n))
        state["batch"] = batch
        state["ops"] = np.zeros(OPS_PER_PAIR[case["shape"]] * (batch.n + 16), dtype=np.int32)
        return state
    state.update(ref_off=_pinned(batch.ref_off), query_off=_pinned(batch.query_off))
    if call == "packed16":
        for name, raw in (("ref", batch.ref), ("query", batch.query)):
            stream = gbsw.pack(kind, raw)
            stream.words = _pinned(stream.words)
            state[name] = stream
    else:
        state.update(ref=_pinned(batch.ref), query=_pinned(batch.query))
    return state


def run(state):
    call, scoring = state["call"], state.get("scoring")
    if call == "server":
        jobs = [state["server"].submit_batch(batch, sc) for sc, batch in state["jobs"]]
        return [job.wait() for job in jobs]
    if call == "dropin":
        if state["kind"] == gbsw.DNA:
            return gbsw.kernel_driver_dna(state["reads"], state["contigs"], DNA_SCORES)
        return gbsw.kernel_driver_aa(state["reads"], state["contigs"], gbsw.scoring.BLOSUM62, *AA_GAPS)
    aligner = state["aligner"]
    if call == "device":
        ref, ref_off, query, query_off = (x.data_ptr() for x in state["inputs"])
        aligner.align_device(scoring, ref, ref_off, query, query_off, state["pairs"], state["longest"],
                             *(x.data_ptr() for x in state["results"]),
                             stream=torch.cuda.current_stream().cuda_stream)
        return state["results"]
    if call == "traceback":
        ops, off = aligner.traceback_batch(state["batch"], scoring, state["results"])
        state["ops"][:len(ops)] = ops.view(np.int32)  # the program's buffer of a whole run's paths
        return state["ops"], off
    if call == "packed16":
        return aligner.align_packed(scoring, state["ref"], state["ref_off"], state["query"], state["query_off"],
                                    int16=True)
    return aligner.align_host(scoring, state["ref"], state["ref_off"], state["query"], state["query_off"],
                              int16=call == "host16")


# Integer operations a cell of the recurrence cannot do without: five additions
# (two gap opens, two gap extensions, the substitution) and five maxima (E, F,
# three for H against both and zero and the running best counted together).
CELL_OPS = 10


def work(case):
    """Of one pass: each input byte once, each result once; forward cells x CELL_OPS
    (the reverse pass's share depends on where the alignments lie; it is left out)."""
    if case["call"] == "server":
        # six jobs in ten are DNA, half the most pairs each on average
        pairs = case["jobs"] * case["pairs"] / 2
        symbols = 0.6 * SHAPES["dna_throughput"][3] + 0.4 * SHAPES["protein"][3]
        cells = 0.6 * SHAPES["dna_throughput"][4] + 0.4 * SHAPES["protein"][4]
        return {"bytes": pairs * (symbols + 16 + 20), "flops": pairs * cells * CELL_OPS}
    kind, _, _, symbols, cells = SHAPES[case["shape"]]
    pairs, call = case["pairs"], case["call"]
    if call == "packed16":
        symbols = symbols / (4 if kind == gbsw.DNA else 1.5)
    out = 10 if call in ("dropin", "host16", "packed16") else 20
    if call == "traceback":
        # the aligned segment: about a third of a DNA pair's cells, four tenths of a
        # protein pair's; results in, about twenty operations out
        return {"bytes": pairs * (symbols + 16 + 20 + 80), "flops": pairs * 0.35 * cells * CELL_OPS}
    return {"bytes": pairs * (symbols + 16 + out), "flops": pairs * cells * CELL_OPS}


def exact(case, seed):
    """Every output is a whole number: it either equals or differs, and has no error to measure."""
    return None
