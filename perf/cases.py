"""Performance cases: the calls a program makes of this framework, over the sizes it makes them at.

A case is one call (or one burst of serving requests) through a public entry point:

  entry "host"     Engine.compute: a batch in host memory in, scores in host memory out
  entry "pinned"   the same from page-locked input and output buffers
  entry "device"   Engine.compute_device: arrays already on the GPU, scores left there
  entry "serving"  Engine.submit_many of single regions, then drain of every ticket
  entry "flat"     forward_pairs_noalloc: a flat pair list in caller-owned device buffers

  kind "short"     one read length, haplotypes half as long again: a variant caller's small regions
  kind "uneven"    regions as an assembler makes them: lognormal read counts (median 40, clipped
                   to 400), 1-16 haplotypes, trimmed reads of 100/150/250 bases, haplotypes 50-400
                   bases longer (the repository's uneven-length configuration)
  kind "stress"    64 reads x 8 haplotypes, 250 x 600, half of the reads unrelated to their region
                   (the precision-stress configuration: half the pairs underflow single precision)
  kind "long"      16 reads of 1,000-2,000 bases x 4 haplotypes of 2,000-5,000 (the long-read
                   configuration)
  kind "mixed"     uneven regions with 5% long-read regions (the streaming configuration)

Sequences and qualities follow gpupairhmm_b200/synth.py's configurations, generated with whole-array
operations so that a batch of thousands of regions takes a fraction of a second.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gpupairhmm_b200 as phmm

MAX_EXACT_WORK = 1.0e11   # cells of the 64-bit sweep, padding included, up to which exact() computes


def listed():
    return [
        # one small region, the unit of a caller that scores regions as it meets them (config 0's
        # record shape); launches and host latency are all of it
        dict(name="region_short_host", entry="host", kind="short", regions=1, read_len=100, reads=32, haps=4,
             gcp=False, layout=1),
        # one region of ordinary size whose arrays another GPU stage left on the device
        dict(name="region_uneven_device", entry="device", kind="uneven", regions=1, gcp=False, layout=1),
        # one long-read region: a few long serial wavefronts
        dict(name="region_long_host", entry="host", kind="long", regions=1, gcp=False, layout=1),
        # a worker's batch of small regions (config 0 as it stands)
        dict(name="records64_short_host", entry="host", kind="short", regions=64, read_len=100, reads=32, haps=4,
             gcp=False, layout=1),
        # a transfer batch of uneven regions on the device: the headline workload's kernels
        dict(name="uneven_2000_device", entry="device", kind="uneven", regions=2000, gcp=False, layout=1),
        # the headline call end to end: page-locked buffers, upload and download inside, large
        # enough to run as overlapped chunks
        dict(name="uneven_4000_pinned", entry="pinned", kind="uneven", regions=4000, gcp=False, layout=1),
        # a mid-size batch from ordinary (pageable) host arrays
        dict(name="uneven_300_host", entry="host", kind="uneven", regions=300, gcp=False, layout=1),
        # the precision-stress shape: half of the pairs need the wide range
        dict(name="stress_300_device", entry="device", kind="stress", regions=300, gcp=False, layout=1),
        # a batch of long-read regions
        dict(name="long_64_device", entry="device", kind="long", regions=64, gcp=False, layout=1),
        # gap-continuation qualities honoured, as the reference's CPU path does
        dict(name="uneven_1000_gcp_host", entry="host", kind="uneven", regions=1000, gcp=True, layout=1),
        # a burst at a scoring service: submit everything that has arrived, collect all of it
        dict(name="burst_400_serving", entry="serving", kind="mixed", regions=400, gcp=False, layout=1),
        # a host that owns every allocation: pairs of related short reads as a flat list
        dict(name="flat_uneven_device", entry="flat", kind="uneven", regions=60, gcp=False, layout=1),
    ]


def draw(rng):
    """One case of the same ranges: every entry and kind, sizes spread over their logarithm."""
    entry = rng.choice(["host", "host", "pinned", "device", "device", "device", "serving", "flat"])
    kind = "mixed" if entry == "serving" else rng.choice(["short", "uneven", "uneven", "stress", "long"])
    if entry == "flat" and kind == "stress":
        kind = "short"   # the flat list is scored in single precision only
    most = {"short": 2500, "uneven": 3000, "stress": 300, "long": 64, "mixed": 400}[kind]
    if entry == "flat":
        most = {"short": 600, "uneven": 120, "long": 4}[kind]
    case = dict(entry=entry, kind=kind, regions=_log_int(rng, 1, most),
                gcp=entry in ("host", "pinned", "device") and kind != "stress" and rng.random() < 0.2,
                layout=rng.randint(1, 10 ** 6))
    if kind == "short":
        case["read_len"] = rng.randint(21, 300)
        case["reads"] = _log_int(rng, 1, 64)
        case["haps"] = rng.randint(1, 16)
    return case


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


# ------------------------------------------------------------------------------------ inputs

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _structure(case):
    """Record structure: reads and haplotypes per region, lengths, and which regions are long-read.  It is
    the case's own ("layout" seeds it); the seed of prepare() makes the sequences and qualities."""
    rng = np.random.default_rng([case["layout"], 17])
    n, kind = case["regions"], case["kind"]
    if kind == "short":
        R, H = np.full(n, case["reads"]), np.full(n, case["haps"])
        rl = np.full(int(R.sum()), case["read_len"])
        hl = np.full(int(H.sum()), case["read_len"] * 3 // 2)
        long = np.zeros(n, bool)
    elif kind == "stress":
        R, H = np.full(n, 64), np.full(n, 8)
        rl, hl = np.full(64 * n, 250), np.full(8 * n, 600)
        long = np.zeros(n, bool)
    else:
        long = np.full(n, kind == "long")
        if kind == "mixed":
            long = np.zeros(n, bool)
            long[rng.choice(n, size=max(1, n // 20), replace=False)] = True
        if n == 1 and case["layout"] == 1:   # the median region
            R, H, Lb = np.full(1, 40), np.full(1, 8), np.full(1, 150)
        else:
            R = np.clip(np.round(40.0 * np.exp(rng.standard_normal(n))), 1, 400).astype(np.int64)
            H = rng.integers(1, 17, size=n)
            Lb = rng.choice([100, 150, 250], p=[0.3, 0.5, 0.2], size=n)
        R, H = np.where(long, 16, R), np.where(long, 4, H)
        lr, lh = np.repeat(long, R), np.repeat(long, H)
        trimmed = np.repeat(Lb, R) - rng.integers(0, 31, size=len(lr))
        assembled = np.repeat(Lb, H) + rng.integers(50, 401, size=len(lh))
        rl = np.where(lr, rng.integers(1000, 2001, size=len(lr)), trimmed)
        hl = np.where(lh, rng.integers(2000, 5001, size=len(lh)), assembled)
        if case["entry"] == "flat" and kind == "long":
            hl = np.maximum(hl // 2, 2000)
    return R.astype(np.int64), H.astype(np.int64), rl.astype(np.int64), hl.astype(np.int64), long


def _padded(lens):
    """Start of every sequence with 1 to 4 bytes of padding behind each, and the array's length."""
    size = lens + (4 - lens % 4)
    end = np.cumsum(size)
    return end - size, int(end[-1])


def _expand(starts, lens, dev):
    """For every base of every sequence: its sequence, its position in it, and its byte in the array."""
    ln = torch.from_numpy(lens).to(dev)
    seq = torch.repeat_interleave(torch.arange(len(lens), device=dev), ln)
    within = torch.arange(int(lens.sum()), device=dev) - torch.from_numpy(np.cumsum(lens) - lens).to(dev)[seq]
    return seq, within, torch.from_numpy(starts).to(dev)[seq] + within


def _batch(case, seed):
    """The case's records as a Batch of host arrays."""
    dev = _device()
    gen = torch.Generator(device=dev).manual_seed(seed * 1000003 + 11)
    R, H, rl, hl, long = _structure(case)
    kind = case["kind"]
    region_of_read, region_of_hap = np.repeat(np.arange(len(R)), R), np.repeat(np.arange(len(H)), H)
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    randint = lambda lo, hi, n: torch.randint(lo, hi, (n,), generator=gen, device=dev)
    acgt = to(np.frombuffer(b"ACGT", np.uint8).copy())

    # haplotypes: prefixes of their region's sequence, about two substitutions each, half of them with
    # one indel (1-5 bases; long-read regions up to 50, but not in a flat list)
    first_hap = np.cumsum(H) - H
    base_len = np.maximum.reduceat(hl, first_hap) + 64
    base_start = np.cumsum(base_len) - base_len
    base = randint(0, 4, int(base_len.sum()))
    ho, hbytes = _padded(hl)
    seq, within, at = _expand(ho, hl, dev)
    nh = len(hl)
    cut = (torch.rand(nh, generator=gen, device=dev) * to(hl)).long()
    wide = long[region_of_hap] & (case["entry"] != "flat")
    size = randint(1, 6, nh) + to(wide.astype(np.int64)) * randint(0, 46, nh)
    size = size * (randint(0, 2, nh) * 2 - 1) * randint(0, 2, nh)   # < 0 insertion (a repeat), > 0 deletion
    src = within + torch.where(within >= cut[seq], size[seq], torch.zeros_like(within))
    src = src.clamp_min(0) + to(base_start[region_of_hap])[seq]
    hap = base[torch.minimum(src, to((base_start + base_len - 1)[region_of_hap])[seq])]
    snp = torch.rand(len(seq), generator=gen, device=dev) < (2.0 / to(hl).double())[seq]
    hap = torch.where(snp, (hap + randint(1, 4, len(seq))) % 4, hap)
    hap_bases = torch.full((hbytes,), ord("N"), dtype=torch.uint8, device=dev)
    hap_bases[at] = acgt[hap]

    # reads: substrings of one of the region's haplotypes with 1% substitutions; in the stress shape
    # every other read is unrelated; in a flat list, scored in single precision only, every read lies
    # within the shortest haplotype of its region and has 0.3% substitutions
    ro, rbytes = _padded(rl)
    seq, within, at = _expand(ro, rl, dev)
    nr = len(rl)
    pick = to(first_hap[region_of_read]) + (torch.rand(nr, generator=gen, device=dev) * to(H[region_of_read])).long()
    span = to(np.minimum.reduceat(hl, first_hap)[region_of_read]) if case["entry"] == "flat" else to(hl)[pick]
    room = (span - to(rl) + 1).clamp_min(1)
    start = to(ho)[pick] + (torch.rand(nr, generator=gen, device=dev) * room).long()
    src = torch.minimum(start[seq] + within, (to(ho)[pick] + to(hl)[pick] - 1)[seq])
    read = hap_bases[src]
    err = torch.rand(len(seq), generator=gen, device=dev) < (0.003 if case["entry"] == "flat" else 0.01)
    if kind == "stress":
        err |= (seq % 2 == 1)
    read = torch.where(err, acgt[randint(0, 4, len(seq))], read)

    lr = to(long[region_of_read])[seq]
    n = len(seq)
    if kind == "stress":
        bq = randint(35, 42, n)
    elif case["entry"] == "flat":
        bq = randint(20, 41, n)
    else:
        bq = torch.where(lr, randint(5, 41, n), randint(10, 41, n))
    iq = torch.where(lr, randint(30, 46, n), torch.full_like(bq, 40))
    dq = torch.where(lr, randint(30, 46, n), torch.full_like(bq, 40))
    gq = randint(10, 41, nr)[seq] if case["gcp"] else torch.full_like(bq, 10)

    def bytes_of(values, pad):
        out = torch.full((rbytes,), pad, dtype=torch.uint8, device=dev)
        out[at] = values.to(torch.uint8)
        return out.cpu().numpy()

    q_pad = ord("N") - 33
    return phmm.Batch(R.astype(np.int32), H.astype(np.int32), bytes_of(read, ord("N")), bytes_of(bq, q_pad),
                      bytes_of(iq, q_pad), bytes_of(dq, q_pad), ro, rl.astype(np.int32), hap_bases.cpu().numpy(),
                      ho, hl.astype(np.int32), bytes_of(gq, q_pad))


def _pairs(batch):
    """(read, haplotype) of every score, in output order: record, then read, then haplotype."""
    R, H = batch.reads_per_record.astype(np.int64), batch.haps_per_record.astype(np.int64)
    haps_of_read = np.repeat(H, R)
    read = np.repeat(np.arange(int(R.sum())), haps_of_read)
    within = np.arange(len(read)) - np.repeat(np.cumsum(haps_of_read) - haps_of_read, haps_of_read)
    return read, np.repeat(np.repeat(np.cumsum(H) - H, R), haps_of_read) + within


def prepare(case, seed):
    batch = _batch(case, seed)
    entry = case["entry"]
    state = dict(case=case)
    if entry == "flat":
        read, hap = _pairs(batch)
        pairs = np.zeros(len(read), dtype=phmm.PAIR_DTYPE)
        pairs["read_offset"], pairs["read_length"] = batch.read_offsets[read], batch.read_lengths[read]
        pairs["hap_offset"], pairs["hap_length"] = batch.hap_offsets[hap], batch.hap_lengths[hap]
        cuda = lambda a: torch.from_numpy(a).to("cuda")
        state.update(arrays=[cuda(a) for a in (batch.read_bases, batch.base_quals, batch.ins_quals, batch.del_quals,
                                               batch.hap_bases)],
                     pairs=cuda(pairs.view(np.uint8)), num_pairs=len(pairs), max_hap=int(batch.hap_lengths.max()),
                     scores=torch.empty(len(pairs), dtype=torch.float32, device="cuda"))
        return state
    state["engine"] = phmm.Engine(device=torch.cuda.current_device(), gcp=case["gcp"])
    if entry == "host":
        state["batch"] = batch
    elif entry == "pinned":
        state.update(batch=batch.pin(), scores=torch.empty(batch.num_pairs, dtype=torch.float32, pin_memory=True))
    elif entry == "device":
        state.update(batch=batch.to_device(), max_read=int(batch.read_lengths.max()),
                     max_hap=int(batch.hap_lengths.max()),
                     scores=torch.empty(batch.num_pairs, dtype=torch.float32, device="cuda"))
    else:
        state["regions"] = phmm.RegionSet([batch.select_records(g, g + 1) for g in range(batch.num_records)])
    return state


def run(state):
    entry = state["case"]["entry"]
    if entry == "flat":
        phmm.forward_pairs_noalloc(torch.cuda.current_device(), *state["arrays"], state["pairs"], state["num_pairs"],
                                   state["max_hap"], state["scores"], torch.cuda.current_stream())
        return state["scores"]
    engine = state["engine"]
    if entry == "host":
        return engine.compute(state["batch"])
    if entry == "pinned":
        return engine.compute(state["batch"], out=state["scores"])
    if entry == "device":
        engine.compute_device(state["batch"], state["scores"], stream=torch.cuda.current_stream(),
                              max_read_length=state["max_read"], max_hap_length=state["max_hap"])
        return state["scores"]
    regions = state["regions"]
    tickets = engine.submit_many(regions)
    return np.concatenate([engine.drain(t, n) for t, n in zip(tickets, regions.num_pairs)])


def work(case):
    """Every input byte read once, every score written once, 11 operations per cell of the recurrence."""
    R, H, rl, hl, _ = _structure(case)
    er, eh = np.cumsum(R), np.cumsum(H)
    cr, ch = np.r_[0, np.cumsum(rl)], np.r_[0, np.cumsum(hl)]
    cells = float(((cr[er] - cr[er - R]) * (ch[eh] - ch[eh - H])).sum())
    read_bytes = (5 if case["gcp"] else 4) * int(rl.sum())
    return {"bytes": read_bytes + int(hl.sum()) + 4 * int((R * H).sum()), "flops": 11.0 * cells}


# ------------------------------------------------------------------------------------ 64 bits

def exact(case, seed):
    """Scores of the recurrence in 64-bit logarithms (natural), one anti-diagonal of many pairs at a time."""
    batch = _batch(case, seed)
    read, hap = _pairs(batch)
    L, H = batch.read_lengths.astype(np.int64)[read], batch.hap_lengths.astype(np.int64)[hap]
    if float((L * (L + H)).sum()) > MAX_EXACT_WORK:
        return None
    dev = _device()
    order = np.lexsort((H, L))
    arrays = [torch.from_numpy(a).to(dev) for a in (batch.read_bases, batch.base_quals, batch.ins_quals,
                                                    batch.del_quals, batch.gcp_quals, batch.hap_bases)]
    out = torch.empty(len(read), dtype=torch.float64, device=dev)
    i = 0
    while i < len(order):
        # pairs of like read length, at most 2^25 positions a chunk
        n = max(1, int(2 ** 25 // max(1, L[order[min(len(order) - 1, i + 2 ** 25 // max(1, L[order[i]]))]])))
        part = order[i:i + n]
        part = part[L[part] <= L[part[0]] + max(8, L[part[0]] // 8)]
        i += len(part)
        out[torch.from_numpy(part).to(dev)] = _log10_pairs(arrays, batch, read[part], hap[part], case["gcp"], dev)
    return out.cpu().numpy()


def _log10_pairs(arrays, batch, read, hap, gcp, dev):
    bases, bqs, iqs, dqs, gqs, haps = arrays
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    L, H = to(batch.read_lengths[read].astype(np.int64)), to(batch.hap_lengths[hap].astype(np.int64))
    Lm, Hm, P = int(L.max()), int(H.max()), len(read)
    ph = torch.tensor([10.0 ** (-q / 10.0) for q in range(128)], dtype=torch.float64).float().to(dev)
    code = torch.full((256,), 4, dtype=torch.uint8, device=dev)
    code[torch.tensor([ord(c) for c in "ACGT"], device=dev)] = torch.arange(4, dtype=torch.uint8, device=dev)

    c = torch.arange(Lm, device=dev)
    at = to(batch.read_offsets[read])[:, None] + torch.minimum(c[None, :], L[:, None] - 1)
    x = code[bases[at].long()]
    # the model's parameters are 32-bit numbers; everything computed from them is in 64 bits
    prob = lambda q: ph[q[at].long().clamp_max(127)]
    p, d, s = prob(bqs), prob(iqs), prob(dqs)
    log = lambda t: torch.log(t.double())
    l_match, l_miss, l_alpha, l_delta, l_sigma = log(1 - p), log(p / 3), log(1 - (d + s)), log(d), log(s)
    if gcp:
        eps = prob(gqs)[:, :1].double()
        beta = (1.0 - eps).float().double()
    else:
        eps = torch.full((P, 1), float(np.float32(0.1)), dtype=torch.float64, device=dev)
        beta = torch.full((P, 1), float(np.float32(0.9)), dtype=torch.float64, device=dev)
    l_eps, l_beta = torch.log(eps), torch.log(beta)

    # haplotype codes laid out so that an anti-diagonal is a slice: rev[Lm + Hm - 1 - j] = hap[j]; rows
    # before the haplotype and after it are masked below
    j = torch.arange(Hm + 2 * Lm, device=dev) - Lm
    src = to(batch.hap_offsets[hap])[:, None] + torch.minimum(j.clamp_min(0)[None, :], H[:, None] - 1)
    rev = torch.flip(code[haps[src].long()], dims=[1])
    ninf = float("-inf")
    new = lambda: torch.full((P, Lm + 1), ninf, dtype=torch.float64, device=dev)
    M1, I1, D1, M2, I2, D2 = new(), new(), new(), new(), new(), new()
    l_init = -torch.log(H.double())
    D1[:, 0] = l_init
    D2[:, 0] = l_init
    total = torch.full((P,), ninf, dtype=torch.float64, device=dev)
    any_n = x == 4
    last = (L - 1)[:, None]
    for k in range(Lm + Hm - 1):   # cell (row k - c, position c); index c + 1, index 0 the column before the read
        first = Hm + Lm - 1 - k
        h = rev[:, first:first + Lm]
        row = k - c
        emit = torch.where((h == x) | (h == 4) | any_n, l_match, l_miss)
        M = emit + torch.logaddexp(l_alpha + M2[:, :-1], l_beta + torch.logaddexp(I2[:, :-1], D2[:, :-1]))
        I = torch.logaddexp(l_delta + M1[:, :-1], l_eps + I1[:, :-1])
        D = torch.logaddexp(l_sigma + M1[:, 1:], l_eps + D1[:, 1:])
        ok = ((row >= 0)[None, :] & (row[None, :] < H[:, None]))
        nM, nI, nD = M2, I2, D2
        nM[:, 1:] = torch.where(ok, M, ninf)
        nI[:, 1:] = torch.where(ok, I, ninf)
        nD[:, 1:] = torch.where(ok, D, ninf)
        nD[:, 0] = l_init
        total = torch.logaddexp(total, torch.logaddexp(nM.gather(1, last + 1), nI.gather(1, last + 1))[:, 0])
        M1, I1, D1, M2, I2, D2 = nM, nI, nD, M1, I1, D1
    return total / math.log(10.0)
