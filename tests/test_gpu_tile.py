"""Exact-tile kernels (wavefront_tile.cuh): every tile's shortest and longest read and
one in between, against the FP64 oracle (parity tolerance, conftest); and the
property the tables rely on, that a pair's score does not depend on the group's
shape, on the reads that share its group, or on which path (one gap quality or
per-position coefficients) its warp took: bitwise."""
import numpy as np
import pytest

import gpupairhmm_b200 as g
import oracle
from conftest import assert_log10_close
from gpupairhmm_b200.synth import ACGT, _Builder

pytestmark = pytest.mark.gpu


def _records(lengths, gaps, seed, extra=(1, 60), reads=3):
    """One record per read length: reads cut from the first haplotype (1% errors),
    the last read unrelated; gap qualities one value per batch ("one"), one per read
    ("read") or one per position ("each"); gcp qualities per read."""
    rng = np.random.default_rng(seed)
    b = _Builder()
    gcp = []
    for L in lengths:
        H = L + rng.integers(*extra, size=2)
        H[1] = max(1, int(H[1]) - L // 2)
        base = ACGT[rng.integers(0, 4, size=int(H.max()))]
        rs = []
        for i in range(reads):
            r = base[:L].copy() if i + 1 < reads else ACGT[rng.integers(0, 4, size=L)]
            m = rng.random(L) < 0.01
            r[m] = ACGT[rng.integers(0, 4, size=int(m.sum()))]
            rs.append(r)
        n = reads * L
        if gaps == "one":
            iq = dq = np.full(n, 40)
        elif gaps == "read":
            iq = dq = np.repeat(rng.integers(20, 46, size=reads), L)
        else:
            iq, dq = rng.integers(10, 46, size=n), rng.integers(10, 46, size=n)
        b.add_concat(np.full(reads, L), np.concatenate(rs), rng.integers(2, 41, size=n).astype(np.uint8),
                     iq.astype(np.uint8), dq.astype(np.uint8), H, np.concatenate([base[:h] for h in H]))
        gcp += [np.repeat(rng.integers(1, 45, size=reads), L)]
    batch = b.build()
    q = np.concatenate(gcp)
    off = np.asarray(batch.read_offsets)
    at = 0
    for o, L in zip(off, batch.read_lengths):
        batch.gcp_quals[o:o + L] = q[at:at + L]
        at += L
    return batch


def _edges(rules):
    out, lo = [], 0
    for max_len, G, R, kind in rules:
        if kind >= 3:
            out += [lo + 1, (lo + 1 + max_len) // 2, max_len]
        lo = max_len
    return sorted(set(out))


@pytest.mark.parametrize("gcp", [False, True])
@pytest.mark.parametrize("gaps", ["one", "read", "each"])
@pytest.mark.parametrize("small", [False, True])
def test_exact_tiles_match_oracle(small, gaps, gcp):
    """small: the default engine's table for few pairs (32 lanes); else the same
    batch on an engine that always takes the table for many."""
    with g.Engine(gcp=gcp) as e:
        rules = e.tile_table()
        if not small:
            # any other table than the default one has no second table
            e.set_tile_table([(rules[0][0] - 1,) + rules[0][1:]] + rules[1:] if rules[0][3] != 0 else
                             [(8, 4, 16 if gcp else 4, 0)] + rules)
        b = _records(_edges(rules), gaps, seed=7 + len(gaps))
        got = e.compute(b)
    assert_log10_close(got, oracle.batch_log10(b, gcp=gcp), what=f"{gaps} gcp={gcp} small={small}")


@pytest.mark.parametrize("gcp", [False, True])
@pytest.mark.parametrize("gaps", ["one", "read", "each"])
def test_score_does_not_depend_on_group_shape(gaps, gcp):
    """Reads of 129-160 (8 x 17..20 or 32 x 5) and 161-320 positions (16 x 11..20 or
    32 x 6..10), many per record so that units pair different reads."""
    b = _records([129, 136, 137, 150, 160, 161, 176, 200, 320], gaps, seed=3, reads=5)
    with g.Engine(gcp=gcp) as e:
        rules = e.tile_table()
        few = e.compute(b)
        e.set_tile_table([(8, 4, 16 if gcp else 4, 0)] + rules)   # the table for many pairs
        many = e.compute(b)
        one = e.compute(b.select_records(3, 4))
    np.testing.assert_array_equal(few, many)
    np.testing.assert_array_equal(one, many[3 * 10:4 * 10])


def test_exact_rules_are_checked():
    with g.Engine() as e:
        e.set_tile_table([(152, 32, 24, 0), (160, 8, 20, 3), (1 << 30, 32, 32, 1)])
        assert e.tile_table()[1] == (160, 8, 20, 3)
        for bad in ([(151, 32, 24, 0), (160, 8, 20, 3), (1 << 30, 32, 32, 1)],   # 152 is one lane's worth short
                    [(152, 32, 24, 0), (161, 8, 20, 3), (1 << 30, 32, 32, 1)],   # longer than the tile
                    [(152, 32, 24, 0), (156, 4, 39, 3), (1 << 30, 32, 32, 1)]):  # not compiled
            with pytest.raises(g.PairHMMError):
                e.set_tile_table(bad)


@pytest.mark.parametrize("gcp", [False, True])
@pytest.mark.parametrize("gaps", ["one", "each"])
def test_fp64_tiles_match_oracle(gaps, gcp):
    """Unrelated high-quality reads at the edges of the FP64 classes (8, 16 and 32 lanes,
    blocks of 4 and 8 warps, and past them), on haplotypes shorter and longer than the
    read: every pair is recomputed in double, some beyond the scaled tier's range.  On
    the tables for few and for many pairs, bitwise the same."""
    rng = np.random.default_rng(5)
    b = _Builder()
    for L in (32, 33, 40, 41, 160, 161, 176, 320, 321, 352, 640, 641, 768, 769, 1024, 1025, 1152, 1793, 2016, 2017,
              2048, 2049, 2304, 2305, 4096, 4097):
        H = np.array([rng.integers(1, 60), max(2, L // 3), L + rng.integers(0, 200)])
        n = 2 * L
        q = rng.integers(35, 46, size=n) if gaps == "each" else np.full(n, 45)
        b.add_concat(np.full(2, L), ACGT[rng.integers(0, 4, size=n)], rng.integers(38, 42, size=n).astype(np.uint8),
                     q.astype(np.uint8), q.astype(np.uint8), H, ACGT[rng.integers(0, 4, size=int(H.sum()))])
    batch = b.build()
    batch.gcp_quals[:] = 10 if not gcp else 20
    want = oracle.batch_log10(batch, gcp=gcp)
    with g.Engine(gcp=gcp) as e:
        few = e.compute(batch)
        st = e.stats()
        rules = e.tile_table()
        e.set_tile_table([(8, 4, 16 if gcp else 4, 0)] + rules)
        many = e.compute(batch)
    assert want.min() < -650 and st.rescued > 0.9 * (want < -70).sum() and st.rescued_ext > 0
    assert_log10_close(few, want, what="FP64 tiles")
    np.testing.assert_array_equal(few, many)


@pytest.mark.parametrize("gaps", ["one", "each", "high"])
@pytest.mark.parametrize("shuffled", [False, True])
def test_flat_list_shapes_match_oracle(gaps, shuffled):
    """The allocation-free entry point at the edges of its shapes (8, 16 and 32 lanes,
    one to five parts; the general form for the shortest reads and for gap qualities
    beyond its exact tiles' range), in list order and with every warp's pairs mixed;
    twice, since a call leaves its queue empty for the next."""
    import torch
    rng = np.random.default_rng(8)
    b = _Builder()
    for L in (1, 2, 8, 9, 16, 17, 152, 153, 160, 161, 176, 177, 320, 321, 352, 640, 641, 704, 1280, 1281, 1344, 1921,
              2600):
        H = np.array([L + 30, L + 1, max(1, L - 3), L + 200])
        base = ACGT[rng.integers(0, 4, size=int(H.max()))]
        reads = [base[:L].copy() for _ in range(3)]
        for r in reads:
            m = rng.random(L) < 0.003
            r[m] = ACGT[rng.integers(0, 4, size=int(m.sum()))]
        n = 3 * L
        q = {"one": np.full(n, 40), "each": rng.integers(20, 46, size=n), "high": rng.integers(55, 94, size=n)}[gaps]
        b.add_concat(np.full(3, L), np.concatenate(reads), rng.integers(20, 41, size=n).astype(np.uint8),
                     q.astype(np.uint8), q.astype(np.uint8), H, np.concatenate([base[:h] for h in H]))
    batch = b.build()
    want = oracle.batch_log10(batch)
    pairs, r0, h0 = [], 0, 0
    for nr, nh in zip(batch.reads_per_record, batch.haps_per_record):
        pairs += [(batch.read_offsets[i], batch.hap_offsets[j], batch.read_lengths[i], batch.hap_lengths[j])
                  for i in range(r0, r0 + nr) for j in range(h0, h0 + nh)]
        r0, h0 = r0 + nr, h0 + nh
    order = rng.permutation(len(pairs)) if shuffled else np.arange(len(pairs))
    pairs = np.array(pairs, dtype=g.PAIR_DTYPE)[order]
    dev = torch.device("cuda:0")
    d = [torch.from_numpy(np.ascontiguousarray(getattr(batch, k))).to(dev)
         for k in ("read_bases", "base_quals", "ins_quals", "del_quals", "hap_bases")]
    dpairs = torch.from_numpy(pairs.view(np.uint8)).to(dev)
    ok = want[order] > -60.0
    assert ok.mean() > 0.9
    for _ in range(2):
        scores = torch.full((len(pairs),), 7.0, dtype=torch.float32, device=dev)
        g.forward_pairs_noalloc(0, *d, dpairs, len(pairs), int(batch.hap_lengths.max()), scores)
        torch.cuda.synchronize(dev)
        assert_log10_close(scores.cpu().numpy()[ok], want[order][ok], what=f"flat list, {gaps}")
