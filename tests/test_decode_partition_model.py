"""The bookkeeping of the balanced decode partition (csrc/ktk_decode_stream.cu), restated in Python.

The kernel cuts the concatenated page lists into equal chunks, one per CTA; a CTA writes the output of a
list it sees whole, or a partial into its "tail" slot (the list starts here and goes on) or its "head" slot
(the list started earlier); the combine pass of CTA c merges the list that starts in c and continues.  This
model runs the same rules on the host and checks the invariants the kernels rely on: every entry is read by
exactly one CTA, every list gets exactly one writer of its output, every slot written is read exactly once.
(The kernels themselves are checked against the oracle in the GPU tests.)
"""
import random


def _walk(units, total, chunk, grid):
    """units: list of (key, start, length, count) in position order.  Returns (outputs, slots, covered)."""
    covered = {k: [0] * cnt for k, _, _, cnt in units}
    out, slots = {}, {}
    for c in range(grid):
        p0, p1 = c * chunk, min((c + 1) * chunk, total)
        if p1 <= p0:
            continue
        for key, start, length, cnt in units:
            if start + length <= p0 or start >= p1 or length == 0:
                continue
            lo, hi = max(p0 - start, 0), min(p1 - start, length)
            first = p0 <= start
            e_lo, e_hi = min(lo, cnt), min(hi, cnt)
            whole = first and e_hi == cnt
            partial = (not whole) and (first or e_hi > e_lo)
            for e in range(e_lo, e_hi):
                covered[key][e] += 1
            if whole:
                assert key not in out
                out[key] = "direct"
            elif partial:
                slot = (c, 1 if first else 0)
                assert slot not in slots and e_hi > e_lo
                slots[slot] = (key, e_lo, e_hi)
    for c in range(grid):                                    # the combine pass
        p0, p1 = c * chunk, min((c + 1) * chunk, total)
        if p1 <= p0 or p1 >= total:
            continue
        key, start, length, cnt = next(u for u in units if u[1] <= p1 - 1 < u[1] + u[2])
        if start < p0 or start + cnt <= p1:
            continue
        pieces, c2 = [], c
        while c2 * chunk < start + cnt:
            k2, a, b = slots.pop((c2, 1 if c2 == c else 0))
            assert k2 == key
            pieces.append((a, b))
            c2 += 1
        pieces.sort()
        assert pieces[0][0] == 0 and pieces[-1][1] == cnt
        assert all(pieces[i][1] == pieces[i + 1][0] for i in range(len(pieces) - 1))
        assert key not in out
        out[key] = "combined"
    return out, slots, covered


def test_padded_rows():
    rng = random.Random(1)
    for _ in range(1500):
        U, wmax = rng.randint(1, 40), rng.randint(1, 70)
        cnts = [rng.choice([0, wmax, rng.randint(0, wmax)]) for _ in range(U)]
        total = U * wmax
        grid = min(rng.choice([1, 2, 3, 7, 16, 444]), max(1, -(-total // rng.choice([1, 4, 16]))))
        chunk = -(-total // grid)
        grid = -(-total // chunk)
        units = [(u, u * wmax, wmax, cnts[u]) for u in range(U)]
        out, slots, covered = _walk(units, total, chunk, grid)
        assert not slots and len(out) == U
        assert all(all(x == 1 for x in cv) for cv in covered.values())


def test_csr_entries():
    rng = random.Random(2)
    for _ in range(1500):
        B, hkv = rng.randint(1, 12), rng.choice([1, 2, 8])
        ns = [rng.choice([0, 0, 1, rng.randint(1, 90)]) for _ in range(B)]
        units, pos = [], 0
        for b, n in enumerate(ns):
            for h in range(hkv):
                units.append(((b, h), pos, n, n))
                pos += n
        total = pos
        grid = rng.choice([1, 2, 5, 17, 444])
        chunk = max(-(-total // grid), rng.choice([1, 4, 16])) if total else 16
        out, slots, covered = _walk(units, total, chunk, grid)
        assert not slots
        assert all(all(x == 1 for x in cv) for cv in covered.values())
        # lists without entries own no position: the combine pass writes their zero rows separately
        assert set(out) == {k for k, _, n, _ in units if n > 0}


def test_rows_shared_by_all_heads():
    """csrc/layers/ktl_attn_shared.cu, balanced: positions are page-list entries, chunks whole tiles of 64 tokens; the joining
    pass reads the second slot of the CTA that a cut sequence starts in, then the first slot of those behind it."""
    rng = random.Random(3)
    for _ in range(1500):
        ps, ctas = rng.choice([16, 32, 64]), rng.choice([1, 2, 9, 148])
        ns = [rng.choice([1, 2, rng.randint(1, 90)]) for _ in range(rng.randint(1, 12))]
        per = 64 // ps
        total = sum(ns)
        chunk = max(-(-(-(-total // ctas)) // per) * per, 4 * per)
        units, pos = [], 0
        for b, n in enumerate(ns):
            units.append((b, pos, n, n))
            pos += n
        out, slots, covered = _walk(units, total, chunk, ctas)
        assert not slots and len(out) == len(ns)
        assert all(all(x == 1 for x in cv) for cv in covered.values())
        for b, start, n, _ in units:                         # what the joining pass derives from the table alone
            c0, pieces = start // chunk, (start + n - 1) // chunk - start // chunk + 1
            assert (pieces == 1) == (out[b] == "direct") and c0 + pieces - 1 < ctas and pieces <= 256


def _item_by_length(first, count, rank):
    """csrc/ktk_prefill_umma.cu, item_of_either where histories differ: 32 probes at a time."""
    at_least = lambda L: sum(min(max(f + c - L, 0), c) for f, c in zip(first, count))
    lo, hi, behind, begun = 0, max(f + c for f, c in zip(first, count)), 0, False
    while hi - lo > 1 or not begun:
        begun = True
        each = (hi - lo + 31) // 32
        have = [at_least(lo + i * each) if lo + i * each < hi else behind for i in range(32)]
        more = [lo + i * each < hi and have[i] > rank for i in range(32)]
        if not more[0]:
            return None
        at = max(i for i in range(32) if more[i])
        assert all(more[:at + 1])
        if at < 31 and lo + (at + 1) * each < hi:
            hi, behind = lo + (at + 1) * each, have[at + 1]
        lo += at * each
    has = [s for s, (f, c) in enumerate(zip(first, count)) if f <= lo < f + c]
    return has[rank - behind], lo - first[has[rank - behind]]


def test_prompt_items_by_length():
    rng = random.Random(4)
    for _ in range(600):
        B = rng.randint(1, 32)
        count = [rng.choice([0, 1, rng.randint(1, 70)]) for _ in range(B)]
        first = [rng.choice([0, rng.randint(0, 3000)]) if c else 0 for c in count]
        items = sorted(((-first[s] - p, s, p) for s in range(B) for p in range(count[s])))
        for rank in {0, len(items) // 3, max(len(items) - 1, 0), len(items), len(items) + 5}:
            want = items[rank][1:] if rank < len(items) else None
            assert _item_by_length(first, count, rank) == want
