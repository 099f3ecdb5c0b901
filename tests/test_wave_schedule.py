"""CPU models of the triangular sweeps' schedules (dplasma_b200/csrc/wave_kernel.cu).

trsm_wave_kernel (more blocks than CTAs): for every CTA the order in which the
producer warp streams W / M / L blocks into the ring must equal the order in which
the consumer warps take them; every block must receive its products in solve order,
then its Z = W acc, then Y = Z - M Y_prev, then its publish; and the CTAs, each
running its program in order with a flag wait before every remote Y, must all finish
(no cycle of waits).  The model restates the kernel's control flow (the owner of the
block after next applies that block's product and forms its Z when Y_q arrives and
defers its other products past its own publish).

trsm_chain_kernel (one block per CTA): the same order of ring blocks on both sides,
no Y stage overwritten while another warp may read it, every CTA waits for earlier
positions only, and the products with the prepared M1 and M2 give the solution."""
import numpy as np
import pytest

RMAX = 4


def blk(qi, P, T):
    return P - 1 - qi if T else qi


def pos(p, P, T):
    return P - 1 - p if T else p


def later(p, q, T):
    return p < q if T else p > q


def producer(c, G, P, T):
    out = []
    owned = [c + i * G for i in range(RMAX) if c + i * G < P]
    first = blk(0, P, T)
    if first % G == c:
        out.append(("W", first))
    if P > 1 and blk(1, P, T) % G == c:
        out.append(("W", blk(1, P, T)))
    for qi in range(P):
        q = blk(qi, P, T)
        nq = blk(qi + 1, P, T) if qi + 1 < P else -1
        nnq = blk(qi + 2, P, T) if qi + 2 < P else -1
        if not any(later(p, q, T) for p in owned):
            continue
        if nq >= 0 and nq % G == c:
            out.append(("M", nq))
            if qi >= 1:
                pq = blk(qi - 1, P, T)
                out += [("L", p, pq) for p in owned if pos(p, P, T) > qi + 1]
        if nnq >= 0 and nnq % G == c:
            out += [("L", nnq, q), ("W", nnq)]
        else:
            out += [("L", p, q) for p in owned if p != nq and later(p, q, T)]
    return out


def consumer(c, G, P, T):
    out = []
    owned = [c + i * G for i in range(RMAX) if c + i * G < P]
    first = blk(0, P, T)
    if first % G == c:
        out += [("W", first), ("PUB", first)]
    if P > 1 and blk(1, P, T) % G == c:
        out.append(("W", blk(1, P, T)))
    for qi in range(P):
        q = blk(qi, P, T)
        nq = blk(qi + 1, P, T) if qi + 1 < P else -1
        nnq = blk(qi + 2, P, T) if qi + 2 < P else -1
        if not any(later(p, q, T) for p in owned):
            continue
        if q % G != c:
            out.append(("WAIT", q))
        if nq >= 0 and nq % G == c:
            out += [("M", nq), ("PUB", nq)]
            if qi >= 1:
                pq = blk(qi - 1, P, T)
                out += [("L", p, pq) for p in owned if pos(p, P, T) > qi + 1]
        if nnq >= 0 and nnq % G == c:
            out += [("L", nnq, q), ("W", nnq)]
        else:
            out += [("L", p, q) for p in owned if p != nq and later(p, q, T)]
    return out


def check(G, P, T):
    seqs = {c: consumer(c, G, P, T) for c in range(G)}
    for c in range(G):
        assert producer(c, G, P, T) == [x for x in seqs[c] if x[0] in ("W", "M", "L")], (G, P, T, c)
    for c in range(G):
        hist = {}
        for x in seqs[c]:
            if x[0] != "WAIT":
                hist.setdefault(x[1], []).append(x)
        for b, h in hist.items():
            pb = pos(b, P, T)
            assert [x[2] for x in h if x[0] == "L"] == [blk(j, P, T) for j in range(pb - 1)], (G, P, T, b)
            kinds = [x[0] for x in h if x[0] != "L"]
            assert kinds == (["W", "PUB"] if pb == 0 else ["W", "M", "PUB"]), (G, P, T, b, kinds)
            iw = [i for i, x in enumerate(h) if x[0] == "W"][0]
            assert all(x[0] != "L" for x in h[iw:]), (G, P, T, b)
    pub, ptr, progress = set(), {c: 0 for c in range(G)}, True
    while progress:
        progress = False
        for c in range(G):
            s = seqs[c]
            while ptr[c] < len(s):
                x = s[ptr[c]]
                if x[0] == "WAIT" and x[1] not in pub:
                    break
                if x[0] == "L":
                    assert x[2] in pub
                if x[0] == "M":
                    assert blk(pos(x[1], P, T) - 1, P, T) in pub
                if x[0] == "PUB":
                    pub.add(x[1])
                ptr[c] += 1
                progress = True
    assert all(ptr[c] == len(seqs[c]) for c in range(G)), (G, P, T)
    assert len(pub) == P


@pytest.mark.parametrize("T", [False, True])
@pytest.mark.parametrize("G", range(2, 12))
def test_wave_schedule_small_grids(G, T):
    for P in range(1, RMAX * G + 1):
        check(G, P, T)


@pytest.mark.parametrize("T", [False, True])
@pytest.mark.parametrize("P", [149, 300, 512, 592])
def test_wave_schedule_b200_grid(P, T):
    check(148, P, T)


# ---------------------------------------------------------------------------
# trsm_chain_kernel
# ---------------------------------------------------------------------------
def chain_producer(pos, P, T):
    p = blk(pos, P, T)
    out = [("L", p, blk(qi, P, T)) for qi in range(max(pos - 2, 0))] + [("W", p)]
    if pos >= 2:
        out.append(("M2", p))
    if pos >= 1:
        out.append(("M1", p))
    return out


def chain_consumer(pos, P, T):
    """the consumer warps' program: ring products, waits for blocks (staged in buffer
    0 or 1), barriers, stores to and reads of the two Y stages"""
    p = blk(pos, P, T)
    out = []

    def product(name, buf):
        out.extend([("RING",) + name, ("READ", buf)])

    def wmul(buf):                                     # acc = W acc, staged in `buf`
        out.extend([("STAGE", buf), ("BAR",)])
        product(("W", p), buf)

    if pos < 3:
        wmul(1)
    for qi in range(pos):
        q, ahead, buf = blk(qi, P, T), pos - qi, qi & 1
        out.extend([("WAIT", q), ("STAGE", buf), ("BAR",)])
        product(("M2", p) if ahead == 2 else ("M1", p) if ahead == 1 else ("L", p, q), buf)
        if ahead == 3:
            wmul((qi + 1) & 1)
            out.append(("BAR",))
    out.append(("SEND", p))
    return out


@pytest.mark.parametrize("T", [False, True])
@pytest.mark.parametrize("P", [1, 2, 3, 4, 5, 9, 32, 148])
def test_chain_order(P, T):
    for pos in range(P):
        seq = chain_consumer(pos, P, T)
        # the ring: what is streamed is what is taken
        assert [x[1:] for x in seq if x[0] == "RING"] == chain_producer(pos, P, T)
        # waits: every earlier position once, in order, then this block is sent
        assert [x[1] for x in seq if x[0] == "WAIT"] == [blk(qi, P, T) for qi in range(pos)]
        assert seq[-1] == ("SEND", blk(pos, P, T)) and [x[0] for x in seq].count("SEND") == 1
        # a stage is written only after a barrier behind the last product that reads it
        # (warps run apart between barriers), and read only after one behind its stores
        open_reads, written = set(), set()
        for x in seq:
            if x[0] == "BAR":
                open_reads.clear()
                written.clear()
            elif x[0] == "STAGE":
                assert x[1] not in open_reads, (P, pos, T)
                written.add(x[1])
            elif x[0] == "READ":
                assert x[1] not in written, (P, pos, T)
                open_reads.add(x[1])


@pytest.mark.parametrize("T", [False, True])
@pytest.mark.parametrize("P", [1, 2, 3, 4, 7])
def test_chain_solves(P, T):
    # 3 x 3 blocks: the program above on numbers
    b, g = 3, np.random.default_rng(P)
    n = P * b
    L = np.tril(g.uniform(-0.5, 0.5, (n, n))) + 2.0 * np.eye(n)
    B = g.uniform(-1.0, 1.0, (n, 2))
    at = lambda M, i, j: M[i * b:(i + 1) * b, j * b:(j + 1) * b]
    op = lambda p, q: at(L, q, p).T if T else at(L, p, q)          # op(L)_pq
    W = [np.linalg.inv(at(L, p, p)).T if T else np.linalg.inv(at(L, p, p)) for p in range(P)]
    near = lambda p, d: p + d if T else p - d                      # d positions before p
    M = {d: [W[p] @ op(p, near(p, d)) if 0 <= near(p, d) < P else None for p in range(P)] for d in (1, 2)}
    Y = {}
    for pos in range(P):                                           # any order that respects the waits
        p = blk(pos, P, T)
        acc, stage = B[p * b:(p + 1) * b].copy(), None
        for x in chain_consumer(pos, P, T):
            if x[0] == "WAIT":
                stage = -Y[x[1]]
            elif x[0] == "RING" and x[1] == "W":
                acc = W[p] @ acc
            elif x[0] == "RING":
                acc = acc + {"L": lambda: op(p, x[3]), "M2": lambda: M[2][p], "M1": lambda: M[1][p]}[x[1]]() @ stage
            elif x[0] == "SEND":
                Y[p] = acc
    X = np.concatenate([Y[p] for p in range(P)])
    ref = np.linalg.solve(L.T if T else L, B)
    assert np.abs(X - ref).max() <= 1e-12 * np.abs(ref).max()
