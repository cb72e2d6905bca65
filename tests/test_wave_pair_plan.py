"""The batch's plan in passes over two register groups, read from the host
image (CPU): what the passes of each instance do, in order, is the circuit --
every layer's mixer on every qubit once, its cost layer between -- and their
blocks and rows of partial sums cover the instance without overlap."""
import ctypes

import numpy as np
import pytest

HEADER = [("head", np.int32, (10,)), ("rounds", np.int32), ("ifwd", np.int32), ("iadj", np.int32),
          ("ipfwd", np.int32), ("ipadj", np.int32), ("pad", np.int32), ("sizes", np.int64, (4,)),
          ("offsets", np.int64, (12,)), ("device_bytes", np.int64)]
WAVE = [(f"{k}_{f}", np.int32) for k in ("fwd", "adj", "pfwd", "padj") for f in ("begin", "count", "blocks")]
PASS = [("inst", np.int32), ("block_begin", np.int32), ("prow", np.int32), ("pair", np.int8), ("init", np.int8),
        ("cost", np.int8), ("hasA", np.int8), ("hasB", np.int8), ("lanesA", np.int8), ("nx", np.int8),
        ("ny", np.int8), ("layerA", np.int16), ("layerB", np.int16), ("x", np.uint8, (4,)), ("y", np.uint8, (4,)),
        ("s", np.uint8, (8,))]


def _image(sizes, layout):
    from quantumflow_gb300 import _native as nat
    from quantumflow_gb300.batched import _Instance
    a = o = 0
    rows = []
    for n, p in sizes:
        rows.append(_Instance(n, p, 2 * n, 0, a, o))
        a, o = a + 2 * p, o + 2 * p + 1
    inst = (_Instance * len(rows))(*rows)
    hb, db = ctypes.c_size_t(), ctypes.c_size_t()
    assert nat.lib.qf_wave_plan(ctypes.addressof(inst), len(rows), layout, None, 0, ctypes.byref(hb),
                                ctypes.byref(db)) == 0
    plan = np.zeros(hb.value, np.uint8)
    assert nat.lib.qf_wave_plan(ctypes.addressof(inst), len(rows), layout, plan.ctypes.data, hb.value, None, None) == 0
    h = plan[:np.dtype(HEADER).itemsize].view(HEADER)[0]
    at = np.dtype(HEADER).itemsize
    waves = plan[at:at + 48 * int(h["rounds"])].view(WAVE)
    # behind the two-group items: reduction segments (16 bytes) and two int32
    # arrays of one entry an output, the first with one more
    nsegs, nout = int(h["head"][8]), int(h["head"][9])
    end = plan.size - 16 * nsegs - 4 * (nout + 1) - 4 * nout
    nfwd, nadj = int(h["ipfwd"]), int(h["ipadj"])
    passes = plan[end - 40 * (nfwd + nadj):end].view(PASS)
    return h, waves, passes[:nfwd], passes[nfwd:]


def _bits(p, side):
    """Bits the mixer of a pass acts on, before ('A') or after ('B') its cost layer."""
    y = [int(b) for b in p["y"][:p["ny"]]]
    x = [int(b) for b in p["x"][:p["nx"]]] if p["pair"] else []
    lanes = list(range(5)) if side == "B" or p["lanesA"] else []
    return lanes + x + y


@pytest.mark.parametrize("dtype,sizes", [("c64", [(13, 1), (14, 3), (16, 2), (17, 5), (20, 6), (22, 1), (30, 2)]),
                                         ("ff", [(11, 1), (12, 3), (13, 2), (15, 4), (18, 6), (19, 1), (21, 3)])])
def test_two_group_passes_are_the_circuit(dtype, sizes):
    from quantumflow_gb300 import _native as nat
    layout, rbf, rba = (nat.LAYOUT_C64, 4, 3) if dtype == "c64" else (nat.LAYOUT_FF, 3, 2)
    h, waves, fwd, adj = _image(sizes, layout)
    assert int(h["ifwd"]) == int(h["iadj"]) == 0
    assert sum(int(w["pfwd_count"]) for w in waves) == len(fwd) == int(h["ipfwd"])
    assert sum(int(w["padj_count"]) for w in waves) == len(adj) == int(h["ipadj"])
    rows = []
    for i, (n, p) in enumerate(sizes):
        done = {}   # layer -> bits mixed so far
        cost = []
        mine = [f for f in fwd if f["inst"] == i]
        assert mine[0]["init"] and not any(f["init"] for f in mine[1:])
        for f in mine:
            for side in "AB":
                if side == "B" and f["cost"]:
                    layer = int(f["layerB"])
                    assert layer == 0 or sorted(done[layer - 1]) == list(range(n))
                    cost.append(layer)
                if f["has" + side]:
                    assert int(f["layer" + side]) == cost[-1]
                    done.setdefault(int(f["layer" + side]), []).extend(_bits(f, side))
            assert len(set(map(int, f["s"][:2 * rbf]))) == 2 * rbf
        assert cost == list(range(p)) and all(sorted(done[l]) == list(range(n)) for l in range(p))
        done, cost = {}, []
        mine = [a for a in adj if a["inst"] == i]
        assert mine[0]["init"] and not any(a["init"] for a in mine[1:])
        for a in mine:
            assert a["hasA"]
            done.setdefault(int(a["layerA"]), []).extend(_bits(a, "A"))
            if a["cost"]:
                assert sorted(done[int(a["layerA"])]) == list(range(n))
                cost.append(int(a["layerA"]))
            if a["hasB"]:
                assert a["cost"] and int(a["layerB"]) == int(a["layerA"]) - 1
                done.setdefault(int(a["layerB"]), []).extend(_bits(a, "B"))
        assert cost == list(range(p))[::-1]
        rows += [(int(a["prow"]), -(-2 ** (n - 5 - 2 * rba) // 4)) for a in mine]
    at = 0
    for first, count in sorted(rows):  # rows of partial sums, without gaps
        assert first == at
        at += count
    for w in waves:  # blocks of each launch
        for kind, items, rb, tiles in (("pfwd", fwd, rbf, 2), ("padj", adj, rba, 4)):
            b = 0
            for f in items[w[kind + "_begin"]:w[kind + "_begin"] + w[kind + "_count"]]:
                assert int(f["block_begin"]) == b
                b += -(-2 ** (sizes[int(f["inst"])][0] - 5 - 2 * rb) // tiles)
            assert b == int(w[kind + "_blocks"])


def test_one_group_counts_need_no_one_group_lists():
    """The header's counts by one group a pass, small and large instances together."""
    from quantumflow_gb300 import _native as nat
    sizes = [(9, 2), (10, 1), (12, 3), (13, 4), (20, 6)]
    h, _, fwd, adj = _image(sizes, nat.LAYOUT_C64)
    count = lambda n, p, rb: p if n - 5 <= rb else 1 + p * (-(-(n - 5) // rb) - 1)
    f, a = [count(n, p, 4) for n, p in sizes], [count(n, p, 3) for n, p in sizes]
    assert h["head"][5] == max(x + y for x, y in zip(f, a))
    assert h["head"][6] == sum(f) and h["head"][7] == sum(a)
    assert h["ifwd"] == sum(f[:3]) and h["iadj"] == sum(a[:3])
    assert {int(x["inst"]) for x in fwd} == {int(x["inst"]) for x in adj} == {3, 4}
