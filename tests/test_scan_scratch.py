"""The recurrence scan's scratch and the memory that the engine leaves for it (host arithmetic, no GPU): the bound that
`activation_bytes` counts holds for every step, and every family with a recurrence counts all of its mixers."""
import random

import pytest

import kofadra_util
import lizazen_util
import sanarax_util
import tonilix_util
from b200attn import _lib, kofadra, lizazen, ops, sanarax, tonilix

SIZES = [(16, 128, 128), (4, 64, 64), (32, 128, 256), (8, 96, 80), (1, 32, 64)]


@pytest.mark.parametrize("H,dk,dv", SIZES)
def test_no_step_asks_for_more_than_the_bound(H, dk, dv):
    lib, r = _lib.load(), random.Random(H + dk)
    for rows, seqs in ((128, 4), (1000, 64), (5003, 16), (8192, 256)):
        for per_channel in (False, True):
            for delta in (False, True):
                bound = ops.scan_scratch_bytes(rows, seqs, [(H, dk, dv, per_channel, delta)])
                for _ in range(400):
                    T = r.randint(1, rows)
                    n = r.randint(1, min(seqs, T))
                    assert 4 * lib.b2_channel_scan_workspace(T, n, H, dk, dv, per_channel, delta) <= bound, (T, n)
    assert ops.scan_scratch_bytes(8192, 64, [(16, 128, 128, True, True)]) > 100 << 20
    assert ops.scan_scratch_bytes(8192, 64, []) == 0


LIMIT = 512 << 20


@pytest.mark.parametrize("H,dk,dv,rows", [(64, 128, 128, 16384), (32, 128, 256, 32768), (64, 128, 128, 32768), (16, 128, 128, 131072), (48, 64, 64, 32768)])
def test_scratch_of_long_steps_has_a_limit_and_the_bound_holds(H, dk, dv, rows):
    """Steps whose scratch would be above the limit go through it in pieces: no step asks for more, and none for more than is kept for it."""
    lib, r, most = _lib.load(), random.Random(H + rows), 0
    for seqs in (1, 64, 200):
        for per_channel in (False, True):
            for delta in (False, True):
                bound = ops.scan_scratch_bytes(rows, seqs, [(H, dk, dv, per_channel, delta)])
                most = max(most, bound)
                for i in range(600):
                    T = r.randint(1, rows) if i % 2 else int(rows ** r.random())
                    n = r.randint(1, min(seqs, T))
                    assert 4 * lib.b2_channel_scan_workspace(T, n, H, dk, dv, per_channel, delta) <= bound, (T, n)
    assert most == LIMIT


def test_scratch_holds_a_chunk_of_any_number_of_heads():
    lib = _lib.load()
    assert LIMIT < 4 * lib.b2_channel_scan_workspace(8192, 1, 4096, 128, 128, False, False) < 3 * LIMIT


def test_fewer_than_two_rows_a_sequence_never_use_scratch():
    lib = _lib.load()                                # ops._scan does not ask then
    for H, dk, dv in SIZES:
        for n in (1, 2, 5, 64, 256, 4096):
            for T in {1, n, 2 * n - 1}:
                assert all(lib.b2_channel_scan_workspace(T, n, H, dk, dv, c, d) == 0 for c in (0, 1) for d in (0, 1))


@pytest.mark.parametrize("module,util,cfgs", [(kofadra, kofadra_util, "abcde"), (tonilix, tonilix_util, "abcdef"), (sanarax, sanarax_util, "abcd"),
                                              (lizazen, lizazen_util, "abcd")])
def test_activation_bytes_count_the_scratch(monkeypatch, module, util, cfgs):
    counted = False
    for name in cfgs:
        raw = getattr(util, "cfg_" + name)()
        raw = util.strip(raw) if hasattr(util, "strip") else raw
        c = module.config_from_dict(raw)
        seen = []
        monkeypatch.setattr(ops, "scan_scratch_bytes", lambda rows, seqs, mixers: seen.append((rows, seqs, list(mixers))) or 0)
        without = c.activation_bytes(300, 5)
        monkeypatch.setattr(ops, "scan_scratch_bytes", lambda rows, seqs, mixers: 12345)
        assert c.activation_bytes(300, 5) == without + 12345
        (rows, seqs, mixers), = seen
        assert (rows, seqs) == (300, 5)
        want = []
        for L in raw["layers"]:
            m, kind = L["mixer"], L["type"]
            right = m.get("right") if isinstance(m.get("right"), dict) else None
            if kind == "delta":
                want.append((m["heads"], m["dim"], m.get("vdim", m["dim"]), False, True))
            elif kind == "channel_delta":
                want.append((m["heads"], m["dim"], m.get("vdim", m["dim"]), True, True))
            elif kind == "lightning":
                want.append((m["heads"], m["dim"], m["vdim"], False, False))
            elif right is not None and module is tonilix:
                want.append((right["heads"], right["dim"], right["vdim"], True, False))
            elif right is not None and "decay" in right:
                want.append((len(right["decay"]), right["dim"], right["vdim"], False, False))
        assert mixers == want, name
        counted = counted or bool(want)
    assert counted
