"""The device TSV parse where its units (16 bytes), its tiles (16 KB) and its number lengths meet, against
the host's own split of the same bytes."""
import numpy as np
import pytest

import ktruss_gb300 as kt

pytestmark = pytest.mark.gpu

UNIT, TILE = 16, 16384


@pytest.fixture(scope="module")
def eng():
    e = kt.Engine(0)
    yield e
    e.close()


def _parse(eng, text: bytes, shift=0, capacity=None):
    torch = pytest.importorskip("torch")
    buf = torch.full((shift + len(text) + 64,), ord("7"), dtype=torch.uint8, device="cuda")  # digits all around
    buf[shift:shift + len(text)] = torch.from_numpy(np.frombuffer(text, np.uint8).copy()).cuda()
    cap = len(text) // 6 + 1 if capacity is None else capacity
    out = torch.full((2, cap + 8), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    try:
        n_e, n_v = eng.parse_tsv(buf.data_ptr() + shift, len(text), out[0].data_ptr(), out[1].data_ptr(), cap)
        status = 0
    except kt.KtrussError as e:
        n_e, n_v, status = 0, 0, e.status
    return status, n_v, out.cpu().numpy().view(np.uint32)[:, :n_e], out.cpu().numpy()[:, n_e:]


def _check(eng, text: bytes, shift=0):
    want = np.array(text.split(), np.uint64).reshape(-1, 3)
    status, n_v, got, rest = _parse(eng, text, shift)
    assert status == 0
    assert np.array_equal(got[1], want[:, 0] - 1) and np.array_equal(got[0], want[:, 1] - 1)
    assert n_v == int(want[:, :2].max(initial=0)) and np.all(rest == -7)


def _line(rng, lengths):
    a, b, x = (str(rng.integers(10 ** (k - 1), min(10 ** k, 2 ** 32))) for k in lengths)
    return f"{a} {b if b != a else int(b) - 1} {x}\n".encode()


@pytest.mark.parametrize("shift", [0, 1, 8, 15])
@pytest.mark.parametrize("where", [UNIT, TILE, 3 * TILE, 9 * TILE])
def test_every_length_at_every_offset(where, shift, eng):
    rng = np.random.default_rng([where, shift])
    for offset in range(0, 3 * UNIT, 1 if where == TILE else 5):
        start = max(where - 3 * UNIT + offset, 0)
        fill = b"".join(_line(rng, rng.integers(2, 8, 3)) for _ in range(max(start // 8, 1)))[:start]
        fill = fill[: fill.rfind(b"\n") + 1].ljust(start, b" ")  # whole lines, then spaces up to the place
        lines = [_line(rng, (k, 11 - k if k < 11 else 1, (k * 3) % 10 + 1)) for k in rng.permutation(np.arange(2, 11))]
        _check(eng, fill + b"".join(lines)[: None if offset % 2 else -1], shift)


@pytest.mark.parametrize("gap", [TILE - 1, TILE, 2 * TILE + 5])
def test_entries_spread_over_tiles(gap, eng):
    space = b" " * gap
    _check(eng, space + b"12" + space + b"4294967295\t" + space + b"0 3 4" + space + b"9\r\n")
    for text, want in ((b"5" + space + b"5 1\n", 2), (b"1 2 3\n7 " + space + b"7" + space + b"2", 2),
                       (b"1 2 3\n0" + space + b"7 2", 9), (b"1 2" + space + b"4294967296", 9),
                       (b"1 2" + space + b"00000000001", 9), (b"1 2" + space + b"3 4", 9),
                       (b"1 2 3" + space + b"4 5 6" + space + b"\x0b", 9)):
        assert _parse(eng, text)[0] == want, text.split()


@pytest.mark.parametrize("entries", [2048, 2049, 5461])
def test_two_byte_tokens_and_capacity(entries, eng):
    text = b"1 2 3 " * (entries - 1) + b"2 1 3"  # as many tokens as a tile can hold
    _check(eng, text)
    assert _parse(eng, text, capacity=entries)[0] == 0
    status, _, _, untouched = _parse(eng, text, capacity=entries - 1)
    assert status == 4 and np.all(untouched == -7)


def test_many_tiles_in_file_order(eng):
    # more tiles than one step of the block that numbers them takes (8,192)
    rng = np.random.default_rng(8)
    ids = rng.integers(1, 2 ** 32, (4, 1 << 16), dtype=np.uint64)
    block = b"".join(b"%d %d %d\n" % (a, b, x) for a, b, x, _ in ids.T if a != b)
    torch = pytest.importorskip("torch")
    reps = 8300 * TILE // len(block) + 1
    text = torch.from_numpy(np.frombuffer(block, np.uint8).copy()).cuda().repeat(reps)
    want = np.array(block.split(), np.uint64).reshape(-1, 3)
    out = torch.empty((2, reps * len(want)), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    n_e, n_v = eng.parse_tsv(text.data_ptr(), text.numel(), out[0].data_ptr(), out[1].data_ptr(), out.shape[1])
    assert n_e == out.shape[1] and n_v == int(want[:, :2].max())
    for row, field in ((1, 0), (0, 1)):
        one = torch.from_numpy((want[:, field] - 1).astype(np.uint32).view(np.int32)).cuda()
        assert bool((out[row].view(reps, -1) == one).all())
